"""The launch shape of the int4 GEMV against a driver that only counts: how many clusters fit is asked for the cluster that the launch then has, also where
whole slices of K-groups make fewer CTAs than the SMs would take, and the deep ring is taken by that answer."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "lithos_b200" / "csrc"
HARNESS = r"""
#include "lb_ops.c"
static int asked, fit[9];
static CUresult count(int* n, CUfunction f, const CUlaunchConfig* cfg) { (void)f; asked = (int)cfg->attrs[0].value.clusterDim.y; *n = fit[asked]; return CUDA_SUCCESS; }
static CUresult current(CUcontext c) { (void)c; return CUDA_SUCCESS; }
int main(int argc, char** argv) {
    static lb_ctx c;
    c.sm_count = 148; c.max_smem_optin = 232448;
    for (int i = 0; i < LBK_COUNT; ++i) c.fn[i] = (CUfunction)1;
    lb_drv.OccupancyMaxActiveClusters = count; lb_drv.CtxSetCurrent = current;
    for (int i = 3; i < argc; ++i) fit[i - 1] = atoi(argv[i]); /* clusters of 2, 3, ... 8 */
    gemv_geom g;
    if (gemv_plan(&c, atoi(argv[1]), atoi(argv[2]), &g) != LB_OK) return 1;
    printf("%d %d %d %d %d %d\n", g.tiles, g.ksplit, g.gps, g.stages, g.early, asked);
    return 0;
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.c").write_text(HARNESS)
    rest = [str(f) for f in sorted((CSRC / "host").glob("*.c")) if f.name != "lb_ops.c"]
    subprocess.check_call(["gcc", "-std=gnu11", "-O0", "-w", "-fopenmp", f"-I{CSRC}/host", f"-I{ROOT}/include", "-I/usr/local/cuda/include", "-o", str(d / "plan"),
                           str(d / "plan.c"), *rest, "-ldl", "-lpthread", "-lm", "-lrt"])
    return lambda K, N, fit: [int(v) for v in subprocess.check_output([str(d / "plan"), str(K), str(N), *map(str, fit)]).split()]


@pytest.mark.parametrize("K,N", [(4224, 9472), (4608, 10496), (2304, 9472), (5120, 17408), (5120, 16384), (8192, 8192), (5120, 34816), (6528, 9600), (3456, 9472)])
def test_cluster_asked_for_is_the_one_launched(plan, K, N):
    whole = [296 // k for k in range(2, 9)]
    tiles, ksplit, gps, stages, early, asked = plan(K, N, whole)
    assert ksplit == 1 or asked == ksplit
    assert (ksplit - 1) * gps < K // 128 <= ksplit * gps
    room = (296 // ksplit - tiles) * ksplit
    if gps <= 4 or room < 0:
        assert not early
    elif room >= 12:
        assert early and stages >= min(gps, 4)


def test_a_cluster_that_does_not_fit_keeps_the_shallow_ring(plan):
    none = [0 if k == 7 else 296 // k for k in range(2, 9)]  # 33 K-groups over 37 tiles: seven slices of five
    assert plan(4224, 9472, [296 // k for k in range(2, 9)])[1:5:3] == [7, 1]
    none[5] = 36
    assert plan(4224, 9472, none)[4] == 0
