/* Per-kernel launch wrappers: argument checks, launch geometry, parameter
 * blocks.  These are the C counterparts of the reference's launch_* helpers
 * (src/launcher.s:1101-2975), one per kernel family. */
#include "lb_internal.h"
#include "../kernels/params.h"
#include <math.h>

#define GEMV_THREADS LB_GEMV_THREADS

/* Geometry of one int4 GEMV launch.
 *  - grid = (column tiles of 128, ksplit); the ksplit CTAs of a tile form one cluster and add
 *    their partial sums on chip, so ksplit <= 8.
 *  - All CTAs of a launch should be co-resident and carry equal work, so that the HBM pipe and
 *    not a tail of late CTAs ends the kernel: ksplit is chosen so that tiles*ksplit comes close
 *    to (and not above) two CTAs per SM.
 *  - A CTA's shared memory (ring of 16 KB stages + its activation slice) is kept under half
 *    of an SM where possible; the CTAs of the NEXT kernel follow those that are done and prefetch
 *    their weights while the others compute (programmatic dependent launch). */
typedef struct { int tiles, ksplit, gps, stages, early; unsigned smem; } gemv_geom;

static int clusters_at_once(lb_ctx* c, int kernel, int k, unsigned threads, unsigned smem, int per_sm, int* slot);
static int gemv_plan(lb_ctx* c, int K, int N, gemv_geom* g) {
    if (K <= 0 || N <= 0 || K % LB_GEMV_GROUP != 0 || N % 32 != 0)
        return lb_fail(c, LB_ERR_INVALID, "int4 GEMV needs K %% 128 == 0 and N %% 32 == 0 (K=%d, N=%d)", K, N);
    int groups = K / LB_GEMV_GROUP;
    g->tiles = (N + LB_GEMV_TILE_N - 1) / LB_GEMV_TILE_N;
    int slots = 2 * c->sm_count;
    int ks = slots / g->tiles;
    if (ks < 1) ks = 1;
    if (ks > LB_GEMV_MAX_SPLITS) ks = LB_GEMV_MAX_SPLITS;
    if (ks > groups) ks = groups;
    g->gps = (groups + ks - 1) / ks;
    g->ksplit = (groups + g->gps - 1) / g->gps;
    /* Two CTAs an SM with a deep ring where all clusters run at once like that and leave room for six CTAs, otherwise shared memory for four, which lets the next launch's
     * clusters in beside them.   us, four / two, with the CTAs of room: none 6016 x 8384 10.4 / 11.5, five 8320 x 13984 18.6 / 20.2, six 8576 x 11232 17.3 / 15.2, eight
     * 17408 x 8192 24.1 / 19.7, twelve 5120 x 17408 15.1 / 12.6; not enough for all 5120 x 10240 11.0 / 15.6.  Slices of up to four K-groups stay with four (3840 x 2048 5.8 /
     * 6.3, 4096 x 4096 6.4 / 6.7), those of 7 to 9, whose ring of four stages is a small part of them, want room for twelve (less: 5760 x 13824 14.4 / 15.0, 5120 x 13824 12.6 / 12.8, 2048 x 36864 12.4 / 12.7, 8192 x
     * 8192 12.7 / 12.8; the exception found 2304 x 37120 14.2 / 12.3). */
    const int k = g->ksplit; /* the cluster that is launched: less than ks where whole slices make fewer of them */
    if (k > 1 && !c->gemv_clusters[k]) LB_CU(c, lb_drv.CtxSetCurrent(c->cu_ctx));
    const int at_once = clusters_at_once(c, LBK_gemv_int4_w256, k, GEMV_THREADS, (unsigned)(c->max_smem_optin / 2 - 2048), 2, &c->gemv_clusters[k]);
    const int two = g->gps > 4 && (at_once - g->tiles) * k >= (g->gps >= 7 && g->gps <= 9 ? 12 : 6);
    /* shared memory: 1 KB alignment slack, ring of 16 KB stages (one group each), the digit
     * table of the K slice (26 bytes per packed row), per-group sums, result buffer, mbarriers */
    int rows = g->gps * LB_GEMV_ROWS;
    size_t dig_words = (size_t)((6 * rows + 2 * (rows >> 2) + 3) & ~3);
    size_t fixed = 1024 + dig_words * 4 + (size_t)((g->gps + 3) & ~3) * 4 + (LB_GEMV_TILE_N + 40) * 4 +
                   (size_t)g->gps * (LB_GEMV_TILE_N * 2 + LB_GEMV_TILE_N / 2); /* + group scales and zero-points */
    fixed += 16; /* the scale-box mbarrier */
    size_t per_stage = LB_GEMV_STAGE_BYTES + 16; /* stage + its two mbarriers */
    size_t sm_total = (size_t)c->max_smem_optin + 1024; /* shared memory of one SM */
    int st = 0;
    for (int per_sm = two ? 2 : 4; per_sm >= 1 && st < 2; per_sm >>= 1) {
        size_t budget = sm_total / per_sm - 1024;
        if (budget > (size_t)c->max_smem_optin) budget = (size_t)c->max_smem_optin;
        st = budget > fixed ? (int)((budget - fixed) / per_stage) : 0;
    }
    if (st < 1) return lb_fail(c, LB_ERR_INVALID, "int4 GEMV: K slice of %d groups does not fit shared memory", g->gps);
    /* the whole slice where six stages hold it, four otherwise (us with 3 / 4 / 6: 5120 x 17408 15.5 / 12.7 / 13.5, 4096 x 11008 with slices of six 10.3 / 10.4 / 9.6; with
     * shared memory for four CTAs an SM, as before, two stages: 15.2 and 10.4) */
    if (st > 6) st = 6;
    if (two && g->gps > 6 && st > 4) st = 4;
    if (st > g->gps) st = g->gps;
    g->stages = st;
    g->early = two;
    g->smem = (unsigned)((fixed + (size_t)st * per_stage + 127) & ~(size_t)127);
    return LB_OK;
}

/* The three tensor maps of one int4 matrix.
 * qweight is viewed as [N/32 column blocks][K/8 packed rows][32 columns] so that ONE tiled load
 * brings a whole stage: box = 8 column blocks x 16 rows x 32 columns, laid down as eight
 * consecutive 2 KB boxes with the 128-byte swizzle.  Parts of the box past the matrix
 * (ragged last tile, last group) are zero-filled and never used.  Scales fp16 [K/128, N] and
 * zero-points u32 [K/128, N/8] come as boxes of box_groups rows x one column tile. */
static int lb_gemv_tensor_maps(lb_ctx* c, uint64_t qweight, uint64_t scales, uint64_t qzeros, int K, int N, int box_groups,
                        unsigned char* tm_w, unsigned char* tm_sc, unsigned char* tm_zr) {
    CUtensorMap tm;
    cuuint64_t dims[3] = {32, (cuuint64_t)(K / 8), (cuuint64_t)(N / 32)};
    cuuint64_t strides[2] = {(cuuint64_t)N * 4, 128};
    cuuint32_t box[3] = {32, LB_GEMV_ROWS, LB_GEMV_TILE_N / 32};
    cuuint32_t estr[3] = {1, 1, 1};
    LB_CU(c, lb_drv.TensorMapEncodeTiled(&tm, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, (void*)qweight, dims, strides, box,
                                         estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
    memcpy(tm_w, &tm, sizeof tm);
    cuuint64_t sdims[2] = {(cuuint64_t)N, (cuuint64_t)(K / 128)};
    cuuint64_t sstr[1] = {(cuuint64_t)N * 2};
    cuuint32_t sbox[2] = {LB_GEMV_TILE_N, (cuuint32_t)box_groups};
    LB_CU(c, lb_drv.TensorMapEncodeTiled(&tm, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, (void*)scales, sdims, sstr, sbox, estr,
                                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
    memcpy(tm_sc, &tm, sizeof tm);
    if (qzeros) {
        cuuint64_t zdims[2] = {(cuuint64_t)(N / 8), (cuuint64_t)(K / 128)};
        cuuint64_t zstr[1] = {(cuuint64_t)(N / 8) * 4};
        cuuint32_t zbox[2] = {LB_GEMV_TILE_N / 8, (cuuint32_t)box_groups};
        LB_CU(c, lb_drv.TensorMapEncodeTiled(&tm, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, (void*)qzeros, zdims, zstr, zbox,
                                             estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
        memcpy(tm_zr, &tm, sizeof tm);
    }
    return LB_OK;
}

LB_API int lb_gemv_int4_fused(lb_ctx* c, uint64_t qweight, uint64_t scales, uint64_t qzeros, uint64_t x, uint64_t y,
                              int K, int N, int x_mode, int y_mode, uint64_t aux0, uint64_t aux1, uint64_t x_out,
                              float eps) {
    if (!c) return LB_ERR_INVALID;
    if (!qweight || !scales || !x || !y) return lb_fail(c, LB_ERR_INVALID, "int4 GEMV: NULL operand");
    if (x_mode < LB_X_F16 || x_mode > LB_X_F32_HEADNORM_SILU || y_mode < LB_Y_F16 || y_mode > LB_Y_SWIGLU_F16)
        return lb_fail(c, LB_ERR_INVALID, "int4 GEMV: unknown x_mode/y_mode %d/%d", x_mode, y_mode);
    if ((x_mode == LB_X_F32_RMSNORM && !aux0) || (x_mode == LB_X_F32_HEADNORM_SILU && (!aux0 || !aux1)))
        return lb_fail(c, LB_ERR_INVALID, "int4 GEMV: norm prologue without its weight/gate operand");
    if (y_mode == LB_Y_SWIGLU_F16 && N % 128 != 0)
        return lb_fail(c, LB_ERR_INVALID, "int4 GEMV: SwiGLU epilogue needs N %% 128 == 0 (N=%d)", N);
    if (((qweight | scales | qzeros | x | y | aux0 | aux1 | x_out) & 15ull) != 0)
        return lb_fail(c, LB_ERR_INVALID, "int4 GEMV: operands must be 16-byte aligned");
    gemv_geom g;
    LB_TRY(gemv_plan(c, K, N, &g));
    lb_gemv_params p;
    memset(&p, 0, sizeof p);
    p.qweight = (const uint32_t*)qweight;
    p.scales = (const uint16_t*)scales;
    p.qzeros = (const uint32_t*)qzeros;
    p.x = (const void*)x;
    p.y = (void*)y;
    p.aux0 = (const void*)aux0;
    p.aux1 = (const void*)aux1;
    p.x_out = (uint16_t*)x_out;
    p.status = (uint32_t*)c->dev_status;
    p.K = K; p.N = N;
    p.ksplit = g.ksplit;
    p.groups_per_split = g.gps;
    p.x_mode = x_mode; p.y_mode = y_mode;
    p.eps = eps;
    p.stages = g.stages;
    p.early = g.early;
    LB_TRY(lb_gemv_tensor_maps(c, qweight, scales, qzeros, K, N, g.gps, p.tmap, p.tmap_sc, p.tmap_zr));
    void* params[] = {&p};
    return lb_launch_cluster(c, LBK_gemv_int4_w256, (unsigned)g.tiles, (unsigned)g.ksplit, 1, GEMV_THREADS, g.smem, params, 1,
                             (unsigned)g.ksplit);
}

LB_API int lb_gemv_int4(lb_ctx* c, uint64_t qweight, uint64_t scales, uint64_t qzeros, uint64_t x, uint64_t y, int K,
                        int N, int flags) {
    if (!c) return LB_ERR_INVALID;
    int x_mode = (flags & LB_GEMV_X_F32) ? LB_X_F32 : LB_X_F16;
    int y_mode = (flags & LB_GEMV_Y_SWIGLU) ? LB_Y_SWIGLU_F16
                 : (flags & LB_GEMV_Y_ACCUM) ? LB_Y_F32_ACCUM
                 : (flags & LB_GEMV_Y_F32)   ? LB_Y_F32
                                             : LB_Y_F16;
    /* a strip-packed copy of this matrix exists (lb_gemv_pack): one CTA per SM streams whole columns, no split-K, no cluster */
    const uint64_t packed = lb_packed_lookup(c, qweight, K, N, y_mode == LB_Y_SWIGLU_F16);
    if (packed) {
        lb_gemv_op o;
        memset(&o, 0, sizeof o);
        o.packed = packed;
        o.x = x; o.y = y; o.K = K; o.N = N; o.x_mode = x_mode; o.y_mode = y_mode; o.eps = 1e-6f;
        return lb_gemv_chain(c, &o, 1);
    }
    return lb_gemv_int4_fused(c, qweight, scales, qzeros, x, y, K, N, x_mode, y_mode, 0, 0, 0, 1e-6f);
}

/* Host-buffer entry: the reference-facing call a launcher without device
 * buffers of its own would make.  Device copies of the weights are cached on
 * the context between calls. */
static struct {
    lb_ctx* owner;
    const void *hq, *hs, *hz;
    int K, N;
    CUdeviceptr dq, ds, dz, dx, dy;
} g_host_cache;

static void host_cache_drop(lb_ctx* c) {
    if (g_host_cache.owner != c) return;
    if (g_host_cache.dq) lb_drv.MemFree(g_host_cache.dq);
    if (g_host_cache.ds) lb_drv.MemFree(g_host_cache.ds);
    if (g_host_cache.dz) lb_drv.MemFree(g_host_cache.dz);
    if (g_host_cache.dx) lb_drv.MemFree(g_host_cache.dx);
    if (g_host_cache.dy) lb_drv.MemFree(g_host_cache.dy);
    memset(&g_host_cache, 0, sizeof g_host_cache);
}

void lb_ops_release(lb_ctx* c) { host_cache_drop(c); }

LB_API int lb_gemv_int4_host(lb_ctx* c, const uint32_t* qweight, const uint16_t* scales, const uint32_t* qzeros,
                             const void* x, void* y, int K, int N, int flags, int weights_resident) {
    if (!c || !qweight || !scales || !x || !y) return lb_fail(c, LB_ERR_INVALID, "lb_gemv_int4_host: NULL operand");
    gemv_geom g;
    LB_TRY(gemv_plan(c, K, N, &g));
    LB_CU(c, lb_drv.CtxSetCurrent(c->cu_ctx));
    size_t qb = (size_t)K / 8 * N * 4, sb = (size_t)K / 128 * N * 2, zb = (size_t)K / 128 * N / 2;
    size_t xb = (size_t)K * ((flags & LB_GEMV_X_F32) ? 4 : 2);
    size_t yb = (size_t)((flags & LB_GEMV_Y_SWIGLU) ? N / 2 : N) *
                ((flags & (LB_GEMV_Y_F32 | LB_GEMV_Y_ACCUM)) && !(flags & LB_GEMV_Y_SWIGLU) ? 4 : 2);
    int hit = weights_resident && g_host_cache.owner == c && g_host_cache.hq == qweight && g_host_cache.hs == scales &&
              g_host_cache.hz == qzeros && g_host_cache.K == K && g_host_cache.N == N;
    if (!hit) {
        host_cache_drop(g_host_cache.owner);
        g_host_cache.owner = c;
        LB_CU(c, lb_drv.MemAlloc(&g_host_cache.dq, qb));
        LB_CU(c, lb_drv.MemAlloc(&g_host_cache.ds, sb));
        if (qzeros) LB_CU(c, lb_drv.MemAlloc(&g_host_cache.dz, zb));
        LB_CU(c, lb_drv.MemAlloc(&g_host_cache.dx, (size_t)K * 4));
        LB_CU(c, lb_drv.MemAlloc(&g_host_cache.dy, (size_t)N * 4));
        LB_CU(c, lb_drv.MemcpyHtoDAsync(g_host_cache.dq, qweight, qb, c->stream));
        LB_CU(c, lb_drv.MemcpyHtoDAsync(g_host_cache.ds, scales, sb, c->stream));
        if (qzeros) LB_CU(c, lb_drv.MemcpyHtoDAsync(g_host_cache.dz, qzeros, zb, c->stream));
        g_host_cache.hq = qweight; g_host_cache.hs = scales; g_host_cache.hz = qzeros;
        g_host_cache.K = K; g_host_cache.N = N;
    }
    LB_CU(c, lb_drv.MemcpyHtoDAsync(g_host_cache.dx, x, xb, c->stream));
    if (flags & LB_GEMV_Y_ACCUM) LB_CU(c, lb_drv.MemcpyHtoDAsync(g_host_cache.dy, y, yb, c->stream));
    LB_TRY(lb_gemv_int4(c, g_host_cache.dq, g_host_cache.ds, g_host_cache.dz, g_host_cache.dx, g_host_cache.dy, K, N,
                        flags));
    LB_CU(c, lb_drv.MemcpyDtoHAsync(y, g_host_cache.dy, yb, c->stream));
    LB_CU(c, lb_drv.StreamSynchronize(c->stream));
    return LB_OK;
}

/* ---- batched int4 projection ---------------------------------------------------------
 * 33..256 tokens (from 9 with LB_GEMM_TCGEN05): gemm_int4_tc (tcgen05, one CTA per SM: 128 columns x a K slice); up to 32 tokens
 * gemm_int4_tc_exact16 / 32 or, as always with LB_GEMM_MMA_SYNC, the mma.sync kernels (two CTAs per SM).  The K slices of a column block are the CTAs
 * of one cluster (<= 8); the slice count fills the SMs without starting a second wave and leaves
 * every slice at least four K-groups. */

/* clusters of k CTAs of a kernel that run at once, asked once per k (slot) */
static int clusters_at_once(lb_ctx* c, int kernel, int k, unsigned threads, unsigned smem, int per_sm, int* slot) {
    if (k <= 1) return c->sm_count * per_sm;
    if (!*slot) {
        CUlaunchConfig cfg;
        memset(&cfg, 0, sizeof cfg);
        CUlaunchAttribute attr;
        memset(&attr, 0, sizeof attr);
        attr.id = CU_LAUNCH_ATTRIBUTE_CLUSTER_DIMENSION;
        attr.value.clusterDim.x = 1; attr.value.clusterDim.y = (unsigned)k; attr.value.clusterDim.z = 1;
        cfg.gridDimX = (unsigned)c->sm_count; cfg.gridDimY = (unsigned)k; cfg.gridDimZ = 1;
        cfg.blockDimX = threads; cfg.blockDimY = cfg.blockDimZ = 1;
        cfg.sharedMemBytes = smem;
        cfg.attrs = &attr; cfg.numAttrs = 1;
        int n = 0;
        if (!c->fn[kernel] || lb_drv.OccupancyMaxActiveClusters(&n, c->fn[kernel], &cfg) != CUDA_SUCCESS || n < 1) n = c->sm_count * per_sm / k;
        *slot = n;
    }
    return *slot;
}

/* K slices (CTAs of a cluster) of the tcgen05 kernels, one CTA per SM: the SMs of a GPC do not all divide by the slices, and one cluster
 * too many doubles the time (4096 -> 2048 at 48 tokens: 14.2 us as 16 clusters of 8, 8.0 as clusters of what fits) */
static int tc_slices(lb_ctx* c, int blocks, int groups) {
    int k = c->sm_count / blocks;
    if (k > 8) k = 8;
    while (k > 1 && (groups / k < 4 || clusters_at_once(c, LBK_gemm_int4_tc_256, k, LB_TC_THREADS, LB_TC_X_HALVES * 256 * 128, 1, &c->tc_clusters[k]) < blocks)) k--;
    return k < 1 ? 1 : k;
}
/* K slices of the mma.sync kernels, two CTAs per SM */
static int mma_slices(const lb_ctx* c, int blocks, int groups) {
    int k = 1;
    while (k < 8 && blocks * k < c->sm_count * 3 / 2 && groups / (k * 2) >= 4) k *= 2;
    return k;
}

/* 17..32 tokens without a flag, and 9..16 where launch_ring does not apply: gemm_int4_tc_exact16 / 32 (1) or the mma.sync kernels (0); neither rounds a weight.  us, mma.sync / tcgen05:
 * matrices split along K: 17408 -> 5120 at 12 tokens 33.9 / 27.1, at 32 47.5 / 31.1; 1024 -> 1024 6.9 / 5.3, 11.4 / 6.3
 * short columns, where the start counts: K = 512 at 9 tokens 4.8 / 4.9, 640 5.5 / 5.3; K = 256 at 17 tokens 5.0 / 5.2, 384 5.7 / 5.5
 * whole columns up to 16 tokens (two CTAs per SM against one): 5120 -> 17408 at 12 tokens 23.9 / 24.5; up to 32 tokens 34.6 / 28.0, 5120 -> 34816 54.7 / 57
 * up to 16 tokens, long columns of which mma.sync makes twice as many slices and all of its clusters run at once (29..32 and 56..70 blocks, fewer
 *   by one above 12 tokens): 17408 -> 7168 at 12 tokens 35.2 / 37.9, 8192 -> 7168 19.6 / 20.3, 6144 -> 7168 16.1 / 16.3 (at 16 16.5 / 16.4), 5120 -> 7168 14.5 / 14.3;
 *   one block more than fits: 8192 -> 9216 31.3 / 20.6
 * or four times as many while two thirds of the SMs have no tcgen05 CTA (46..49 blocks): 17408 -> 5888 35.6 / 37.6, 11008 -> 5888 26.2 / 25.6 */
static int exact_on_tc(lb_ctx* c, int B, int blocks, int groups) {
    if (groups <= (B > 16 ? 2 : 4)) return 0;
    if (B > 16) return blocks <= c->sm_count;
    if (2 * blocks > c->sm_count) return 0;
    const int tc = tc_slices(c, blocks, groups), mma = mma_slices(c, blocks, groups);
    if (groups >= (B > 12 ? 64 : 48) && mma >= 2 * tc && blocks < clusters_at_once(c, LBK_gemm_int4_mma_b16, mma, 256, 4 * 16 * 320, 2, &c->mma_clusters[mma]) - (B > 12)) return 0;
    if (groups >= 112 && mma >= 4 * tc && 3 * blocks * tc < 2 * c->sm_count) return 0;
    return 1;
}

/* X [B, K] fp16, box = 64 k (128 bytes) x nt tokens, laid down with the 128-byte swizzle */
static int map_tokens(lb_ctx* c, lb_bgemm_params* p, int nt) {
    CUtensorMap tm;
    cuuint64_t dims[2] = {(cuuint64_t)p->K, (cuuint64_t)p->B}, strides[1] = {(cuuint64_t)p->K * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)nt}, estr[2] = {1, 1};
    LB_CU(c, lb_drv.TensorMapEncodeTiled(&tm, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, (void*)p->x, dims, strides, box, estr,
                                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
    memcpy(p->tmap_x, &tm, sizeof tm);
    return LB_OK;
}

/* gemm_int4_ring8 / 16 run 2 to 16 tokens at every size, more column blocks than SMs too (us, the kernels before / ring: 5120 -> 17408 at 2 tokens 19.0 / 12.2, 12 24.4 /
 * 15.2; 17408 -> 5120 28.2 / 15.4, 27.5 / 18.7; 1024 -> 1024 5.1 / 4.2, 5.7 / 4.8; 8192 -> 2048 9.6 / 6.7, 8.9 / 8.0; one block more than SMs, 5120 -> 19072, at 2 29.6 /
 * 22.0, 16 40.1 / 28.2; 5120 -> 34816 32.4 / 24.3, 39.9 / 29.8; 2048 -> 24576 15.0 / 11.4, 22.8 / 14.1; 4096 -> 37888 26.4 / 21.7, 33.1 / 26.0), but for those of 9 to 16
 * tokens that ran on the kernels of LB_GEMM_MMA_SYNC before there was a ring: their callers may compare rows with and without the flag, and keep the kernel for that
 * alone.  It is the slower one (8192 -> 7168 at 12 tokens 19.6 / 14.1, 14336 -> 5888 31.8 / 21.1), and such a matrix's rows of 2 to 8 tokens, which are the ring's,
 * differ from these in the last bits; the header says which sizes they are.  Whole columns of more than 1024, which the same rule would keep, are the decode batches
 * that the ring is for (5120 -> 17408). */
static int pinned_to_mma(lb_ctx* c, int B, int blocks, int groups) {
    return B > 8 && !exact_on_tc(c, B, blocks, groups) && (2 * blocks <= c->sm_count || groups <= 8);
}
/* gemm_int4_ring8 / 16 */
static int launch_ring(lb_ctx* c, lb_bgemm_params* p, int blocks, int groups) {
    const int nt = p->B > 8 ? 16 : 8, ksplit = tc_slices(c, blocks, groups);
    CUtensorMap tm; /* qweight as [N/32 column blocks][K/8 packed rows][32 columns] */
    cuuint64_t dims[3] = {32, (cuuint64_t)(p->K / 8), (cuuint64_t)(p->N / 32)}, strides[2] = {(cuuint64_t)p->N * 4, 128};
    cuuint32_t box[3] = {32, 16, 4}, estr[3] = {1, 1, 1};
    LB_CU(c, lb_drv.TensorMapEncodeTiled(&tm, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, (void*)p->qweight, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
    memcpy(p->tmap_w, &tm, sizeof tm);
    LB_TRY(map_tokens(c, p, nt));
    void* params[] = {p};
    return lb_launch_cluster(c, nt > 8 ? LBK_gemm_int4_ring16 : LBK_gemm_int4_ring8, (unsigned)blocks, (unsigned)ksplit, 1, LB_RING_THREADS, (unsigned)LB_RING_SMEM(nt), params, 1, (unsigned)ksplit);
}

int lb_gemm_int4_epi(lb_ctx* c, uint64_t qweight, uint64_t scales, uint64_t qzeros, uint64_t x, uint64_t y, int K, int N, int B, int flags, int epi) {
    if (!c || !qweight || !scales || !x || !y || K <= 0 || N <= 0 || K % 128 || N % 16 || B < 1 || B > LB_GEMM_MAX_BATCH ||
        (flags & ~(LB_GEMV_Y_F32 | LB_GEMM_MMA_SYNC | LB_GEMM_TCGEN05)) ||
        ((flags & LB_GEMM_MMA_SYNC) && (flags & LB_GEMM_TCGEN05)) || ((flags & LB_GEMM_TCGEN05) && B <= 8) ||
        ((flags & LB_GEMM_MMA_SYNC) && B > 64))
        return lb_fail(c, LB_ERR_INVALID, "lb_gemm_int4: bad argument (K %% 128, N %% 16, 1 <= B <= %d, flags LB_GEMV_Y_F32, LB_GEMM_MMA_SYNC (up to 64 tokens) or LB_GEMM_TCGEN05 (9 tokens or more))",
                       LB_GEMM_MAX_BATCH);
    lb_bgemm_params p;
    memset(&p, 0, sizeof p);
    p.qweight = (const uint32_t*)qweight; p.scales = (const uint16_t*)scales; p.qzeros = (const uint32_t*)qzeros;
    p.x = (const uint16_t*)x; p.y = (void*)y;
    p.K = K; p.N = N; p.B = B; p.y_f32 = (flags & LB_GEMV_Y_F32) != 0; p.epi = epi;
    if (epi && (B <= 32 || (flags & ~LB_GEMV_Y_F32) || (epi == LB_BG_SWIGLU && N % 128))) return lb_fail(c, LB_ERR_INVALID, "lb_gemm_int4: an epilogue of the kernels of 33 tokens or more");
    p.status = (uint32_t*)c->dev_status;
    /* one token: the GEMV kernel (TMA-streamed, integer tensor-core products) is the faster path, with the same result type */
    if (B == 1 && !(flags & LB_GEMM_MMA_SYNC) && N % 32 == 0 && ((qweight | scales | qzeros | x | y) & 15ull) == 0)
        if (lb_gemv_int4(c, qweight, scales, qzeros, x, y, K, N, flags & LB_GEMV_Y_F32) == LB_OK) return LB_OK; /* else: the batched kernel */
    const int blocks = (N + 127) / 128, groups = K / 128;
    void* params[] = {&p};
    if (x & 15) return lb_fail(c, LB_ERR_INVALID, "lb_gemm_int4: x must be 16-byte aligned");
    const int mma_ok = ((qweight & 7) | (scales & 3)) == 0; /* the mma.sync kernels load the words and scales of two columns at once */
    if ((flags & LB_GEMM_MMA_SYNC) && !mma_ok) return lb_fail(c, LB_ERR_INVALID, "lb_gemm_int4: LB_GEMM_MMA_SYNC wants qweight 8-byte and scales 4-byte aligned");
    const int ring_ok = N % 32 == 0 && ((qweight | scales | qzeros) & 15) == 0; /* what its bulk copies want */
    if (ring_ok && B > 1 && B <= 16 && !(flags & (LB_GEMM_MMA_SYNC | LB_GEMM_TCGEN05)) && !pinned_to_mma(c, B, blocks, groups)) return launch_ring(c, &p, blocks, groups);
    const int exact = B <= 32 && !(flags & (LB_GEMM_MMA_SYNC | LB_GEMM_TCGEN05)) && (!mma_ok || (B > 8 && exact_on_tc(c, B, blocks, groups)));
    if (exact || (B > 32 && !(flags & LB_GEMM_MMA_SYNC)) || (flags & LB_GEMM_TCGEN05)) {
        const int nt = exact ? (B > 16 ? 32 : 16) : LB_TC_NT(B), halves = nt > LB_TC_HALVES_FROM;
        LB_TRY(map_tokens(c, &p, nt));
        const int ksplit = tc_slices(c, blocks, groups);
        const unsigned smem = halves ? (unsigned)(LB_TC_X_HALVES * nt * 128) : (unsigned)((exact ? 7 : LB_TC_STAGES(nt)) * nt * 256); /* activation stages; the partial tile [nt][132] fp32 fits over them */
        return lb_launch_cluster(c, exact ? (nt > 16 ? LBK_gemm_int4_tc_exact32 : LBK_gemm_int4_tc_exact16) : halves ? (epi ? LBK_gemm_int4_tc_256_epi : LBK_gemm_int4_tc_256) : epi ? LBK_gemm_int4_tc_epi : LBK_gemm_int4_tc, (unsigned)blocks, (unsigned)ksplit, 1,
                                 exact ? (nt > 16 ? LB_TC_EXACT32_THREADS : LB_TC_EXACT16_THREADS) : LB_TC_THREADS, smem, params, 1, (unsigned)ksplit);
    }
    const int rows = B > 32 ? 64 : B > 16 ? 32 : B > 8 ? 16 : 8; /* token rows the CTA stages */
    const int kernel = B > 32 ? LBK_gemm_int4_mma_b64 : B > 16 ? LBK_gemm_int4_mma_b32 : B > 8 ? LBK_gemm_int4_mma_b16 : LBK_gemm_int4_mma_b8;
    const unsigned smem = (unsigned)((B > 16 ? 3 : 4) * rows * 320); /* activation ring (the partial tile reuses it) */
    const int ksplit = mma_slices(c, blocks, groups);
    return lb_launch_cluster(c, kernel, (unsigned)blocks, (unsigned)ksplit, 1, 256, smem, params, 1, (unsigned)ksplit);
}

LB_API int lb_gemm_int4(lb_ctx* c, uint64_t qweight, uint64_t scales, uint64_t qzeros, uint64_t x, uint64_t y, int K, int N,
                        int B, int flags) {
    return lb_gemm_int4_epi(c, qweight, scales, qzeros, x, y, K, N, B, flags, LB_BG_STORE);
}

LB_API int lb_gptq_dequant(lb_ctx* c, uint64_t qweight, uint64_t scales, uint64_t qzeros, uint64_t w_out, int K, int N) {
    if (!c || !qweight || !scales || !w_out || K % 128 || N % 8) return lb_fail(c, LB_ERR_INVALID, "lb_gptq_dequant: bad argument");
    void* params[] = {&qweight, &scales, &qzeros, &w_out, &K, &N};
    return lb_launch(c, LBK_gptq_dequant_f32, (unsigned)((N + 255) / 256), (unsigned)(K / 8), 1, 256, 0, params, 0);
}

LB_API int lb_gptq_unpack(lb_ctx* c, uint64_t qweight, uint64_t q_out, int K, int N) {
    if (!c || !qweight || !q_out || K % 8) return lb_fail(c, LB_ERR_INVALID, "lb_gptq_unpack: bad argument");
    void* params[] = {&qweight, &q_out, &K, &N};
    return lb_launch(c, LBK_gptq_unpack_u8, (unsigned)((N + 255) / 256), (unsigned)(K / 8), 1, 256, 0, params, 0);
}

/* shared memory of dense_bf16_stream: 8 warps x 2 ring slots of one row, the fp32 activations, reduction scratch, mbarriers */
static size_t dense_stream_smem(int K) { return (size_t)8 * 2 * K * 2 + (size_t)K * 4 + 40 * 4 + 16 * 8; }
static int dense_streams(const lb_ctx* c, int N, int K) {
    return K % 8 == 0 && N >= 8 * c->sm_count &&
           dense_stream_smem(K) <= (size_t)c->max_smem_optin - (size_t)((c->fn_static_smem[LBK_dense_bf16_stream] + 1023) & ~1023);
}

/* CTAs of the dense GEMV = arg-max candidates it leaves */
int lb_dense_ctas(lb_ctx* c, int N, int K) {
    if (dense_streams(c, N, K)) return c->sm_count; /* one CTA per SM, rows streamed through shared memory */
    int ctas = (N + 7) / 8, cap = c->sm_count * 8;  /* each CTA strides over rows, 8 warps = 8 rows at a time */
    return ctas > cap ? cap : ctas;
}

int lb_dense_launch(lb_ctx* c, uint64_t w, uint64_t x, uint64_t y, int N, int K, int x_mode, uint64_t norm_w, float eps,
                    uint64_t part_val, uint64_t part_idx) {
    if (!c || !w || !x || !y || K % 8 || N <= 0) return lb_fail(c, LB_ERR_INVALID, "dense bf16 GEMV: bad argument");
    lb_dense_params p;
    memset(&p, 0, sizeof p);
    p.w = (const uint16_t*)w; p.x = (const void*)x; p.y = (float*)y; p.norm_w = (const void*)norm_w;
    p.N = N; p.K = K; p.x_mode = x_mode; p.eps = eps;
    p.part_val = (float*)part_val; p.part_idx = (int32_t*)part_idx;
    p.status = (uint32_t*)c->dev_status;
    int ctas = lb_dense_ctas(c, N, K);
    void* params[] = {&p};
    if (dense_streams(c, N, K))
        return lb_launch(c, LBK_dense_bf16_stream, (unsigned)ctas, 1, 1, 256, (unsigned)dense_stream_smem(K), params, 1);
    return lb_launch(c, LBK_dense_bf16_gemv, (unsigned)ctas, 1, 1, 256, (unsigned)(K * 4 + 256), params, 1);
}

LB_API int lb_dense_bf16_gemv(lb_ctx* c, uint64_t w, uint64_t x, uint64_t y, int N, int K, int x_is_f32) {
    return lb_dense_launch(c, w, x, y, N, K, x_is_f32 ? LB_X_F32 : LB_X_F16, 0, 1e-6f, 0, 0);
}

LB_API int lb_deltanet_step(lb_ctx* c, uint64_t state, uint64_t q, uint64_t k, uint64_t v, uint64_t z, uint64_t g,
                            uint64_t beta, uint64_t out, int HV, int HK, int n_steps, int in_is_f32) {
    if (!c || !state || !q || !k || !v || !g || !beta || !out || HV <= 0 || HK <= 0 || HV % HK || n_steps < 1)
        return lb_fail(c, LB_ERR_INVALID, "lb_deltanet_step: bad argument");
    lb_deltanet_params p;
    memset(&p, 0, sizeof p);
    p.state = (float*)state; p.q = (const void*)q; p.k = (const void*)k; p.v = (const void*)v;
    p.z = (const float*)z; p.g = (const float*)g; p.beta = (const float*)beta; p.out = (float*)out;
    p.HV = HV; p.HK = HK;
    void* params[] = {&p, &n_steps};
    /* two steps: the kernel of few steps while its CTAs are at most two per SM (fp32, two steps / run: 48 heads 3.74 / 3.96 us, 96 heads 4.99 / 4.66) */
    const int few = n_steps == 1 || (n_steps == 2 && 2 * HV <= c->sm_count);
    /* More than twelve steps: 16 columns per CTA instead of 32 where the fullest SM then has less than twice as many of them and holds them
     * at a time (four).  us, 32 / 16 columns, bf16: 48 heads (two
     * CTAs / three) 8 steps 4.8 / 5.1, 16 7.3 / 7.1, 64 21.5 / 19.5, 256 78.4 / 68.9; 16 heads (one / one) 16 steps 5.0 / 4.5, 256 52.1 / 42.1; 24 and 32 heads
     * (one / two) 24 steps 6.6 / 7.2, 256 52.1 / 53.5.  fp32: 48 heads 9 steps 5.5 / 5.7, 12 6.2 / 6.3, 15 7.0 / 7.0, 24 9.4 / 9.1, 256 77.5 / 67.0; 16 heads 15 steps
     * 5.3 / 4.7, 256 50.9 / 41.4; 24 heads 24 steps 6.5 / 7.2, 256 51.0 / 51.8; 64 (two / four) 9 steps 5.5 / 7.0, 256 77.3 / 84.8; 96 (three / six, of which four fit at
     * a time) 9 steps 6.9 / 10.1, 256 108 / 127 */
    const int ctas32 = (4 * HV + c->sm_count - 1) / c->sm_count, ctas16 = (8 * HV + c->sm_count - 1) / c->sm_count; /* on the fullest SM */
    const int narrow = !few && n_steps > 12 && ctas16 < 2 * ctas32 && ctas16 <= 4;
    const int kernel = few ? (n_steps == 1 ? (in_is_f32 ? LBK_deltanet_one_f32 : LBK_deltanet_one_bf16) : (in_is_f32 ? LBK_deltanet_two_f32 : LBK_deltanet_two_bf16))
                     : narrow ? (in_is_f32 ? LBK_deltanet_step16_f32 : LBK_deltanet_step16_bf16)
                              : (in_is_f32 ? LBK_deltanet_step_f32 : LBK_deltanet_step_bf16);
    return lb_launch(c, kernel, (unsigned)HV, narrow ? 8 : 4, 1, 128, 0, params, 1);
}

LB_API int lb_decay_gate(lb_ctx* c, uint64_t a, uint64_t a_log, uint64_t dt_bias, uint64_t b, uint64_t g_out,
                         uint64_t beta_out, int n) {
    if (!c || !a || !a_log || !dt_bias || !g_out || n <= 0) return lb_fail(c, LB_ERR_INVALID, "lb_decay_gate: bad argument");
    lb_decay_params p = {(const float*)a, (const float*)a_log, (const float*)dt_bias, (const float*)b,
                         (float*)g_out, (float*)beta_out, n};
    void* params[] = {&p};
    return lb_launch(c, LBK_decay_gate_beta, (unsigned)((n + 127) / 128), 1, 1, 128, 0, params, 1);
}

/* attn_decode_mma: slices of 128 rows (a block of 16 per warp), and no more of them than make one wave of one CTA per SM: the CTAs of a KV head wait for
 * each other.  24 / 4 heads at 100 000 rows: 69 us as 37 slices a head, 102 with the 64 (two waves) of the kernel before; 48 / 8 heads, 18 slices / 64: 2400 rows 13.6 / 25.2, 8192 20.9 / 54.5,
 * 100 000 129 / 188; 8 / 8 heads 8192 rows 18.6 / 39.7 */
int lb_attn_mma_splits(lb_ctx* c, int pos, int HKV) {
    const int cap = (c->sm_count < 512 ? c->sm_count : 512) / HKV; /* the scratch holds 512 records of 8 heads */
    const int s = (pos + 127) / 128;
    return s > cap ? (cap < 1 ? 1 : cap) : s < 1 ? 1 : s;
}

/* a context with a shorter limit for its waits: one look */
int lb_attn_stay(const lb_ctx* c) { return c->wait_limit_ns && c->wait_limit_ns < 200 * LB_ATTN_STAY ? 0 : LB_ATTN_STAY; }

unsigned lb_attn_mma_smem(int G) { /* as attn_mma_body lays it out */
    return (unsigned)(16 * 576 + 8 * G * 260 * 4 + 2 * 256 * 2 + 2 * 64 * 4 + 2 * 8 * 8 * 4);
}

LB_API int lb_attention_decode(lb_ctx* c, uint64_t q, uint64_t k_new, uint64_t v_new, uint64_t gate, uint64_t q_norm_w,
                               uint64_t k_norm_w, uint64_t k_cache, uint64_t v_cache, uint64_t out, int pos, int HQ,
                               int HKV, int in_is_f32, int rot_dims, float rope_theta, float eps) {
    if (!c || !q || !k_new || !v_new || !k_cache || !v_cache || !out || pos < 0 || HKV <= 0 || HQ % HKV)
        return lb_fail(c, LB_ERR_INVALID, "lb_attention_decode: bad argument");
    int G = HQ / HKV;
    if (!(G == 1 || G == 2 || G == 3 || G == 4 || G == 6) || HKV > 8)
        return lb_fail(c, LB_ERR_INVALID, "lb_attention_decode: unsupported head ratio %d/%d", HQ, HKV);
    if ((q_norm_w == 0) != (k_norm_w == 0)) return lb_fail(c, LB_ERR_INVALID, "lb_attention_decode: q/k norm weights must come together");
    if (rot_dims < 0 || rot_dims > 128 || rot_dims % 8) return lb_fail(c, LB_ERR_INVALID, "lb_attention_decode: bad rot_dims");
    lb_attn_params p;
    memset(&p, 0, sizeof p);
    p.q = (const void*)q; p.k_new = (const void*)k_new; p.v_new = (const void*)v_new; p.gate = (const void*)gate;
    p.q_norm_w = (const uint16_t*)q_norm_w; p.k_norm_w = (const uint16_t*)k_norm_w;
    p.k_cache = (uint16_t*)k_cache; p.v_cache = (uint16_t*)v_cache; p.out = (float*)out;
    p.scratch = (float*)c->attn_scratch; p.counters = (uint32_t*)(c->gemv_counters + 2048 * 4);
    p.pos = pos; p.HQ = HQ; p.HKV = HKV;
    p.splits = lb_attn_mma_splits(c, pos, HKV);
    p.stay = lb_attn_stay(c);
    p.status = (uint32_t*)c->dev_status;
    p.in_dtype = in_is_f32 ? 1 : 0;
    p.gate_stride = 256; p.q_stride = 256;
    p.rot_dims = rot_dims; p.rope_theta = rope_theta; p.eps = eps;
    for (int i = 0; i < rot_dims / 2; i++) p.rope_freq[i] = exp2(-log2((double)rope_theta) * (double)i / (double)(rot_dims / 2));
    void* params[] = {&p};
    return lb_launch(c, LBK_attn_decode_mma, (unsigned)HKV, (unsigned)p.splits, 1, 256, lb_attn_mma_smem(G), params, 1);
}

/* tensor maps of a chunk's keys and values: `rows` rows of `ld` bf16 values, read in boxes of 64 features x box_rows */
static int ac_map(lb_ctx* c, unsigned char* out, CUdeviceptr p, int width, int ld, int rows, int box_rows) {
    CUtensorMap tm;
    cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows}, es[2] = {1, 1};
    LB_CU(c, lb_drv.TensorMapEncodeTiled(&tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)p, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
    memcpy(out, &tm, sizeof tm);
    return LB_OK;
}
int lb_ac_fill(lb_ctx* c, lb_ac_maps* m, CUdeviceptr k, int k_ld, CUdeviceptr tail, int tail_w, int tail_ld, CUdeviceptr v, int v_ld, int vdim, int rows) {
    memset(m, 0, sizeof *m);
    LB_TRY(ac_map(c, m->k, k, k_ld, k_ld, rows, 128));
    if (tail) LB_TRY(ac_map(c, m->tail, tail, tail_w, tail_ld, rows, 128));
    return ac_map(c, m->v, v, v_ld, v_ld, rows, 8192 / vdim);
}

/* Key blocks of a tile are dealt to several CTAs where the tiles of a launch leave half of the SMs idle or more: as many parts as make one wave, of two blocks at
 * least (a part pays its queries' way in and its rows' way out). */
int lb_ac_launch(lb_ctx* c, int kernel, int merge, int rows, int kv_heads, int keys, int vdim, CUdeviceptr scratch, size_t bytes, void* p, lb_ac_maps* maps) {
    lb_ac_split sp;
    memset(&sp, 0, sizeof sp);
    sp.tiles = (rows + LB_AC_ROWS - 1) / LB_AC_ROWS;
    sp.part = (float*)scratch;
    const size_t one = (size_t)kv_heads * sp.tiles * LB_AC_ROWS * (vdim + 4) * 4;
    int parts = c->sm_count / (sp.tiles * kv_heads);
    if (parts > (keys + 127) / 256) parts = (keys + 127) / 256;
    if (parts > 16) parts = 16;
    if (one && (size_t)parts > bytes / one) parts = (int)(bytes / one);
    sp.parts = parts > 1 ? parts : 1;
    void* params[] = {p, maps, &sp};
    LB_TRY(lb_launch(c, kernel, (unsigned)sp.tiles, (unsigned)kv_heads, (unsigned)sp.parts, LB_AC_THREADS, LB_AC_SMEM, params, 1));
    if (sp.parts == 1) return LB_OK;
    return lb_launch(c, merge, (unsigned)sp.tiles, (unsigned)kv_heads, (unsigned)(vdim / 32), 256, 0, params, 1);
}

LB_API int lb_rmsnorm(lb_ctx* c, uint64_t x, uint64_t res, uint64_t w, uint64_t y, uint64_t sum_out, int rows, int D,
                      float eps, int one_plus_w) {
    if (!c || !x || !w || !y || rows <= 0 || D <= 0) return lb_fail(c, LB_ERR_INVALID, "lb_rmsnorm: bad argument");
    void* params[] = {&x, &res, &w, &y, &sum_out, &D, &eps, &one_plus_w};
    return lb_launch(c, LBK_rmsnorm_f32, (unsigned)rows, 1, 1, 256, 0, params, 1);
}

LB_API int lb_argmax(lb_ctx* c, uint64_t x, int n, uint64_t out_idx) {
    if (!c || !x || !out_idx || n <= 0) return lb_fail(c, LB_ERR_INVALID, "lb_argmax: bad argument");
    uint64_t zero = 0;
    void* params[] = {&x, &n, &out_idx, &zero, &zero, &zero};
    return lb_launch(c, LBK_argmax_f32, 1, 1, 1, 1024, 0, params, 1);
}

LB_API int lb_sample_topk(lb_ctx* c, uint64_t x, int n, float temperature, int top_k, uint64_t seed, uint64_t counter, uint64_t out_idx,
                          uint64_t probs_out, uint64_t idx_out) {
    if (!c || !x || !out_idx || n <= 0 || top_k < 1 || top_k > 64) return lb_fail(c, LB_ERR_INVALID, "lb_sample_topk: bad argument (1 <= top_k <= 64)");
    uint64_t zero = 0;
    void* params[] = {&x, &n, &out_idx, &zero, &zero, &temperature, &top_k, &seed, &counter, &probs_out, &idx_out};
    return lb_launch(c, LBK_topk_sample_f32, 1, 1, 1, 1024, 0, params, 1);
}

LB_API int lb_embed(lb_ctx* c, uint64_t table, uint64_t token, uint64_t out, int D) {
    if (!c || !table || !token || !out || D <= 0) return lb_fail(c, LB_ERR_INVALID, "lb_embed: bad argument");
    void* params[] = {&table, &token, &out, &D};
    return lb_launch(c, LBK_embed_bf16, (unsigned)((D + 1023) / 1024), 1, 1, 256, 0, params, 1);
}
