// Gated DeltaNet single-token recurrence for sm_100a.
//
// Restates inference/deltanet_fused.ls:97-149 (and delta_update.ls:24-54):
//   r_j   = sum_i k_i S_ij                  (pre-update, un-decayed state)
//   d_j   = beta (v_j - r_j)
//   S_ij <- g S_ij + k_i d_j
//   o_j   = sum_i S_ij(new) q_i             [ * silu(z_j) when z is given ]
// with decay g = exp(-exp(A_log) softplus(a + dt_bias)), beta = sigmoid(b)
// (inference/decay_gate.ls:28-57, inference/recur.ls:45-55).
//
// The reference walks the 64 KB head state twice from global memory with one
// thread per column.  Columns j of a head are independent, so here a CTA owns
// a 32-column slab of one head and holds it in REGISTERS (128 threads x 32
// fp32): the state is read from HBM once and written once per step, and when
// n_steps > 1 it stays on chip for the whole run of steps.
#include "deltanet_core.cuh"

// A warp owns 8 columns of a head, all 128 rows of them: lane (rg, cg) holds 16 rows (four neighbouring ones of every 32, so that the
// lanes' 16-byte reads of a token's k or q are one conflict-free wavefront) of 2 columns, the rows in pairs for packed multiply-adds; cg is
// the fast part of the lane number, so that a half-warp's 8-byte accesses to the state fill whole sectors.  A
// step needs nothing from another warp: both sums over the rows end in three shuffles, and what the warps of a CTA share, the operands of
// DN_RUN tokens in fp32, costs one block barrier per DN_RUN tokens.  A thread loads its piece of the run after next into registers and
// stores it a run later, so the chain of a step (dot, three shuffles, update) meets no trip to L2.  The read-outs of four tokens are summed
// together (seven shuffles instead of 24), in the order of a single one: the same bits for one step and for many.
// 48 heads, bf16 (us before -> after; before: a column's rows in four lanes, 16 reads of k and q and a barrier a token): 5.0 -> 4.2 at 4 steps,
// 38 -> 24 at 64, 144 -> 86 at 256.  Two warps per scheduler now take 620 cycles a token, of which 256 are the
// multiply-adds' and 440 one warp's chain; reading the next token's k ahead moved it by 3 % either way.
#define DN_RUN 8
template <typename T> struct dn_in; // element type of q, k, v: 16 bytes of them, and how they go to shared memory as fp32
template <> struct dn_in<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void put(float* dst, uint4 u) { *reinterpret_cast<uint4*>(dst) = u; }
};
template <> struct dn_in<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void put(float* dst, uint4 u) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(u.x << 16, u.x & 0xffff0000u, u.y << 16, u.y & 0xffff0000u);
        *reinterpret_cast<uint4*>(dst + 4) = make_uint4(u.z << 16, u.z & 0xffff0000u, u.w << 16, u.w & 0xffff0000u);
    }
};
__device__ __forceinline__ uint64_t dn_pack(float x, float y) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 dn_unpack(uint64_t a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ uint64_t dn_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t dn_mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float dn_sum4(uint64_t a, uint64_t b) { // two running pair sums
    const float2 x = dn_unpack(a), y = dn_unpack(b);
    return (x.x + x.y) + (y.x + y.y);
}

// a lane's two columns of a state row: 8 bytes at once where the state's address allows it (PAIRS)
template <bool PAIRS> __device__ __forceinline__ float2 dn_row(const float* r) {
    if (!PAIRS) return make_float2(r[0], r[1]);
    return *reinterpret_cast<const float2*>(r);
}
template <bool PAIRS> __device__ __forceinline__ void dn_load_rows(const float* S, uint64_t (&s)[4][2][2]) {
    float2 x[4][2][2];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i >> 2][(i >> 1) & 1][i & 1] = dn_row<PAIRS>(S + (size_t)(32 * (i >> 2) + (i & 3)) * DN_D);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            s[j][e][0] = dn_pack(x[j][e][0].x, x[j][e][1].x);
            s[j][e][1] = dn_pack(x[j][e][0].y, x[j][e][1].y);
        }
}
__device__ __forceinline__ void dn_load_state(const float* S, bool pairs, uint64_t (&s)[4][2][2]) {
    if (pairs) dn_load_rows<true>(S, s);
    else dn_load_rows<false>(S, s);
}
__device__ __forceinline__ void dn_store_state(float* S, bool pairs, const uint64_t (&s)[4][2][2]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float* r = S + (size_t)(32 * j + 2 * e) * DN_D;
            const float2 x = dn_unpack(s[j][e][0]), y = dn_unpack(s[j][e][1]);
            if (pairs) {
                *reinterpret_cast<float2*>(r) = make_float2(x.x, y.x);
                *reinterpret_cast<float2*>(r + DN_D) = make_float2(x.y, y.y);
            } else {
                r[0] = x.x; r[1] = y.x;
                r[DN_D] = x.y; r[DN_D + 1] = y.y;
            }
        }
}
// r_j = sum_i k_i S_ij (pre-update state): four running sums per column
__device__ __forceinline__ void dn_recall(const uint64_t (&k)[4][2], const uint64_t (&s)[4][2][2], uint64_t (&a)[2][2]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int e = 0; e < 2; ++e) a[c][e] = j ? dn_fma2(k[j][e], s[j][e][c], a[c][e]) : dn_mul2(k[j][e], s[j][e][c]);
}
__device__ __forceinline__ void dn_decay(float g, uint64_t (&s)[4][2][2]) {
    const uint64_t g2 = dn_pack(g, g);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int c = 0; c < 2; ++c) s[j][e][c] = dn_mul2(g2, s[j][e][c]);
}
// S_ij += k_i d_j on the decayed state, o_j = sum_i S_ij q_i
__device__ __forceinline__ void dn_update(const uint64_t (&k)[4][2], const uint64_t (&q)[4][2], float d0, float d1, uint64_t (&s)[4][2][2], uint64_t (&a)[2][2]) {
    const uint64_t d[2] = {dn_pack(d0, d0), dn_pack(d1, d1)};
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                s[j][e][c] = dn_fma2(k[j][e], d[c], s[j][e][c]);
                a[c][e] = j ? dn_fma2(q[j][e], s[j][e][c], a[c][e]) : dn_mul2(q[j][e], s[j][e][c]);
            }
}
__device__ __forceinline__ void dn_reduce(float& x, float& y) { // over the eight row groups
#pragma unroll
    for (int m = 4; m < 32; m <<= 1) {
        x += __shfl_xor_sync(0xffffffffu, x, m);
        y += __shfl_xor_sync(0xffffffffu, y, m);
    }
}
__device__ __forceinline__ void dn_read(const float* row, uint64_t (&r)[4][2]) { // a lane's rows of k or q, from shared memory
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(row + 32 * j);
        r[j][0] = u.x;
        r[j][1] = u.y;
    }
}

// One or two steps, where a trip to memory is all that counts: a thread holds 32 rows of one column (rows 8 q4 + 32 j + i), so that a warp's loads
// of the state are whole sectors, all of them in flight at once, ahead of g, beta and v and behind one load per thread of k and q.  The sums are those
// of a run, in the same order: four running sums per group of four rows, groups 2 q4 and 2 q4 + 1 first, then the column's four lanes.
// A single step lets its successor start as soon as its loads are on their way; two steps do not (4.8 -> 6.0 us at 96 heads).
// us a step at 16 / 32 / 48 / 96 value heads, states not in L2 (in brackets what a run of one or two steps takes with deltanet_body): one, bf16 2.35 /
// 2.47 / 3.07 / 4.07, fp32 2.30 / 2.41 / 3.03 / 4.13; two, bf16 2.57 / 2.71 / 3.59 / 4.71 [3.07 / 3.28 / 3.99 / 4.82], fp32 2.56 / 2.78 / 3.74 / 4.99
// [3.04 / 3.30 / 3.96 / 4.66].
__device__ __forceinline__ float dn_column_sum(const float (&c)[8]) {
    float x = ((c[0] + c[1]) + (c[2] + c[3])) + ((c[4] + c[5]) + (c[6] + c[7]));
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    return x + __shfl_xor_sync(0xffffffffu, x, 2);
}
template <typename T, int STEPS>
__device__ __forceinline__ void deltanet_few(const lb_deltanet_params& p) {
    const int h = blockIdx.x, kh = h / (p.HV / p.HK), q4 = threadIdx.x & 3, j0 = blockIdx.y * DN_COLS + (threadIdx.x >> 2);
    float* S = p.state + (size_t)h * DN_D * DN_D + (size_t)(8 * q4) * DN_D + j0;
    const size_t oi = (size_t)h * DN_D + j0, ld = (size_t)p.HV * DN_D;
    constexpr int N = dn_in<T>::N, PIECES = 2 * DN_D / N; // 16-byte pieces of a token's k and q
    static_assert(STEPS * PIECES <= DN_THREADS, "a thread brings at most one piece");
    __shared__ __align__(16) float kq[STEPS][2][DN_D];
    float s[4][8], c[8], g[STEPS], beta[STEPS], v[STEPS];
    pdl_wait();
    uint4 piece = make_uint4(0u, 0u, 0u, 0u);
    const int pu = threadIdx.x / PIECES, pe = threadIdx.x % PIECES;
    if (threadIdx.x < STEPS * PIECES)
        piece = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(pe < DN_D / N ? p.k : p.q) + ((size_t)pu * p.HK + kh) * DN_D) + pe % (DN_D / N));
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i) asm volatile("ld.global.f32 %0, [%1];" : "=f"(s[j][i]) : "l"(S + (size_t)(32 * j + i) * DN_D) : "memory");
    if (STEPS == 1) pdl_launch_dependents();
#pragma unroll
    for (int u = 0; u < STEPS; ++u) {
        g[u] = p.g[u * p.HV + h];
        beta[u] = p.beta[u * p.HV + h];
        v[u] = sizeof(T) == 2 ? bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(p.v)[oi + u * ld]) : reinterpret_cast<const float*>(p.v)[oi + u * ld];
    }
    if (threadIdx.x < STEPS * PIECES) dn_in<T>::put(&kq[pu][pe / (DN_D / N)][pe % (DN_D / N) * N], piece);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < STEPS; ++u) {
        float k[4][8], q[4][8];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 8; i += 4) {
                *reinterpret_cast<float4*>(&k[j][i]) = *reinterpret_cast<const float4*>(&kq[u][0][32 * j + 8 * q4 + i]);
                *reinterpret_cast<float4*>(&q[j][i]) = *reinterpret_cast<const float4*>(&kq[u][1][32 * j + 8 * q4 + i]);
            }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            c[i] = __fmul_rn(k[0][i], s[0][i]);
#pragma unroll
            for (int j = 1; j < 4; ++j) c[i] = __fmaf_rn(k[j][i], s[j][i], c[i]);
        }
        const float d = beta[u] * (v[u] - dn_column_sum(c));
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[j][i] = __fmaf_rn(k[j][i], d, __fmul_rn(g[u], s[j][i]));
                c[i] = j ? __fmaf_rn(q[j][i], s[j][i], c[i]) : __fmul_rn(q[j][i], s[j][i]);
            }
        float o = dn_column_sum(c);
        if (STEPS > 1 && u == STEPS - 1) pdl_launch_dependents();
        if (q4 == 0) {
            if (p.z) o *= siluf_dev(p.z[oi + u * ld]);
            p.out[oi + u * ld] = o;
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i) S[(size_t)(32 * j + i) * DN_D] = s[j][i];
}

// n_steps consecutive tokens: q,k are [n_steps][HK][128], v (z, out) are
// [n_steps][HV][128], g and beta are [n_steps][HV].
template <typename T>
__device__ __forceinline__ void deltanet_body(const lb_deltanet_params& p, int n_steps) {
    constexpr int N = dn_in<T>::N, PIECES = DN_RUN * 2 * DN_D / N, PER = PIECES / DN_THREADS; // 16-byte pieces of a run's k and q
    constexpr int VP = DN_RUN * DN_COLS / N;
    __shared__ __align__(16) float kq[2][DN_RUN][2][DN_D], vs[2][DN_RUN][DN_COLS], gb[2][2][DN_RUN];
    const int h = blockIdx.x, jb = blockIdx.y;
    const int kh = h / (p.HV / p.HK);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, rg = lane >> 2, cg = lane & 3;
    const int jl = warp * 8 + cg * 2; // this lane's first column of the slab
    float* S = p.state + (size_t)h * DN_D * DN_D + (size_t)(4 * rg) * DN_D + jb * DN_COLS + jl;
    const bool pairs = (reinterpret_cast<uintptr_t>(p.state) & 7) == 0;

    pdl_wait();
    uint4 piece[PER], vpiece = make_uint4(0u, 0u, 0u, 0u);
    float gpiece = 0.f;
    auto load = [&](int s0) { // this thread's pieces of tokens s0 .. s0 + DN_RUN - 1 (those that there are)
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int e = i * DN_THREADS + t, tok = e / (2 * DN_D / N), which = (e / (DN_D / N)) & 1, c = e % (DN_D / N);
            if (s0 + tok < n_steps)
                piece[i] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(which ? p.q : p.k) + ((size_t)(s0 + tok) * p.HK + kh) * DN_D) + c);
        }
        if (t < VP) {
            const int tok = t / (DN_COLS / N), c = t % (DN_COLS / N);
            if (s0 + tok < n_steps)
                vpiece = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.v) + ((size_t)(s0 + tok) * p.HV + h) * DN_D + jb * DN_COLS) + c);
        } else if (t >= DN_THREADS - 2 * DN_RUN) {
            const int e = t - (DN_THREADS - 2 * DN_RUN), tok = e % DN_RUN;
            if (s0 + tok < n_steps) gpiece = __ldg((e < DN_RUN ? p.g : p.beta) + (size_t)(s0 + tok) * p.HV + h);
        }
    };
    auto store = [&](int st) {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int e = i * DN_THREADS + t;
            dn_in<T>::put(&kq[st][e / (2 * DN_D / N)][(e / (DN_D / N)) & 1][(e % (DN_D / N)) * N], piece[i]);
        }
        if (t < VP) dn_in<T>::put(&vs[st][t / (DN_COLS / N)][(t % (DN_COLS / N)) * N], vpiece);
        else if (t >= DN_THREADS - 2 * DN_RUN) gb[st][(t - (DN_THREADS - 2 * DN_RUN)) / DN_RUN][t % DN_RUN] = gpiece;
    };
    static_assert(VP <= DN_THREADS - 2 * DN_RUN && DN_THREADS % DN_RUN == 0, "threads for v, g and beta");
#pragma unroll
    for (int i = 0; i < PER; ++i) piece[i] = make_uint4(0u, 0u, 0u, 0u);
    load(0);
    uint64_t s[4][2][2]; // [run of 32 rows][rows 4 rg + (0, 1) / (2, 3) of it][column]
    dn_load_state(S, pairs, s);
    store(0);
    if (DN_RUN < n_steps) load(DN_RUN);

    for (int s0 = 0, st = 0; s0 < n_steps; s0 += DN_RUN, st ^= 1) {
        __syncthreads(); // the run's operands are visible, and everybody is done with the other stage
        if (s0 + DN_RUN < n_steps) {
            store(st ^ 1);
            if (s0 + 2 * DN_RUN < n_steps) load(s0 + 2 * DN_RUN);
        }
#pragma unroll
        for (int u0 = 0; u0 < DN_RUN; u0 += 4) {
            if (s0 + u0 >= n_steps) break;
            float o[8]; // read-outs of four tokens, two columns each: this lane's rows
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                o[2 * u] = o[2 * u + 1] = 0.f;
                if (s0 + u0 + u >= n_steps) continue;
                uint64_t kk[4][2], qq[4][2], a[2][2];
                dn_read(kq[st][u0 + u][0] + 4 * rg, kk);
                dn_read(kq[st][u0 + u][1] + 4 * rg, qq);
                const float g = gb[st][0][u0 + u], beta = gb[st][1][u0 + u];
                const float2 v = *reinterpret_cast<const float2*>(&vs[st][u0 + u][jl]);
                dn_recall(kk, s, a);
                float r0 = dn_sum4(a[0][0], a[0][1]), r1 = dn_sum4(a[1][0], a[1][1]);
                dn_decay(g, s); // independent of the sums: in their shadow
                dn_reduce(r0, r1);
                dn_update(kk, qq, beta * (v.x - r0), beta * (v.y - r1), s, a);
                o[2 * u] = dn_sum4(a[0][0], a[0][1]);
                o[2 * u + 1] = dn_sum4(a[1][0], a[1][1]);
            }
            // sums over the eight row groups: lane rg is left with token (rg & 1) * 2 + (rg >> 1 & 1), column rg >> 2
#pragma unroll
            for (int m = 1, len = 4; m < 8; m <<= 1, len >>= 1)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (i < len) {
                        const float give = rg & m ? o[i] : o[len + i], keep = rg & m ? o[len + i] : o[i];
                        o[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4 * m);
                    }
            const int step = s0 + u0 + (rg & 1) * 2 + ((rg >> 1) & 1);
            if (step < n_steps) {
                const size_t oi = ((size_t)step * p.HV + h) * DN_D + jb * DN_COLS + jl + (rg >> 2);
                float y = o[0];
                if (p.z) y *= siluf_dev(p.z[oi]);
                p.out[oi] = y;
            }
        }
    }
    pdl_launch_dependents();
    dn_store_state(S, pairs, s);
}

extern "C" __global__ void __launch_bounds__(DN_THREADS) deltanet_step_bf16(const __grid_constant__ lb_deltanet_params p,
                                                                            int n_steps) {
    deltanet_body<__nv_bfloat16>(p, n_steps);
}
extern "C" __global__ void __launch_bounds__(DN_THREADS) deltanet_one_bf16(const __grid_constant__ lb_deltanet_params p) { deltanet_few<__nv_bfloat16, 1>(p); }
extern "C" __global__ void __launch_bounds__(DN_THREADS) deltanet_one_f32(const __grid_constant__ lb_deltanet_params p) { deltanet_few<float, 1>(p); }
extern "C" __global__ void __launch_bounds__(DN_THREADS) deltanet_two_bf16(const __grid_constant__ lb_deltanet_params p) { deltanet_few<__nv_bfloat16, 2>(p); }
extern "C" __global__ void __launch_bounds__(DN_THREADS) deltanet_two_f32(const __grid_constant__ lb_deltanet_params p) { deltanet_few<float, 2>(p); }
extern "C" __global__ void __launch_bounds__(DN_THREADS) deltanet_step_f32(const __grid_constant__ lb_deltanet_params p,
                                                                           int n_steps) {
    deltanet_body<float>(p, n_steps);
}

// g = exp(-exp(A_log) softplus(a + dt_bias)), beta = sigmoid(b); natural log
// as in models/.../deltanet/unroll.ls (DecayGate: softplus = ln(1+e^x)).
extern "C" __global__ void decay_gate_beta(const __grid_constant__ lb_decay_params p) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const float t = p.a[i] + p.dt_bias[i];
    const float sp = t > 20.f ? t : log1pf(expf(t));
    p.g[i] = expf(-expf(p.a_log[i]) * sp);
    if (p.b && p.beta) p.beta[i] = 1.0f / (1.0f + expf(-p.b[i]));
}

// ---------------------------------------------------------------------------
// The whole DeltaNet mixer of one layer in ONE kernel: what the reference runs
// as in_proj_a/b, conv1d x3, activate, l2norm x2, decay_gate, gate_sigmoid and
// the recurrence (src/launcher.s:832-844; models/.../deltanet/kernels.ls:4-14):
//   a,b   = in_proj_a/b . xn                       (bf16 rows, fp32 accumulate)
//   c     = silu(conv1d(qkv))                      (4 taps, inference/recur.ls:12-40)
//   q     = l2norm(c_q) / sqrt(128), k = l2norm(c_k), v = c_v     (per head)
//   g     = exp(-exp(A_log) softplus(a + dt_bias)), beta = sigmoid(b)
//   state update + read-out as in deltanet_body above.
// CTA = (value head, 32-column slab).  The conv history is a ring of 4 slots
// indexed by position, so the CTAs that share a key head can all read the three
// previous slots while one of them writes the current one.
// ---------------------------------------------------------------------------
extern "C" __global__ void __launch_bounds__(DN_THREADS) deltanet_layer_fused(const __grid_constant__ lb_dn_layer_params p) {
    __shared__ dn_unit_smem sm;
    deltanet_layer_unit<true, false>(p, blockIdx.x, blockIdx.y, threadIdx.x, sm, [] { __syncthreads(); }, 0, nullptr, [] {});
}
