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

// A warp owns 4 CL columns of a head, all 128 rows of them: lane (rg, cg) holds 16 rows (four neighbouring ones of every 32, so that the
// lanes' 16-byte reads of a token's k or q are free of conflicts) of CL columns, the rows in pairs for packed multiply-adds; cg is
// the fast part of the lane number, so that neighbouring lanes' accesses to the state are neighbours.  A
// step needs nothing from another warp: both sums over the rows end in three shuffles, and what the warps of a CTA share, the operands of
// DN_RUN tokens in fp32, costs one block barrier per DN_RUN tokens.  A thread loads its piece of the run after next into registers and
// stores it a run later, so the chain of a step (dot, three shuffles, update) meets no trip to L2.  The read-outs of four tokens are summed
// together, in the order of a single one: the same bits for one step and for many.
// DN_RUN whole tokens are one stretch of code without a branch, in which a token's read-out and decay and the next token's operands lie in the shadow of the
// recall's shuffles.  What a step costs then is its instructions and that chain (140 instructions of a warp at CL = 2, 390 cycles alone on a scheduler) and,
// with three CTAs on an SM, what shared memory delivers (16 bytes to every lane per read, 8 reads a token and warp).  CL = 1 has twice the warps to
// balance and hide the chain with, CL = 2 half the start.  us a call, before -> CL = 2, CL = 1 (the rule stands at lb_deltanet_step): 256 steps of 16 heads 64.6 -> 52.1, 42.1;
// 24 64.6 -> 52.1, 53.5; 32 64.8 -> 52.3, 53.6; 48 86.6 -> 78.4, 68.9; 8 steps of 48 heads 5.06 -> 4.77, 5.06.
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

// a lane's CL columns of a state row: 8 bytes at once where the state's address allows it (PAIRS)
template <int CL, bool PAIRS> __device__ __forceinline__ void dn_load_rows(const float* S, uint64_t (&s)[4][2][CL]) {
    __align__(8) float x[4][4][CL];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float* r = S + (size_t)(32 * (i >> 2) + (i & 3)) * DN_D;
        if (PAIRS) *reinterpret_cast<float2*>(x[i >> 2][i & 3]) = *reinterpret_cast<const float2*>(r);
        else
#pragma unroll
            for (int c = 0; c < CL; ++c) x[i >> 2][i & 3][c] = r[c];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int c = 0; c < CL; ++c) s[j][e][c] = dn_pack(x[j][2 * e][c], x[j][2 * e + 1][c]);
}
template <int CL> __device__ __forceinline__ void dn_load_state(const float* S, bool pairs, uint64_t (&s)[4][2][CL]) {
    if (CL == 2 && pairs) dn_load_rows<CL, CL == 2>(S, s);
    else dn_load_rows<CL, false>(S, s);
}
template <int CL> __device__ __forceinline__ void dn_store_state(float* S, bool pairs, const uint64_t (&s)[4][2][CL]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float* r = S + (size_t)(32 * j + 2 * e) * DN_D;
            const float2 x = dn_unpack(s[j][e][0]), y = dn_unpack(s[j][e][CL - 1]);
            if (CL == 2 && pairs) {
                *reinterpret_cast<float2*>(r) = make_float2(x.x, y.x);
                *reinterpret_cast<float2*>(r + DN_D) = make_float2(x.y, y.y);
            } else {
                r[0] = x.x; r[DN_D] = x.y;
                if (CL == 2) { r[1] = y.x; r[DN_D + 1] = y.y; }
            }
        }
}
// sum_i k_i S_ij over this lane's rows: four running sums per column
template <int CL> __device__ __forceinline__ void dn_dot(const uint64_t (&k)[4][2], const uint64_t (&s)[4][2][CL], float (&r)[CL]) {
    uint64_t a[CL][2];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int c = 0; c < CL; ++c)
#pragma unroll
            for (int e = 0; e < 2; ++e) a[c][e] = j ? dn_fma2(k[j][e], s[j][e][c], a[c][e]) : dn_mul2(k[j][e], s[j][e][c]);
#pragma unroll
    for (int c = 0; c < CL; ++c) r[c] = dn_sum4(a[c][0], a[c][1]);
}
template <int CL> __device__ __forceinline__ void dn_decay(float g, uint64_t (&s)[4][2][CL]) {
    const uint64_t g2 = dn_pack(g, g);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int c = 0; c < CL; ++c) s[j][e][c] = dn_mul2(g2, s[j][e][c]);
}
// d_j = beta (v_j - r_j), S_ij += k_i d_j on the decayed state
template <int CL> __device__ __forceinline__ void dn_write(const uint64_t (&k)[4][2], float beta, const float (&v)[CL], const float (&r)[CL], uint64_t (&s)[4][2][CL]) {
#pragma unroll
    for (int c = 0; c < CL; ++c) {
        const float dj = beta * (v[c] - r[c]);
        const uint64_t d = dn_pack(dj, dj);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) s[j][e][c] = dn_fma2(k[j][e], d, s[j][e][c]);
    }
}
template <int CL> __device__ __forceinline__ void dn_reduce(float (&r)[CL]) { // over the eight row groups
#pragma unroll
    for (int m = 4; m < 32; m <<= 1)
#pragma unroll
        for (int c = 0; c < CL; ++c) r[c] += __shfl_xor_sync(0xffffffffu, r[c], m);
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
template <typename T, int CL>
__device__ __forceinline__ void deltanet_body(const lb_deltanet_params& p, int n_steps) {
    constexpr int THREADS = DN_THREADS, COLS = CL * THREADS / 8, N = dn_in<T>::N, PIECES = DN_RUN * 2 * DN_D / N, PER = PIECES / THREADS; // 16-byte pieces of a run's k and q
    constexpr int VP = DN_RUN * COLS / N;
    __shared__ __align__(16) float kq[2][DN_RUN][2][DN_D], vs[2][DN_RUN][COLS], gb[2][2][DN_RUN];
    const int h = blockIdx.x, jb = blockIdx.y;
    const int kh = h / (p.HV / p.HK);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, rg = lane >> 2, cg = lane & 3;
    const int jl = CL * (warp * 4 + cg); // this lane's first column of the CTA's
    float* S = p.state + (size_t)h * DN_D * DN_D + (size_t)(4 * rg) * DN_D + jb * COLS + jl;
    const bool pairs = (reinterpret_cast<uintptr_t>(p.state) & 7) == 0;

    pdl_wait();
    uint4 piece[PER], vpiece = make_uint4(0u, 0u, 0u, 0u);
    float gpiece = 0.f;
    auto load = [&](int s0) { // this thread's pieces of tokens s0 .. s0 + DN_RUN - 1 (those that there are)
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int e = i * THREADS + t, tok = e / (2 * DN_D / N), which = (e / (DN_D / N)) & 1, c = e % (DN_D / N);
            if (s0 + tok < n_steps)
                piece[i] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(which ? p.q : p.k) + ((size_t)(s0 + tok) * p.HK + kh) * DN_D) + c);
        }
        if (t < VP) {
            const int tok = t / (COLS / N), c = t % (COLS / N);
            if (s0 + tok < n_steps)
                vpiece = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.v) + ((size_t)(s0 + tok) * p.HV + h) * DN_D + jb * COLS) + c);
        } else if (t >= THREADS - 2 * DN_RUN) {
            const int e = t - (THREADS - 2 * DN_RUN), tok = e % DN_RUN;
            if (s0 + tok < n_steps) gpiece = __ldg((e < DN_RUN ? p.g : p.beta) + (size_t)(s0 + tok) * p.HV + h);
        }
    };
    auto store = [&](int st) {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int e = i * THREADS + t;
            dn_in<T>::put(&kq[st][e / (2 * DN_D / N)][(e / (DN_D / N)) & 1][(e % (DN_D / N)) * N], piece[i]);
        }
        if (t < VP) dn_in<T>::put(&vs[st][t / (COLS / N)][(t % (COLS / N)) * N], vpiece);
        else if (t >= THREADS - 2 * DN_RUN) gb[st][(t - (THREADS - 2 * DN_RUN)) / DN_RUN][t % DN_RUN] = gpiece;
    };
    static_assert(VP <= THREADS - 2 * DN_RUN && THREADS % DN_RUN == 0, "threads for v, g and beta");
#pragma unroll
    for (int i = 0; i < PER; ++i) piece[i] = make_uint4(0u, 0u, 0u, 0u);
    load(0);
    uint64_t s[4][2][CL]; // [run of 32 rows][rows 4 rg + (0, 1) / (2, 3) of it][column]
    dn_load_state(S, pairs, s);
    store(0);
    if (DN_RUN < n_steps) load(DN_RUN);

    // sums of four tokens' read-outs over the eight row groups: lane rg is left with token (rg & 1) * 2 + (rg >> 1 & 1), column rg >> 2 of two (one: twice)
    auto put_out = [&](float (&o)[4 * CL], int first) {
#pragma unroll
        for (int m = 1, len = 2 * CL; m < 8; m <<= 1, len >>= 1)
#pragma unroll
            for (int i = 0; i < 2 * CL; ++i) {
                if (i < len) {
                    const float give = rg & m ? o[i] : o[len + i], keep = rg & m ? o[len + i] : o[i];
                    o[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4 * m);
                } else if (len == 0 && i == 0) o[0] += __shfl_xor_sync(0xffffffffu, o[0], 4 * m);
            }
        const int step = first + (rg & 1) * 2 + ((rg >> 1) & 1);
        if (step < n_steps && (CL == 2 || rg < 4)) {
            const size_t oi = ((size_t)step * p.HV + h) * DN_D + jb * COLS + jl + (CL == 2 ? rg >> 2 : 0);
            float y = o[0];
            if (p.z) y *= siluf_dev(p.z[oi]);
            p.out[oi] = y;
        }
    };
    auto values = [&](int st, int u, float (&v)[CL]) {
        if (CL == 2) {
            const float2 x = *reinterpret_cast<const float2*>(&vs[st][u][jl]);
            v[0] = x.x;
            v[CL - 1] = x.y;
        } else v[0] = vs[st][u][jl];
    };
    auto run_full = [&](int st, int s0) {
        uint64_t kk[4][2], qq[4][2];
        dn_read(kq[st][0][0] + 4 * rg, kk);
        float o[4 * CL], r[CL], v[CL], y[CL];
#pragma unroll
        for (int u = 0; u < DN_RUN; ++u) {
            uint64_t kn[4][2];
            dn_dot(kk, s, r); // recall from the old state
            const float g = gb[st][0][u], beta = gb[st][1][u];
            values(st, u, v);
            if (u + 1 < DN_RUN) dn_read(kq[st][u + 1][0] + 4 * rg, kn);
            if (u > 0) {
                dn_dot(qq, s, y); // read-out of the token before
#pragma unroll
                for (int c = 0; c < CL; ++c) o[CL * ((u - 1) & 3) + c] = y[c];
            }
            dn_read(kq[st][u][1] + 4 * rg, qq);
            dn_decay(g, s);
            dn_reduce(r);
            if (u == 4) put_out(o, s0);
            dn_write(kk, beta, v, r, s);
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) kk[j][e] = kn[j][e];
        }
        dn_dot(qq, s, y);
#pragma unroll
        for (int c = 0; c < CL; ++c) o[CL * 3 + c] = y[c];
        put_out(o, s0 + 4);
    };
    auto run_part = [&](int st, int s0) { // fewer than DN_RUN tokens
#pragma unroll
        for (int u0 = 0; u0 < DN_RUN; u0 += 4) {
            if (s0 + u0 >= n_steps) break;
            float o[4 * CL];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                float r[CL], v[CL], y[CL];
#pragma unroll
                for (int c = 0; c < CL; ++c) o[CL * u + c] = 0.f;
                if (s0 + u0 + u >= n_steps) continue;
                uint64_t kk[4][2], qq[4][2];
                dn_read(kq[st][u0 + u][0] + 4 * rg, kk);
                dn_read(kq[st][u0 + u][1] + 4 * rg, qq);
                const float g = gb[st][0][u0 + u], beta = gb[st][1][u0 + u];
                values(st, u0 + u, v);
                dn_dot(kk, s, r);
                dn_decay(g, s); // independent of the sum: in its shadow
                dn_reduce(r);
                dn_write(kk, beta, v, r, s);
                dn_dot(qq, s, y);
#pragma unroll
                for (int c = 0; c < CL; ++c) o[CL * u + c] = y[c];
            }
            put_out(o, s0 + u0);
        }
    };

    for (int s0 = 0, st = 0; s0 < n_steps; s0 += DN_RUN, st ^= 1) {
        __syncthreads(); // the run's operands are visible, and everybody is done with the other stage
        if (s0 + DN_RUN < n_steps) {
            store(st ^ 1);
            if (s0 + 2 * DN_RUN < n_steps) load(s0 + 2 * DN_RUN);
        }
        if (s0 + DN_RUN <= n_steps) run_full(st, s0);
        else run_part(st, s0);
    }
    pdl_launch_dependents();
    dn_store_state(S, pairs, s);
}

// grid (HV, 4) / (HV, 8): 32 / 16 columns per CTA.  At CL = 2 the registers of three CTAs an SM: left to itself the compiler stops at 128 for fp32 and spills (us,
// 128 -> 168 registers: 24 heads 24 steps 7.3 -> 6.5, 256 60.3 -> 51.0; 96 heads 256 steps 108, the loop without straight runs 109)
#define DN_RUNS(name, T, CL, ...) \
    extern "C" __global__ void __launch_bounds__(__VA_ARGS__) name(const __grid_constant__ lb_deltanet_params p, int n_steps) { deltanet_body<T, CL>(p, n_steps); }
DN_RUNS(deltanet_step_bf16, __nv_bfloat16, 2, DN_THREADS, 3)
DN_RUNS(deltanet_step_f32, float, 2, DN_THREADS, 3)
DN_RUNS(deltanet_step16_bf16, __nv_bfloat16, 1, DN_THREADS)
DN_RUNS(deltanet_step16_f32, float, 1, DN_THREADS)
extern "C" __global__ void __launch_bounds__(DN_THREADS) deltanet_one_bf16(const __grid_constant__ lb_deltanet_params p) { deltanet_few<__nv_bfloat16, 1>(p); }
extern "C" __global__ void __launch_bounds__(DN_THREADS) deltanet_one_f32(const __grid_constant__ lb_deltanet_params p) { deltanet_few<float, 1>(p); }
extern "C" __global__ void __launch_bounds__(DN_THREADS) deltanet_two_bf16(const __grid_constant__ lb_deltanet_params p) { deltanet_few<__nv_bfloat16, 2>(p); }
extern "C" __global__ void __launch_bounds__(DN_THREADS) deltanet_two_f32(const __grid_constant__ lb_deltanet_params p) { deltanet_few<float, 2>(p); }
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
