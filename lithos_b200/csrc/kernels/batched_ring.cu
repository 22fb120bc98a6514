// Batched int4 projection of 2 to 16 tokens on sm_100a (HBM-bound: the packed words once): Y[b][n] = sum_k W(k,n) X[b][k], operands as in batched.cu.
// No weight is rounded: A = the exact integers q - z, the fp16 group scale multiplies a K-group's fp32 sum.
//
// One CTA per SM = 128 columns x a K slice, eight warps.  What bounds the other kernels of these sizes is not the words' way
// from HBM but what a K-group costs beside it: hand-overs between converting, issuing and reading warps (gemm_int4_tc_exact*, 0.5 us a K-group), or loads
// through registers that cannot be kept far enough ahead (gemm_int4_mma_*).  Here
//   * a ring of K-groups (21 of 10.6 KB up to 8 tokens, 17 of 12.6 KB up to 16) is filled by bulk copies: packed words by one tiled TMA
//     (16 packed rows x 128 columns as four boxes of 32 columns, 128-byte swizzle), the tokens' activations by two, scales and zero-points as plain runs;
//   * a warp takes a K-group WHOLE (warp w: groups w, w + 8, ...): all 128 columns and all tokens, from its slot straight into
//     mma.sync.m16n8k16 operands, and asks for the K-group that follows in the slot when it has read it.  It meets nobody until the end: one wait per 8 KB
//     of weights.  (A ninth warp for the copies would cost the registers of three.)
// The order of k in a product is free, so it is chosen for the words: lane (g, t) has packed rows 2t, 2t + 1, 2t + 8, 2t + 9 of columns 4g..4g + 3 of a box
// (16-byte reads without bank conflicts under the swizzle); w & 0x000f000f, w & 0x00f000f0 and the same of w >> 8, or-ed with 0x6400, are the
// fp16 pairs (1024 + q0, 1024 + q4), (1024 + 16 q1, 1024 + 16 q5), (q2, q6), (q3, q7): one add or fma each makes them q - z, nine instructions per
// eight weights; the activations' pairs are made once per K-group and lane (16 tokens) by byte permutes.
// The warps' sums are added in warp order, K slices (the CTAs of a cluster) in rank order: a result does not depend on timing, nor on how many rows there are.
#include "common.cuh"
#include "params.h"

#define RG_WARPS 8
#define RG_COLS 128
#define RG_PS 132 // floats per token of a partial tile

__device__ __forceinline__ void rg_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t rg_and_or(uint32_t a, uint32_t mask, uint32_t bits) { // (a & mask) | bits
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(mask), "r"(bits));
    return r;
}
__device__ __forceinline__ uint32_t rg_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 rg_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
// a packed word as four fp16 pairs: (q0, q4), (q1, q5), (q2, q6), (q3, q7), each minus z; add1 = -(1024 + z) twice, add16 = -(64 + z) twice
__device__ __forceinline__ void rg_word(uint32_t w, __half2 add1, __half2 add16, uint32_t (&a)[4]) {
    const __half2 sixteenth = rg_h2(0x2C002C00u);
    const uint32_t v = w >> 8;
    a[0] = rg_bits(__hadd2(rg_h2(rg_and_or(w, 0x000f000fu, 0x64006400u)), add1));
    a[1] = rg_bits(__hfma2(rg_h2(rg_and_or(w, 0x00f000f0u, 0x64006400u)), sixteenth, add16));
    a[2] = rg_bits(__hadd2(rg_h2(rg_and_or(v, 0x000f000fu, 0x64006400u)), add1));
    a[3] = rg_bits(__hfma2(rg_h2(rg_and_or(v, 0x00f000f0u, 0x64006400u)), sixteenth, add16));
}
// eight activations of one token as the pairs that belong to rg_word's
__device__ __forceinline__ void rg_acts(const uint4& x, uint32_t (&b)[4]) {
    b[0] = __byte_perm(x.x, x.z, 0x5410);
    b[1] = __byte_perm(x.x, x.z, 0x7632);
    b[2] = __byte_perm(x.y, x.w, 0x5410);
    b[3] = __byte_perm(x.y, x.w, 0x7632);
}
__device__ __forceinline__ uint32_t rg_pick(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

__device__ __forceinline__ void rg_tma3(uint32_t dst, const void* tmap, int row, int block, uint64_t* bar, uint64_t pol) { // 32 columns x 16 rows x 4 blocks
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(dst),
                 "l"(tmap), "r"(0), "r"(row), "r"(block), "r"(smem_u32(bar)), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void rg_tma2(uint32_t dst, const void* tmap, int k, uint64_t* bar) { // 64 k x all tokens
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(tmap), "r"(k), "r"(0),
                 "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ uint32_t rg_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void rg_cluster_sync() {
    __syncwarp(); // .aligned: the whole warp together, also behind code of some lanes only
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 rg_ld_cluster4(const float* local_ptr, uint32_t rank) {
    uint32_t remote; float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local_ptr)), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}

// NT: blocks of eight tokens.  dynamic shared memory: slots [S][words 8192 | activations NT x 2048], then [S][scales 256 | zero-points 64];
// partial sums [8 warps][8 NT][RG_PS] over the slots at the end
template <int NT>
__device__ __forceinline__ void gemm_int4_ring_body(const lb_bgemm_params& p, unsigned char* sm) {
    constexpr int TOK = 8 * NT, S = LB_RING_SLOTS(TOK), XB = TOK * 256, SLOT = 8192 + XB;
    static_assert(RG_WARPS * TOK * RG_PS * 4 <= S * SLOT, "the partial sums lie over the slots");
    __shared__ __align__(8) uint64_t full[S];
    __shared__ uint32_t round_of[S]; // how often a slot has been asked for again: whoever waits for its next K-group has to know that the phase before is over
    unsigned char* sz = sm + (size_t)S * SLOT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int groups = p.K / 128, KS = (int)gridDim.y, n0 = (int)blockIdx.x * RG_COLS, cols = min(RG_COLS, p.N - n0);
    const int g_begin = (int)(((long long)blockIdx.y * groups) / KS), g_end = (int)(((long long)(blockIdx.y + 1) * groups) / KS), n = g_end - g_begin;
    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], 1);
            round_of[s] = 0u;
        }
        mbar_fence_init();
    }
    __syncthreads();
    pdl_wait();
    bool failed = false;
    float sum[4][2][NT][4]; // [box][tile of 16 columns][token block]: columns 32 box + 4g + 2 tile (0, 1) and + 1 (2, 3), tokens 2t and 2t + 1
#pragma unroll
    for (int i = 0; i < 4 * 2 * NT * 4; ++i) (&sum[0][0][0][0])[i] = 0.f;
    const uint64_t pol = l2_policy_evict_first();
    auto request = [&](int i) { // one lane: K-group i of the slice into its slot
        const int s = i % S, grp = g_begin + i;
        const uint32_t dst = smem_u32(sm) + (uint32_t)(s * SLOT), s_bytes = (uint32_t)cols * 2u, z_bytes = p.qzeros ? (uint32_t)cols / 2u : 0u;
        mbar_arrive_expect_tx(&full[s], SLOT + s_bytes + z_bytes);
        if (i >= S) *const_cast<volatile uint32_t*>(&round_of[s]) = (uint32_t)(i / S);
        rg_tma3(dst, p.tmap_w, grp * 16, n0 / 32, &full[s], pol);
        bulk_g2s(sz + s * 320, p.scales + (size_t)grp * p.N + n0, s_bytes, &full[s], pol);
        if (p.qzeros) bulk_g2s(sz + s * 320 + 256, p.qzeros + (size_t)grp * (p.N / 8) + n0 / 8, z_bytes, &full[s], pol);
        rg_tma2(dst + 8192, p.tmap_x, grp * 128, &full[s]);
        rg_tma2(dst + 8192 + XB / 2, p.tmap_x, grp * 128 + 64, &full[s]);
    };
    // another warp asks for a slot's next K-group when it has read this one: a parity alone would not tell a warp that is two rounds ahead
    auto asked = [&](int s, uint32_t round) -> bool {
        const volatile uint32_t* r = &round_of[s];
        if (*r == round) return true;
        const uint64_t t0 = globaltimer_ns();
        for (uint32_t it = 0; it < (1u << 24); ++it) {
            if (*r == round) return true;
            if ((it & 255u) == 255u && globaltimer_ns() - t0 > LB_WAIT_NS) break;
        }
        return false;
    };
    if (lane == 0)
        for (int i = warp; i < S && i < n; i += RG_WARPS) request(i);
    __syncwarp();
    {
        for (int i = warp; i < n; i += RG_WARPS) {
            const int s = i % S;
            if (!__all_sync(0xffffffffu, asked(s, (uint32_t)(i / S)) && mbar_wait(&full[s], (uint32_t)(i / S) & 1u))) {
                failed = true;
                if (lane == 0 && p.status) atomicExch(p.status, RG_FAIL_FULL);
                break;
            }
            const unsigned char *w_s = sm + (size_t)s * SLOT, *x_s = w_s + 8192, *sz_s = sz + s * 320;
            // token 8 nt + g, packed row 2t + (e & 1) + 8 (e >> 1): 16 bytes
            auto acts = [&](int e, int nt, uint32_t (&b)[4]) {
                const int chunk = 2 * t + (e & 1);
                rg_acts(*reinterpret_cast<const uint4*>(x_s + (e >> 1) * (XB / 2) + (8 * nt + g) * 128 + ((chunk ^ g) << 4)), b);
            };
            uint32_t xb[4][NT][4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) acts(e, nt, xb[e][nt]);
#pragma unroll
            for (int box = 0; box < 4; ++box) {
                const uint32_t zw = p.qzeros ? *reinterpret_cast<const uint32_t*>(sz_s + 256 + 16 * box + 4 * (g >> 1)) >> (16 * (g & 1)) : 0x8888u;
                __half2 add1[4], add16[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint32_t z = (zw >> (4 * c)) & 15u;
                    add1[c] = rg_h2((0xE400u + z) * 0x10001u);         // -(1024 + z)
                    add16[c] = rg_h2((0xD400u + (z << 4)) * 0x10001u); // -(64 + z)
                }
                float acc[2][NT][4];
#pragma unroll
                for (int j = 0; j < 2 * NT * 4; ++j) (&acc[0][0][0])[j] = 0.f;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int row = 2 * t + (e & 1); // + 8 (e >> 1)
                    const uint4 w = *reinterpret_cast<const uint4*>(w_s + box * 2048 + (row + 8 * (e >> 1)) * 128 + ((g ^ row) << 4));
#pragma unroll
                    for (int tile = 0; tile < 2; ++tile) {
                        uint32_t a[4], b[4];
                        rg_word(rg_pick(w, 2 * tile), add1[2 * tile], add16[2 * tile], a);
                        rg_word(rg_pick(w, 2 * tile + 1), add1[2 * tile + 1], add16[2 * tile + 1], b);
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) {
                            const uint32_t (&x)[4] = xb[e][nt];
                            rg_mma(acc[tile][nt], a[0], b[0], a[1], b[1], x[0], x[1]);
                            rg_mma(acc[tile][nt], a[2], b[2], a[3], b[3], x[2], x[3]);
                        }
                    }
                }
                const uint2 su = *reinterpret_cast<const uint2*>(sz_s + 64 * box + 8 * g);
                const float2 s01 = __half22float2(rg_h2(su.x)), s23 = __half22float2(rg_h2(su.y));
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        sum[box][0][nt][j] = fmaf(j < 2 ? s01.x : s01.y, acc[0][nt][j], sum[box][0][nt][j]);
                        sum[box][1][nt][j] = fmaf(j < 2 ? s23.x : s23.y, acc[1][nt][j], sum[box][1][nt][j]);
                    }
            }
            __syncwarp(); // the slot has been read
            if (lane == 0 && i + S < n) request(i + S);
            __syncwarp();
        }
    }
    pdl_launch_dependents();
    failed = __syncthreads_or(failed ? 1 : 0) != 0; // every copy has landed and been read: the slots are free
    if (failed && tid == 0) // nothing may still be on its way into this CTA's shared memory when it ends
        for (int s = 0; s < S && s < n; ++s) mbar_wait(&full[s], round_of[s] & 1u);
    float* part = reinterpret_cast<float*>(sm); // [8 warps][TOK][RG_PS]
    {
        float* mine = part + (size_t)warp * TOK * RG_PS;
#pragma unroll
        for (int box = 0; box < 4; ++box)
#pragma unroll
            for (int tile = 0; tile < 2; ++tile)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        *reinterpret_cast<float2*>(mine + (8 * nt + 2 * t + j) * RG_PS + 32 * box + 4 * g + 2 * tile) =
                            make_float2(sum[box][tile][nt][j], sum[box][tile][nt][2 + j]);
    }
    __syncthreads();
    const bool wide = p.y_f32 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;
    auto put = [&](int b, int c, float4 v) {
        const size_t o = (size_t)b * p.N + n0 + c;
        if (wide) *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.y) + o) = v;
        else if (p.y_f32) {
            float* y = reinterpret_cast<float*>(p.y) + o;
            y[0] = v.x; y[1] = v.y; y[2] = v.z; y[3] = v.w;
        } else {
            __half* y = reinterpret_cast<__half*>(p.y) + o;
            y[0] = __float2half_rn(v.x); y[1] = __float2half_rn(v.y); y[2] = __float2half_rn(v.z); y[3] = __float2half_rn(v.w);
        }
    };
    // a warp per token, four columns per lane: the sums of the eight warps, in warp order
        for (int b = warp; b < (KS > 1 ? TOK : p.B); b += RG_WARPS) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < RG_WARPS; ++w) {
                const float4 a = *reinterpret_cast<const float4*>(part + ((size_t)w * TOK + b) * RG_PS + 4 * lane);
                v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
            }
            if (KS > 1) *reinterpret_cast<float4*>(part + (size_t)b * RG_PS + 4 * lane) = v; // where this lane read the first warp's
            else if (!failed && 4 * lane < cols) put(b, 4 * lane, v);
        }
    if (KS > 1) {
        rg_cluster_sync(); // every CTA of the cluster has its tile in place
        const int rank = (int)rg_rank();
        if (!failed && 4 * lane < cols)
            for (int b = rank + KS * warp; b < p.B; b += KS * RG_WARPS) { // rank r adds the tokens r, r + KS, ...
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                for (int q = 0; q < KS; ++q) {
                    const float4 a = rg_ld_cluster4(part + (size_t)b * RG_PS + 4 * lane, (uint32_t)q);
                    v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
                }
                put(b, 4 * lane, v);
            }
        rg_cluster_sync(); // nobody leaves while a neighbour still reads its tile
    }
}
extern "C" __global__ void __launch_bounds__(LB_RING_THREADS, 1) gemm_int4_ring8(const __grid_constant__ lb_bgemm_params p) { // 2..8 tokens
    extern __shared__ __align__(1024) unsigned char rg_sm[];
    gemm_int4_ring_body<1>(p, rg_sm);
}
extern "C" __global__ void __launch_bounds__(LB_RING_THREADS, 1) gemm_int4_ring16(const __grid_constant__ lb_bgemm_params p) { // 9..16 tokens
    extern __shared__ __align__(1024) unsigned char rg_sm[];
    gemm_int4_ring_body<2>(p, rg_sm);
}
