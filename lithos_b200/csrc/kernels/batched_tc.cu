// Batched int4 projection on the 5th-generation tensor cores (tcgen05 + TMEM) for up to 256 tokens on sm_100a:
// Y[b][n] = sum_k W(k,n) X[b][k], W in the GPTQ buffers of the batch-1 GEMV (qweight [K/8,N], scales fp16
// [K/128,N], qzeros [K/128,N/8] or NULL = zero-point 8; inference/gemv.ls:44-130), X fp16 [B,K],
// Y fp32 or fp16 [B,N].  The product is one
// tcgen05.mma of 128 weight columns x NT tokens x 16 k per instruction, accumulated in tensor memory.
//
// One CTA = 128 output columns x one K slice: 16 converting warps, one issuing thread, one activation thread.
//   * Four warps (a thread per column) take a WHOLE K-group (128 k), the sets of four warps take K-groups in turn: scale, zero-point,
//     addresses, waits and hand-overs are paid once per 16 packed words of a thread, and while one set waits (for its words, its stage, its
//     stores) the others convert.  Packed words come two K-groups of the set ahead in registers (64 KB per SM on the way).  A packed word
//     is 8 consecutive k of one column: four fp16 pairs (q - z) * s - q - z exact through the 0x6400 exponent trick, then one fp16 multiply -
//     which go to TENSOR memory (tcgen05.st; lane = weight column, a 32-bit column = two consecutive k: the A operand of tcgen05.mma read
//     from tensor memory).
//   * The activations of a K-group arrive by two tiled TMA loads (64 k x NT tokens each, 128-byte swizzle by the copy engine, tokens past
//     the batch zero-filled) in the shared-memory half of the same stage.
//   * The issuing thread waits for the stage's "full" mbarrier (one arrival per warp of the set + the bytes of the copy), issues the eight
//     products (k = 16 each: the descriptor's start address steps 32 bytes inside the swizzle atom) and commits them to "free".
// What bound it before was the issuing thread, not the conversion: its K-group took 0.85 us whatever the tokens, also with loads, conversion and
// stores taken out.  Its role is now entered by elect.sync (37.3 -> 26.8 us, 5120 -> 17408 at 16 tokens), its warp's other lanes rest instead of
// polling beside it (-> 22.4), waits off its path are suspended ones and it waits for one barrier per K-group (-> 19.8).
// Now, us at 48 / 100 / 256 tokens, before -> after: 5120 -> 17408 36.6 -> 20.3, 40.9 -> 22.9, 48.3 -> 41.8; 17408 -> 5120 42.7 -> 23.2, 48.2 -> 25.0,
// 57.8 -> 46.5.  Up to 128 tokens the issuing thread (about 750 cycles per K-group) and the conversion (1100 cycles of a set, 4 sets) bound it; at 256 the
// activations' trip from L2 (64 KB per K-group and SM, 1024 cycles at 64 B per cycle) and the products (1104 cycles: 128 x N x 16 with A in tensor memory
// takes about 10 + N / 2).  So a product carries no more tokens than there are, in steps of 16 (before: 64, 128 or 256), and up to 160 whole stages of
// activations, one barrier a K-group.  us, before -> after: 5120 -> 17408 at 75 tokens 26.1 -> 24.6, 136 39.5 -> 29.9, 150 40.5 -> 31.9, 192 42.7 -> 36.6, 240
// 45.6 -> 44.0; 17408 -> 5120 at 150 43.9 -> 34.3; 2048 -> 4096 at 150 11.4 -> 10.0.
// EXACT (up to 32 tokens): the weights go in as q - z, exact; every K-group has an accumulator of its own (four in turn), and
// four more warps (a thread per column) read it and add scale * sum in fp32, so no weight is ever rounded.
// Epilogue: without a K split straight from tensor memory (or the EXACT sums in registers) to global memory, 32 neighbouring columns of a token
// per store; K slices (the CTAs of a cluster) leave partial tiles in shared memory, which are added in rank order through distributed shared
// memory.  Every wait is bounded and reports through the status word; TMEM is freed on every path.
#include "tcgen05.cuh"
#include "params.h"

#define TC_COLS 128    // weight columns per CTA = M of the product
#define TC_STAGES 7    // most stages: weights in tensor memory, activations in shared memory
#define TC_ACCS 4      // EXACT: accumulators, used in turn
#define TC_PSTRIDE 132 // floats per row of the partial tile
#define TC_TMEM_COLS 512 // accumulator in columns 0.. (one per token; EXACT: four of 32), weight stages of 64 columns behind it

__device__ __forceinline__ uint32_t tc_cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void tc_cluster_sync() {
    __syncwarp(); // .aligned: the whole warp together, also behind code of some lanes only
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 tc_ld_cluster4(const float* local_ptr, uint32_t rank) { // 16-byte aligned
    uint32_t remote; float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local_ptr)), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t tc_lop3_and_or(uint32_t a, uint32_t mask, uint32_t bits) { // (a & mask) | bits
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(mask), "r"(bits));
    return r;
}
__device__ __forceinline__ uint32_t tc_h2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 tc_bits_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
// byte I of a packed word (q0 | q1 << 4) as the fp16 pair ((q0 - z) s, (q1 - z) s), EXACT: (q0 - z, q1 - z): (1024 + q0, 1024 + 16 q1) by
// mask-and-or, (q0 - z, q1 - z) by one fma with (1, 1/16) and (-(1024 + z), -(64 + z)), both exact, then the scale
template <int EXACT, int I>
__device__ __forceinline__ uint32_t tc_pair(uint32_t w, __half2 mul, __half2 add, __half2 s) {
    const uint32_t v = __byte_perm(w, 0u, 0x4040u | I | (I << 8));
    const __half2 q = __hfma2(tc_bits_h2(tc_lop3_and_or(v, 0x00f0000fu, 0x64006400u)), mul, add);
    return tc_h2_bits(EXACT ? q : __hmul2(q, s));
}
template <int EXACT>
__device__ __forceinline__ uint4 tc_word(uint32_t w, __half2 mul, __half2 add, __half2 s) {
    return make_uint4(tc_pair<EXACT, 0>(w, mul, add, s), tc_pair<EXACT, 1>(w, mul, add, s), tc_pair<EXACT, 2>(w, mul, add, s), tc_pair<EXACT, 3>(w, mul, add, s));
}

// One tiled TMA load of 64 k of the activations of a K-group: box 64 k (128 bytes) x NT tokens of X [B, K], written with
// the 128-byte swizzle: the K-major operand tile with the tokens as rows.  Tokens past the batch are filled with zeros
// by the copy engine.
__device__ __forceinline__ void tc_tma_x(uint32_t dst_smem, const void* tmap, int k, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst_smem),
                 "l"(tmap), "r"(k), "r"(0), "r"(smem_u32(bar))
                 : "memory");
}

struct tc_group { // a thread's share of one K-group: the 16 packed words (8 k each) of one column
    uint32_t w[16];
    uint32_t s;  // its fp16 scale (u16 load)
    uint32_t zw; // the zero-point word of its octet, as loaded (the nibble is taken out when the group is used)
};

#define TC_SBO 1024                    // bytes between groups of 8 rows: 8 rows of 128 bytes (one 128-byte swizzle atom)

template <bool EPI>
__device__ __forceinline__ void tc_store_y(const lb_bgemm_params& p, size_t o, float v) {
    if (EPI && p.epi == LB_BG_ADD) reinterpret_cast<float*>(p.y)[o] += v;
    else if (p.y_f32) reinterpret_cast<float*>(p.y)[o] = v;
    else reinterpret_cast<__half*>(p.y)[o] = __float2half_rn(v);
}

// a lane's four columns (lanes 0..15: gates, lanes 16..31: the ups that belong to them) of token b, SwiGLU: the whole warp together
__device__ __forceinline__ void tc_store_glu(const lb_bgemm_params& p, int b, float4 v) {
    const int lane = threadIdx.x & 31;
    const float4 u = make_float4(__shfl_down_sync(0xffffffffu, v.x, 16), __shfl_down_sync(0xffffffffu, v.y, 16), __shfl_down_sync(0xffffffffu, v.z, 16), __shfl_down_sync(0xffffffffu, v.w, 16));
    if (lane >= 16) return;
    const __half2 lo = __floats2half2_rn(siluf_dev(v.x) * u.x, siluf_dev(v.y) * u.y), hi = __floats2half2_rn(siluf_dev(v.z) * u.z, siluf_dev(v.w) * u.w);
    *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(p.y) + (size_t)b * (p.N / 2) + (size_t)blockIdx.x * 64 + 4 * lane) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

// SETS: converting sets of four warps (a set = the 128 columns); the exact kernels have fewer, their reading warps need the registers (spilling there cost
// 20 %: 17408 -> 5120 at 32 tokens 38.2 us with three sets, 31.3 with two; at 16 tokens 31.0 with registers for 32 tokens, 27.1 with those for 16).
// HALVES (161..256 tokens): a K-group of activations is 64 KB, so they have a ring of their own of 64-k halves, seven of which fit beside four weight stages.
// EPI: p.epi counts.  Kernels of their own, since its branches beside each store cost every call without one 0.4 to 0.7 us (24 tokens, 4096 -> 4096 9.1 -> 9.6, 2048 -> 17408
// at 28 12.1 -> 12.8).
template <int EXACT, int SETS, bool HALVES, bool EPI> // EXACT: 0, or the tokens the product carries (16, 32)
__device__ __forceinline__ void gemm_int4_tc_body(const lb_bgemm_params& p, unsigned char* tc_smem) {
    __shared__ __align__(8) uint64_t bar_free[TC_STAGES]; // a stage's products are done (tcgen05.commit)
    __shared__ __align__(8) uint64_t bar_full[TC_STAGES]; // a stage's weights are in place (one arrival per warp of the set) and its activations have landed (transaction bytes)
    __shared__ __align__(8) uint64_t bar_read[TC_ACCS]; // EXACT: a K-group's accumulator has been read (one arrival per reading warp)
    __shared__ __align__(8) uint64_t bar_x[LB_TC_X_HALVES], bar_xfree[LB_TC_X_HALVES]; // HALVES: a half of a K-group's activations has landed; its products are done
    __shared__ __align__(8) uint64_t bar_done;
    __shared__ uint32_t tmem_base_slot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int NT = EXACT ? EXACT : LB_TC_NT(p.B); // tokens the product carries (rows past B are zero)
    const uint32_t a0 = EXACT ? TC_ACCS * 32u : NT > 64 ? (uint32_t)NT : 64u; // first column of the weight stages
    // Stages: what tensor memory and shared memory hold.  At least SETS: a set waits for the K-group `stages` back with the parity of an mbarrier, and with fewer
    // stages it could be two phases ahead of it.
    const int stages = (int)((TC_TMEM_COLS - a0) / 64u); // LB_TC_STAGES: 256 tokens 4, 128 tokens 6, up to 64 7 (EXACT: 6)
    const uint32_t x_stage_bytes = (uint32_t)NT * 256u, x_half = (uint32_t)NT * 128u; // a 64-k half: NT rows of 128 bytes
    unsigned char* x_smem = tc_smem;                          // [stages][NT * 256], HALVES: [LB_TC_X_HALVES][NT * 128]
    float* pt = reinterpret_cast<float*>(tc_smem);            // [NT][TC_PSTRIDE], over the activation stages once the products are done
    const int groups = p.K / 128, KS = (int)gridDim.y;
    const int g_begin = (int)(((long long)blockIdx.y * groups) / KS), g_end = (int)(((long long)(blockIdx.y + 1) * groups) / KS);
    const int n_groups = g_end - g_begin;

    if (tid == 0) {
        for (int s = 0; s < TC_STAGES; ++s) {
            mbar_init(&bar_free[s], 1);
            mbar_init(&bar_full[s], HALVES ? 4 : 4 + 1);
        }
        for (int s = 0; HALVES && s < LB_TC_X_HALVES; ++s) {
            mbar_init(&bar_x[s], 1);
            mbar_init(&bar_xfree[s], 1);
        }
        for (int s = 0; s < TC_ACCS; ++s) mbar_init(&bar_read[s], 4);
        mbar_init(&bar_done, 1);
        mbar_fence_init();
    }
    if (warp == 0) {
        __syncwarp(); // lane 0 comes from the barriers; the allocation is one of the whole warp
        tmem_alloc(&tmem_base_slot, TC_TMEM_COLS);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_slot;
    const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16; // a warp reaches the tensor-memory lanes 32 (warp % 4) .. + 31
    const int n = blockIdx.x * TC_COLS + 32 * (warp & 3) + lane; // this thread's column
    const bool live = n < p.N;
    // Lanes past the last column (N % 32 == 16) load the last column's words, so that no load splits a warp in front of its tensor-memory
    // instructions, which the whole warp has to execute together; their products stay in lanes that nobody stores.  A warp without any column loads nothing.
    const bool any_live = n - lane < p.N;
    const int nl = min(n, p.N - 1);
    pdl_wait();

    bool failed = false;
    float sum[EXACT ? EXACT : 1]; // EXACT: the reading warps' sums, one per token
    constexpr int CV_WARPS = 4 * SETS;
    if (warp < CV_WARPS) {
        // ---------------- converting warps: set i takes the K-groups i, i + SETS, ... ----------------
        const int set = warp >> 2;
        const size_t N = (size_t)p.N;
        const uint32_t* qptr = p.qweight + (size_t)(g_begin + set) * 16 * N + nl;
        const uint16_t* sptr = p.scales + (size_t)(g_begin + set) * N + nl;
        const uint32_t* zptr = p.qzeros ? p.qzeros + (size_t)(g_begin + set) * (N / 8) + (nl >> 3) : nullptr;
        tc_group ring[2]; // the set's next two K-groups
        auto load_words = [&](tc_group& w, int c) { // a quarter of a K-group's words; the last one steps to the next K-group
#pragma unroll
            for (int j = 0; j < 4; ++j) w.w[4 * c + j] = __ldg(qptr + (size_t)(4 * c + j) * N);
            if (c == 3) {
                if (!EXACT) w.s = __ldg(sptr);
                w.zw = zptr ? __ldg(zptr) : 0x88888888u;
                qptr += 16 * SETS * N;
                sptr += SETS * N;
                if (zptr) zptr += SETS * (N / 8);
            }
        };
#pragma unroll
        for (int u = 0; u < 2; ++u) {
#pragma unroll
            for (int j = 0; j < 16; ++j) ring[u].w[j] = 0u;
            ring[u].s = 0u;
            ring[u].zw = 0x88888888u;
            if (any_live && set + SETS * u < n_groups) {
#pragma unroll
                for (int c = 0; c < 4; ++c) load_words(ring[u], c);
            }
        }
        const __half2 mul = tc_bits_h2(0x2C003C00u); // (1, 1/16)
        const int zshift = 4 * (nl & 7);
        int st = set; // stage (and its phase) of the K-group the set works on
        uint32_t ph = 0u;
        for (int g0 = set; g0 < n_groups && !failed; g0 += 2 * SETS) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int g = g0 + SETS * u;
                if (g < n_groups && !failed) {
                    const uint32_t z = (ring[u].zw >> zshift) & 0xFu;
                    const __half2 add = tc_bits_h2((0xE400u + z) | ((0xD400u + (z << 4)) << 16)); // (-(1024 + z), -(64 + z))
                    const __half2 sc = tc_bits_h2((ring[u].s & 0xFFFFu) * 0x10001u);
                    const bool more = any_live && g + 2 * SETS < n_groups;
                    // the stage held the K-group `stages` back: wait until its products are done (lane 0 waits for its warp; the vote orders the
                    // others behind it).  Suspended waits, here and wherever else a wait is not on the critical path: lanes that spin on
                    // mbarriers slow every other wait of the SM down.
                    if (g >= stages && lane == 0 && !mbar_wait(&bar_free[st], ph ^ 1u)) {
                        failed = true;
                        if (p.status) atomicExch(p.status, TC_FAIL_FREE);
                    }
                    failed = __any_sync(0xffffffffu, failed); // the warp goes on, or leaves the loop, together
                    tc_fence_after();
                    const uint32_t stage = tmem + lanes + a0 + (uint32_t)(64 * st);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint4 v0 = tc_word<EXACT>(ring[u].w[4 * c], mul, add, sc), v1 = tc_word<EXACT>(ring[u].w[4 * c + 1], mul, add, sc);
                        const uint4 v2 = tc_word<EXACT>(ring[u].w[4 * c + 2], mul, add, sc), v3 = tc_word<EXACT>(ring[u].w[4 * c + 3], mul, add, sc);
                        if (more) load_words(ring[u], c);
                        tmem_st16(stage + (uint32_t)(16 * c), v0, v1, v2, v3);
                    }
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bar_full[st]);
                    for (st += SETS; st >= stages; st -= stages) ph ^= 1u;
                }
            }
        }
    } else if (warp == CV_WARPS) {
        // ---------------- issuing thread: eight products per K-group as soon as its weights and activations are in place ----------------
        if (tc_elect()) {
            const uint32_t idesc = tc_idesc(TC_COLS, (uint32_t)NT);
            const uint64_t x_desc0 = tc_smem_desc(smem_u32(x_smem), 16, TC_SBO);
            int s = 0, xs = 0;
            uint32_t ph = 0u, xph = 0u;
            bool full = false;
            for (int it = 0; it < n_groups && !failed; ++it) {
                const int b = it & (TC_ACCS - 1);
                if (EXACT && it >= TC_ACCS && !tc_wait(&bar_read[b], (uint32_t)(it / TC_ACCS - 1) & 1u)) {
                    failed = true;
                    if (p.status) atomicExch(p.status, TC_FAIL_FREE);
                    break;
                }
                if (!full && !tc_wait(&bar_full[s], ph)) {
                    failed = true;
                    if (p.status) atomicExch(p.status, TC_FAIL_FULL);
                    break;
                }
                tc_fence_after();
                const int s_now = s;
                if (++s == stages) { s = 0; ph ^= 1u; }
                full = tc_test_wait(&bar_full[s], ph); // the next K-group's state is on its way (about 200 cycles) while this one's products are issued
                const uint32_t d = tmem + (EXACT ? (uint32_t)(32 * b) : 0u), a = tmem + a0 + (uint32_t)(64 * s_now);
                const uint64_t x_desc = x_desc0 + (uint64_t)((s_now * x_stage_bytes) >> 4); // the start-address field counts 16-byte units
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) { // k = 16 kk .. + 15
                    uint64_t xd = x_desc + (uint64_t)(((kk >> 2) * x_half + (kk & 3) * 32) >> 4);
                    if (HALVES) {
                        if ((kk & 3) == 0) {
                            if (!failed && !tc_wait(&bar_x[xs], xph)) {
                                failed = true;
                                if (p.status) atomicExch(p.status, TC_FAIL_FULL);
                            }
                            tc_fence_after();
                        }
                        xd = x_desc0 + (uint64_t)((xs * x_half + (kk & 3) * 32) >> 4);
                    }
                    tc_mma_ta(d, a + (uint32_t)(8 * kk), xd, idesc, kk > 0 || (!EXACT && it > 0) ? 1u : 0u);
                    if (HALVES && (kk & 3) == 3) {
                        tc_commit(&bar_xfree[xs]);
                        if (++xs == LB_TC_X_HALVES) { xs = 0; xph ^= 1u; }
                    }
                }
                tc_commit(&bar_free[s_now]);
            }
            tc_commit(&bar_done); // fires when every product issued above is done
        }
        __syncwarp(); // the other lanes rest here: waiting for the end below, they would share this warp's issue with its one busy lane
    } else if (warp == CV_WARPS + 1) {
        // ---------------- activation thread: tiled TMA loads of 64 k, as far ahead as there are stages ----------------
        if (tc_elect()) {
            int j = 0, s = 0;
            uint32_t ph = 1u;
            if (HALVES) {
                for (; j < 2 * n_groups; ++j) {
                    if (j >= LB_TC_X_HALVES && !mbar_wait(&bar_xfree[s], ph)) {
                        failed = true;
                        if (p.status) atomicExch(p.status, TC_FAIL_FREE);
                        break;
                    }
                    mbar_arrive_expect_tx(&bar_x[s], x_half);
                    tc_tma_x(smem_u32(x_smem + (size_t)s * x_half), p.tmap_x, g_begin * 128 + j * 64, &bar_x[s]);
                    if (++s == LB_TC_X_HALVES) { s = 0; ph ^= 1u; }
                }
                if (failed) // nothing may still be on its way into this CTA's shared memory when it ends
                    for (int i = j > LB_TC_X_HALVES ? j - LB_TC_X_HALVES : 0; i < j; ++i) mbar_wait(&bar_x[i % LB_TC_X_HALVES], (uint32_t)((i / LB_TC_X_HALVES) & 1));
            } else {
                for (; j < n_groups; ++j) {
                    if (j >= stages && !mbar_wait(&bar_free[s], ph)) {
                        failed = true;
                        if (p.status) atomicExch(p.status, TC_FAIL_FREE);
                        break; // the issuing thread then gives up on this stage's barrier and reports too
                    }
                    mbar_arrive_expect_tx(&bar_full[s], x_stage_bytes);
                    tc_tma_x(smem_u32(x_smem + (size_t)s * x_stage_bytes), p.tmap_x, (g_begin + j) * 128, &bar_full[s]);
                    tc_tma_x(smem_u32(x_smem + (size_t)s * x_stage_bytes + x_half), p.tmap_x, (g_begin + j) * 128 + 64, &bar_full[s]);
                    if (++s == stages) { s = 0; ph ^= 1u; }
                }
                if (failed)
                    for (int i = j > stages ? j - stages : 0; i < j; ++i) mbar_wait(&bar_full[i % stages], (uint32_t)((i / stages) & 1));
            }
        }
        __syncwarp();
    } else if (EXACT) {
        // ---------------- reading warps: sum += scale * (the K-group's products) ----------------
        const uint16_t* sptr = p.scales + (size_t)g_begin * p.N + nl;
        uint16_t sc[TC_ACCS];
#pragma unroll
        for (int u = 0; u < TC_ACCS; ++u) sc[u] = any_live && u < n_groups ? __ldg(sptr + (size_t)u * p.N) : (uint16_t)0;
        float part[EXACT ? EXACT : 1]; // the sums of up to eight K-groups: two levels, so that a long K slice is no less exact than a short one
#pragma unroll
        for (int j = 0; j < EXACT; ++j) sum[j] = part[j] = 0.f;
        int st = 0;
        uint32_t ph = 0u;
        for (int i0 = 0; i0 < n_groups && !failed; i0 += TC_ACCS) {
#pragma unroll
            for (int u = 0; u < TC_ACCS; ++u) {
                const int it = i0 + u;
                if (it < n_groups && !failed) {
                    const float s = __half2float(__ushort_as_half(sc[u]));
                    if (any_live && it + TC_ACCS < n_groups) sc[u] = __ldg(sptr + (size_t)(it + TC_ACCS) * p.N);
                    if (lane == 0 && !mbar_wait(&bar_free[st], ph)) {
                        failed = true;
                        if (p.status) atomicExch(p.status, TC_FAIL_FREE);
                    }
                    failed = __any_sync(0xffffffffu, failed);
                    if (++st == stages) { st = 0; ph ^= 1u; }
                    tc_fence_after();
                    uint32_t r[16];
                    tmem_ld16(tmem + lanes + (uint32_t)(32 * u), r);
                    tmem_ld_wait();
                    if (EXACT > 16) { // half of the tokens after the other: sums, parts and all 32 results would not fit the registers
#pragma unroll
                        for (int j = 0; j < 16; ++j) part[j] = fmaf(s, __uint_as_float(r[j]), part[j]);
                        tmem_ld16(tmem + lanes + (uint32_t)(32 * u + 16), r);
                        tmem_ld_wait();
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bar_read[u]);
#pragma unroll
                    for (int j = 0; j < 16; ++j) part[EXACT - 16 + j] = fmaf(s, __uint_as_float(r[j]), part[EXACT - 16 + j]);
                }
            }
            if ((i0 & TC_ACCS) || i0 + TC_ACCS >= n_groups) {
#pragma unroll
                for (int j = 0; j < EXACT; ++j) {
                    sum[j] += part[j];
                    part[j] = 0.f;
                }
            }
        }
    }
    pdl_launch_dependents();
    const bool done = mbar_wait(&bar_done, 0);
    if (!done && tid == 0 && p.status) atomicExch(p.status, TC_FAIL_DONE);
    tc_fence_after();
    failed = __syncthreads_or((failed || !done) ? 1 : 0) != 0;
    // accumulator: TMEM lane = column of the tile, TMEM column = token
    if (!failed && EXACT && warp >= CV_WARPS + 2) {
#pragma unroll
        for (int j = 0; j < EXACT; ++j) {
            if (KS > 1) pt[j * TC_PSTRIDE + 32 * (warp & 3) + lane] = sum[j];
            else if (live && j < p.B) tc_store_y<EPI>(p, (size_t)j * p.N + n, sum[j]);
        }
    }
    const bool glu = EPI && p.epi == LB_BG_SWIGLU, tiled = KS > 1 || glu; // through the tile in shared memory
    if (!failed && !EXACT && warp < CV_WARPS) {
        for (int c = warp >> 2; c < NT / 16; c += SETS) { // the sets share the tokens
            uint32_t r[16];
            __syncwarp(); // the stores before are some lanes' only
            tmem_ld16(tmem + lanes + (uint32_t)(c * 16), r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const int b = c * 16 + j;
                if (tiled) pt[b * TC_PSTRIDE + 32 * (warp & 3) + lane] = __uint_as_float(r[j]);
                else if (live && b < p.B) tc_store_y<EPI>(p, (size_t)b * p.N + n, __uint_as_float(r[j]));
            }
        }
    }
    tc_fence_before();
    if (KS == 1 && glu) {
        __syncthreads();
        if (!failed)
            for (int b = warp; b < p.B; b += (int)(blockDim.x >> 5)) tc_store_glu(p, b, *reinterpret_cast<const float4*>(pt + b * TC_PSTRIDE + 4 * lane));
    }
    if (KS > 1) {
        tc_cluster_sync(); // every CTA of the cluster has its tile in place
        const int rank = (int)tc_cluster_rank();
        const int cols = min(TC_COLS, p.N - (int)blockIdx.x * TC_COLS), c = 4 * lane; // a warp per token, four columns per thread (N is a multiple of 16)
        const bool wide = p.y_f32 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;
        if (!failed && c < cols) {
            for (int b = rank + KS * warp; b < p.B; b += KS * (int)(blockDim.x >> 5)) { // rank r adds the tokens r, r + KS, ...
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                for (int q = 0; q < KS; ++q) {
                    const float4 t = tc_ld_cluster4(pt + b * TC_PSTRIDE + c, (uint32_t)q);
                    v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
                }
                const size_t o = (size_t)b * p.N + (size_t)blockIdx.x * TC_COLS + c;
                if (glu) {
                    tc_store_glu(p, b, v); // whole blocks of 128 columns: every lane is here
                    continue;
                }
                if (wide) {
                    float4* y = reinterpret_cast<float4*>(reinterpret_cast<float*>(p.y) + o);
                    if (EPI && p.epi == LB_BG_ADD) {
                        const float4 a = *y;
                        v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
                    }
                    *y = v;
                }
                else {
                    tc_store_y<EPI>(p, o, v.x); tc_store_y<EPI>(p, o + 1, v.y); tc_store_y<EPI>(p, o + 2, v.z); tc_store_y<EPI>(p, o + 3, v.w);
                }
            }
        }
        tc_cluster_sync(); // nobody leaves while a neighbour still reads its tile
    }
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, TC_TMEM_COLS);
    }
}

extern "C" __global__ void __launch_bounds__(LB_TC_THREADS, 1) gemm_int4_tc(const __grid_constant__ lb_bgemm_params p) { // 9..160 tokens
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    gemm_int4_tc_body<0, 4, false, false>(p, tc_smem);
}
extern "C" __global__ void __launch_bounds__(LB_TC_THREADS, 1) gemm_int4_tc_256(const __grid_constant__ lb_bgemm_params p) { // 161..256 tokens
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    gemm_int4_tc_body<0, 4, true, false>(p, tc_smem);
}
extern "C" __global__ void __launch_bounds__(LB_TC_THREADS, 1) gemm_int4_tc_epi(const __grid_constant__ lb_bgemm_params p) { // 33..160 tokens
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    gemm_int4_tc_body<0, 4, false, true>(p, tc_smem);
}
extern "C" __global__ void __launch_bounds__(LB_TC_THREADS, 1) gemm_int4_tc_256_epi(const __grid_constant__ lb_bgemm_params p) { // 161..256 tokens
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    gemm_int4_tc_body<0, 4, true, true>(p, tc_smem);
}
extern "C" __global__ void __launch_bounds__(LB_TC_EXACT16_THREADS, 1) gemm_int4_tc_exact16(const __grid_constant__ lb_bgemm_params p) { // up to 16 tokens where neither the ring nor mma.sync takes them
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    gemm_int4_tc_body<16, 3, false, false>(p, tc_smem);
}
extern "C" __global__ void __launch_bounds__(LB_TC_EXACT32_THREADS, 1) gemm_int4_tc_exact32(const __grid_constant__ lb_bgemm_params p) { // 17..32 tokens
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    gemm_int4_tc_body<32, 2, false, false>(p, tc_smem);
}
