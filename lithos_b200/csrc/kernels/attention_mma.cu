// GQA decode attention on the tensor cores (sm_100a): same contract, parameter block and results as
// attn_decode_split (attention.cu; inference/attend.ls:85-191, attend_full.ls:186-248).
//   * A CTA is (KV head, slice of positions), one CTA per SM at most; a warp takes blocks of 16 rows and reads them from global memory
//     straight into the operand registers of its products: which feature is which k (keys) or m (values) of a product is free, so a lane's
//     16-byte pieces of a row are its fragments as they are (keys) or after one byte permute per register (values).  Nothing is staged in
//     shared memory, no lane waits for another warp, and the next block's keys are on their way as soon as this block's scores are done,
//     its values as soon as its read-outs are: 8 to 16 KB per warp in flight, 8 warps.
//   * The first block of every warp is requested at kernel start, before griddepcontrol.wait (cache rows below the current position are
//     never written by this step).
//   * S = Q K^T as mma.sync.m16n8k16 bf16.  Q is the normalised, rotated, pre-scaled fp32 query split into two bf16 terms: the leading
//     terms of the KV head's query heads are rows 0..G-1 of the A operand and the remainders rows 8..8+G-1 of the same one, so one product
//     per fragment of keys gives both and the scores carry 16 bits of Q; K is bf16 in the cache.
//   * O^T = V^T P^T: the probabilities come out of the first product in exactly the B-fragment layout (head g, rows 2t and 2t+1) and go in
//     as two bf16 terms as well.
//   * Online soft-max per head over the warp's blocks, warps merged through shared memory in warp order, slices by all CTAs of a KV
//     head together, each its share of the outputs, in slice order: run-to-run identical.  A launch has no more CTAs than the GPU has SMs, but
//     nothing promises it all of them: a CTA that has waited for the others some 50 us leaves its share to those that come later, the last of which waits for nobody.
//     (A cooperative launch, which does promise them, takes 4 us longer.)
// mma.sync rather than tcgen05: M is the 1..6 query heads of a KV head.
// HBM-bound at long contexts (K and V rows once), a chain of latencies at short ones.  24 / 4 heads, us a call, before -> after (before: rows staged in
// shared memory by 512-byte bulk copies, one block per warp in flight, up to 64 slices per KV head = two waves beyond 4736 rows, and there a single CTA
// merging all of them): 300 rows 18.4 -> 9.5, 4096 14.4 -> 10.6, 8192 31.0 -> 14.3, 20 000 42.2 -> 22.0, 100 000 101.7 -> 69.1 (5.9 TB/s);
// 12 / 2 heads, 100 000 rows 51.7 -> 40.7; 48 / 8 heads, 8192 rows 54.5 -> 20.9.
#include "attention_core.cuh"

#define AM_ROWS 16
#define AM_QS 576  // bytes per row of queries: 512 + 64, so that the 16-byte reads of two neighbouring rows by four lanes each fill all banks
#define AM_HS 260  // floats per head of a warp's partial result

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// (x, y) as a bf16 pair (x in the low half) and the bf16 pair of what the rounding left over
__device__ __forceinline__ void split_bf16x2(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const float2 hf = __bfloat1622float2(h);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - hf.x, y - hf.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ uint32_t am_add(uint32_t* a, uint32_t v) {
    uint32_t old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(a), "r"(v) : "memory");
    return old;
}
// the last CTA to be done with a KV head's records puts the words back to zero (the flags are)
__device__ __forceinline__ void am_done(const lb_attn_params& p, uint32_t* word, uint32_t* finished) {
    if (atomicAdd(finished, 1u) == (uint32_t)p.splits - 1u) {
        *word = 0u;
        *finished = 0u;
    }
}
// 16 bytes of a cache row, read once: not kept in L1, first to leave L2
__device__ __forceinline__ uint4 ld_row16(const unsigned char* a, uint64_t pol) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v4.u32 {%0,%1,%2,%3}, [%4], %5;"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(a), "l"(pol) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t word(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// A block of 16 rows in registers.  Keys: [rows 0-7 / 8-15][32 features], lane (g, t) has features 8t..8t+7 of row g.  Values: [row 2t, 2t+1, 2t+8,
// 2t+9][64 features], lane (g, t) has features 8g..8g+7.
struct am_keys { uint4 w[2][8]; };
struct am_values { uint4 w[4][4]; };

template <int G>
struct am_warp { // a warp's running maximum and sum of head g in the lanes of row group g, and O^T[feature][head]
    float m, l, acc[16][4]; // acc[4 seg + j]: features 64 seg + 8g + 2j (0, 1) and + 1 (2, 3), heads 2t, 2t+1

    // qs: this lane's place in the leading terms of head g (features 8t..); the remainders lie 8 rows behind
    __device__ __forceinline__ void scores(const am_keys& k, const unsigned char* qs, float (&s)[2][4]) const {
        float e[2][4]; // even and odd k-steps apart: chains of eight products
#pragma unroll
        for (int i = 0; i < 2; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = e[i][0] = e[i][1] = e[i][2] = e[i][3] = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const uint4 h = *reinterpret_cast<const uint4*>(qs + c * 64), r = *reinterpret_cast<const uint4*>(qs + 8 * AM_QS + c * 64);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                mma_bf16(s[i], h.x, r.x, h.y, r.y, k.w[i][c].x, k.w[i][c].y);
                mma_bf16(e[i], h.z, r.z, h.w, r.w, k.w[i][c].z, k.w[i][c].w);
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] += e[i][j];
    }
    // scores of 16 rows -> probabilities; the first row of a block is always valid
    __device__ __forceinline__ void softmax(const float (&s)[2][4], int nvalid, int t, uint32_t (&ph)[2], uint32_t (&pl)[2]) {
        float sv[4] = {s[0][0] + s[0][2], s[0][1] + s[0][3], s[1][0] + s[1][2], s[1][1] + s[1][3]}; // head g, rows 2t, 2t+1, 2t+8, 2t+9
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (2 * t + (i & 1) + 8 * (i >> 1) >= nvalid) sv[i] = -INFINITY;
        float mx = fmaxf(fmaxf(sv[0], sv[1]), fmaxf(sv[2], sv[3]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float m_new = fmaxf(m, mx), corr = exp2f(m - m_new); // exp2f(-inf) = 0 on the first block
        float pr[4], ps = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            pr[i] = exp2f(sv[i] - m_new);
            ps += pr[i];
        }
        ps += __shfl_xor_sync(0xffffffffu, ps, 1);
        ps += __shfl_xor_sync(0xffffffffu, ps, 2);
        l = fmaf(l, corr, ps);
        m = m_new;
        split_bf16x2(pr[0], pr[1], ph[0], pl[0]);
        split_bf16x2(pr[2], pr[3], ph[1], pl[1]);
        // the accumulators of this lane belong to heads 2t and 2t+1: their factors live in row groups 2t, 2t+1
        if (__any_sync(0xffffffffu, corr != 1.f)) {
            const float c0 = __shfl_sync(0xffffffffu, corr, 8 * t), c1 = __shfl_sync(0xffffffffu, corr, 8 * t + 4);
#pragma unroll
            for (int b = 0; b < 16; ++b) { acc[b][0] *= c0; acc[b][1] *= c1; acc[b][2] *= c0; acc[b][3] *= c1; }
        }
    }
    __device__ __forceinline__ void read_out(const am_values& v, const uint32_t (&ph)[2], const uint32_t (&pl)[2]) {
#pragma unroll
        for (int seg = 0; seg < 4; ++seg)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t r0 = word(v.w[0][seg], j), r1 = word(v.w[1][seg], j), r2 = word(v.w[2][seg], j), r3 = word(v.w[3][seg], j);
                const uint32_t a0 = __byte_perm(r0, r1, 0x5410), a1 = __byte_perm(r0, r1, 0x7632), a2 = __byte_perm(r2, r3, 0x5410), a3 = __byte_perm(r2, r3, 0x7632);
                mma_bf16(acc[4 * seg + j], a0, a1, a2, a3, ph[0], ph[1]);
                mma_bf16(acc[4 * seg + j], a0, a1, a2, a3, pl[0], pl[1]);
            }
    }
};

// A warp's head vector (lane: 8 neighbouring features in v): RMS norm, rotation, scale, as warp_norm_rope, the result in v
__device__ __forceinline__ void am_norm_rope(float (&v)[8], const uint16_t* w, const float* cs, const float* sn, int rot_dims, float eps, float scale) {
    const int lane = threadIdx.x & 31;
    float ww[8], ss = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        ww[j] = w ? bf16_bits_to_f32(w[lane * 8 + j]) : 1.f;
        ss += v[j] * v[j];
    }
    if (w) {
        ss = warp_sum(ss);
        const float r = rsqrtf(ss * (1.0f / AT_D) + eps);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = v[j] * r * ww[j];
    }
    if (lane * 8 < rot_dims) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = lane * 4 + j;
            if (2 * i < rot_dims) {
                const float a = v[2 * j], b = v[2 * j + 1];
                v[2 * j] = a * cs[i] - b * sn[i];
                v[2 * j + 1] = a * sn[i] + b * cs[i];
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] *= scale;
}

// the gate of this thread's first output of a share
template <int G>
__device__ __forceinline__ float am_gate(const lb_attn_params& p, int kv, int share) {
    if (!p.gate) return 0.f;
    const int per = (G * AT_D + p.splits - 1) / p.splits, ol = p.splits > 16 ? threadIdx.x & 63 : threadIdx.x, o = share * per + ol;
    return ol < per && o < G * AT_D ? ld_in(p.gate, (size_t)(kv * G + o / AT_D) * p.gate_stride + o % AT_D, p.in_dtype) : 0.f;
}

// A share of a KV head's outputs (as many shares as slices) from the records of all its slices, GR slice groups (group `sub`: slices sub, sub + GR, ...) of
// 256 / GR threads; the groups' results are combined in group order.  gate0: am_gate.  red: [3][GR][256 / GR] floats.
template <int G, int GR>
__device__ __forceinline__ void am_finish(const lb_attn_params& p, int kv, int share, float gate0, float* red) {
    constexpr int W = 256 / GR;
    const int t = threadIdx.x, sub = t / W, ol = t % W, per = (G * AT_D + p.splits - 1) / p.splits; // the share: outputs [share * per, (share + 1) * per)
    const float* kvrec = p.scratch + (size_t)kv * p.splits * G * AT_REC;
    for (int ob = 0; ob < per; ob += W) {
        const int o = share * per + ob + ol;
        const bool live = ob + ol < per && o < G * AT_D;
        const int g = live ? o / AT_D : 0, dim = live ? o % AT_D : 0;
        float M = -INFINITY, L = 0.f, A = 0.f;
        for (int s0 = sub; s0 < p.splits; s0 += 16 * GR) { // 16 slices a time, all loads in flight at once
            float mv[16], lv[16], av[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const int s = s0 + GR * j;
                const bool on = live && s < p.splits;
                const float* r = kvrec + ((size_t)(on ? s : 0) * G + g) * AT_REC;
                mv[j] = on ? __ldcg(r + 256) : -INFINITY;
                lv[j] = on ? __ldcg(r + 257) : 0.f;
                av[j] = on ? __ldcg(r + dim) : 0.f;
            }
            float mx = M;
#pragma unroll
            for (int j = 0; j < 16; ++j) mx = fmaxf(mx, mv[j]);
            const float c = M == -INFINITY ? 0.f : exp2f(M - mx);
            L *= c;
            A *= c;
            M = mx;
#pragma unroll
            for (int j = 0; j < 16; ++j) { // slice order inside the group
                const float w = mv[j] == -INFINITY ? 0.f : exp2f(mv[j] - mx);
                L = fmaf(lv[j], w, L);
                A = fmaf(av[j], w, A);
            }
        }
        if (GR > 1) {
            __syncthreads(); // the previous block of outputs has been combined
            red[t] = M; red[256 + t] = L; red[512 + t] = A;
            __syncthreads();
            if (sub == 0) {
                float mx = M;
#pragma unroll
                for (int q = 1; q < GR; ++q) mx = fmaxf(mx, red[q * W + ol]);
                L = A = 0.f;
#pragma unroll
                for (int q = 0; q < GR; ++q) {
                    const float m = red[q * W + ol], w = m == -INFINITY ? 0.f : exp2f(m - mx);
                    L = fmaf(red[256 + q * W + ol], w, L);
                    A = fmaf(red[512 + q * W + ol], w, A);
                }
            }
        }
        if (sub == 0 && live) {
            const int hq = kv * G + g;
            float out = A / L;
            if (p.gate) out *= sigmoidf_dev(ob == 0 ? gate0 : ld_in(p.gate, (size_t)hq * p.gate_stride + dim, p.in_dtype));
            p.out[(size_t)hq * AT_D + dim] = out;
        }
    }
}

// puts a flag on the CTA's share and says so in the word: AM_LEFT, or the word where everybody had arrived and nobody else has taken the share
#define AM_LEFT 0xffffu
__device__ __noinline__ uint32_t am_leave(uint32_t* word, uint32_t* flag, uint32_t all) {
    atomicExch(flag, 1u);
    const uint32_t v = am_add(word, 0x10000u);
    return (v & 0xffffu) != all || atomicExch(flag, 0u) == 0u ? AM_LEFT : v;
}
// the shares that other CTAs have left; apart, so that the ordinary way does not carry its registers
template <int G>
__device__ __noinline__ void am_take_over(const lb_attn_params& p, int kv, uint32_t* flags, float* red) {
    __shared__ int s_next;
    for (int share = 0;; ++share) {
        __syncthreads(); // everybody is done with the share before
        if (threadIdx.x == 0) {
            while (share < p.splits && atomicExch(flags + share, 0u) == 0u) ++share;
            s_next = share;
        }
        __syncthreads();
        share = s_next;
        if (share >= p.splits) return;
        const float gate0 = am_gate<G>(p, kv, share);
        if (p.splits > 16) am_finish<G, 4>(p, kv, share, gate0, red);
        else am_finish<G, 1>(p, kv, share, gate0, red);
    }
}

template <int G>
__device__ __forceinline__ void attn_mma_body(const lb_attn_params& p, unsigned char* sm) {
    const int kv = blockIdx.x, split = blockIdx.y;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int fg = lane >> 2, ft = lane & 3;
    // shared memory
    unsigned char* qs = sm;                                             // [16][576 B] bf16: leading terms of the queries, then the remainders
    float* part = reinterpret_cast<float*>(qs + 16 * AM_QS);            // [8 warps][G][260]
    __nv_bfloat16* kn_s = reinterpret_cast<__nv_bfloat16*>(part + AT_WARPS * G * AM_HS); // [256] new key, new value
    __nv_bfloat16* vn_s = kn_s + AT_D;
    float* cs_s = reinterpret_cast<float*>(vn_s + AT_D);                // [64]
    float* sn_s = cs_s + 64;                                            // [64]
    float* wm = sn_s + 64;                                              // [8][8] per-warp max
    float* wl = wm + AT_WARPS * AT_GMAX;                                // [8][8] per-warp sum

    // The position comes from device memory written by the previous STEP (not the previous kernel), and cache rows
    // below it are not written by this step: the first block of every warp can be requested at once.
    const int pos = p.pos_ptr ? p.pos_ptr[0] : p.pos;
    if (p.max_ctx > 0 && (pos < 0 || pos >= p.max_ctx)) { // the position lies outside the caches: report it, touch nothing
        if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0 && p.status) atomicExch(p.status, LB_DEV_POS_RANGE);
        return;
    }
    const int chunk = (((pos + p.splits - 1) / p.splits) + AM_ROWS - 1) & ~(AM_ROWS - 1); // rows per slice, whole blocks
    const int t0 = split * chunk, t1 = min(pos, t0 + chunk);
    const int n_blocks = t1 > t0 ? (t1 - t0 + AM_ROWS - 1) / AM_ROWS : 0;
    const size_t row_bytes = (size_t)p.HKV * AT_D * 2;
    const uint64_t pol = l2_policy_evict_first();
    const unsigned char* kc = reinterpret_cast<const unsigned char*>(p.k_cache) + (size_t)kv * AT_D * 2;
    const unsigned char* vc = reinterpret_cast<const unsigned char*>(p.v_cache) + (size_t)kv * AT_D * 2;
    am_keys K;
    am_values V;
    auto load_keys = [&](int b) { // rows past the slice end repeat its last row (finite values; their scores are masked)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const unsigned char* r = kc + (size_t)min(t0 + b * AM_ROWS + 8 * i + fg, t1 - 1) * row_bytes + ft * 16;
#pragma unroll
            for (int c = 0; c < 8; ++c) K.w[i][c] = ld_row16(r + c * 64, pol);
        }
    };
    auto load_values = [&](int b) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const unsigned char* r = vc + (size_t)min(t0 + b * AM_ROWS + 2 * ft + (i & 1) + 8 * (i >> 1), t1 - 1) * row_bytes + fg * 16;
#pragma unroll
            for (int c = 0; c < 4; ++c) V.w[i][c] = ld_row16(r + c * 128, pol);
        }
    };
    if (warp < n_blocks) {
        load_keys(warp);
        load_values(warp);
    }
    const bool last = split == p.splits - 1; // this CTA also appends and attends the token being decoded
    const float qscale = rsqrtf((float)AT_D) * 1.4426950408889634f; // scores kept in log2 units
    // cos/sin of this position once per CTA: the angle is formed and reduced modulo 2*pi in double, the trigonometry
    // itself is fp32 on |r| <= pi; freq comes from the host in double
    if (t < p.rot_dims / 2) {
        double freq; // indexed in the parameter space itself: a plain index makes a local copy of the whole block, from which everything is then read
        asm("ld.param.f64 %0, [%1];" : "=d"(freq) : "l"(__cvta_generic_to_grid_constant(p.rope_freq + t)));
        const double a = (double)pos * freq;
        const double k = rint(a * 0.15915494309189535);
        const float r = (float)fma(-k, 6.283185307179586, a);
        sincosf(r, &sn_s[t], &cs_s[t]);
    }
    pdl_wait();
    // warp w < G: query head w, warp G of the last slice: the new key
    const bool is_q = warp < G, is_k = last && warp == G;
    float x[8];
    if (is_q || is_k) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
            x[j] = is_q ? ld_in(p.q, (size_t)(kv * G + warp) * p.q_stride + lane * 8 + j, p.in_dtype) : ld_in(p.k_new, (size_t)kv * AT_D + lane * 8 + j, p.in_dtype);
    }
    __nv_bfloat16 vb = __float2bfloat16_rn(0.f);
    if (last) vb = __float2bfloat16_rn(ld_in(p.v_new, (size_t)kv * AT_D + t, p.in_dtype));
    __syncthreads();
    if (is_q || is_k) am_norm_rope(x, is_q ? p.q_norm_w : p.k_norm_w, cs_s, sn_s, p.rot_dims, p.eps, is_q ? qscale : 1.0f);
    uint4 hi, lo;
    split_bf16x2(is_q ? x[0] : 0.f, is_q ? x[1] : 0.f, hi.x, lo.x);
    split_bf16x2(is_q ? x[2] : 0.f, is_q ? x[3] : 0.f, hi.y, lo.y);
    split_bf16x2(is_q ? x[4] : 0.f, is_q ? x[5] : 0.f, hi.z, lo.z);
    split_bf16x2(is_q ? x[6] : 0.f, is_q ? x[7] : 0.f, hi.w, lo.w);
    *reinterpret_cast<uint4*>(qs + warp * AM_QS + lane * 16) = hi; // rows G..7 are zero
    *reinterpret_cast<uint4*>(qs + (8 + warp) * AM_QS + lane * 16) = lo;
    if (is_k) {
        const size_t row = ((size_t)pos * p.HKV + kv) * AT_D + lane * 8;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const __nv_bfloat16 kb = __float2bfloat16_rn(x[j]);
            kn_s[lane * 8 + j] = kb;
            reinterpret_cast<__nv_bfloat16*>(p.k_cache)[row + j] = kb; // KV append
        }
    }
    if (last) {
        vn_s[t] = vb;
        reinterpret_cast<__nv_bfloat16*>(p.v_cache)[((size_t)pos * p.HKV + kv) * AT_D + t] = vb;
    }
    __syncthreads();
    pdl_launch_dependents();

    am_warp<G> a;
    a.m = -INFINITY;
    a.l = 0.f;
#pragma unroll
    for (int b = 0; b < 16; ++b) a.acc[b][0] = a.acc[b][1] = a.acc[b][2] = a.acc[b][3] = 0.f;
    const unsigned char* ql = qs + fg * AM_QS + ft * 16;
    for (int b = warp; b < n_blocks; b += AT_WARPS) {
        const bool more = b + AT_WARPS < n_blocks;
        float s[2][4];
        uint32_t ph[2], pl[2];
        a.scores(K, ql, s);
        if (more) load_keys(b + AT_WARPS);
        a.softmax(s, min(AM_ROWS, t1 - (t0 + b * AM_ROWS)), ft, ph, pl);
        a.read_out(V, ph, pl);
        if (more) load_values(b + AT_WARPS);
    }
    if (last && warp == AT_WARPS - 1) { // the token being decoded: a block whose 16 rows all repeat it, one of them valid
        float s[2][4];
        uint32_t ph[2], pl[2];
#pragma unroll
        for (int c = 0; c < 8; ++c) K.w[0][c] = K.w[1][c] = *reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned char*>(kn_s) + c * 64 + ft * 16);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) V.w[i][c] = *reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned char*>(vn_s) + c * 128 + fg * 16);
        a.scores(K, ql, s);
        a.softmax(s, 1, ft, ph, pl);
        a.read_out(V, ph, pl);
    }

    // ---- merge the 8 warps (fixed order): every warp brings its result to the common maximum, then thread t owns feature t ----
    if (ft == 0) {
        wm[warp * AT_GMAX + fg] = a.m;
        wl[warp * AT_GMAX + fg] = a.l;
    }
    __syncthreads();
    if (2 * ft < G) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int g = 2 * ft + e;
            if (g >= G) continue;
            float M = -INFINITY;
#pragma unroll
            for (int w = 0; w < AT_WARPS; ++w) M = fmaxf(M, wm[w * AT_GMAX + g]);
            const float mw = wm[warp * AT_GMAX + g], sc = mw == -INFINITY ? 0.f : exp2f(mw - M);
            float* dst = part + (warp * G + g) * AM_HS + 8 * fg;
#pragma unroll
            for (int seg = 0; seg < 4; ++seg)
#pragma unroll
                for (int j = 0; j < 4; j += 2)
                    *reinterpret_cast<float4*>(dst + 64 * seg + 2 * j) =
                        make_float4(a.acc[4 * seg + j][e] * sc, a.acc[4 * seg + j][2 + e] * sc, a.acc[4 * seg + j + 1][e] * sc, a.acc[4 * seg + j + 1][2 + e] * sc);
        }
    }
    __syncthreads();
    float Ag[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        Ag[g] = 0.f;
#pragma unroll
        for (int w = 0; w < AT_WARPS; ++w) Ag[g] += part[(w * G + g) * AM_HS + t];
    }
    float M = -INFINITY, L = 0.f; // of head t, in the first G threads
    if (t < G) {
#pragma unroll
        for (int w = 0; w < AT_WARPS; ++w) M = fmaxf(M, wm[w * AT_GMAX + t]);
#pragma unroll
        for (int w = 0; w < AT_WARPS; ++w) {
            const float mw = wm[w * AT_GMAX + t];
            L = fmaf(wl[w * AT_GMAX + t], mw == -INFINITY ? 0.f : exp2f(mw - M), L);
        }
    }
    if (p.splits == 1) {
        if (t < G) wl[t] = L; // the first warp's sums: their readers above are these threads themselves
        __syncthreads();
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int hq = kv * G + g;
            float o = Ag[g] / wl[g];
            if (p.gate) o *= sigmoidf_dev(ld_in(p.gate, (size_t)hq * p.gate_stride + t, p.in_dtype));
            p.out[(size_t)hq * AT_D + t] = o;
        }
        return;
    }

    // ---- merge the position slices: every CTA of a KV head leaves its record, and each finishes its own share of the (head, feature) outputs when all
    // of them are there.  The arrivals are the low half of a word; a CTA that does not want to wait any longer puts a flag on its share, adds to the high half and
    // leaves, unless that addition finds everybody arrived.  So whoever finds everybody there, the last arrival at least, also sees whether shares were left, and
    // does those whose flags it takes off: each share is done once. ----
    float* rec = p.scratch + ((size_t)(kv * p.splits + split) * G) * AT_REC;
#pragma unroll
    for (int g = 0; g < G; ++g) __stcg(rec + g * AT_REC + t, Ag[g]);
    if (t < G) {
        __stcg(rec + t * AT_REC + 256, M);
        __stcg(rec + t * AT_REC + 257, L);
    }
    const bool groups = p.splits > 16;
    const float gate0 = am_gate<G>(p, kv, split); // on its way during the wait
    __syncthreads(); // the whole record is written
    uint32_t *word = p.counters + kv, *finished = p.counters + 8 + kv, *flags = p.counters + 16 + kv * p.splits;
    bool left = false; // of thread 0: others have left their shares
    int leave = 0;
    if (t == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(word) : "memory");
        const uint64_t w0 = globaltimer_ns();
        const uint32_t mask = (uint32_t)p.stay; // the timer is read once per mask + 1 polls
        uint32_t v;
        bool ok = false;
        for (uint32_t it = 0; it < LB_WAIT_SPINS; ++it) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
            if ((v & 0xffffu) == (uint32_t)p.splits) { ok = true; break; }
            if ((it & mask) == mask && globaltimer_ns() - w0 >= 200ull * mask) break;
        }
        if (!ok) v = am_leave(word, flags + split, (uint32_t)p.splits);
        leave = v == AM_LEFT;
        left = v >> 16;
    }
    if (!__syncthreads_or(leave)) {
        if (groups) am_finish<G, 4>(p, kv, split, gate0, part);
        else am_finish<G, 1>(p, kv, split, gate0, part);
    }
    if (__syncthreads_or(left)) am_take_over<G>(p, kv, flags, part);
    if (t == 0) am_done(p, word, finished);
}

extern "C" __global__ void __launch_bounds__(AT_THREADS, 1) attn_decode_mma(const __grid_constant__ lb_attn_params p) {
    extern __shared__ __align__(128) unsigned char am_sm[];
    const int G = p.HQ / p.HKV;
    switch (G) {
        case 1: attn_mma_body<1>(p, am_sm); break;
        case 2: attn_mma_body<2>(p, am_sm); break;
        case 3: attn_mma_body<3>(p, am_sm); break;
        case 4: attn_mma_body<4>(p, am_sm); break;
        case 6: attn_mma_body<6>(p, am_sm); break;
        default: break; // host rejects other ratios
    }
}
