// Causal attention of a prompt chunk on the 5th-generation tensor cores, shared by the int4 hybrid (prefill.cu) and the list-of-layers models
// (window_attention.cu).  A CTA owns 128 query rows of one KV head (row R = (token R / G, head R % G)) and walks the keys 128 at a time:
//   S = Q K^T   128 x 128 x dim,  both operands from shared memory, Q as two bf16 terms (16 bits), K bf16: two products per k-step
//   O += P V    128 x vdim x 128, P as two bf16 terms from TENSOR memory, V from shared memory as it lies in the cache (MN-major operand)
// Warps: one thread brings keys and values by tiled TMA in units of 16 KB (64 features x 128 keys, or vdim features x 8192 / vdim keys) into one ring,
// one thread issues products, four warps (thread = query row = tensor-memory lane, so no soft-max quantity ever crosses lanes) turn scores into
// probabilities.  P overwrites the scores it came from; there are three such buffers (two at 256 value features, where the accumulator takes half of the
// tensor memory), so the scores of block i + 1 are made while block i is with the soft-max warps.
// The maximum a row's probabilities refer to follows its running maximum only when that is more than 8 (in log2 units) ahead, and then the accumulator is
// rescaled in tensor memory (the conditional rescaling of FlashAttention-4); sums of up to 256 x as large terms cost no precision in fp32, and almost no block rescales.
// Few query rows behind many keys leave SMs idle: the key blocks of a tile are then dealt to `parts` CTAs (grid.z), which leave unnormalised rows, maxima and sums
// in scratch, and attn_chunk_merge adds them in order (lb_ac_launch chooses; us: hybrid 75 tokens behind 2000 1625 -> 1545, 5 tokens 1102 -> 1003, Vobunex 100
// behind 2000 930 -> 907, Nufalorn 150 behind 2000 1009 -> 984).
// Every wait is bounded and reports through the status word; TMEM is freed on every path.
// Bound by the products where a CTA has many keys, and by its start and end where it has few: the tensor pipe is busy for 42 % of the active cycles of the SM with most
// blocks at 1536 tokens of 128-feature heads, for 37 % where 256 tokens of the hybrid's heads (256 features) behind 1536 are dealt to three CTAs a
// tile (ncu).  Before (mma.sync, 16 query rows per warp, keys and values re-read from shared memory through ldmatrix for every 16 rows, the reason it stood at a tenth of the tensor cores' rate), whole prompts, us: int4 hybrid 75 tokens
// behind 2000 1837 -> 1648, Nufalorn 3000 7185 -> 6869 and 40 behind 1500 861 -> 746, Vobunex 4001 6120 -> 5194 and 100 behind 2000 1168 -> 929.
#pragma once
#include "tcgen05.cuh"
#include "params.h"

#define AC_ROWS LB_AC_ROWS
#define AC_KEYS 128
#define AC_UNIT LB_AC_UNIT

__device__ __forceinline__ void ac_tma(uint32_t dst_smem, const void* tmap, int x, int row, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst_smem),
                 "l"(tmap), "r"(x), "r"(row), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ float ac_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// (x, y) as a bf16 pair and the pair of what the rounding left over
__device__ __forceinline__ void ac_split(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xffff0000u));
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

struct ac_shared {
    __align__(8) uint64_t full[LB_AC_MAX_UNITS], empty[LB_AC_MAX_UNITS], s_done[3], p_ready[3], pv_done[3];
    uint32_t tmem;
};

// C says what a row is: const uint16_t *qh, *ql; size_t q_at(R): its first element in them; int lim(R), low(R): the keys low..lim are visible;
// float m0(R), l0(): the maximum and the sum to start from; table(sm): what store() wants in shared memory, by the 128 threads of the soft-max warps;
// store(sm, R, d, v, inv): features d..d+15 of its result, v * inv.
// dim: features of a key, own of them at k[row][kv * own ..], the rest (shared by the KV heads) at tail[row][..]; multiples of 64.  vdim 64, 128 or 256.
template <class C>
__device__ __forceinline__ void attn_chunk_tc(const C& c, const lb_ac_maps& maps, ac_shared& sh, unsigned char* sm, int kv, int R0, int n_rows, int first_key, int last_key,
                                              int dim, int own, int vdim, int units, uint32_t* status, const lb_ac_split& sp) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, z = blockIdx.z;
    const int blocks = (last_key - first_key) / AC_KEYS + 1, b0 = blocks * z / sp.parts, n = blocks * (z + 1) / sp.parts - b0; // n 0: a part without keys
    first_key += b0 * AC_KEYS;
    float* part = sp.parts > 1 ? sp.part + ((((size_t)kv * sp.tiles + R0 / AC_ROWS) * sp.parts + z) * AC_ROWS) * (vdim + 4) : nullptr; // [128][vdim | maximum, sum]
    const int NB = vdim > 128 ? 2 : 3, kc = dim / 64, vu = vdim / 64, vr = 8192 / vdim;
    unsigned char* ring = sm + (size_t)2 * kc * AC_UNIT; // behind the queries: [2 terms][kc][128 rows][128 bytes], 128-byte swizzle
    if (tid == 0) {
        for (int s = 0; s < units; ++s) {
            mbar_init(&sh.full[s], 1);
            mbar_init(&sh.empty[s], 1);
        }
        for (int s = 0; s < 3; ++s) {
            mbar_init(&sh.s_done[s], 1);
            mbar_init(&sh.p_ready[s], 4);
            mbar_init(&sh.pv_done[s], 1);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        __syncwarp();
        tmem_alloc(&sh.tmem, 512);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem, tmem_o = tmem + (NB == 2 ? 256u : 384u);
    pdl_wait();

    if (warp > 0) { // the queries; rows past the chunk repeat the last one (they are never stored)
        const int pieces = dim / 8;
        for (int i = tid - 32; i < AC_ROWS * pieces; i += LB_AC_THREADS - 32) {
            const int r = i / pieces, f = i - r * pieces;
            const size_t at = c.q_at(min(R0 + r, n_rows - 1)) + 8 * f;
            unsigned char* dst = sm + (size_t)(f >> 3) * AC_UNIT + r * 128 + (((f & 7) ^ (r & 7)) << 4);
            *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(c.qh + at);
            *reinterpret_cast<uint4*>(dst + (size_t)kc * AC_UNIT) = *reinterpret_cast<const uint4*>(c.ql + at);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("bar.sync 1, %0;" ::"n"(LB_AC_THREADS - 32) : "memory");
    }

    if (warp == 0) {
        // ---------------- keys and values: K 0, K 1, V 0, K 2, V 1, ... ----------------
        if (tc_elect()) {
            int u = 0, issued = 0;
            uint32_t ph = 0;
            bool ok = true;
            auto room = [&]() -> bool {
                if (issued >= units && !tc_wait(&sh.empty[u], ph ^ 1u)) {
                    if (status) atomicExch(status, AC_FAIL_EMPTY);
                    return false;
                }
                mbar_arrive_expect_tx(&sh.full[u], AC_UNIT);
                return true;
            };
            auto next = [&] {
                ++issued;
                if (++u == units) { u = 0; ph ^= 1u; }
            };
            for (int i = -1; i < n && ok; ++i) {
                for (int f = 0; f < kc && ok && i + 1 < n; ++f) {
                    if (!(ok = room())) break;
                    const bool mine = 64 * f < own;
                    ac_tma(smem_u32(ring) + (uint32_t)u * AC_UNIT, mine ? maps.k : maps.tail, mine ? kv * own + 64 * f : 64 * f - own, first_key + (i + 1) * AC_KEYS, &sh.full[u]);
                    next();
                }
                for (int j = 0; j < vu && ok && i >= 0; ++j) {
                    if (!(ok = room())) break;
                    for (int f = 0; f < vu; ++f)
                        ac_tma(smem_u32(ring) + (uint32_t)(u * AC_UNIT + f * vr * 128), maps.v, kv * vdim + 64 * f, first_key + i * AC_KEYS + j * vr, &sh.full[u]);
                    next();
                }
            }
            if (!ok) // nothing may still be on its way into this CTA's shared memory when it ends
                for (int s = 0; s < units && s < issued; ++s) {
                    if (--u < 0) { u = units - 1; ph ^= 1u; }
                    tc_wait(&sh.full[u], ph);
                }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- products: S 0, S 1, PV 0, S 2, PV 1, ... ----------------
        if (tc_elect()) {
            const uint32_t s_idesc = tc_idesc_bf16(AC_ROWS, AC_KEYS), o_idesc = tc_idesc_bf16(AC_ROWS, (uint32_t)vdim) | (1u << 16); // bit 16: B is MN-major
            const uint64_t q_desc = tc_smem_desc(smem_u32(sm), 16, 1024), k_desc = tc_smem_desc(smem_u32(ring), 16, 1024);
            // V: 64 features (128 bytes) x 8 keys are a swizzle atom; from 8 keys to the next 1024 bytes, from 64 features to the next vr x 128
            const uint64_t v_desc = tc_smem_desc(smem_u32(ring), (uint32_t)vr * 128u, 1024);
            int u = 0;
            uint32_t ph = 0;
            bool ok = true;
            auto landed = [&]() -> bool {
                if (!tc_wait(&sh.full[u], ph)) {
                    if (status) atomicExch(status, AC_FAIL_FULL);
                    return ok = false;
                }
                tc_fence_after();
                return true;
            };
            auto done = [&] {
                tc_commit(&sh.empty[u]);
                if (++u == units) { u = 0; ph ^= 1u; }
            };
            for (int i = -1; i < n && ok; ++i) {
                if (i + 1 < n) { // scores of block i + 1, once the read-out of the block that had the buffer is done
                    const int b = (i + 1) % NB;
                    if (i + 1 >= NB && !tc_wait(&sh.pv_done[b], (uint32_t)((i + 1) / NB - 1) & 1u)) {
                        ok = false;
                        if (status) atomicExch(status, AC_FAIL_SCORES);
                        break;
                    }
                    tc_fence_after();
                    const uint32_t d = tmem + (uint32_t)(128 * b);
                    for (int f = 0; f < kc && landed(); ++f) {
                        const uint64_t qd = q_desc + (uint64_t)((f * AC_UNIT) >> 4), kd = k_desc + (uint64_t)((u * AC_UNIT) >> 4);
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) {
                            tc_mma(d, qd + (uint64_t)(2 * kk), kd + (uint64_t)(2 * kk), s_idesc, f > 0 || kk > 0 ? 1u : 0u);
                            tc_mma(d, qd + (uint64_t)((kc * AC_UNIT) >> 4) + (uint64_t)(2 * kk), kd + (uint64_t)(2 * kk), s_idesc, 1u);
                        }
                        done();
                    }
                    if (!ok) break;
                    tc_commit(&sh.s_done[b]);
                }
                if (i >= 0) {
                    const int b = i % NB;
                    if (!tc_wait(&sh.p_ready[b], (uint32_t)(i / NB) & 1u)) {
                        ok = false;
                        if (status) atomicExch(status, AC_FAIL_SCORES);
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a = tmem + (uint32_t)(128 * b); // leading terms in 64 columns (two keys each), the remainders in the next 64
                    for (int j = 0; j < vu && landed(); ++j) {
                        const uint64_t vd = v_desc + (uint64_t)((u * AC_UNIT) >> 4);
                        for (int kk = 0; kk < vr / 16; ++kk) {
                            const uint32_t p = a + (uint32_t)((j * vr + kk * 16) >> 1);
                            tc_mma_ta(tmem_o, p, vd + (uint64_t)(128 * kk), o_idesc, i > 0 || j > 0 || kk > 0 ? 1u : 0u);
                            tc_mma_ta(tmem_o, p + 64u, vd + (uint64_t)(128 * kk), o_idesc, 1u);
                        }
                        done();
                    }
                    if (!ok) break;
                    tc_commit(&sh.pv_done[b]);
                }
            }
        }
        __syncwarp();
    } else {
        // ---------------- soft-max: thread = query row ----------------
        const int quad = warp & 3, R = R0 + 32 * quad + lane, Rc = min(R, n_rows - 1);
        const uint32_t lanes = (uint32_t)(32 * quad) << 16;
        const int lim = c.lim(Rc), low = c.low(Rc);
        float m = z == 0 ? c.m0(Rc) : -INFINITY, l = z == 0 ? c.l0() : 0.f;
        bool ok = true;
        for (int i = 0; i < n; ++i) {
            const int b = i % NB, key0 = first_key + i * AC_KEYS;
            ok = __all_sync(0xffffffffu, tc_wait(&sh.s_done[b], (uint32_t)(i / NB) & 1u));
            if (!ok) break;
            tc_fence_after();
            const uint32_t buf = tmem + lanes + (uint32_t)(128 * b);
            uint32_t s[8][16];
#pragma unroll
            for (int j = 0; j < 8; ++j) tmem_ld16(buf + (uint32_t)(16 * j), s[j]);
            tmem_ld_wait();
            if (!__all_sync(0xffffffffu, key0 >= low && key0 + AC_KEYS - 1 <= lim)) {
#pragma unroll
                for (int j = 0; j < 128; ++j)
                    if (key0 + j > lim || key0 + j < low) s[j >> 4][j & 15] = 0xff800000u; // -inf
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int j = 0; j < 128; ++j) mx[j & 3] = fmaxf(mx[j & 3], __uint_as_float(s[j >> 4][j & 15]));
            const float mb = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            const bool ahead = mb > m + 8.f;
            if (__any_sync(0xffffffffu, ahead)) {
                const float m_new = ahead ? mb : m, f = ahead ? exp2f(m - m_new) : 1.f;
                m = m_new;
                l *= f;
                if (i > 0) {
                    ok = __all_sync(0xffffffffu, tc_wait(&sh.pv_done[(i - 1) % NB], (uint32_t)((i - 1) / NB) & 1u));
                    if (!ok) break;
                    tc_fence_after();
                    for (int d = 0; d < vdim; d += 16) {
                        uint32_t r[16];
                        tmem_ld16(tmem_o + lanes + (uint32_t)d, r);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * f);
                        tmem_st16(tmem_o + lanes + (uint32_t)d, make_uint4(r[0], r[1], r[2], r[3]), make_uint4(r[4], r[5], r[6], r[7]), make_uint4(r[8], r[9], r[10], r[11]),
                                  make_uint4(r[12], r[13], r[14], r[15]));
                    }
                }
            }
            const float mu = m == -INFINITY ? 0.f : m; // nothing seen so far: every score of the block is -infinity, every probability 0
            float ps[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < 4; ++j) { // 32 keys: 16 pairs
                uint32_t h[16], r[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float p0 = ac_exp2(__uint_as_float(s[2 * j + (e >> 3)][2 * (e & 7)]) - mu), p1 = ac_exp2(__uint_as_float(s[2 * j + (e >> 3)][2 * (e & 7) + 1]) - mu);
                    ps[(2 * e) & 3] += p0;
                    ps[(2 * e + 1) & 3] += p1;
                    ac_split(p0, p1, h[e], r[e]);
                }
                tmem_st16(buf + (uint32_t)(16 * j), make_uint4(h[0], h[1], h[2], h[3]), make_uint4(h[4], h[5], h[6], h[7]), make_uint4(h[8], h[9], h[10], h[11]),
                          make_uint4(h[12], h[13], h[14], h[15]));
                tmem_st16(buf + 64u + (uint32_t)(16 * j), make_uint4(r[0], r[1], r[2], r[3]), make_uint4(r[4], r[5], r[6], r[7]), make_uint4(r[8], r[9], r[10], r[11]),
                          make_uint4(r[12], r[13], r[14], r[15]));
            }
            l += (ps[0] + ps[1]) + (ps[2] + ps[3]);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.p_ready[b]);
        }
        if (ok && n > 0) ok = __all_sync(0xffffffffu, tc_wait(&sh.pv_done[(n - 1) % NB], (uint32_t)((n - 1) / NB) & 1u));
        tc_fence_after();
        pdl_launch_dependents();
        if (!ok && lane == 0 && status) atomicExch(status, AC_FAIL_SCORES);
        ok = __all_sync(0xffffffffu, ok);
        float* mine = part ? part + (size_t)(32 * quad + lane) * (vdim + 4) : nullptr;
        if (part) {
            mine[vdim] = m;
            mine[vdim + 1] = l;
        } else {
            c.table(sm, R0); // every product is done: queries and ring are free
            asm volatile("bar.sync 2, 128;" ::: "memory");
        }
        const float inv = 1.0f / l;
        for (int d = 0; d < vdim && ok; d += 16) {
            uint32_t r[16];
            __syncwarp(); // the stores before are some lanes' only
            if (n > 0) {
                tmem_ld16(tmem_o + lanes + (uint32_t)d, r);
                tmem_ld_wait();
            } else
#pragma unroll
                for (int j = 0; j < 16; ++j) r[j] = 0u;
            if (part) {
#pragma unroll
                for (int j = 0; j < 16; j += 4) *reinterpret_cast<uint4*>(mine + d + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
            } else if (R < n_rows) c.store(sm, R0, R, d, r, inv);
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// The parts of a tile, in order: grid (tiles, KV heads, 128 vdim / 4096), block 256, a thread 16 features of a row
template <class C>
__device__ __forceinline__ void attn_chunk_merge(const C& c, int kv, int n_rows, int vdim, const lb_ac_split& sp) {
    pdl_wait();
    const int per = vdim / 16, i = (int)blockIdx.z * 256 + threadIdx.x, row = i / per, d = 16 * (i - row * per), tile = (int)blockIdx.x, R = tile * AC_ROWS + row;
    if (R < n_rows) {
        const float* base = sp.part + ((((size_t)kv * sp.tiles + tile) * sp.parts) * AC_ROWS + row) * (vdim + 4);
        const size_t step = (size_t)AC_ROWS * (vdim + 4);
        float M = -INFINITY, L = 0.f, o[16];
        for (int z = 0; z < sp.parts; ++z) M = fmaxf(M, base[z * step + vdim]);
#pragma unroll
        for (int j = 0; j < 16; ++j) o[j] = 0.f;
        for (int z = 0; z < sp.parts; ++z) {
            const float w = exp2f(base[z * step + vdim] - M), l = base[z * step + vdim + 1];
            L = fmaf(w, l, L);
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
                const float4 v = *reinterpret_cast<const float4*>(base + z * step + d + j);
                o[j] = fmaf(w, v.x, o[j]); o[j + 1] = fmaf(w, v.y, o[j + 1]); o[j + 2] = fmaf(w, v.z, o[j + 2]); o[j + 3] = fmaf(w, v.w, o[j + 3]);
            }
        }
        uint32_t r[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(o[j]);
        c.store(nullptr, 0, R, d, r, 1.0f / L);
    }
}
