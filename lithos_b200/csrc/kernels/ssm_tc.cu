// A prompt chunk through the state-space recurrence (ssm.cu) on the 5th-generation tensor cores, for states of 128 rows and heads of 64 value columns (padded).
// A CTA owns a head's whole state (thread = row and half of the columns, in registers) and walks blocks of 128 tokens.  With c_i the sum of
// a = -exp(A_log) dt over the block's tokens up to i:
//   G  = C B^T                                     128 x 128 x 128, operands as they lie in the convolution's output
//   Y1 = C S                                       128 x  64 x 128, S as three bf16 terms from shared memory
//   Y2 = M x, M_ij = exp(c_i - c_j) dt_j G_ij (j <= i)  128 x 64 x 128, M as three bf16 terms from TENSOR memory
//   D  = B^T (w x), w_j = exp(c_end - c_j) dt_j    128 x  64 x 128, w x as three bf16 terms; B read as its own transpose
//   y  = exp(c_i) Y1 + Y2 + skip x,   S <- exp(c_end) S + D
// B, C and x are bf16; three bf16 terms carry all 24 bits of the fp32 factors; sums are fp32, c_i - c_j comes from sums in fp64 kept as two floats.
// Segments (gridDim.z = P > 1; segment g is tokens g * seg ..) as in ssm.cu: LOCAL (first launch, P - 1 segments) leaves what each makes of a zero state
// (segment 0: of the sequence's state) and its summed log decay, and keeps the sequence's state in the last place; the second launch makes a segment's start
// from those before it, and the last leaves the sequence's state.  The workspace holds a state in the order of the threads.
// Tokens past the chunk are zero-filled by the copy engine, their step size is 0 and they are not stored.
// Every wait is bounded and reports through the status word; TMEM is freed on every path.
// Bound by the chain of a block: products, exponentials and splits, products again, with a barrier of the block between them; the tensor pipe is busy for 18 % of the
// active cycles, the warps wait for barriers and shared memory most (ncu).  The mma.sync kernels of ssm.cu (64 tokens x 32 columns, 262 products of 16 cycles a warp) were bound by that unit and made
// C B^T twice.  Vobunex prompts, us, before -> after: 4001 tokens 5126 -> 4790, 1500 behind 300 2236 -> 2064, 600 1398 -> 1284, 100 behind 2000 916 -> 904.
#include "tcgen05.cuh"
#include "mma_sync.cuh"
#include "params.h"

#define ST_UNIT 16384 /* 128 rows of 64 bf16 columns, 128-byte swizzle */
// tensor memory: G | M's three terms | Y1 | Y2 | D
#define ST_G 0u
#define ST_M 128u
#define ST_Y1 320u
#define ST_Y2 384u
#define ST_D 448u
static_assert(LB_SSM_TC_TOKENS == 128 && LB_SSM_TC_SMEM == 14 * ST_UNIT + 2048 + 128, "layout");

__device__ __forceinline__ void st_tma(uint32_t dst_smem, const void* tmap, int x, int row, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst_smem),
                 "l"(tmap), "r"(x), "r"(row), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]),
                 "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ uint32_t st_at(int row, int piece) { return (uint32_t)(row * 128 + ((piece ^ (row & 7)) << 4)); } // a 16-byte piece of a row

// grid (H, 1, segments), block 256
template <bool LOCAL>
__device__ __forceinline__ void ssm_tc_body(const lb_ssm_params& p, const lb_ac_maps& maps) {
    extern __shared__ __align__(1024) unsigned char st_sm[];
    unsigned char *b_s = st_sm, *x_s = b_s + 4 * ST_UNIT, *c_s = x_s + 2 * ST_UNIT, *s_s = c_s + 2 * ST_UNIT, *w_s = s_s + 3 * ST_UNIT; // B and x: two stages
    float4* cum = reinterpret_cast<float4*>(w_s + 3 * ST_UNIT); // [128] of the block: c as two floats, dt
    uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(cum) + 2048);
    uint64_t *bar_in = bars, *bar_c = bars + 2, *bar_g = bars + 3, *bar_y1 = bars + 4, *bar_y2 = bars + 5, *bar_d = bars + 6;
    uint32_t* slot = reinterpret_cast<uint32_t*>(bars + 8);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, quad = warp & 3, half = warp >> 2, row = 32 * quad + lane; // row: of the state, of the block's tokens
    const int h = blockIdx.x, g = h / (p.H / p.G);
    const float a_neg = -expf(bf16_bits_to_f32(p.a_log[h])), dskip = bf16_bits_to_f32(p.d[h]);
    const int seg = blockIdx.z, P = LOCAL ? gridDim.z + 1 : gridDim.z, tok_lo = seg * p.seg, tok_hi = min(p.T, tok_lo + p.seg);
    const int n_blk = (tok_hi - tok_lo + 127) / 128;
    if (t == 0) {
        for (int i = 0; i < 7; ++i) mbar_init(&bars[i], 1);
        mbar_fence_init();
    }
    if (warp == 0) {
        __syncwarp();
        tmem_alloc(slot, 512);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *slot, lanes = (uint32_t)(32 * quad) << 16;
    if (!LOCAL) { // M's columns of later tokens are never written again
        const uint4 z = make_uint4(0u, 0u, 0u, 0u);
        for (int c = 96 * half; c < 96 * half + 96; c += 16) tmem_st16(tmem + lanes + ST_M + (uint32_t)c, z, z, z, z);
    }
    pdl_wait();

    auto fetch = [&](int blk) { // one thread: B and x of a block
        const int st = blk & 1, tok = tok_lo + blk * 128, xb = p.H * 64 + g * 128;
        mbar_arrive_expect_tx(&bar_in[st], 3 * ST_UNIT);
        st_tma(smem_u32(b_s) + (uint32_t)(2 * st) * ST_UNIT, maps.k, xb, tok, &bar_in[st]);
        st_tma(smem_u32(b_s) + (uint32_t)(2 * st + 1) * ST_UNIT, maps.k, xb + 64, tok, &bar_in[st]);
        st_tma(smem_u32(x_s) + (uint32_t)st * ST_UNIT, maps.k, h * 64, tok, &bar_in[st]);
    };
    auto fetch_c = [&](int blk) { // one thread
        const int tok = tok_lo + blk * 128, xc = p.H * 64 + (p.G + g) * 128;
        mbar_arrive_expect_tx(bar_c, 2 * ST_UNIT);
        st_tma(smem_u32(c_s), maps.k, xc, tok, bar_c);
        st_tma(smem_u32(c_s) + ST_UNIT, maps.k, xc + 64, tok, bar_c);
    };
    if (t == 0) {
        fetch(0);
        if (!LOCAL) fetch_c(0);
    }

    // the state: row `row`, columns 32 half .. + 31
    float s[32];
    float* mine = p.state + ((size_t)h * p.N + row) * p.V + 32 * half;
    const bool quads = (p.V & 3) == 0 && (reinterpret_cast<uintptr_t>(p.state) & 15) == 0;
    float4* ws = reinterpret_cast<float4*>(p.seg_state) + (size_t)h * 2048 + t;
    const size_t ws_seg = (size_t)p.H * 2048;
    auto put = [&](int at) {
#pragma unroll
        for (int i = 0; i < 8; ++i) ws[at * ws_seg + i * 256] = make_float4(s[4 * i], s[4 * i + 1], s[4 * i + 2], s[4 * i + 3]);
    };
#pragma unroll
    for (int i = 0; i < 32; ++i) s[i] = 0.f;
    if (LOCAL ? seg == 0 : P == 1) {
        if (row < p.N) {
            if (quads) {
#pragma unroll
                for (int i = 0; i < 32; i += 4)
                    if (32 * half + i < p.V) {
                        const float4 v = *reinterpret_cast<const float4*>(mine + i);
                        s[i] = v.x; s[i + 1] = v.y; s[i + 2] = v.z; s[i + 3] = v.w;
                    }
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (32 * half + i < p.V) s[i] = mine[i];
            }
        }
        if (LOCAL) put(P - 1);
    } else if (!LOCAL) {
        const int from = seg == 0 ? P - 1 : 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 v = ws[from * ws_seg + i * 256];
            s[4 * i] = v.x; s[4 * i + 1] = v.y; s[4 * i + 2] = v.z; s[4 * i + 3] = v.w;
        }
        for (int q = 1; q < seg; ++q) {
            const float d = expf(p.seg_decay[(size_t)q * p.H + h]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 v = ws[q * ws_seg + i * 256];
                s[4 * i] = fmaf(d, s[4 * i], v.x); s[4 * i + 1] = fmaf(d, s[4 * i + 1], v.y); s[4 * i + 2] = fmaf(d, s[4 * i + 2], v.z); s[4 * i + 3] = fmaf(d, s[4 * i + 3], v.w);
            }
        }
    }
    auto put_terms = [&]() { // the state as the B operand of Y1: rows of 64 columns
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t a[4], b[4], c[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) ms_split3(s[8 * i + 2 * e], s[8 * i + 2 * e + 1], a[e], b[e], c[e]);
            unsigned char* d = s_s + st_at(row, 4 * half + i);
            *reinterpret_cast<uint4*>(d) = make_uint4(a[0], a[1], a[2], a[3]);
            *reinterpret_cast<uint4*>(d + ST_UNIT) = make_uint4(b[0], b[1], b[2], b[3]);
            *reinterpret_cast<uint4*>(d + 2 * ST_UNIT) = make_uint4(c[0], c[1], c[2], c[3]);
        }
    };
    double log_decay = 0.;
    float4 next[4]; // of warp 1: c and dt of a block, a lane has four tokens
    auto sums = [&](int blk) {
        const int i0 = tok_lo + blk * 128 + 4 * lane;
        float d[4];
        double c[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i] = i0 + i < tok_hi ? p.dt[(size_t)(i0 + i) * p.H + h] : 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) c[i] = (double)(a_neg * d[i]) + (i > 0 ? c[i - 1] : 0.);
        double s = c[3];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += v;
        }
        s -= c[3];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double v = s + c[i];
            const float hi = (float)v;
            next[i] = make_float4(hi, (float)(v - (double)hi), d[i], 0.f);
        }
        if (LOCAL) log_decay += __shfl_sync(0xffffffffu, s + c[3], 31);
    };
    auto put_sums = [&]() {
#pragma unroll
        for (int i = 0; i < 4; ++i) cum[4 * lane + i] = next[i];
    };
    if (!LOCAL) put_terms();
    if (warp == 1) {
        sums(0);
        put_sums();
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tmem_st_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    const uint32_t g_idesc = tc_idesc_bf16(128, 128), y_idesc = tc_idesc_bf16(128, 64) | (1u << 16), d_idesc = y_idesc | (1u << 15); // bit 16: B is MN-major, 15: A
    const uint64_t b_desc = tc_smem_desc(smem_u32(b_s), 16, 1024), bt_desc = tc_smem_desc(smem_u32(b_s), ST_UNIT, 1024), c_desc = tc_smem_desc(smem_u32(c_s), 16, 1024),
                   x_desc = tc_smem_desc(smem_u32(x_s), ST_UNIT, 1024), s_desc = tc_smem_desc(smem_u32(s_s), ST_UNIT, 1024), w_desc = tc_smem_desc(smem_u32(w_s), ST_UNIT, 1024);
    constexpr uint64_t U = ST_UNIT >> 4;
    bool ok = true;
    int blk = 0;
    for (; blk < n_blk; ++blk) {
        const int st = blk & 1, tok0 = tok_lo + blk * 128;
        const uint32_t ph = (uint32_t)blk & 1u, ph_in = (uint32_t)(blk >> 1) & 1u;
        if (warp == 0 && tc_elect()) {
            if (!LOCAL) {
                ok = tc_wait(&bar_in[st], ph_in) && tc_wait(bar_c, ph);
                tc_fence_after();
                if (ok) {
                    for (int f = 0; f < 2; ++f)
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            tc_mma(tmem + ST_G, c_desc + f * U + 2 * kk, b_desc + (2 * st + f) * U + 2 * kk, g_idesc, f > 0 || kk > 0 ? 1u : 0u);
                    tc_commit(bar_g);
                    for (int term = 2; term >= 0; --term)
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk)
                            tc_mma(tmem + ST_Y1, c_desc + (kk >> 2) * U + 2 * (kk & 3), s_desc + term * U + 128 * kk, y_idesc, term < 2 || kk > 0 ? 1u : 0u);
                    tc_commit(bar_y1);
                }
            }
            if (ok && blk + 1 < n_blk) fetch(blk + 1); // everybody is done with that stage
        }
        __syncwarp();
        ok = ok && tc_wait(&bar_in[st], ph_in);
        const float4 last = cum[127];
        if (ok) { // scaled x: the B operand of D
            const float4 cj = cum[t & 127];
            const float w = cj.z * expf((last.x - cj.x) + (last.y - cj.y));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t at = st_at(t & 127, 4 * (t >> 7) + i);
                const uint4 v = *reinterpret_cast<const uint4*>(x_s + st * ST_UNIT + at);
                const uint32_t u[4] = {v.x, v.y, v.z, v.w};
                uint32_t a[4], b[4], c[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) ms_split3(w * __uint_as_float(u[e] << 16), w * __uint_as_float(u[e] & 0xffff0000u), a[e], b[e], c[e]);
                *reinterpret_cast<uint4*>(w_s + at) = make_uint4(a[0], a[1], a[2], a[3]);
                *reinterpret_cast<uint4*>(w_s + ST_UNIT + at) = make_uint4(b[0], b[1], b[2], b[3]);
                *reinterpret_cast<uint4*>(w_s + 2 * ST_UNIT + at) = make_uint4(c[0], c[1], c[2], c[3]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        const float4 ci = cum[row];
        if (!LOCAL) { // M: a warp has 32 rows and every other 16 columns of those up to its last row
            ok = __all_sync(0xffffffffu, ok && tc_wait(bar_g, ph));
            if (ok) {
                tc_fence_after();
#pragma unroll 2
                for (int jg = half; jg < 2 * quad + 2; jg += 2) {
                    uint32_t v[16], m[3][8];
                    tmem_ld16(tmem + lanes + ST_G + (uint32_t)(16 * jg), v);
                    tmem_ld_wait();
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        float e[2];
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const int j = 16 * jg + 2 * q + i;
                            const float4 cj = cum[j];
                            e[i] = j <= row ? expf((ci.x - cj.x) + (ci.y - cj.y)) * cj.z : 0.f;
                        }
                        ms_split3(__uint_as_float(v[2 * q]) * e[0], __uint_as_float(v[2 * q + 1]) * e[1], m[0][q], m[1][q], m[2][q]);
                    }
#pragma unroll
                    for (int term = 0; term < 3; ++term) tmem_st8(tmem + lanes + ST_M + (uint32_t)(64 * term + 8 * jg), m[term]);
                }
                tmem_st_wait();
            }
        }
        tc_fence_before();
        ok = __syncthreads_and(ok);
        if (!ok) break;
        tc_fence_after();
        if (warp == 0 && tc_elect()) {
            if (!LOCAL) {
                for (int term = 2; term >= 0; --term)
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)
                        tc_mma_ta(tmem + ST_Y2, tmem + ST_M + (uint32_t)(64 * term + 8 * kk), x_desc + st * U + 128 * kk, y_idesc, term < 2 || kk > 0 ? 1u : 0u);
                tc_commit(bar_y2);
            }
            for (int term = 2; term >= 0; --term)
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                    tc_mma(tmem + ST_D, bt_desc + 2 * st * U + 128 * kk, w_desc + term * U + 128 * kk, d_idesc, term < 2 || kk > 0 ? 1u : 0u);
            tc_commit(bar_d);
            if (!LOCAL && blk + 1 < n_blk && (ok = tc_wait(bar_y1, ph))) fetch_c(blk + 1); // C has been read
        }
        __syncwarp();
        if (warp == 1 && blk + 1 < n_blk) sums(blk + 1);
        const float e_end = expf(last.x + last.y);
        if (!LOCAL) {
            ok = __all_sync(0xffffffffu, ok && tc_wait(bar_y1, ph) && tc_wait(bar_y2, ph));
            if (ok) {
                tc_fence_after();
                const float e = expf(ci.x + ci.y);
                const int tok = tok0 + row;
                float* dst = p.y + ((size_t)tok * p.H + h) * p.V + 32 * half;
                uint32_t y1[2][16], y2[2][16];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    tmem_ld16(tmem + lanes + ST_Y1 + (uint32_t)(32 * half + 16 * i), y1[i]);
                    tmem_ld16(tmem + lanes + ST_Y2 + (uint32_t)(32 * half + 16 * i), y2[i]);
                }
                tmem_ld_wait();
                if (tok < tok_hi) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint4 v = *reinterpret_cast<const uint4*>(x_s + st * ST_UNIT + st_at(row, 4 * half + i));
                        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
                        float o[8];
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            const float xv = __uint_as_float(q & 1 ? u[q >> 1] & 0xffff0000u : u[q >> 1] << 16);
                            const int c = 8 * i + q;
                            o[q] = fmaf(dskip, xv, fmaf(e, __uint_as_float(y1[c >> 4][c & 15]), __uint_as_float(y2[c >> 4][c & 15])));
                        }
                        const int col = 32 * half + 8 * i;
                        if ((p.V & 3) == 0) {
                            if (col < p.V) *reinterpret_cast<float4*>(dst + 8 * i) = make_float4(o[0], o[1], o[2], o[3]);
                            if (col + 4 < p.V) *reinterpret_cast<float4*>(dst + 8 * i + 4) = make_float4(o[4], o[5], o[6], o[7]);
                        } else {
#pragma unroll
                            for (int q = 0; q < 8; ++q)
                                if (col + q < p.V) dst[8 * i + q] = o[q];
                        }
                    }
                }
                __syncwarp();
            }
        }
        ok = __all_sync(0xffffffffu, ok && tc_wait(bar_d, ph));
        if (ok) {
            tc_fence_after();
            uint32_t d[2][16];
            tmem_ld16(tmem + lanes + ST_D + (uint32_t)(32 * half), d[0]);
            tmem_ld16(tmem + lanes + ST_D + (uint32_t)(32 * half + 16), d[1]);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) s[i] = fmaf(e_end, s[i], __uint_as_float(d[i >> 4][i & 15]));
            if (!LOCAL && blk + 1 < n_blk) put_terms();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        tc_fence_before();
        ok = __syncthreads_and(ok); // everybody is done with the block's sums, x, and what tensor memory holds
        if (!ok) break;
        if (blk + 1 < n_blk) {
            if (warp == 1) put_sums();
            __syncthreads();
        }
        tc_fence_after();
    }
    pdl_launch_dependents();
    if (!ok) {
        if (t == 0) {
            if (p.status) atomicExch(p.status, ST_FAIL);
            // nothing may still be on its way into this CTA's shared memory when it ends
            tc_wait(&bar_in[blk & 1], (uint32_t)(blk >> 1) & 1u);
            if (blk + 1 < n_blk) tc_wait(&bar_in[(blk + 1) & 1], (uint32_t)((blk + 1) >> 1) & 1u);
            if (!LOCAL) {
                tc_wait(bar_c, (uint32_t)blk & 1u);
                if (blk + 1 < n_blk) tc_wait(bar_c, (uint32_t)(blk + 1) & 1u);
            }
        }
    } else if (LOCAL) {
        put(seg);
        if (t == 32) p.seg_decay[(size_t)seg * p.H + h] = (float)log_decay;
    } else if (seg == P - 1 && row < p.N) {
        if (quads) {
#pragma unroll
            for (int i = 0; i < 32; i += 4)
                if (32 * half + i < p.V) *reinterpret_cast<float4*>(mine + i) = make_float4(s[i], s[i + 1], s[i + 2], s[i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (32 * half + i < p.V) mine[i] = s[i];
        }
    }
    __syncthreads();
    if (warp == 0) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}
extern "C" __global__ void __launch_bounds__(256) ssm_tc(const __grid_constant__ lb_ssm_params p, const __grid_constant__ lb_ac_maps maps) { ssm_tc_body<false>(p, maps); }
extern "C" __global__ void __launch_bounds__(256) ssm_tc_local(const __grid_constant__ lb_ssm_params p, const __grid_constant__ lb_ac_maps maps) { ssm_tc_body<true>(p, maps); }
