// Prompt pass (prefill): the small kernels between the batched int4 projections (gemm_int4_*) when a chunk of up to 128
// prompt tokens goes through a layer at once.  The layers run the same element-wise / recurrence kernels as decoding
// (compiler/megakernel-link.ls:281-525 layer order); here every kernel takes a chunk [T, ...] and leaves exactly the
// state a token-by-token decode of the same tokens leaves: DeltaNet state, convolution ring (slot = position & 3), KV rows.
// All activations are fp32 except the projection inputs, which are rounded to fp16 (the decode step's contract).
#include "common.cuh"
#include "params.h"

// X[t, :] = float(E[token[t], :])                                   grid T, block 256
extern "C" __global__ void pf_embed(const uint16_t* __restrict__ table, const int* __restrict__ tokens, float* __restrict__ X, int D) {
    pdl_wait(); // launched with programmatic stream serialization: nothing of the previous kernel is read before this
    const uint16_t* src = table + (size_t)tokens[blockIdx.x] * D;
    float* dst = X + (size_t)blockIdx.x * D;
    if ((D & 7) == 0 && (reinterpret_cast<uintptr_t>(table) & 15) == 0) { // whole 16-byte pieces
        for (int i = threadIdx.x; i < D / 8; i += blockDim.x) {
            const uint4 u = __ldg(reinterpret_cast<const uint4*>(src) + i);
            reinterpret_cast<float4*>(dst)[2 * i] = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
            reinterpret_cast<float4*>(dst)[2 * i + 1] = make_float4(__uint_as_float(u.z << 16), __uint_as_float(u.z & 0xffff0000u), __uint_as_float(u.w << 16), __uint_as_float(u.w & 0xffff0000u));
        }
        return;
    }
    for (int i = threadIdx.x; i < D; i += blockDim.x) dst[i] = bf16_bits_to_f32(src[i]);
}

// [x[t, :] += add[t, :] when add is given;]  y16[t, :] = fp16( x[t, :] * rsqrt(mean x^2 + eps) * (1 + w) )
// grid T, block 256, D a multiple of 4                                                 (inference/reduce.ls:21-147)
extern "C" __global__ void __launch_bounds__(256) pf_rmsnorm_f16(float* __restrict__ X, const float* __restrict__ add,
                                                                 const uint16_t* __restrict__ w, __half* __restrict__ Y, int D, float eps) {
    pdl_wait(); // launched with programmatic stream serialization: nothing of the previous kernel is read before this
    __shared__ float red[33];
    float4* x4 = reinterpret_cast<float4*>(X + (size_t)blockIdx.x * D);
    const float4* a4 = add ? reinterpret_cast<const float4*>(add + (size_t)blockIdx.x * D) : nullptr;
    float ss = 0.f;
    for (int i = threadIdx.x; i < D / 4; i += 256) {
        float4 v = x4[i];
        if (a4) {
            const float4 a = a4[i];
            v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
            x4[i] = v;
        }
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
    ss = block_sum(ss, red);
    const float rinv = rsqrtf(ss / (float)D + eps);
    for (int i = threadIdx.x; i < D / 4; i += 256) { // the thread re-reads what it wrote itself
        const float4 v = x4[i];
        const uint2 ww = *reinterpret_cast<const uint2*>(w + 4 * i);
        const __half2 lo = __floats2half2_rn(v.x * rinv * (1.0f + __uint_as_float(ww.x << 16)), v.y * rinv * (1.0f + __uint_as_float(ww.x & 0xffff0000u)));
        const __half2 hi = __floats2half2_rn(v.z * rinv * (1.0f + __uint_as_float(ww.y << 16)), v.w * rinv * (1.0f + __uint_as_float(ww.y & 0xffff0000u)));
        uint2 o;
        o.x = *reinterpret_cast<const uint32_t*>(&lo);
        o.y = *reinterpret_cast<const uint32_t*>(&hi);
        *reinterpret_cast<uint2*>(Y + (size_t)blockIdx.x * D + 4 * i) = o;
    }
}

// The DeltaNet front end of a chunk: causal 4-tap convolution over time, SiLU, per-head L2 norm of q and k, q / sqrt(128).
// One block per (token, head of q, k or v): grid (T, 2*HK + HV), thread = channel.  The three earlier tokens of a channel are
// rows of the same projection buffer, or, before the chunk's first token, slots of the ring history (slot = position & 3),
// which this kernel only reads: pf_ab_gate records the chunk's last positions afterwards.
// proj [T, ld]: q | k | v | z columns of the fused projection.  Writes q, k [T, HK, 128], v [T, HV, 128] (fp32).
//                                                                        (inference/recur.ls:12-40, reduce.ls:153-207)
extern "C" __global__ void __launch_bounds__(128) pf_dn_frontend(const float* __restrict__ proj, int ld, const uint16_t* __restrict__ conv_w,
                                                                 const float* __restrict__ ring, float* __restrict__ q, float* __restrict__ k,
                                                                 float* __restrict__ v, int HK, int HV, int pos0, int T) {
    pdl_wait(); // launched with programmatic stream serialization: nothing of the previous kernel is read before this
    __shared__ float red[4];
    const int QK = HK * 128, C = 2 * QK + HV * 128;
    const int s = blockIdx.x, b = blockIdx.y, t = threadIdx.x;
    const int kind = b < HK ? 0 : b < 2 * HK ? 1 : 2, head = kind == 0 ? b : kind == 1 ? b - HK : b - 2 * HK;
    const int c = (kind == 0 ? 0 : kind == 1 ? QK : 2 * QK) + head * 128 + t;
    auto past = [&](int back) { // the channel's raw value `back` tokens ago
        return s >= back ? proj[(size_t)(s - back) * ld + c] : ring[(size_t)((pos0 + s - back) & 3) * C + c];
    };
    float y = bf16_bits_to_f32(conv_w[c]) * proj[(size_t)s * ld + c];
    y = fmaf(bf16_bits_to_f32(conv_w[C + c]), past(1), y);
    y = fmaf(bf16_bits_to_f32(conv_w[2 * C + c]), past(2), y);
    y = fmaf(bf16_bits_to_f32(conv_w[3 * C + c]), past(3), y);
    y = siluf_dev(y);
    if (kind == 2) { v[((size_t)s * HV + head) * 128 + t] = y; return; }
    float n2 = warp_sum(y * y);
    if ((t & 31) == 0) red[t >> 5] = n2;
    __syncthreads();
    n2 = (red[0] + red[1]) + (red[2] + red[3]);
    if (kind == 0) q[((size_t)s * HK + head) * 128 + t] = y * rsqrtf(n2) * 0.08838834764831845f;
    else k[((size_t)s * HK + head) * 128 + t] = y * rsqrtf(n2);
}

// decay and beta of a chunk: a = in_proj_a . xn, b = in_proj_b . xn per value head, then
// g = exp(-exp(A_log) softplus(a + dt_bias)), beta = sigmoid(b).  A block is 16 tokens x 8 NT of the 2 HV rows (a's, then b's), its eight warps take the hidden
// dimension in turn, 32 at a time, U (even) of those in flight.  The products are mma.sync m16n8k8 tf32, in which fp16 activations and
// bf16 weights are exact (sums fp32): a lane's 16-byte pieces of a token and of a row are its operands of four k-steps, the order of k being free.  The tensor core
// truncates its sums, so chains of two products start from zero and are added pairwise: as far from 64 bits as the fp32 multiply-adds before (48 heads, 5120: g 2.1e-7
// against 2.2e-7 rms, beta 1.2e-7 against 1.3e-7; one chain over all k was ten times as far off).
// Bound by the loads' way in.  Before, one head x 8 tokens per block read the tokens 48 times.  NT = 3 reads them less often, NT = 1 makes three times the blocks and
// keeps the SMs busy with a few tokens (the launch decides).  48 heads, hidden 5120, us, before -> after: 16 tokens 8.3 -> 8.3, 75 9.5 -> 8.3, 128 12.3 -> 8.3,
// 256 17.0 -> 10.3; with the ring's launch gone, whole prompts: 4096 tokens 33 090 -> 32 350, 800 behind 500 7400 -> 7240, 75 behind 2000 1517 -> 1492.
// Besides, the ring slots of the chunk's last (up to four) tokens, ring[(pos0 + s) & 3][c] = proj[s][c]: the history the next chunk, or the decode step, continues
// from (pf_dn_frontend, the launch before, has read what was there).
// grid (ceil(T / 16), ceil(2 HV / (8 NT))), block 256; H a multiple of 8
__device__ __forceinline__ uint4 pf_ld16(const uint4* a) { // volatile: all loads of a stretch are issued before the first is used
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(a) : "memory");
    return v;
}
template <int NT, int U>
__device__ __forceinline__ void pf_ab_gate_body(const __half* __restrict__ xn, const uint16_t* __restrict__ proj_a, const uint16_t* __restrict__ proj_b, const float* __restrict__ a_log,
                                                const uint16_t* __restrict__ dt_bias, float* __restrict__ g, float* __restrict__ beta, int HV, int H, int T,
                                                const float* __restrict__ proj, int ld, float* __restrict__ ring, int C, int pos0) {
    pdl_wait(); // launched with programmatic stream serialization: nothing of the previous kernel is read before this
    __shared__ float red[8][16][8 * NT + 1];
    const int s0 = blockIdx.x * 16, r0 = blockIdx.y * (8 * NT), t = threadIdx.x, warp = t >> 5, lane = t & 31, fg = lane >> 2, ft = lane & 3;
    const uint4* x[2];
    const uint4* w[NT];
#pragma unroll
    for (int i = 0; i < 2; ++i) x[i] = reinterpret_cast<const uint4*>(xn + (size_t)min(s0 + fg + 8 * i, T - 1) * H) + ft; // tokens past the chunk repeat the last one
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        const int r = min(r0 + 8 * i + fg, 2 * HV - 1);
        w[i] = reinterpret_cast<const uint4*>(r < HV ? proj_a + (size_t)r * H : proj_b + (size_t)(r - HV) * H) + ft;
    }
    float acc[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    const int pieces = H / 8;
    for (int j0 = 4 * warp; j0 < pieces; j0 += 32 * U) {
        uint4 xv[U][2], wv[U][NT];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = j0 + 32 * u;
            const bool in = j + ft < pieces;
#pragma unroll
            for (int i = 0; i < 2; ++i) xv[u][i] = pf_ld16(x[i] + (in ? j : -ft));
#pragma unroll
            for (int i = 0; i < NT; ++i) wv[u][i] = pf_ld16(w[i] + (in ? j : -ft));
        }
#pragma unroll
        for (int u = 0; u < U; ++u) // past the end: zeros
            if (j0 + 32 * u + ft >= pieces) {
                xv[u][0] = xv[u][1] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int i = 0; i < NT; ++i) wv[u][i] = make_uint4(0u, 0u, 0u, 0u);
            }
        float sum[NT][4], pair[NT][4], part[NT][4], stretch[NT][4]; // chains of two products, added pairwise
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int s = 0; s < 4; ++s) { // a k-step: two of the lane's eight k
                float2 a[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t h = s == 0 ? xv[u][i].x : s == 1 ? xv[u][i].y : s == 2 ? xv[u][i].z : xv[u][i].w;
                    a[i] = __half22float2(*reinterpret_cast<const __half2*>(&h));
                }
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    const uint32_t b = s == 0 ? wv[u][i].x : s == 1 ? wv[u][i].y : s == 2 ? wv[u][i].z : wv[u][i].w;
                    if (s % 2 == 0) part[i][0] = part[i][1] = part[i][2] = part[i][3] = 0.f;
                    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                        : "+f"(part[i][0]), "+f"(part[i][1]), "+f"(part[i][2]), "+f"(part[i][3])
                        : "r"(__float_as_uint(a[0].x)), "r"(__float_as_uint(a[1].x)), "r"(__float_as_uint(a[0].y)), "r"(__float_as_uint(a[1].y)), "r"(b << 16), "r"(b & 0xffff0000u));
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if (s == 1) pair[i][e] = part[i][e];
                        if (s != 3) continue;
                        const float v = pair[i][e] + part[i][e];
                        if (u % 2 == 0) stretch[i][e] = v;
                        else sum[i][e] = u == 1 ? stretch[i][e] + v : sum[i][e] + (stretch[i][e] + v);
                        if (u == U - 1) acc[i][e] += sum[i][e];
                    }
                }
            }
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        red[warp][fg][8 * i + 2 * ft] = acc[i][0];
        red[warp][fg][8 * i + 2 * ft + 1] = acc[i][1];
        red[warp][fg + 8][8 * i + 2 * ft] = acc[i][2];
        red[warp][fg + 8][8 * i + 2 * ft + 1] = acc[i][3];
    }
    __syncthreads();
    for (int e = t; e < 16 * 8 * NT; e += 256) {
        const int s = e / (8 * NT), c = e - 8 * NT * s, r = r0 + c;
        if (s0 + s >= T || r >= 2 * HV) continue;
        const float v = ((red[0][s][c] + red[1][s][c]) + (red[2][s][c] + red[3][s][c])) + ((red[4][s][c] + red[5][s][c]) + (red[6][s][c] + red[7][s][c]));
        if (r < HV) {
            const float tt = v + bf16_bits_to_f32(dt_bias[r]);
            const float sp = tt > 20.f ? tt : log1pf(expf(tt));
            g[(size_t)(s0 + s) * HV + r] = expf(-expf(a_log[r]) * sp);
        } else beta[(size_t)(s0 + s) * HV + r - HV] = 1.0f / (1.0f + expf(-v));
    }
    const int last = T > 4 ? T - 4 : 0, blocks = gridDim.x * gridDim.y;
    for (int i = (blockIdx.y * gridDim.x + blockIdx.x) * 256 + t; i < (T - last) * C; i += blocks * 256) {
        const int s = last + i / C, c = i % C;
        ring[(size_t)((pos0 + s) & 3) * C + c] = proj[(size_t)s * ld + c];
    }
}
#define PF_AB_GATE(name, NT, U)                                                                                                                                            \
    extern "C" __global__ void __launch_bounds__(256) name(const __half* xn, const uint16_t* proj_a, const uint16_t* proj_b, const float* a_log, const uint16_t* dt_bias,     \
                                                           float* g, float* beta, int HV, int H, int T, const float* proj, int ld, float* ring, int C, int pos0) {          \
        pf_ab_gate_body<NT, U>(xn, proj_a, proj_b, a_log, dt_bias, g, beta, HV, H, T, proj, ld, ring, C, pos0);                                                           \
    }
PF_AB_GATE(pf_ab_gate, 3, 4)
PF_AB_GATE(pf_ab_gate_few, 1, 10)

// y16[t, h, :] = fp16( o * rsqrt(mean_head o^2 + eps) * w * silu(z) ): the out projection's input.  One warp per (token, head).
// o [T, HV, 128]; z = proj + z_off with row stride ld.            grid (T, ceil(HV/4)), block 128
extern "C" __global__ void __launch_bounds__(128) pf_headnorm_gate_f16(const float* __restrict__ o, const float* __restrict__ proj, int ld,
                                                                       int z_off, const float* __restrict__ w, __half* __restrict__ y,
                                                                       int HV, float eps) {
    pdl_wait(); // launched with programmatic stream serialization: nothing of the previous kernel is read before this
    const int s = blockIdx.x, h = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (h >= HV) return;
    const float4 v = *reinterpret_cast<const float4*>(o + ((size_t)s * HV + h) * 128 + lane * 4);
    const float4 z = *reinterpret_cast<const float4*>(proj + (size_t)s * ld + z_off + h * 128 + lane * 4);
    const float4 ww = *reinterpret_cast<const float4*>(w + lane * 4);
    const float r = rsqrtf(warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w) * (1.0f / 128.0f) + eps);
    __half* dst = y + ((size_t)s * HV + h) * 128 + lane * 4;
    dst[0] = __float2half_rn(v.x * r * ww.x * siluf_dev(z.x));
    dst[1] = __float2half_rn(v.y * r * ww.y * siluf_dev(z.y));
    dst[2] = __float2half_rn(v.z * r * ww.z * siluf_dev(z.z));
    dst[3] = __float2half_rn(v.w * r * ww.w * siluf_dev(z.w));
}

// SwiGLU of a chunk: gu [T, 2I] in interleaved 64-wide (gate, up) blocks -> y16 [T, I] = silu(gate) * up    (kernels.ls:61-66)
// four outputs per thread; total4 = T * I / 4 (fits 32 bits: a chunk has at most 256 tokens)
extern "C" __global__ void pf_swiglu_f16(const float* __restrict__ gu, __half* __restrict__ y, int I, int total4) {
    pdl_wait(); // launched with programmatic stream serialization: nothing of the previous kernel is read before this
    const int I4 = I / 4;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total4; i += gridDim.x * blockDim.x) {
        const int s = i / I4, n = (i - s * I4) * 4, blk = n >> 6, j = n & 63;
        const float* row = gu + (size_t)s * 2 * I + (size_t)blk * 128;
        const float4 gt = *reinterpret_cast<const float4*>(row + j), up = *reinterpret_cast<const float4*>(row + 64 + j);
        const __half2 lo = __floats2half2_rn(siluf_dev(gt.x) * up.x, siluf_dev(gt.y) * up.y);
        const __half2 hi = __floats2half2_rn(siluf_dev(gt.z) * up.z, siluf_dev(gt.w) * up.w);
        uint2 o;
        o.x = *reinterpret_cast<const uint32_t*>(&lo);
        o.y = *reinterpret_cast<const uint32_t*>(&hi);
        *reinterpret_cast<uint2*>(y + (size_t)i * 4) = o;
    }
}

// x += y, four values per thread (n4 = n / 4)
extern "C" __global__ void pf_add(float4* __restrict__ x, const float4* __restrict__ y, int n4) {
    pdl_wait(); // launched with programmatic stream serialization: nothing of the previous kernel is read before this
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += gridDim.x * blockDim.x) {
        float4 a = x[i];
        const float4 b = y[i];
        a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
        x[i] = a;
    }
}

// ---- causal attention of a chunk ---------------------------------------------------------------------------------
// The decode step runs q/k norm, RoPE, the KV append and the attention of ONE token in one kernel (attention_mma.cu;
// inference/attend.ls:85-191, attend_full.ls:186-248).  For a chunk of T prompt tokens the same work is two kernels:
// pf_attn_prepare does the per-token part with the decode kernel's own routine (same bits in the cache rows and the
// same queries), pf_attn_chunk then attends all T tokens at once, token s over the cache rows [0, pos0 + s].
#include "attention_core.cuh"

// grid T, block 256: token s of the chunk.  Queries -> (qh, ql) as two bf16 terms, pre-scaled by log2(e)/sqrt(256);
// key -> norm, RoPE, bf16 -> cache row pos0+s; value -> bf16 -> cache row pos0+s.
extern "C" __global__ void __launch_bounds__(256) pf_attn_prepare(const __grid_constant__ lb_pf_attn_params p) {
    pdl_wait();
    __shared__ float cs_s[128], sn_s[128];
    __shared__ __align__(16) float row_s[8][AT_D];
    const int s = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int pos = p.pos0 + s;
    if (t < p.rot_dims / 2) { // the decode kernel's angle reduction: product and reduction modulo 2 pi in double
        const double a = (double)pos * p.rope_freq[t];
        const double k = rint(a * 0.15915494309189535);
        const float r = (float)fma(-k, 6.283185307179586, a);
        sincosf(r, &sn_s[t], &cs_s[t]);
    }
    __syncthreads();
    const float qscale = rsqrtf((float)AT_D) * 1.4426950408889634f; // scores in log2 units
    const float* row = p.proj + (size_t)s * p.ld;
    const size_t nq = (size_t)2 * p.HQ * AT_D, nkv = (size_t)p.HKV * AT_D;
    for (int r = warp; r < p.HQ + p.HKV; r += 8) {
        float* dst = row_s[warp];
        if (r < p.HQ) {
            warp_norm_rope(row, (size_t)r * 512, 1, p.q_norm_w, dst, cs_s, sn_s, p.rot_dims, p.eps, qscale);
            __syncwarp();
            const size_t o = ((size_t)s * p.HQ + r) * AT_D + lane * 8;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float q = dst[lane * 8 + j];
                const __nv_bfloat16 h = __float2bfloat16_rn(q);
                reinterpret_cast<__nv_bfloat16*>(p.qh)[o + j] = h;
                reinterpret_cast<__nv_bfloat16*>(p.ql)[o + j] = __float2bfloat16_rn(q - __bfloat162float(h));
            }
        } else {
            const int kv = r - p.HQ;
            warp_norm_rope(row + nq, (size_t)kv * AT_D, 1, p.k_norm_w, dst, cs_s, sn_s, p.rot_dims, p.eps, 1.0f);
            __syncwarp();
            const size_t o = ((size_t)pos * p.HKV + kv) * AT_D + lane * 8;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                reinterpret_cast<__nv_bfloat16*>(p.k_cache)[o + j] = __float2bfloat16_rn(dst[lane * 8 + j]);
                reinterpret_cast<__nv_bfloat16*>(p.v_cache)[o + j] = __float2bfloat16_rn(row[nq + nkv + (size_t)kv * AT_D + lane * 8 + j]);
            }
        }
        __syncwarp();
    }
}

// grid (ceil(T*G / 128), HKV), block LB_AC_THREADS: all tokens of the chunk, token s over the cache rows [0, pos0 + s].  Query row R of a KV head = (token
// R / G, head R % G), so a cache row is read once per 128 rows instead of once per token; the tiles that see most keys start first.
#include "attention_tc.cuh"
struct pf_chunk_rows {
    const lb_pf_attn_params& p;
    int kv, G;
    const uint16_t *qh, *ql;
    __device__ __forceinline__ size_t q_at(int R) const { return ((size_t)(R / G) * p.HQ + kv * G + R % G) * AT_D; }
    __device__ __forceinline__ int lim(int R) const { return p.pos0 + R / G; }
    __device__ __forceinline__ int low(int) const { return 0; }
    __device__ __forceinline__ float m0(int) const { return -INFINITY; }
    __device__ __forceinline__ float l0() const { return 0.f; }
    __device__ __forceinline__ void table(unsigned char*, int) const {}
    // out[s][hq][d..d+15] = fp16( O / l * sigmoid(gate) )
    __device__ __forceinline__ void store(unsigned char*, int, int R, int d, const uint32_t (&r)[16], float inv) const {
        const int s = R / G, hq = kv * G + R % G;
        const float* gate = p.proj + (size_t)s * p.ld + (size_t)hq * 512 + 256 + d;
        uint32_t o[8];
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
            const float4 g = *reinterpret_cast<const float4*>(gate + j);
            const __half2 a = __floats2half2_rn(__uint_as_float(r[j]) * inv * sigmoidf_dev(g.x), __uint_as_float(r[j + 1]) * inv * sigmoidf_dev(g.y));
            const __half2 b = __floats2half2_rn(__uint_as_float(r[j + 2]) * inv * sigmoidf_dev(g.z), __uint_as_float(r[j + 3]) * inv * sigmoidf_dev(g.w));
            o[j / 2] = *reinterpret_cast<const uint32_t*>(&a);
            o[j / 2 + 1] = *reinterpret_cast<const uint32_t*>(&b);
        }
        uint4* dst = reinterpret_cast<uint4*>(p.out + ((size_t)s * p.HQ + hq) * AT_D + d);
        dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
        dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
};
extern "C" __global__ void __launch_bounds__(LB_AC_THREADS, 1) pf_attn_chunk(const __grid_constant__ lb_pf_attn_params p, const __grid_constant__ lb_ac_maps maps, const lb_ac_split sp) {
    extern __shared__ __align__(1024) unsigned char pa_sm[];
    __shared__ ac_shared sh;
    const int G = p.HQ / p.HKV, n_rows = p.T * G, R0 = (int)(gridDim.x - 1 - blockIdx.x) * AC_ROWS;
    const pf_chunk_rows c = {p, (int)blockIdx.y, G, p.qh, p.ql};
    attn_chunk_tc(c, maps, sh, pa_sm, (int)blockIdx.y, R0, n_rows, 0, p.pos0 + min(R0 + AC_ROWS - 1, n_rows - 1) / G, AT_D, AT_D, AT_D, LB_AC_UNITS(AT_D), p.status, sp);
}
extern "C" __global__ void __launch_bounds__(256) pf_attn_merge(const __grid_constant__ lb_pf_attn_params p, const __grid_constant__ lb_ac_maps, const lb_ac_split sp) {
    const pf_chunk_rows c = {p, (int)blockIdx.y, p.HQ / p.HKV, p.qh, p.ql};
    attn_chunk_merge(c, (int)blockIdx.y, p.T * c.G, AT_D, sp);
}
