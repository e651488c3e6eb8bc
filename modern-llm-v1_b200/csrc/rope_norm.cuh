// Fused RoPE + per-head RMSNorm (QK-Norm) on the way into the attention kernels, and its backward.
//
// The reference prepares q and k for attention with five passes over each tensor
// (llm/src/model/modern_gpt.cu:351-370): split_heads ([B,T,H*d] -> [B*H,T,d], llm/src/model/attention.cu:344-364),
// rope_apply_inplace (llm/src/model/rope.cu:25-44,146-163) and rmsnorm_forward over rows of length d
// (llm/src/model/rmsnorm.cu:24-53), FP32 throughout; the backward mirrors it (modern_gpt.cu:527-552:
// rmsnorm_backward, llm/src/model/rmsnorm.cu:55-101, rope_apply_backward_inplace, llm/src/model/rope.cu:46-65,
// merge_heads).  Here one kernel reads a row of the projection output where it lies (either layout, FP32 or
// BF16), rotates it, normalises it, scales it by gamma and writes it as BF16 in the layout the attention
// kernels take; the backward does the inverse chain in one pass and reduces d_gamma without atomics.
//
//   r[2i]   = x[2i] cos(t, i) - x[2i+1] sin(t, i)          r[2i+1] = x[2i] sin(t, i) + x[2i+1] cos(t, i)
//   rstd    = rsqrt(mean_d r[d]^2 + eps)                    y[d]    = r[d] rstd gamma[d]
//   g[d]    = dy[d] gamma[d]       s = sum_d g[d] r[d]      dr[d]   = rstd g[d] - rstd^3 / D s r[d]
//   dx[2i]  = dr[2i] cos + dr[2i+1] sin                     dx[2i+1] = -dr[2i] sin + dr[2i+1] cos
//   d_gamma[d] += sum over rows of dy[d] r[d] rstd
//
// The work is bound by HBM bandwidth (one read and one write of the tensors).  A lane owns 8 consecutive elements of a row
// (16-byte accesses), so a row takes D / 8 lanes and a warp works on 32 / (D / 8) consecutive tokens at a time.  A warp's
// item is such a group of tokens and a chunk of heads: the cosines and sines of its tokens are loaded once and stay in
// registers for all heads of the chunk, and so do the token's addresses.  (Loaded per row they were as many bytes through
// L2 as x and y together, and the row's decoding as many instructions as its arithmetic.)  kUnroll rows are loaded
// before the first is used; together with 24 warps per SM that is enough in flight.
// Measured on B200 against rows walked one by one with staged loads, q and k together: FP32 B=16 T=1024 16/4 D=128
// 69.6 -> 42.4 us forward (5.97 TB/s), 92.7 -> 72.6 us backward (5.80 TB/s); BF16 B=4 T=8192 16/4 D=128 82.8 -> 65.0 and
// 107.8 -> 97.3; BF16 B=32 T=512 6/2 D=64 11.0 -> 9.6 and 16.7 -> 16.5, of which some 4 us each are launch and latency.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "ptx.cuh"

namespace b200attn {

struct RopeNormParams {
    const void* x;       // input rows (forward) / the forward's input again (backward)
    void* y;             // forward: BF16 output;  backward: d_x output (same type and layout as x)
    const uint16_t* dy;  // backward: BF16 gradient of y, in y's layout
    float* rstd;         // [B, H, T]: written by the forward, read by the backward
    const float* gamma;  // [D]
    const float* cos_t;  // [T, D/2]
    const float* sin_t;  // [T, D/2]
    float* partial;      // backward: [gridDim.x, D] partial d_gamma sums
    float* d_gamma;      // backward: [D], accumulated into by rope_norm_dgamma_kernel
    int B, T, H;
    unsigned n_tokens;   // B * T
    unsigned n_items;    // groups of tokens x chunks of heads
    int chunk;           // heads per item
    FastDiv div_t, div_chunks;  // division by T and by the number of chunks
    long long x_st, x_sh, x_sb;  // element strides of x (and of d_x): token, head, batch
    long long y_st, y_sh, y_sb;  // element strides of y (and of dy)
    float eps;
};

constexpr int kRopeNormThreads = 256;  // 8 warps
constexpr int kRopeNormFwdBlocks = 3, kRopeNormBwdBlocks = 3;  // CTAs per SM that the register budgets are made for

__device__ __forceinline__ float rn_bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float rn_bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ uint32_t rn_pack_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// sum over the LPR lanes that share a row (LPR a power of two, lanes of a row are adjacent)
template <int LPR>
__device__ __forceinline__ float rn_row_sum(float v) {
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// 8 consecutive elements starting at element offset `off`
template <bool F32>
__device__ __forceinline__ void rn_load8(const void* base, long long off, float (&v)[8]) {
    if (F32) {
        const float4* ptr = reinterpret_cast<const float4*>(static_cast<const float*>(base) + off);
        const float4 a = ptr[0], c = ptr[1];
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = c.x, v[5] = c.y, v[6] = c.z, v[7] = c.w;
    } else {
        const uint4 a = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(base) + off);
        v[0] = rn_bf16_lo(a.x), v[1] = rn_bf16_hi(a.x), v[2] = rn_bf16_lo(a.y), v[3] = rn_bf16_hi(a.y);
        v[4] = rn_bf16_lo(a.z), v[5] = rn_bf16_hi(a.z), v[6] = rn_bf16_lo(a.w), v[7] = rn_bf16_hi(a.w);
    }
}
template <bool F32>
__device__ __forceinline__ void rn_store8(void* base, long long off, const float (&v)[8]) {
    if (F32) {
        float4* ptr = reinterpret_cast<float4*>(static_cast<float*>(base) + off);
        ptr[0] = make_float4(v[0], v[1], v[2], v[3]);
        ptr[1] = make_float4(v[4], v[5], v[6], v[7]);
    } else {
        *reinterpret_cast<uint4*>(static_cast<uint16_t*>(base) + off) =
            make_uint4(rn_pack_bf16x2(v[0], v[1]), rn_pack_bf16x2(v[2], v[3]), rn_pack_bf16x2(v[4], v[5]),
                       rn_pack_bf16x2(v[6], v[7]));
    }
}

// The forward arithmetic of one row, shared by every kernel that prepares q or k (so that a row gives the same
// bits whichever kernel computes it).  rn_rotate8: RoPE on a lane's 8 elements (4 pairs; cs, sn = the 4 cosines
// and sines of the lane's pairs at the row's position) and the lane's share of the row's sum of squares.
__device__ __forceinline__ float rn_rotate8(const float (&v)[8], const float4& cs, const float4& sn, float (&rot)[8]) {
    const float c[4] = {cs.x, cs.y, cs.z, cs.w}, s[4] = {sn.x, sn.y, sn.z, sn.w};
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float x0 = v[2 * i], x1 = v[2 * i + 1];
        rot[2 * i] = x0 * c[i] - x1 * s[i];
        rot[2 * i + 1] = x0 * s[i] + x1 * c[i];
        ss += rot[2 * i] * rot[2 * i] + rot[2 * i + 1] * rot[2 * i + 1];
    }
    return ss;
}
template <int D>
__device__ __forceinline__ float rn_rstd(float row_sum_sq, float eps) {
    return rsqrtf(row_sum_sq / float(D) + eps);
}
__device__ __forceinline__ void rn_scale8(const float (&rot)[8], float rstd, const float (&gm)[8], float (&out)[8]) {
#pragma unroll
    for (int e = 0; e < 8; ++e) out[e] = rot[e] * rstd * gm[e];
}

// 8 elements as they lie in memory, and as numbers
template <bool F32>
struct RnRaw {
    uint4 w[F32 ? 2 : 1];
    __device__ __forceinline__ void load(const void* base, long long off) {
        const uint4* ptr = F32 ? reinterpret_cast<const uint4*>(static_cast<const float*>(base) + off)
                               : reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(base) + off);
        w[0] = __ldcs(ptr);
        if (F32) w[F32 ? 1 : 0] = __ldcs(ptr + 1);
    }
    __device__ __forceinline__ void clear() { w[0] = w[F32 ? 1 : 0] = make_uint4(0u, 0u, 0u, 0u); }
    __device__ __forceinline__ void get(float (&v)[8]) const {
        if (F32) {
            const uint4 a = w[0], c = w[F32 ? 1 : 0];
            v[0] = __uint_as_float(a.x), v[1] = __uint_as_float(a.y), v[2] = __uint_as_float(a.z), v[3] = __uint_as_float(a.w);
            v[4] = __uint_as_float(c.x), v[5] = __uint_as_float(c.y), v[6] = __uint_as_float(c.z), v[7] = __uint_as_float(c.w);
        } else {
            const uint4 a = w[0];
            v[0] = rn_bf16_lo(a.x), v[1] = rn_bf16_hi(a.x), v[2] = rn_bf16_lo(a.y), v[3] = rn_bf16_hi(a.y);
            v[4] = rn_bf16_lo(a.z), v[5] = rn_bf16_hi(a.z), v[6] = rn_bf16_lo(a.w), v[7] = rn_bf16_hi(a.w);
        }
    }
};

// A warp's item: D / 8 lanes per token; lane's token, and the heads [h0, h1) that are the item's
template <int D>
struct RnItem {
    bool live;  // the lane has a token
    int b, t, h0, h1;
    __device__ __forceinline__ RnItem(const RopeNormParams& p, unsigned item, int sub) {
        const unsigned group = fastdiv(item, p.div_chunks);
        h0 = int(item - group * p.div_chunks.d) * p.chunk;
        h1 = min(h0 + p.chunk, p.H);
        unsigned token = group * (256u / D) + unsigned(sub);
        live = token < p.n_tokens;
        if (!live) token = 0;
        b = int(fastdiv(token, p.div_t));
        t = int(token - unsigned(b) * unsigned(p.T));
    }
};

// One tensor's forward: the items `item`, item + n_warps, ... of this warp; returns how far the last step went beyond the
// tensor's items, which is where the warp begins in the next tensor.  (A function of its own, called once per tensor with
// the kernel parameter itself, so that every field stays a constant-bank operand; selecting the struct at run time would
// move it to local memory.)
template <int D, bool F32>
__device__ __forceinline__ unsigned rope_norm_fwd_tensor(const RopeNormParams& p, unsigned item, unsigned n_warps) {
    constexpr int LPR = D / 8;  // lanes per row
    constexpr int kUnroll = 4;
    const int lane = threadIdx.x & 31;
    const int sub = lane / LPR, li = lane % LPR;  // token within the group, position within the row
    float gm[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) gm[e] = p.gamma[li * 8 + e];
    for (; item < p.n_items; item += n_warps) {
        const RnItem<D> it(p, item, sub);
        const float4 cs = *reinterpret_cast<const float4*>(p.cos_t + static_cast<long long>(it.t) * (D / 2) + li * 4);
        const float4 sn = *reinterpret_cast<const float4*>(p.sin_t + static_cast<long long>(it.t) * (D / 2) + li * 4);
        const long long x_off = it.b * p.x_sb + it.t * p.x_st + li * 8, y_off = it.b * p.y_sb + it.t * p.y_st + li * 8;
        float* rstd_t = p.rstd + static_cast<long long>(it.b) * p.H * p.T + it.t;
        for (int h = it.h0; h < it.h1; h += kUnroll) {
            RnRaw<F32> raw[kUnroll];
#pragma unroll
            for (int k = 0; k < kUnroll; ++k) {
                raw[k].clear();
                if (it.live && h + k < it.h1) raw[k].load(p.x, x_off + (h + k) * p.x_sh);
            }
#pragma unroll
            for (int k = 0; k < kUnroll; ++k) {
                if (h + k >= it.h1) break;
                float v[8], rot[8], out[8];
                raw[k].get(v);
                const float ss = rn_row_sum<LPR>(rn_rotate8(v, cs, sn, rot));  // every lane takes part in the shuffles
                const float rstd = rn_rstd<D>(ss, p.eps);
                rn_scale8(rot, rstd, gm, out);
                if (it.live) {
                    rn_store8<false>(p.y, y_off + (h + k) * p.y_sh, out);
                    if (li == 0) rstd_t[static_cast<long long>(h + k) * p.T] = rstd;
                }
            }
        }
    }
    return item - p.n_items;
}

// one launch takes q and k (n_tensors = 2), one after the other
template <int D, bool F32>
__global__ void __launch_bounds__(kRopeNormThreads, kRopeNormFwdBlocks)
rope_norm_fwd_kernel(const __grid_constant__ RopeNormParams p0, const __grid_constant__ RopeNormParams p1,
                     const int n_tensors) {
    const unsigned warp = (blockIdx.x * kRopeNormThreads + threadIdx.x) >> 5, n_warps = (gridDim.x * kRopeNormThreads) >> 5;
    grid_dep_wait();  // launched with programmatic stream serialization: the inputs come from the kernel before
    const unsigned next = rope_norm_fwd_tensor<D, F32>(p0, warp, n_warps);
    if (n_tensors > 1) rope_norm_fwd_tensor<D, F32>(p1, next, n_warps);
}

// One tensor's backward, in the same manner; leaves this CTA's d_gamma sums in p.partial.
template <int D, bool F32>
__device__ __forceinline__ unsigned rope_norm_bwd_tensor(const RopeNormParams& p, unsigned item, unsigned n_warps, float (*s_part)[D]) {
    constexpr int LPR = D / 8;
    constexpr int kUnroll = 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = lane / LPR, li = lane % LPR;
    float gm[8], dg[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        gm[e] = p.gamma[li * 8 + e];
        dg[e] = 0.f;
    }
    for (; item < p.n_items; item += n_warps) {
        const RnItem<D> it(p, item, sub);
        const float4 cs = *reinterpret_cast<const float4*>(p.cos_t + static_cast<long long>(it.t) * (D / 2) + li * 4);
        const float4 sn = *reinterpret_cast<const float4*>(p.sin_t + static_cast<long long>(it.t) * (D / 2) + li * 4);
        const float c[4] = {cs.x, cs.y, cs.z, cs.w}, sv[4] = {sn.x, sn.y, sn.z, sn.w};
        const long long x_off = it.b * p.x_sb + it.t * p.x_st + li * 8, y_off = it.b * p.y_sb + it.t * p.y_st + li * 8;
        const float* rstd_t = p.rstd + static_cast<long long>(it.b) * p.H * p.T + it.t;
        for (int h = it.h0; h < it.h1; h += kUnroll) {
            RnRaw<F32> raw_x[kUnroll];
            RnRaw<false> raw_dy[kUnroll];
            float rstd[kUnroll];
#pragma unroll
            for (int k = 0; k < kUnroll; ++k) {
                raw_x[k].clear();
                raw_dy[k].clear();
                rstd[k] = 0.f;
                if (it.live && h + k < it.h1) {
                    raw_x[k].load(p.x, x_off + (h + k) * p.x_sh);
                    raw_dy[k].load(p.dy, y_off + (h + k) * p.y_sh);
                    rstd[k] = rstd_t[static_cast<long long>(h + k) * p.T];
                }
            }
#pragma unroll
            for (int k = 0; k < kUnroll; ++k) {
                if (h + k >= it.h1) break;
                float v[8], dyv[8], rot[8], g[8];
                raw_x[k].get(v);
                raw_dy[k].get(dyv);
                const float rs = rstd[k];
                float s = 0.f;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float x0 = v[2 * i], x1 = v[2 * i + 1];
                    rot[2 * i] = x0 * c[i] - x1 * sv[i];
                    rot[2 * i + 1] = x0 * sv[i] + x1 * c[i];
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    g[e] = dyv[e] * gm[e];
                    s += g[e] * rot[e];
                    dg[e] += dyv[e] * rot[e] * rs;
                }
                s = rn_row_sum<LPR>(s);
                const float coeff = rs * rs * rs * (1.f / float(D)) * s;
                float dx[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float d0 = rs * g[2 * i] - coeff * rot[2 * i];
                    const float d1 = rs * g[2 * i + 1] - coeff * rot[2 * i + 1];
                    dx[2 * i] = d0 * c[i] + d1 * sv[i];
                    dx[2 * i + 1] = -d0 * sv[i] + d1 * c[i];
                }
                if (it.live) rn_store8<F32>(p.y, x_off + (h + k) * p.x_sh, dx);
            }
        }
    }
    // d_gamma: a lane holds sums for its 8 columns over its rows.  Add the lanes that own the same columns
    // (they differ in `sub`), then the warps of the CTA, both in a fixed order.
#pragma unroll
    for (int e = 0; e < 8; ++e) {
#pragma unroll
        for (int o = LPR; o < 32; o <<= 1) dg[e] += __shfl_xor_sync(0xffffffffu, dg[e], o);
    }
    if (sub == 0) {
#pragma unroll
        for (int e = 0; e < 8; ++e) s_part[warp][li * 8 + e] = dg[e];
    }
    __syncthreads();
    for (int d = threadIdx.x; d < D; d += kRopeNormThreads) {
        float acc = 0.f;
#pragma unroll
        for (int w = 0; w < kRopeNormThreads / 32; ++w) acc += s_part[w][d];
        p.partial[static_cast<long long>(blockIdx.x) * D + d] = acc;
    }
    return item - p.n_items;
}

template <int D, bool F32>
__global__ void __launch_bounds__(kRopeNormThreads, kRopeNormBwdBlocks)
rope_norm_bwd_kernel(const __grid_constant__ RopeNormParams p0, const __grid_constant__ RopeNormParams p1,
                     const int n_tensors) {
    __shared__ float s_part[2][kRopeNormThreads / 32][D];
    const unsigned warp = (blockIdx.x * kRopeNormThreads + threadIdx.x) >> 5, n_warps = (gridDim.x * kRopeNormThreads) >> 5;
    grid_dep_wait();
    const unsigned next = rope_norm_bwd_tensor<D, F32>(p0, warp, n_warps, s_part[0]);
    if (n_tensors > 1) rope_norm_bwd_tensor<D, F32>(p1, next, n_warps, s_part[1]);
}

// d_gamma[d] += sum of the CTAs' partial sums, for one or two tensors.  A CTA takes 8 columns (one 32-byte sector of every
// part): thread (r, c) adds parts r, r + 32, ... of column c in order, then the 32 sums of a column are added in order, so
// the result is bit-reproducible.  The kernel is latency and nothing else: a thread's sixteen loads, enough for the 444 parts of
// three CTAs per SM, and the old d_gamma are all issued before the first is used (in a loop unrolled by eight the last six parts
// cost a round trip through L2 each): forward and backward FP32 B=16 T=1024 16/4 D=128 115.0 -> 113.4 us, BF16 B=32 T=512 6/2
// D=64 29.0 -> 27.9.  With 128 threads and four columns a CTA it was 1.8 us slower, with 512 the same, with 1024 slower where the
// backward kernel has filled the SMs.  (Done by the last CTA of the backward kernel instead, the same sums took 25 us: one CTA
// cannot keep enough loads in flight.  Bringing this kernel or the next in early made no difference.)
constexpr int kDgammaThreads = 256, kDgammaRows = kDgammaThreads / 8, kDgammaLoads = 16;
template <int D>
__global__ void __launch_bounds__(kDgammaThreads) rope_norm_dgamma_kernel(const float* __restrict__ partial0, float* __restrict__ d_gamma0,
                                                                          const float* __restrict__ partial1, float* __restrict__ d_gamma1,
                                                                          int n_parts) {
    __shared__ float s_sum[kDgammaRows][9];
    const int ts = blockIdx.x / (D / 8), c = threadIdx.x & 7, r = threadIdx.x >> 3, d = (blockIdx.x % (D / 8)) * 8 + c;
    const float* partial = ts ? partial1 : partial0;
    float* d_gamma = ts ? d_gamma1 : d_gamma0;
    float acc = 0.f;
    grid_dep_wait();  // the partial sums come from the kernel before this one
    const float old = r == 0 ? d_gamma[d] : 0.f;
    for (int i0 = r; i0 < n_parts; i0 += kDgammaLoads * kDgammaRows) {
        float v[kDgammaLoads];
#pragma unroll
        for (int k = 0; k < kDgammaLoads; ++k) {
            const int i = i0 + k * kDgammaRows;
            v[k] = i < n_parts ? partial[static_cast<long long>(i) * D + d] : 0.f;
        }
#pragma unroll
        for (int k = 0; k < kDgammaLoads; ++k) acc += v[k];
    }
    s_sum[r][c] = acc;
    __syncthreads();
    if (r == 0) {
        acc = 0.f;
#pragma unroll
        for (int i = 0; i < kDgammaRows; ++i) acc += s_sum[i][c];
        d_gamma[d] = old + acc;
    }
}

}  // namespace b200attn
