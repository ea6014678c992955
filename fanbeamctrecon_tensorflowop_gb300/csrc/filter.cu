// Ramp filter of every detector row: q[i] = sum_j h[i - j] p[j], i, j in
// [0, C) -- the middle C samples of ippsConv_32f's full linear convolution of
// the row with the 2C-1 taps (FBP/transform.cu:166-174,
// FDK/GPURecon_GPU.cu:207-215), which ran serially on the host CPU in the
// reference.  Direct FP32 form, for the widths that the tensor-core filter
// cannot take: a block stages R rows and the taps in shared memory, and a thread
// forms four outputs of all R rows.  Four values of a row are one broadcast
// 16-byte load, the four taps that a step of four adds to the sliding window
// another: 16 R FMAs for R + 1 loads, so the FMA pipe is the bound.  For the
// Ram-Lak window the even taps (n != 0) are exactly zero: outputs of one parity
// are the centre tap plus a convolution of the row's other parity with the odd
// taps.  Each output sums its terms in the order of j in one FMA chain.
// 719 x 733 sinograms, us for 1 / 16 / 32 slices: Shepp-Logan 36 / 283 / 540,
// Ram-Lak 21 / 164 / 318 (92 / 597 / 1119 and 55 / 422 / 797 with one output per
// thread and a load per term); 23 TFLOP/s of FP32 for the 32.
#include <cstdint>

#include "common.cuh"

namespace ctk {
namespace {

constexpr int kThreads = 256;

// Shared memory of the direct form: the taps' window and R rows.  Dense: taps
// h[n], n = -4 Q .. 4 Q + 3 (Q quads of outputs, zero beyond +-(C-1)), rows of 4 Q
// floats.  Odd-only: two windows of odd taps (one per output parity) over the
// half length, rows as two halves (even and odd j).
__host__ __device__ inline int quads_of(int n) { return (n + 3) / 4; }
__host__ __device__ inline size_t direct_floats(int C, int R, bool odd) {
    const int Q = quads_of(odd ? (C + 1) / 2 : C);
    return odd ? 2 * (size_t)(8 * Q + 4) + (size_t)R * 8 * Q + 1
               : (size_t)(8 * Q + 4) + (size_t)R * 4 * Q;
}

// acc[r][o] += sum_j taps(4 g + o - j) row_r[j], j < 4 Q; tq: the window's quads,
// tq[Q + k] holding taps 4 k .. 4 k + 3.
template <int R>
__device__ __forceinline__ void conv_quad(float (&acc)[R][4], const float4 *tq, const float4 *rows,
                                          int rstride4, int g, int Q) {
    float4 hi = tq[Q + g];
    for (int b = 0; b < Q; ++b) {
        const float4 lo = tq[Q + g - b - 1];
        // w[3 + o - jj] = tap 4 (g - b) + o - jj
        const float w[7] = {lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float4 p = rows[r * rstride4 + b];
            const float pv[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
            for (int jj = 0; jj < 4; ++jj)
#pragma unroll
                for (int o = 0; o < 4; ++o) acc[r][o] = fmaf(w[3 + o - jj], pv[jj], acc[r][o]);
        }
        hi = lo;
    }
}

template <bool ODD_ONLY, int R>
__global__ void __launch_bounds__(kThreads)
    ramp_direct_kernel(const float *__restrict__ in, float *__restrict__ out,
                       const float *__restrict__ taps, int C, int rows) {
    extern __shared__ float4 sm4[];
    float *st = reinterpret_cast<float *>(sm4);
    const int half = ODD_ONLY ? (C + 1) / 2 : C, Q = quads_of(half), win = 8 * Q + 4;
    float *sp = st + (ODD_ONLY ? 2 : 1) * win;          // row r at r * rlen
    const int rlen = ODD_ONLY ? 8 * Q : 4 * Q;          // (even j, then odd j)
    const int r0 = blockIdx.x * R, nr = min(R, rows - r0);
    for (int k = threadIdx.x; k < win; k += blockDim.x) {
        const int m = k - 4 * Q;
        if (ODD_ONLY) {
            // output 2a + q, input 2b + 1 - q: tap 2 (a - b) + 2 q - 1
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int n = 2 * m + 2 * q - 1;
                st[q * win + k] = n > -C && n < C ? __ldg(taps + n + C - 1) : 0.0f;
            }
        } else {
            st[k] = m > -C && m < C ? __ldg(taps + m + C - 1) : 0.0f;
        }
    }
    for (int k = threadIdx.x; k < R * rlen; k += blockDim.x) {
        const int r = k / rlen, e = k - r * rlen;
        const int j = ODD_ONLY ? (e < 4 * Q ? 2 * e : 2 * (e - 4 * Q) + 1) : e;
        sp[k] = r < nr && j < C ? __ldg(in + (size_t)(r0 + r) * C + j) : 0.0f;
    }
    __syncthreads();
    const int units = ODD_ONLY ? 2 * Q : Q;
    const float h0 = __ldg(taps + C - 1);
    for (int u0 = 0; u0 < units; u0 += blockDim.x) {
        const int u = u0 + threadIdx.x;
        const int q = ODD_ONLY ? (u >= Q) : 0, g = u - q * Q;
        if (u >= units) continue;
        float acc[R][4];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int o = 0; o < 4; ++o)
                acc[r][o] = ODD_ONLY ? h0 * sp[r * rlen + q * 4 * Q + 4 * g + o] : 0.0f;
        conv_quad<R>(acc, reinterpret_cast<const float4 *>(st + q * win),
                     reinterpret_cast<const float4 *>(sp + (ODD_ONLY ? (1 - q) * 4 * Q : 0)),
                     rlen / 4, g, Q);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (r >= nr) break;
            float *o = out + (size_t)(r0 + r) * C;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = ODD_ONLY ? 2 * (4 * g + k) + q : 4 * g + k;
                if (i < C) o[i] = acc[r][k];
            }
        }
    }
}

// Pre-weights over [batch][V][rows][C]: wv[v][c] (short scan) and wr[r][c]
// (cosine), either may be NULL.  A warp takes one row at a time; VEC: rows as
// float4 (C a multiple of 4, 16-byte aligned).  HBM-bound: a clinical cone-beam
// volume's projections (224 MB in, 224 MB out) took 255 us with 64-bit divisions per
// element, 75 us now (6.0 TB/s).
template <bool VEC>
__global__ void __launch_bounds__(256)
    preweight_kernel(const float *__restrict__ in, float *__restrict__ out,
                     const float *__restrict__ wv, const float *__restrict__ wr, long long total,
                     int C, int rows, int V) {
    const int lane = threadIdx.x & 31;
    for (long long e = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); e < total;
         e += (long long)gridDim.x * 8) {
        const int r = (int)(e % rows), v = (int)(e / rows % V);
        const float *pv = wv ? wv + (size_t)v * C : nullptr, *pr = wr ? wr + (size_t)r * C : nullptr;
        const float *src = in + e * C;
        float *dst = out + e * C;
        if constexpr (VEC) {
#pragma unroll 4
            for (int i = lane; i < C / 4; i += 32) {
                const float4 x = __ldg(reinterpret_cast<const float4 *>(src) + i);
                float4 w = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
                if (pv) w = __ldg(reinterpret_cast<const float4 *>(pv) + i);
                if (pr) {
                    const float4 u = __ldg(reinterpret_cast<const float4 *>(pr) + i);
                    w.x *= u.x;
                    w.y *= u.y;
                    w.z *= u.z;
                    w.w *= u.w;
                }
                reinterpret_cast<float4 *>(dst)[i] =
                    make_float4(x.x * w.x, x.y * w.y, x.z * w.z, x.w * w.w);
            }
        } else {
            for (int i = lane; i < C; i += 32) {
                float w = 1.0f;
                if (pv) w = __ldg(pv + i);
                if (pr) w *= __ldg(pr + i);
                dst[i] = src[i] * w;
            }
        }
    }
}

}  // namespace

int apply_preweight(const ct_plan *p, const float *in, float *out, int batch, void *stream) {
    const long long total = (long long)batch * p->g.n_views * p->n_rows;
    const long long blocks = (total + 7) / 8;
    const int C = p->g.n_cols;
    auto go = [&](auto kern) {
        kern<<<(int)(blocks < p->sms * 8 ? blocks : p->sms * 8), 256, 0, (cudaStream_t)stream>>>(
            in, out, p->d_parker, p->d_cosw, total, C, p->n_rows, p->g.n_views);
    };
    // the weight tables start on 256-byte boundaries; the caller's buffers may not
    const bool vec = C % 4 == 0 && (reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) % 16 == 0;
    vec ? go(preweight_kernel<true>) : go(preweight_kernel<false>);
    ct_count_launch();
    return (int)cudaGetLastError();
}

namespace {

template <bool ODD, int R>
int launch_direct(const ct_plan *p, const float *in, float *out, int rows, cudaStream_t stream) {
    const int C = p->g.n_cols;
    const size_t smem = sizeof(float) * direct_floats(C, R, ODD);
    cudaError_t e = cudaFuncSetAttribute(ramp_direct_kernel<ODD, R>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const int units = ODD ? 2 * quads_of((C + 1) / 2) : quads_of(C);
    const int threads = units < kThreads ? (units + 31) / 32 * 32 : kThreads;
    ramp_direct_kernel<ODD, R><<<(rows + R - 1) / R, threads, smem, stream>>>(in, out, p->d_taps, C,
                                                                              rows);
    ct_count_launch();
    return (int)cudaGetLastError();
}

}  // namespace

// The width limit of the direct form, as the shared memory of eight rows and the
// taps: up to 5,810 channels (fewer rows per block fit wherever this does).
size_t ramp_direct_smem(int C) { return sizeof(float) * ((2 * C - 1 + 3) / 4 * 4 + 8 * C); }

int ramp_filter(const ct_plan *p, const float *in, float *out, int rows, void *stream) {
    if (p->filter_algo == CT_FILTER_TOEPLITZ_TC) return ramp_filter_tc(p, in, out, rows, stream);
    if (rows == 0) return 0;
    const bool odd = p->opts.filter_window == CT_WINDOW_RAMLAK;
    const cudaStream_t s = (cudaStream_t)stream;
    // rows per block: eight while that leaves several blocks per SM and they fit
    auto fits = [&](int R) {
        return sizeof(float) * direct_floats(p->g.n_cols, R, odd) <= 227 * 1024;
    };
    if (rows >= 8 * p->sms * 2 && fits(8))
        return odd ? launch_direct<true, 8>(p, in, out, rows, s)
                   : launch_direct<false, 8>(p, in, out, rows, s);
    if (rows >= 4 * p->sms && fits(4))
        return odd ? launch_direct<true, 4>(p, in, out, rows, s)
                   : launch_direct<false, 4>(p, in, out, rows, s);
    if (rows >= 2 * p->sms && fits(2))
        return odd ? launch_direct<true, 2>(p, in, out, rows, s)
                   : launch_direct<false, 2>(p, in, out, rows, s);
    return odd ? launch_direct<true, 1>(p, in, out, rows, s)
               : launch_direct<false, 1>(p, in, out, rows, s);
}

}  // namespace ctk
