// The forward projector's per-warp work, shared by the per-plan kernel and the
// uneven-batch kernel, and the quad images of the cone projector.
#pragma once

#include <climits>

#include <cuda_bf16.h>

#include "cellwalk.cuh"

namespace ctk {

__device__ __forceinline__ void store_val(float *p, float v) { *p = v; }
__device__ __forceinline__ void store_val(__nv_bfloat16 *p, float v) { *p = __float2bfloat16(v); }
__device__ __forceinline__ float load_val(const float *p) { return __ldg(p); }
__device__ __forceinline__ float load_val(const __nv_bfloat16 *p) {
    return __bfloat162float(__ldg(p));
}

// Two FP32 lanes in one 64-bit register for the f32x2 FMA (each lane rounds
// as fmaf does).
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long r) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
    return v;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// x rounded down (up) to an integer by an FP32 add that rounds toward -inf
// (+inf), |x| < 2^22: no conversion instructions.  The sum's low bits hold
// the integer (kMagicInt + it).
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
constexpr int kMagicInt = 0x4B400000;
__device__ __forceinline__ float ceil_magic(float x) { return __fadd_ru(x, kMagic) - kMagic; }

// The texel images a warp reads: per layout (0: rows along x; 1: the
// transposed image) [nx+2][nx+2] texels, texel (x, y) of -1 .. nx at
// (y + 1)(nx + 2) + x + 1 with its value clamped to the image's edge (samples
// lie inside the FOV circle of radius nx/2 texels, so no cell beyond -1 ..
// nx-1 is visited).  A texel holds TS slices (4 TS bytes); slices 8k .. 8k+7
// of a wider group are planes of their own.
struct TexelImages {
    const char *base;  // layout 0 of the group's first plane
    size_t plane;      // bytes between planes
    size_t layout;     // bytes from layout 0 to layout 1
};

// One texel of a lane's ray, loaded when its weight is not zero and added
// later: the loads of a row go out before the next row's weights are formed
// (32 clinical slices: 4.4 -> 3.9 ms).  They are predicated in assembly: a
// branch per texel would return from each load before the next is issued.
// (Groups of eight slices as two 16-byte loads instead of one of 32 bytes:
// 5.5 ms.)
template <int TS, int NP>
struct Texel {
    static constexpr int R = TS == 8 ? 2 * NP : 1;  // float4 registers
    float4 v[R];
    __device__ __forceinline__ void load(const TexelImages &im, const char *p, bool ok, float w) {
        if (!CT_DCHECK(w == 0.0f || ok)) w = 0.0f;
        if constexpr (TS == 1) {
            asm volatile("{.reg .pred p; setp.neu.f32 p, %2, 0f00000000;"
                         " @p ld.global.nc.f32 %0, [%1];}"
                         : "=f"(v[0].x)
                         : "l"(p), "f"(w));
        } else if constexpr (TS == 2) {
            asm volatile("{.reg .pred p; setp.neu.f32 p, %3, 0f00000000;"
                         " @p ld.global.nc.v2.f32 {%0, %1}, [%2];}"
                         : "=f"(v[0].x), "=f"(v[0].y)
                         : "l"(p), "f"(w));
        } else if constexpr (TS == 4) {
            asm volatile("{.reg .pred p; setp.neu.f32 p, %5, 0f00000000;"
                         " @p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];}"
                         : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[0].z), "=f"(v[0].w)
                         : "l"(p), "f"(w));
        } else {
#pragma unroll
            for (int k = 0; k < NP; ++k)
                asm volatile("{.reg .pred p; setp.neu.f32 p, %9, 0f00000000;"
                             " @p ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];}"
                             : "=f"(v[2 * k].x), "=f"(v[2 * k].y), "=f"(v[2 * k].z),
                               "=f"(v[2 * k].w), "=f"(v[2 * k + 1].x), "=f"(v[2 * k + 1].y),
                               "=f"(v[2 * k + 1].z), "=f"(v[2 * k + 1].w)
                             : "l"(p + k * im.plane), "f"(w));
        }
    }
};

// A lane's sums.  The running sums are moved to totals every kFlushRows image
// rows: an FP32 sum of a whole ray's thousand terms rounds at its own size
// each time (clinical phantoms: 4.8e-7 relative L2 from FP64, 1.2e-7 with the
// totals, at 1% of the time; 64^2 phantoms 1.9e-7 and 1.2e-7).  Groups of two slices and
// more keep the totals in shared memory (`tot`, [SB/2][threads]).
constexpr int kFlushRows = 32;
template <int TS, int NP>
struct RayAcc {
    static constexpr int SB = TS * NP;  // slices of the walk
    static constexpr int N2 = SB / 2 ? SB / 2 : 1;
    static constexpr bool kShared = TS > 1;
    float one, one_total;  // SB == 1
    unsigned long long two[N2];
    unsigned long long *tot;  // this thread's totals in shared memory, or unused
    __device__ __forceinline__ void init(unsigned long long *shared) {
        tot = shared + threadIdx.x;
        one = one_total = 0.0f;
#pragma unroll
        for (int s = 0; s < N2; ++s) {
            two[s] = 0ull;
            if constexpr (kShared) tot[s * blockDim.x] = 0ull;
        }
    }
    __device__ __forceinline__ void flush() {
        one_total += one;
        one = 0.0f;
#pragma unroll
        for (int s = 0; s < N2; ++s) {
            if constexpr (kShared) tot[s * blockDim.x] = add2(tot[s * blockDim.x], two[s]);
            two[s] = 0ull;
        }
    }
    // += w * texel where w is not zero; the same fused multiply-add per slice
    // for every group size
    __device__ __forceinline__ void add(const Texel<TS, NP> &t, float w) {
        if (w == 0.0f) return;  // not loaded
        asm volatile("");  // keeps the adds conditional (not computed and selected)
        if constexpr (TS == 1) {
            one = fmaf(w, t.v[0].x, one);
        } else {
            const unsigned long long ww = pack2(w, w);
            two[0] = fma2(ww, pack2(t.v[0].x, t.v[0].y), two[0]);
            if constexpr (TS >= 4) {
#pragma unroll
                for (int k = 0; k < Texel<TS, NP>::R; ++k) {
                    if (k) two[2 * k] = fma2(ww, pack2(t.v[k].x, t.v[k].y), two[2 * k]);
                    two[2 * k + 1] = fma2(ww, pack2(t.v[k].z, t.v[k].w), two[2 * k + 1]);
                }
            }
        }
    }
    __device__ __forceinline__ float value(int s) const {
        if constexpr (SB == 1) return one_total;
        const float2 v = unpack2(tot[(s / 2) * blockDim.x]);
        return (s & 1) ? v.y : v.x;
    }
};

// One warp = 32 consecutive channels of one view (unit gw: view gw / wpv,
// channels 32 * (gw % wpv) + lane); warps never straddle views.  Each lane
// walks its ray along its major axis (v), through the texel image whose rows
// lie across it, and the warp's lanes step through those rows together, so
// that adjacent lanes (adjacent rays) read adjacent texels of one row.  Lanes
// of another layout or direction (a warp at a diagonal) walk in a second pass.
//
// Coordinates run along the ray: u and v are negated where the ray's step is
// negative, so both grow with the sample index.  The N samples of cell row j
// (v in [j, j+1)) span less than one texel of u (|du| <= |dv|), hence at most
// two cells; with x = u - q the position from the first cell's lower texel
// column q, the bilinear weights of columns q, q+1, q+2 are the hats 1-x+r,
// x-2r, r, r = max(x-1, 0), times 1-psi (texel row j) and psi (row j+1),
// psi = v - j.  The fractions phi and psi of the next row's first sample
// follow from this row's (their sums round at 1, not at nx).  The sums over the
// samples need sum x, sum psi and sum x psi over the row and over its second
// cell (the two lanes of f32x2 instructions).
// Row j+1's part is carried to the next step, where the next cell row adds
// its own: every texel the ray touches is then read once, with one weight,
// where a sum per cell reads four taps of each cell: 2.8 texels instead of
// 5.8 taps per image row on average.  A sample within rounding of a cell
// boundary may be counted to the neighbouring cell: the interpolant is
// continuous there.
//
// out: the [V][C] sinogram of slice 0, slices `ostride` apart; nsl valid
// slices; totals: RayAcc's shared memory (groups of two slices and more).
// The rows are walked in kFpParts shares, whose sums are added in order; a share
// begins with the carried weights of the row before it.  A block's kFpParts
// warps take one each (warp `part`; the sums meet in `totals`, [slices][threads],
// between a block-wide barrier and the stores of warp 0).
constexpr int kFpParts = 4;
template <int TS, int NP, typename OutT>
__device__ __forceinline__ void fp_warp(const TexelImages &im, OutT *__restrict__ out,
                                        size_t ostride, const float4 *__restrict__ ray,
                                        const int *__restrict__ nsamp, int V, int C, int wpv,
                                        int nx, float w, int nsl, int gw,
                                        unsigned long long *totals, int part) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int TB = 4 * TS;  // bytes of a texel
    // Groups of four and eight slices read the fourth texel of a row, which most
    // rows do not touch, after the first is added: its registers go to more blocks
    // per SM (8 slices 1094 -> 1059 us, 4 slices 838 -> 823).  One slice loses by it
    // (659 -> 676), and 16 hold too much for a fifth block either way (1823 -> 1936).
    constexpr bool kLate = TS >= 4 && NP == 1;
    const int lane = threadIdx.x & 31;
    const int v = gw / wpv;
    const int c = (gw - v * wpv) * 32 + lane;
    const bool has_c = c < C;
    const int r = v * C + (has_c ? c : C - 1);
    const int n = has_c ? __ldg(nsamp + r) : 0;
    const bool valid = n > 0;
    const float4 q4 = valid ? __ldg(ray + r) : make_float4(0.f, 0.f, 0.f, 0.f);
    const bool along_x = fabsf(q4.z) > fabsf(q4.w);
    const float su = along_x ? q4.w : q4.z, sv = along_x ? q4.z : q4.w;
    const float pu = (along_x ? q4.y : q4.x) - 0.5f, pv = (along_x ? q4.x : q4.y) - 0.5f;
    const float s = fabsf(su), t = fabsf(sv);
    const float u0 = su < 0.0f ? -pu : pu, v0 = sv < 0.0f ? -pv : pv;
    const float is = s > 0.0f ? fminf(1.0f / s, 1e30f) : 1e30f;
    const float it = valid ? 1.0f / t : 0.0f;
    const float um0 = __fadd_rd(u0, kMagic), phi0 = u0 - (um0 - kMagic);
    const int q0 = __float_as_int(um0) - kMagicInt;
    const int sgn = su < 0.0f ? -TB : TB;
    const int cls = valid ? (along_x ? 2 : 0) + (sv < 0.0f ? 1 : 0) : -1;
    const int P = nx + 2;
    const unsigned long long ss = pack2(s, s), tt = pack2(t, t);
    const unsigned long long kHalf = pack2(0.5f, 0.5f), kMinusHalf = pack2(-0.5f, -0.5f);
    const unsigned long long kMinusOne = pack2(-1.0f, -1.0f);
    const float st = s * t * (1.0f / 12.0f);
    const unsigned long long st12 = pack2(st, st);
    const int jf = (int)floorf(v0), jl = (int)floorf(fmaf(t, (float)(n - 1), v0));
    RayAcc<TS, NP> acc;
    acc.init(totals);
#pragma unroll 1
    for (int pass = 0; pass < 4; ++pass) {
        const bool on = cls == pass;
        if (!__any_sync(FULL, on)) continue;
        const int J0 = __reduce_min_sync(FULL, on ? jf : INT_MAX);
        // + 1: the row of the last carried weights; + 1: a last sample that
        // rounding puts in the next row
        const int J1 = __reduce_max_sync(FULL, on ? jl : INT_MIN) + 2;
        const int nrow = J1 - J0 + 1;
        const int Ja = J0 + nrow * part / kFpParts, Jb = J0 + nrow * (part + 1) / kFpParts - 1;
        // bytes to the next row, and texel -1 of the current one
        const ptrdiff_t step = (ptrdiff_t)(pass & 1 ? -P : P) * TB;
        const char *row = im.base + (pass & 2 ? im.layout : 0) +
                          (ptrdiff_t)((pass & 1 ? -Ja : Ja) + 1) * P * TB;
        // position of the first sample not yet taken: u = q + sh + phi, v = j + psi;
        // samples left; row j's carried weights (columns q, q+1, q+2); column q's
        // byte offset in its row
        float phi = phi0, psi = v0 - (float)Ja, left = on ? (float)n : 0.0f;
        float e0 = 0.0f, e1 = 0.0f, e2 = 0.0f;
        int sh = 0;
        unsigned off = (unsigned)(q0 * sgn + TB), offw = off;
        if (part > 0) {
            // from the first sample of the row before the share
            const float k = fminf(left, fmaxf(ceil_magic(((float)(Ja - 1) - v0) * it), 0.0f));
            const float u = fmaf(s, k, u0), um = __fadd_rd(u, kMagic);
            phi = u - (um - kMagic);
            psi = fmaf(t, k, v0) - (float)(Ja - 1);
            left -= k;
            off = offw = (unsigned)((__float_as_int(um) - kMagicInt) * sgn + TB);
        }
        float w0, w1, w2, w3, w4;
        // the weights w0 .. w4 of columns q .. q+4 (at offw) of the next row
        auto weights = [&]() {
            // samples of the row, and of its first and second cell
            const float N = fminf(left, fmaxf(ceil_magic(fmaf(-psi, it, it)), 0.0f));
            const float N1 = fminf(N, ceil_magic(fmaf(-phi, is, is)));
            const float m = N - N1;
            const float phi2 = fmaf(s, N1, phi) - 1.0f, psi2 = fmaf(t, N1, psi);
            // f32x2 lane 0: the row; lane 1: its second cell.  About the middle
            // sample h = (n-1)/2: sum x = n x_h, sum psi = n psi_h and
            // sum x psi = n x_h psi_h + s t n (n^2 - 1) / 12
            const unsigned long long nn = pack2(N, m), h = fma2(nn, kHalf, kMinusHalf);
            const unsigned long long xh = fma2(ss, h, pack2(phi, phi2));
            const unsigned long long yh = fma2(tt, h, pack2(psi, psi2));
            const unsigned long long X2 = mul2(nn, xh), Y2 = mul2(nn, yh);
            const unsigned long long Z2 =
                fma2(X2, yh, mul2(mul2(nn, st12), fma2(nn, nn, kMinusOne)));
            const float2 X = unpack2(X2), Y = unpack2(Y2), Z = unpack2(Z2);
            // weights of rows j (d) and j+1 (f), columns q + sh + 0, 1, 2 (f2 = Z.y)
            const float d2 = X.y - Z.y, yz = Y.x - Z.x;
            const float d1 = fmaf(-2.0f, d2, X.x - Z.x), d0 = (N - X.x) - yz + d2;
            w0 = e0 + (sh == 0 ? d0 : 0.0f);
            w1 = e1 + (sh == 0 ? d1 : d0);
            w2 = e2 + (sh == 0 ? d2 : d1);
            w3 = sh == 0 ? 0.0f : d2;
            w4 = 0.0f;
            if (sh > 1) {  // both boundaries within one sample step (slopes near one)
                w1 = e1;
                w2 = e2 + d0;
                w3 = d1;
                w4 = d2;
            }
            offw = off;
            e0 = yz + Z.y;
            e1 = fmaf(-2.0f, Z.y, Z.x);
            e2 = Z.y;
            left -= N;
            off += sh * sgn;
            const float x = fmaf(s, N, phi), xm = __fadd_rd(x, kMagic);
            sh = __float_as_int(xm) - kMagicInt;
            phi = x - (xm - kMagic);
            psi = fmaf(t, N, psi) - 1.0f;
        };
        if (part > 0) weights();  // its lower part only: carried into row Ja
        weights();
#pragma unroll 1
        for (int jb = Ja; jb <= Jb; jb += kFlushRows) {
            const int je = min(jb + kFlushRows - 1, Jb);
#pragma unroll 1
            for (int j = jb; j <= je; ++j, row += step) {
                // debug builds: the row and the columns are in the image
                auto in = [&](int k) {
                    return (unsigned)((pass & 1 ? -j : j) + 1) < (unsigned)P &&
                           offw + k * sgn < (unsigned)(P * TB);
                };
                Texel<TS, NP> t0, t1, t2, t3;
                t0.load(im, row + offw, in(0), w0);
                t1.load(im, row + (offw + sgn), in(1), w1);
                t2.load(im, row + (offw + 2 * sgn), in(2), w2);
                const char *p3 = row + (offw + 3 * sgn);
                const bool in3 = in(3);
                if constexpr (!kLate) t3.load(im, p3, in3, w3);
                const float c0 = w0, c1 = w1, c2 = w2, c3 = w3, c4 = w4;
                const char *p4 = row + (offw + 4 * sgn);
                const bool in4 = in(4);
                weights();
                acc.add(t0, c0);
                acc.add(t1, c1);
                acc.add(t2, c2);
                if constexpr (!kLate) {
                    acc.add(t3, c3);
                } else if (c3 != 0.0f) {
                    t0.load(im, p3, in3, c3);
                    acc.add(t0, c3);
                }
                if (c4 != 0.0f) {
                    t0.load(im, p4, in4, c4);
                    acc.add(t0, c4);
                }
            }
            acc.flush();
        }
    }
    if constexpr (TS == 1) reinterpret_cast<float *>(totals)[threadIdx.x] = acc.value(0);
    __syncthreads();
    if (part > 0 || !has_c) return;
#pragma unroll
    for (int k = 0; k < TS * NP; ++k) {
        float val = acc.value(k);
#pragma unroll
        for (int q = 1; q < kFpParts; ++q) {
            if constexpr (TS == 1) {
                val += reinterpret_cast<float *>(totals)[q * 32 + lane];
            } else {
                const float2 e = unpack2(totals[(k / 2) * (32 * kFpParts) + q * 32 + lane]);
                val += (k & 1) ? e.y : e.x;
            }
        }
        if (k < nsl) store_val(out + (size_t)k * ostride + (size_t)v * C + c, val * w);
    }
}

// Quad images (layout 0 walks (u, v) = (x, y); layout 1 the transposed image,
// (u, v) = (y, x)): for every bilinear cell (cu, cv) of the walked layout the
// four clamp-to-edge taps (cu,cv), (cu+1,cv), (cu,cv+1), (cu+1,cv+1) as one
// float4.  Samples lie inside the FOV circle of radius nx/2 texels, so cells
// run over [-1, nx-1] in both axes of both layouts; quad (qi, qj) holds cell
// (qi-1, qj-1) and a layout is (nx+1)^2 quads.
template <typename T>
__device__ __forceinline__ void build_quad(const T *__restrict__ im, float4 *__restrict__ dst,
                                           int nx, int ny, int layout, int qi, int qj) {
    const int cu = qi - 1, cv = qj - 1;
    float4 t;
    float *tv = &t.x;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int du = k & 1, dv = k >> 1;
        int x = layout ? cv + dv : cu + du;
        int y = layout ? cu + du : cv + dv;
        x = min(max(x, 0), nx - 1);
        y = min(max(y, 0), ny - 1);
        tv[k] = load_val(im + (size_t)y * nx + x);
    }
    *dst = t;
}

}  // namespace ctk
