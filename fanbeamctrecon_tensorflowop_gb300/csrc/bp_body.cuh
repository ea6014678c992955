// The backprojector's per-tile work, shared by the per-plan kernel and the
// uneven-batch kernel (geometry and arithmetic are described in bp.cu).
#pragma once

#include "fp_body.cuh"

namespace ctk {

struct BpArgs {
    int V, C, nx, ny;
    float xmin, ymin, dx, dy;
    float R;
    float inv_dcol;   // 1/dcol
    float pos_off;    // shift - left/dcol + 1/2: y = atan*inv_dcol + pos_off = col + 1/2
    float fC;         // n_cols
    double fov_r2;
    float ycoef[9];   // y = z * sum ycoef[k] z^(2k) + pos_off, z = t/U: the atan fit over
                      // 1/dcol (zero-padded to degree 8)
    int tex;          // texture-unit weights (tex_weight) instead of exact FP32 ones
};

// The arguments of a plan (host).
inline BpArgs bp_args(const ct_plan *p) {
    BpArgs a;
    a.V = p->g.n_views;
    a.C = p->g.n_cols;
    a.nx = p->g.nx;
    a.ny = p->g.ny;
    a.xmin = p->g.xmin;
    a.ymin = p->g.ymin;
    a.dx = p->g.dx;
    a.dy = p->g.dy;
    a.R = p->g.sid;
    const double inv = 1.0 / (double)p->g.dcol;
    a.inv_dcol = (float)inv;
    a.pos_off = (float)((double)p->g.shift - (double)p->g.left * inv + 0.5);
    a.fC = (float)a.C;
    a.fov_r2 = (double)p->g.rfov * (double)p->g.rfov;
    // degree-4 fits are the degree-8 polynomial with zero high coefficients
    for (int k = 0; k < 9; ++k) a.ycoef[k] = (float)((double)p->atan_coef[k] / (double)p->g.dcol);
    a.tex = p->opts.texture_weights;
    return a;
}

// Column position y = col + 1/2 at z = t / U.
template <int DEG>
__device__ __forceinline__ float bp_column(float z, const float *ycoef, float inv_dcol, float off) {
    if constexpr (DEG == 0) {
        return fmaf(atanf(z), inv_dcol, off);
    } else {
        const float s = z * z;
        float p = ycoef[DEG];
#pragma unroll
        for (int k = DEG - 1; k >= 0; --k) p = fmaf(p, s, ycoef[k]);
        return fmaf(z, p, off);
    }
}

// y = col + 1/2 >= 0: i = trunc(y) = floor(col - 1/2) + 1 and f = frac(y),
// without float-to-int conversion instructions (valid for 0 <= y < 2^22).
__device__ __forceinline__ void split_pos(float y, int &i, float &f) {
    const float m = __fadd_rz(y, 12582912.0f);
    i = __float_as_int(m) - 0x4B400000;
    f = y - (m - 12582912.0f);
}

// The GPU texture unit's linear-filter weight for a fraction f in [0, 1): f
// rounded to a multiple of 1/256, ties up (8 fractional bits; measured on
// GB300 against texture objects with the reference's sampler state).  The
// reference interpolates its sinogram rows through the texture unit
// (BP/transform.cu:90, FBP/transform.cu:85, FDK/GPURecon_GPU.cu:45); plans
// created with texture_weights = 1 reproduce it.  f * 256 + 1/2 is exact in
// FP32, so this is the rounding itself, not an approximation of it.
__device__ __forceinline__ float tex_weight(float f) {
    return floorf(fmaf(f, 256.0f, 0.5f)) * (1.0f / 256.0f);
}

__device__ __forceinline__ unsigned long long add_rz2(unsigned long long a,
                                                      unsigned long long b) {
    unsigned long long d;
    asm("add.rz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// The sums of one pixel over views for the TS * NP slices of a group: NP planes
// of TS = 1 slice (the sinograms themselves, [V][C]) or 4 slices ([V][C][4]).
template <int TS, int NP>
struct BpAcc {
    static constexpr int N = TS == 1 ? NP : 2 * NP;
    float one[N];              // TS == 1
    unsigned long long two[N];  // TS == 4: slice pairs
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            one[k] = 0.0f;
            two[k] = 0ull;
        }
    }
    // += wa * (tap at byte offset a of the row) + wb * (tap at offset b)
    __device__ __forceinline__ void add(const char *row, size_t plane, int a, int b, bool ok,
                                        float wa, float wb) {
        if constexpr (TS == 1) {
            float va[NP], vb[NP];
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                va[p] = CT_DLOAD(ok, reinterpret_cast<const float *>(row + p * plane + a));
                vb[p] = CT_DLOAD(ok, reinterpret_cast<const float *>(row + p * plane + b));
            }
#pragma unroll
            for (int p = 0; p < NP; ++p) one[p] = fmaf(wa, va[p], fmaf(wb, vb[p], one[p]));
        } else {
            // Two planes' taps at a time: with all four in flight the registers allow
            // three blocks of 16 slices per SM instead of four (BP 926 -> 876 us, FBP
            // 1049 -> 1010; one plane at a time 925 and 1060).
            constexpr int H = NP < 2 ? NP : 2;
            const unsigned long long a2 = pack2(wa, wa), b2 = pack2(wb, wb);
#pragma unroll
            for (int h = 0; h < NP; h += H) {
                float4 va[H], vb[H];
#pragma unroll
                for (int p = 0; p < H && h + p < NP; ++p) {
                    const char *r = row + (h + p) * plane;
                    va[p] = CT_DLOAD(ok, reinterpret_cast<const float4 *>(r + a));
                    vb[p] = CT_DLOAD(ok, reinterpret_cast<const float4 *>(r + b));
                }
#pragma unroll
                for (int p = 0; p < H && h + p < NP; ++p) {
                    unsigned long long *t = two + 2 * (h + p);
                    t[0] = fma2(a2, pack2(va[p].x, va[p].y),
                                fma2(b2, pack2(vb[p].x, vb[p].y), t[0]));
                    t[1] = fma2(a2, pack2(va[p].z, va[p].w),
                                fma2(b2, pack2(vb[p].z, vb[p].w), t[1]));
                }
            }
        }
    }
    __device__ __forceinline__ float value(int s) const {
        if constexpr (TS == 1) return one[s];
        const float2 v = unpack2(two[s / 2]);
        return (s & 1) ? v.y : v.x;
    }
};

// Adds views 2 p0 .. 2 p1 - 1 (below V) of pixel (px, py) to acc: per view
//   U = R + px c + py s, t = -px s + py c, y = atan(t/U)/dcol + offset = col + 1/2,
// the taps trunc(y) - 1 and trunc(y), weights (1-f, f) times 1/(U^2 + t^2) when
// WEIGHTED.  The geometry of two views is one f32x2 evaluation (pairs: per
// view pair (c0, c1, s0, s1)).
// COVER: every pixel of the FOV lies at y in (1, C) in every view (plans with
// bp_cover) and the weights are exact: no range test and no clamp.
// Otherwise pixels with y outside (1/2, C + 1/2) add nothing, the taps are
// clamped to the row, and a.tex selects the texture unit's weights.
template <int TS, int NP, bool WEIGHTED, int DEG, bool COVER>
__device__ __forceinline__ void bp_views(BpAcc<TS, NP> &acc, const char *__restrict__ sino,
                                         size_t plane, const float4 *__restrict__ pairs,
                                         const BpArgs &a, float px, float py, int p0, int p1) {
    constexpr int TB = 4 * TS;
    const unsigned long long px2 = pack2(px, px), py2 = pack2(py, py), nx2 = pack2(-px, -px);
    const unsigned long long R2 = pack2(a.R, a.R), off2 = pack2(a.pos_off, a.pos_off);
    const unsigned long long mg2 = pack2(kMagic, kMagic);
    const ptrdiff_t rstep = (ptrdiff_t)a.C * TB;
    const char *row = sino + 2 * p0 * rstep;
    for (int p = p0; p < p1; ++p, row += 2 * rstep) {
        const float4 cs = __ldg(pairs + p);
        const unsigned long long c2 = pack2(cs.x, cs.y), s2 = pack2(cs.z, cs.w);
        const unsigned long long U2 = fma2(px2, c2, fma2(py2, s2, R2));
        const unsigned long long t2 = fma2(py2, c2, mul2(nx2, s2));
        const float2 U = unpack2(U2);
        const unsigned long long z2 =
            mul2(t2, pack2(__fdividef(1.0f, U.x), __fdividef(1.0f, U.y)));
        unsigned long long y2;
        if constexpr (DEG == 0) {
            const float2 z = unpack2(z2);
            y2 = fma2(pack2(atanf(z.x), atanf(z.y)), pack2(a.inv_dcol, a.inv_dcol), off2);
        } else {
            const unsigned long long q2 = mul2(z2, z2);
            unsigned long long g2 = pack2(a.ycoef[DEG], a.ycoef[DEG]);
#pragma unroll
            for (int k = DEG - 1; k >= 0; --k) g2 = fma2(g2, q2, pack2(a.ycoef[k], a.ycoef[k]));
            y2 = fma2(z2, g2, off2);
        }
        float2 w = make_float2(1.0f, 1.0f);
        if constexpr (WEIGHTED) {
            const float2 l = unpack2(fma2(U2, U2, mul2(t2, t2)));
            w = make_float2(__fdividef(1.0f, l.x), __fdividef(1.0f, l.y));
        }
        // i = trunc(y) and f = frac(y), 0 <= y < 2^22, without conversions
        const float2 yv = unpack2(y2);
        if constexpr (!COVER)
            y2 = pack2(fminf(fmaxf(yv.x, 0.0f), a.fC), fminf(fmaxf(yv.y, 0.0f), a.fC));
        const unsigned long long m2 = add_rz2(y2, mg2);
        const float2 m = unpack2(m2), f = unpack2(sub2(y2, sub2(m2, mg2)));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (h && 2 * p + 1 >= a.V) break;  // the last view of an odd number
            const float y = h ? yv.y : yv.x;
            const int i = __float_as_int(h ? m.y : m.x) - kMagicInt;
            float fb = h ? f.y : f.x;
            const float wg = h ? w.y : w.x;
            const char *r = row + h * rstep;
            if constexpr (COVER) {
                const bool ok = i >= 1 && i < a.C;
                acc.add(r, plane, (i - 1) * TB, i * TB, ok, WEIGHTED ? (1.0f - fb) * wg : 1.0f - fb,
                        WEIGHTED ? fb * wg : fb);
            } else {
                if (!(y > 0.5f && y < a.fC + 0.5f)) continue;
                // y beyond C: the clamped taps coincide, any fraction serves
                if (a.tex) fb = tex_weight(fb);
                const int i0 = max(i - 1, 0), i1 = min(i, a.C - 1);
                const bool ok = (unsigned)i0 < (unsigned)a.C && (unsigned)i1 < (unsigned)a.C;
                acc.add(r, plane, i0 * TB, i1 * TB, ok, WEIGHTED ? (1.0f - fb) * wg : 1.0f - fb,
                        WEIGHTED ? fb * wg : fb);
            }
        }
    }
}

// The views of a pixel are summed in kBpShares shares, then the shares in order:
// first view pair of share g.
constexpr int kBpShares = 8;
__device__ __forceinline__ int bp_share(int V, int g) {
    return (int)((long long)((V + 1) / 2) * g / kBpShares);
}

// Pixel centre (ix, iy), and whether it lies in the image and the FOV disc
// (elsewhere the isocentre stands in for it: its sums are dropped).  The centre
// is the FP64 sum rounded once, as fmaf gives it; the disc test is FP64's, made
// in FP32 except within 1e-6 of the rim (its own error is 3e-7; 1e-30: radii whose
// squares FP32 cannot hold).  All of a block's warps, or a volume's slice groups,
// make this test for the same pixels, and the FP64 pipe is narrow: with FP64 alone
// it took 60 us of any 512^2 BP, the time of 60 views.
template <class Args>
__device__ __forceinline__ bool bp_pixel(const Args &a, int ix, int iy, float &px, float &py) {
    const float x = fmaf(a.dx, (float)ix + 0.5f, a.xmin);
    const float y = fmaf(a.dy, (float)iy + 0.5f, a.ymin);
    const float r2 = (float)a.fov_r2;
    const float d = fmaf(x, x, y * y) - r2;
    bool in = d < 0.0f;
    if (!(fabsf(d) > fmaf(r2, 1e-6f, 1e-30f))) {
        const double xd = (double)a.xmin + (double)a.dx * (ix + 0.5);
        const double yd = (double)a.ymin + (double)a.dy * (iy + 0.5);
        in = xd * xd + yd * yd <= a.fov_r2;
    }
    in = in && ix < a.nx && iy < a.ny;
    px = in ? x : 0.0f;
    py = in ? y : 0.0f;
    return in;
}

// A warp's 8 x 4 pixels: lanes 0 .. 15 a 4 x 4 block, lanes 16 .. 31 the one
// to its right, so that the 16 lanes of a 16-byte load's pass read the fewest
// detector columns.
__device__ __forceinline__ int bp_lane_x(int lane) { return (lane & 3) + ((lane >> 4) << 2); }
__device__ __forceinline__ int bp_lane_y(int lane) { return (lane >> 2) & 3; }

}  // namespace ctk
