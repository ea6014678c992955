// Gather-form transpose of the pixel-driven backprojector (BP and the
// 1/L^2-weighted FBP / FDK-2D form): deterministic, no atomics.
//
// The backprojector adds, per pixel p inside the FOV disc and view, the
// linearly interpolated detector value at column coordinate y = col + 1/2
// (texel centres at +1/2, clamped taps) when 1/2 < y < C + 1/2
// (BP/transform.cu:76-92, FBP/transform.cu:70-87).  Its transpose sends x_p w
// to the two taps: (1 - f) to max(i-1, 0) and f to min(i, C-1), i = trunc(y),
// f = y - i.  Gathered per detector column: strip b = the pixels with
// trunc(y) = b lies between the rays y = b and y = b + 1 from the source, so
// a lane owns strip b, walks the image lines (rows or columns) across it, and
// sums A_b = sum (1 - f) x w and B_b = sum f x w over its pixels; channel c
// is then B_c + A_{c+1} (channel 0 adds A_0, channel C-1 adds B_C: the
// clamped taps).  A warp holds strips 31k .. 31k+31 and writes channels
// 31k .. 31k+30, so every channel is written by one lane: no atomics, and
// each lane sums in a fixed order.
//
// Geometry per (view, strip group), from host FP64 tables (ct_build_bpt_tables):
// each boundary ray's crossing of the first line and its step per line, in
// 32.32 fixed point along the line, so that the crossings are exact integers
// plus fractions; two lanes sharing a boundary read the same table entry, so
// every pixel belongs to exactly one strip.  A pixel's offset from its
// strip's lower boundary along the line is then small and exact in FP32,
// and its angle from that boundary, atan(n / L) with n its normal distance
// and L its distance along the ray, needs no large coordinate: f is accurate
// to ~1e-7 of a channel, where the absolute column coordinate in FP32 (up to
// ~900 channels) carries ~6e-5 -- noise the ramp filter of the FBP adjoint
// amplifies about 80-fold (the scatter form reached 1.5e-4 relative L2 at
// 512^2 / 984 x 888; the contract is 1e-4).
//
// A crossing and its line step are stored along the direction of growing angle
// and biased by 2^32 - 1, so that a strip is always [lower, upper), the high
// word of its sum is the first pixel and the complement of the low word that
// pixel's offset.  A strip is about one pixel wide: a line's first two pixels
// are loaded ahead of their weights, without a loop.
//
// Slices: 1, 4, 8 or 16 slices share every lane's geometry; the images come as
// planes of one or four slices in both layouts (rows [plane][y][x] for row
// walks, columns [plane][x][y] for column walks) so that adjacent lanes --
// adjacent strips -- read adjacent 4- or 16-byte pixels; pixels outside the FOV
// are zeros there.  Blocks are 4 warps = 4 adjacent views of one channel group
// (their strips cross nearly the same pixels) or, in small geometries, a
// quarter of one view's lines each, ordered channel-group-major as the forward
// projector's.
//
// Bound: issue (85% busy with one slice), load latency and L1 with 16 (issue 60%,
// L1 62%).  BP adjoint, clinical geometry, against groups of at least four slices
// with a loop over each strip's pixels clipped to the line's FOV span (us):
//   slices     1     2     4     8    13    16    32
//   before   838   838   839  1090  1347  1350  2690
//   now      464   523   523   662  1001  1001  2010
#include <type_traits>

#include "bp_body.cuh"

namespace ctk {
namespace {

struct BptArgs {
    int V, C, W, nx, ny;
    int vq;           // blocks per channel group
    float inv_dcol;   // 1 / dcol
};

constexpr int kGatherParts = 4;  // warps of a block
// Geometries of fewer blocks than this (channel groups x view quads) split each
// view's lines among a block's warps: four times the blocks, a quarter as long,
// where whole views leave the GPU part empty or end on a long last wave.  The
// price is the L1 lines that four adjacent views share, which larger geometries
// (and 16 slices) feel.  BP adjoint, 1 / 4 / 8 / 16 slices, whole -> split (us):
// 64^2, 90 x 96 (92 blocks) 31 / 35 / 35 / 41 -> 20 / 20 / 20 / 21; 180^2, 346 x 312
// (957) 57 / 64 / 71 / 77 -> 41 / 46 / 54 / 78; 220^2, 420 x 400 (1365) 70 / 78 / 87 /
// 124 -> 60 / 68 / 83 / 119; 240^2, 460 x 450 (1725) 76 / 84 / 97 / 149 -> 72 / 83 /
// 101 / 148; 512^2, 984 x 888 464 / 523 / 662 / 1002 -> 464 / 567 / 737 / 1159.  A rule
// on the geometry alone, so that a slice gives the same bits in every batch.
constexpr int kSplitBlocks = 1500;
// Resident blocks per SM (BP adjoint of the clinical geometry, us): one slice 464
// with 12 (468 with 9, 631 with 14: spills), four 523 with 10 (581 with 9), eight
// 662 with 8 (672 with 7, 1045 with 9), sixteen 1001 with 5 (1170 with 4, 2521
// with 6).
constexpr int gather_min_blocks(int sb) {
    return sb == 1 ? 12 : sb == 4 ? 10 : sb == 8 ? 8 : 5;
}

// Wide strips (below), 512^2, 984 views, 220 and 110 channels, BP adjoint of 1 / 4 / 8 /
// 16 slices, us, with the pixels' loop unrolled twice: 432 / 551 / 789 / 1430 and 389 /
// 606 / 1119 / 2061 (with the blocks above 426 / 550 / 788 / 1349 and 405 / 602 / 1109 /
// 2326; not unrolled 381 / 530 / 765 / 1281 and 420 / 695 / 1205 / 2455).
constexpr int wide_min_blocks(int sb) { return sb == 1 ? 8 : sb == 4 ? 6 : sb == 8 ? 5 : 4; }

// The (1-f) and f sums of a strip for TS * NQ slices; slice pairs in f32x2.
template <int TS, int NQ>
struct StripSums {
    static constexpr int N = TS == 1 ? NQ : 2 * NQ;
    float a1[N], b1[N];
    unsigned long long a2[N], b2[N];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            a1[k] = b1[k] = 0.0f;
            a2[k] = b2[k] = 0ull;
        }
    }
};

// A pixel of a line for the group's planes, loaded when `on`.
template <int TS, int NQ>
struct LinePixel {
    float4 v[NQ];
    __device__ __forceinline__ void load(const char *p, size_t plane, bool on) {
#pragma unroll
        for (int k = 0; k < NQ; ++k) {
            if constexpr (TS == 1)
                asm volatile("{.reg .pred p; setp.ne.s32 p, %2, 0; @p ld.global.nc.f32 %0, [%1];}"
                             : "=f"(v[k].x)
                             : "l"(p + k * plane), "r"((int)on));
            else
                asm volatile(
                    "{.reg .pred p; setp.ne.s32 p, %5, 0;"
                    " @p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];}"
                    : "=f"(v[k].x), "=f"(v[k].y), "=f"(v[k].z), "=f"(v[k].w)
                    : "l"(p + k * plane), "r"((int)on));
        }
    }
    __device__ __forceinline__ void add(StripSums<TS, NQ> &s, float wa, float wb) const {
        if constexpr (TS == 1) {
#pragma unroll
            for (int k = 0; k < NQ; ++k) {
                s.a1[k] = fmaf(wa, v[k].x, s.a1[k]);
                s.b1[k] = fmaf(wb, v[k].x, s.b1[k]);
            }
        } else {
            const unsigned long long pa = pack2(wa, wa), pb = pack2(wb, wb);
#pragma unroll
            for (int k = 0; k < NQ; ++k) {
                const unsigned long long x01 = pack2(v[k].x, v[k].y), x23 = pack2(v[k].z, v[k].w);
                s.a2[2 * k] = fma2(pa, x01, s.a2[2 * k]);
                s.a2[2 * k + 1] = fma2(pa, x23, s.a2[2 * k + 1]);
                s.b2[2 * k] = fma2(pb, x01, s.b2[2 * k]);
                s.b2[2 * k + 1] = fma2(pb, x23, s.b2[2 * k + 1]);
            }
        }
    }
};

// Planes of TS slices, TS * NQ slices per launch slice group (blockIdx.y).
// SPLIT: a block's four warps take a quarter of one view's lines each, and their
// sums are added in order; else a view each.
// WIDE (plans with bpt_wide: strips of six pixels and more): one loop over the strip's
// pixels inside the image, where a far source's strips may be 10^8 pixels wide.  Narrow
// strips take the first two pixels ahead of that loop, which costs wide ones more than
// it saves (BP adjoint, 512^2, 984 views, 1 / 4 / 8 / 16 slices, narrow -> wide form, us:
// 888 channels 472 / 530 / 670 / 1004 -> 562 / 592 / 736 / 1039; 300, up to 5.0 pixels,
// 411 / 498 / 688 / 1150 -> 418 / 515 / 700 / 1239; 220, 6.9, 463 / 741 / 883 / 1524 ->
// 432 / 551 / 789 / 1430; 110 507 / 801 / 1347 / 2643 -> 389 / 606 / 1119 / 2061; 40 1137
// / 1468 / 1731 / 4035 -> 621 / 802 / 1400 / 2666).
template <bool WEIGHTED, int TS, int NQ, bool SPLIT, bool WIDE>
__global__ void __launch_bounds__(32 * kGatherParts,
                                  WIDE ? wide_min_blocks(TS * NQ) : gather_min_blocks(TS * NQ))
    bp_gather_kernel(const char *__restrict__ rows, const char *__restrict__ cols, size_t plane,
                     float *__restrict__ sino, int nsl, const int4 *__restrict__ wtab,
                     const longlong2 *__restrict__ btab, const float4 *__restrict__ rtab,
                     BptArgs a) {
    constexpr int TB = 4 * TS, SB = TS * NQ;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k = blockIdx.x / a.vq, q = blockIdx.x - k * a.vq;
    const int v = SPLIT ? q : q * kGatherParts + warp;
    if (v >= a.V) return;  // warp-uniform, and never with SPLIT
    const size_t e = (size_t)v * a.W + k;
    const int4 wi = __ldg(wtab + e);
    const bool colwalk = wi.x & 1, pos = (wi.x >> 1) & 1;
    const int lines = wi.z - wi.y + 1, skip = SPLIT ? lines * warp / kGatherParts : 0;
    const int J0 = wi.y + skip;
    const int J1 = SPLIT ? wi.y + lines * (warp + 1) / kGatherParts - 1 : wi.z;
    const int strip = k * kBptOut + lane;
    const longlong2 bl = __ldg(btab + e * 33 + lane);
    // lanes past the last strip get an empty one
    const longlong2 bh = strip <= a.C ? __ldg(btab + e * 33 + lane + 1) : bl;
    const float4 rr = __ldg(rtab + e * 32 + lane);
    const int npx = colwalk ? a.ny : a.nx;
    // debug builds: pixel i of line j is in the image
    auto in = [&](int i, int j) {
        return (unsigned)i < (unsigned)npx && (unsigned)j < (unsigned)(colwalk ? a.nx : a.ny);
    };
    const char *line = (colwalk ? cols : rows) + (size_t)blockIdx.y * NQ * plane +
                       (size_t)J0 * npx * TB;
    const size_t lstep = (size_t)npx * TB;
    const float na = rr.z, da = rr.w;                              // per pixel
    const float nb = na * 2.3283064365386963e-10f, db = da * 2.3283064365386963e-10f;  // 2^-32
    const float c0 = a.inv_dcol, c1 = a.inv_dcol * (-1.0f / 3.0f), c2 = a.inv_dcol * 0.2f;

    StripSums<TS, NQ> sum;
    sum.clear();
    long long Xl = bl.x, Xh = bh.x;
    float tf = 0.0f;
    if constexpr (SPLIT) {
        Xl += skip * bl.y;
        Xh += skip * bh.y;
        tf = (float)skip;
    }
    // (1-f, f) times the weight, from the normal distance n and the distance L
    // along the lower boundary ray: f = atan(n/L)/dcol, |n/L| <= dcol
    auto weights = [&](float n, float L, float &wa, float &wb) {
        const float q = __fdividef(n, L), q2 = q * q;
        wb = q * fmaf(q2, fmaf(q2, c2, c1), c0);
        wa = 1.0f - wb;
        if (WEIGHTED) {
            const float w = __fdividef(1.0f, fmaf(L, L, n * n));  // 1 / (U^2 + t^2)
            wa *= w;
            wb *= w;
        }
    };
    for (int j = J0; j <= J1; ++j, line += lstep, Xl += bl.y, Xh += bh.y, tf += 1.0f) {
        // pixels i .. ih - 1 of the strip (in the direction of growing angle); pixel i
        // is (2^32 - 1 - low word) / 2^32 past the boundary
        const int i = (int)(Xl >> 32), ih = (int)(Xh >> 32);
        LinePixel<TS, NQ> x;
        const float d = __uint2float_rn(~(unsigned)Xl), Lb = fmaf(tf, rr.y, rr.x);
        const float n0 = d * nb, L0 = fmaf(d, db, Lb);
        float wa, wb;
        if constexpr (WIDE) {
            const int ge = min(ih, pos ? npx : 1);  // (-g < npx)
#pragma unroll 2
            for (int g = max(i, pos ? 0 : 1 - npx); g < ge; ++g) {
                const float m = __uint2float_rn((unsigned)g - (unsigned)i);
                if (!CT_DCHECK(in(pos ? g : -g, j))) continue;
                x.load(line + (ptrdiff_t)(pos ? g : -g) * TB, plane, true);
                weights(fmaf(m, na, n0), fmaf(m, da, L0), wa, wb);
                x.add(sum, wa, wb);
            }
            continue;
        }
        const int cnt = ih - i, i0 = pos ? i : -i;
        const bool on0 = cnt > 0 && (unsigned)i0 < (unsigned)npx && CT_DCHECK(in(i0, j));
        x.load(line + (ptrdiff_t)i0 * TB, plane, on0);
        if (on0) {
            weights(n0, L0, wa, wb);
            x.add(sum, wa, wb);
        }
        // A line's second pixel is loaded after the first is added: with both held at
        // once the registers allowed a fifth fewer blocks (1 / 4 / 8 / 16 slices 499 /
        // 557 / 721 / 1198 us, now 464 / 523 / 662 / 1001; FBP adjoint 620 / 674 / 854 /
        // 1330 -> 578 / 663 / 814 / 1204).  In the loop below instead: 464 / 518 / 656 /
        // 1032 and 612 / 653 / 799 / 1210.
        const int i1 = pos ? i + 1 : -i - 1;
        if (cnt > 1 && (unsigned)i1 < (unsigned)npx && CT_DCHECK(in(i1, j))) {
            x.load(line + (ptrdiff_t)i1 * TB, plane, true);
            weights(n0 + na, L0 + da, wa, wb);
            x.add(sum, wa, wb);
        }
        for (int m = 2; m < cnt; ++m) {  // detectors coarser than the pixels
            const int im = pos ? i + m : -i - m;
            if ((unsigned)im >= (unsigned)npx || !CT_DCHECK(in(im, j))) continue;
            x.load(line + (ptrdiff_t)im * TB, plane, true);
            weights(fmaf((float)m, na, n0), fmaf((float)m, da, L0), wa, wb);
            x.add(sum, wa, wb);
        }
    }
    // channel c = strip c's f sum + strip c+1's (1-f) sum (+ the clamped taps)
    const int c = strip;
    const bool writes = lane < kBptOut && c < a.C;
    const size_t sstride = (size_t)a.V * a.C;
    const int s0 = blockIdx.y * SB;
    float *out = sino + (size_t)s0 * sstride + (size_t)v * a.C + c;
    auto store = [&](int h, float av, float bv) {
        const float an = __shfl_down_sync(0xffffffffu, av, 1);
        const float bn = __shfl_down_sync(0xffffffffu, bv, 1);
        float r = bv + an;
        if (c == 0) r += av;
        if (c == a.C - 1) r += bn;
        if (writes && s0 + h < nsl) out[(size_t)h * sstride] = r;
    };
    auto sums = [&](int h, float &av, float &bv) {
        if constexpr (TS == 1) {
            av = sum.a1[h];
            bv = sum.b1[h];
        } else {
            const float2 ap = unpack2(sum.a2[h / 2]), bp = unpack2(sum.b2[h / 2]);
            av = h & 1 ? ap.y : ap.x;
            bv = h & 1 ? bp.y : bp.x;
        }
    };
    if constexpr (!SPLIT) {
#pragma unroll
        for (int h = 0; h < SB; ++h) {
            float av, bv;
            sums(h, av, bv);
            store(h, av, bv);
        }
    } else {
        // a slice per warp and step: all at once would take 16 KB of a block's L1
        constexpr int HC = SB < kGatherParts ? SB : kGatherParts;
        __shared__ float part[kGatherParts][2 * HC][32];
#pragma unroll
        for (int h0 = 0; h0 < SB; h0 += HC) {
            if (h0) __syncthreads();
#pragma unroll
            for (int h = 0; h < HC; ++h)
                sums(h0 + h, part[warp][2 * h][lane], part[warp][2 * h + 1][lane]);
            __syncthreads();
            if (warp < HC) {
                float av = part[0][2 * warp][lane], bv = part[0][2 * warp + 1][lane];
#pragma unroll
                for (int g = 1; g < kGatherParts; ++g) {
                    av += part[g][2 * warp][lane];
                    bv += part[g][2 * warp + 1][lane];
                }
                store(h0 + warp, av, bv);
            }
        }
    }
}

// Planes of TS slices (slices TS q .. of img; zero past `batch` and outside the
// FOV disc, so that the walk needs no clipping to it): rows[q][y][x][TS] and
// cols[q][x][y][TS], through a shared-memory tile.
template <int TS>
__global__ void __launch_bounds__(256)
    bpt_planes_kernel(const float *__restrict__ img, float *__restrict__ rows,
                      float *__restrict__ cols, const int2 *__restrict__ fov_row, int nx, int ny,
                      int batch) {
    __shared__ float tile[TS][32][33];
    const int q = blockIdx.z;
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
    const size_t plane = (size_t)nx * ny;
    auto store = [](float *p, const float *v) {
        if constexpr (TS == 1)
            *p = v[0];
        else
            *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    };
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int x = x0 + threadIdx.x, y = y0 + r;
        float v[TS];
        bool in = x < nx && y < ny;
        if (in) {
            const int2 fr = __ldg(fov_row + y);
            in = x >= fr.x && x <= fr.y;
        }
#pragma unroll
        for (int s = 0; s < TS; ++s) {
            const int b = TS * q + s;
            v[s] = in && b < batch ? __ldg(img + (size_t)b * plane + (size_t)y * nx + x) : 0.0f;
            tile[s][r][threadIdx.x] = v[s];
        }
        if (x < nx && y < ny) store(rows + (q * plane + (size_t)y * nx + x) * TS, v);
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int x = x0 + r, y = y0 + threadIdx.x;
        float v[TS];
#pragma unroll
        for (int s = 0; s < TS; ++s) v[s] = tile[s][threadIdx.x][r];
        if (x < nx && y < ny) store(cols + (q * plane + (size_t)x * ny + y) * TS, v);
    }
}

constexpr int kChunk = 64;  // slices per pass

// Slices per plane, and planes per group and in all, of a chunk of nb slices.
int plane_slices(int nb) { return nb == 1 ? 1 : 4; }
int group_planes(int nb) { return nb <= 4 ? 1 : nb <= 8 ? 2 : 4; }
int padded_planes(int nb) {
    const int ts = plane_slices(nb), nq = group_planes(nb);
    return ((nb + ts - 1) / ts + nq - 1) / nq * nq;
}

template <int TS, int NQ>
void launch_gather(const ct_plan *p, const BptArgs &a, unsigned groups, cudaStream_t s,
                   const float *rows, const float *cols, float *sino, int nsl, int weighted) {
    auto go = [&](auto kern) {
        kern<<<dim3((unsigned)(a.W * a.vq), groups), 32 * kGatherParts, 0, s>>>(
            reinterpret_cast<const char *>(rows), reinterpret_cast<const char *>(cols),
            (size_t)a.nx * a.ny * TS * sizeof(float), sino, nsl,
            reinterpret_cast<const int4 *>(p->d_bpt_warp),
            reinterpret_cast<const longlong2 *>(p->d_bpt_bnd),
            reinterpret_cast<const float4 *>(p->d_bpt_ray), a);
    };
    auto form = [&](auto split, auto wide) {
        weighted ? go(bp_gather_kernel<true, TS, NQ, split.value, wide.value>)
                 : go(bp_gather_kernel<false, TS, NQ, split.value, wide.value>);
    };
    const std::true_type yes;
    const std::false_type no;
    if (a.vq == a.V && a.V > 1)
        p->bpt_wide ? form(yes, yes) : form(yes, no);
    else
        p->bpt_wide ? form(no, yes) : form(no, no);
}

}  // namespace

bool bp_gather_usable(const ct_plan *p) {
    return p->d_bpt_warp != nullptr && p->opts.texture_weights == 0;
}

size_t bp_gather_work_bytes(const ct_plan *p, int batch) {
    if (!bp_gather_usable(p) || batch <= 0) return 0;
    const int nb = batch < kChunk ? batch : kChunk;
    return 2 * sizeof(float) * (size_t)plane_slices(nb) * padded_planes(nb) * p->g.nx * p->g.ny;
}

int bp_gather(const ct_plan *p, const float *img, float *sino, int batch, int weighted,
              void *work, void *stream) {
    cudaStream_t s = (cudaStream_t)stream;
    BptArgs a;
    a.V = p->g.n_views;
    a.C = p->g.n_cols;
    a.W = p->bpt_W;
    a.nx = p->g.nx;
    a.ny = p->g.ny;
    const int quads = (a.V + kGatherParts - 1) / kGatherParts;
    const bool split = a.W * quads < kSplitBlocks;
    a.vq = split ? a.V : quads;
    a.inv_dcol = (float)(1.0 / (double)p->g.dcol);
    const size_t plane = (size_t)a.nx * a.ny, sl = (size_t)a.V * a.C;
    for (int b0 = 0; b0 < batch; b0 += kChunk) {
        const int nb = batch - b0 < kChunk ? batch - b0 : kChunk;
        const int ts = plane_slices(nb), nq = group_planes(nb), pq = padded_planes(nb);
        float *rows = static_cast<float *>(work);
        float *cols = rows + (size_t)pq * plane * ts;
        auto build = [&](auto kern) {
            kern<<<dim3((a.nx + 31) / 32, (a.ny + 31) / 32, pq), dim3(32, 8), 0, s>>>(
                img + (size_t)b0 * plane, rows, cols, reinterpret_cast<const int2 *>(p->d_fov_row),
                a.nx, a.ny, nb);
        };
        ts == 1 ? build(bpt_planes_kernel<1>) : build(bpt_planes_kernel<4>);
        float *out = sino + (size_t)b0 * sl;
        const unsigned groups = (unsigned)(pq / nq);
        if (ts == 1)
            launch_gather<1, 1>(p, a, groups, s, rows, cols, out, nb, weighted);
        else if (nq == 1)
            launch_gather<4, 1>(p, a, groups, s, rows, cols, out, nb, weighted);
        else if (nq == 2)
            launch_gather<4, 2>(p, a, groups, s, rows, cols, out, nb, weighted);
        else
            launch_gather<4, 4>(p, a, groups, s, rows, cols, out, nb, weighted);
        ct_count_launch(2);
    }
    return (int)cudaGetLastError();
}

}  // namespace ctk
