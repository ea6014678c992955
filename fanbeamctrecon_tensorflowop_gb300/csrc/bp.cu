// Pixel-driven fan-beam backprojection (unweighted BP and 1/L^2-weighted FBP /
// FDK-2D) and its transpose.
//
// Per pixel centre (x, y) inside the FOV disc and view beta, with
// c = -cos(beta), s = -sin(beta):
//   U = R + x c + y s,  t = -x s + y c,  col = (atan(t/U) - left)/dcol + shift,
// and when 0 < col < n_cols the pixel gains the linearly interpolated,
// clamped detector value at col (texel centres at +1/2), times 1/(U^2+t^2) in
// the weighted form (BP/transform.cu:76-92, FBP/transform.cu:70-87,
// FDK/GPURecon_GPU.cu:25-49).
//
// One launch covers all views and slices.  A block's eight warps sum the same
// 8 x 4 pixels over an eighth of the views each (a 256^2 slice alone fills the
// GPU that way), and the image is written once.  A thread evaluates a
// pixel's geometry for two views at a time as f32x2 instructions and shares it
// among up to 16 slices, whose detector values come as planes of four slices
// (bp_planes_kernel) in one 16-byte load per tap: a pass of 16 lanes covers a
// 4 x 4 block of pixels, whose taps lie on few lines.  t/U uses the SFU
// reciprocal; atan(z) is a polynomial in z^2 fitted per plan over the FOV's
// |z| range (to FP32 atanf accuracy, 3e-8 absolute), with atanf kept for fans
// wider than 90 degrees.  Plans whose FOV lies inside the detector in every
// view (bp_cover) need no range test and no clamp.  Plans with texture_weights
// = 1 round the interpolation weight as the reference's texture unit does
// (tex_weight); the default keeps exact FP32.
//
// Bound: issue for one slice (74% busy), the L1 data path beyond (88% busy).
// Clinical geometry (512^2, 984 x 888; before: 32 x 8 ROWS pixel blocks over
// all views, and tap images of four slices read 32 bytes at a time), us:
//   slices            1     2     3     4     5     8    13    16    32
//   BP  before      721   990  1419   558  1133   965  2087  1894  2909
//       now         184   231   276   267   459   460   870   870  1709
//   FBP before      788  1205  1614   553  1042  1115  2150  2086  3445
//       now         267   332   331   331   525   532   977  1012  1954
// (1, 2, 4 shares of the views instead of 8: one slice 251 / 214 / 204 us, 32
// slices 2378 / 2090 / 1987 with two blocks of 16 slices per SM.)
#include <cstdint>

#include "bp_body.cuh"

namespace ctk {
namespace {

constexpr int kTile = 32;  // tile edge of the scatter transpose
// slices per transpose thread for batches of 4 or more (32 clinical slices:
// 1 -> 16.2 ms, 4 -> 15.5, 8 -> 17.2); smaller batches take one per thread
constexpr int kBptSlices = 4;
constexpr int kRowsPerThr = 4;

// Resident blocks per SM (clinical geometry, BP / FBP, us, with the disc test in FP64, which
// took some 8 us of each): four slices 274 / 342
// with 7 (288 / 368 with 6, 284 / 374 with 5), eight 487 / 547 with 5 (481 / 573 with
// 7), twelve 679 / 776 with 5 (697 / 780 with 4), sixteen 876 / 1010 with 4 (926 / 1049
// with 3 and all planes at once); one 187 / 278 with 4 (198 / 281 with 5); three read
// as sinograms 276 (BP) with 8 (276 with 7, 290 with 6 and 5).
constexpr int bp_min_blocks(int sb) {
    return sb == 1 ? 4 : sb == 2 ? 5 : sb == 3 ? 8 : sb <= 4 ? 7 : sb <= 12 ? 5 : 4;
}

// A block is kBpShares warps over the same 8 x 4 pixels: warp g takes the g-th
// share of the view pairs, and the warps' sums are added in shared memory in
// order.  blockIdx.z: slice group (group bytes apart).
template <int TS, int NP, bool WEIGHTED, int DEG, bool COVER>
__global__ void __launch_bounds__(256, bp_min_blocks(TS * NP))
    bp_fan_kernel(const char *__restrict__ sino, size_t plane, size_t group,
                  float *__restrict__ img, const float4 *__restrict__ pairs, BpArgs a,
                  int batch) {
    constexpr int SB = TS * NP;
    __shared__ float4 part[kBpShares][32];
    const int lane = threadIdx.x & 31, g = warp_index();
    const int ix = blockIdx.x * 8 + bp_lane_x(lane), iy = blockIdx.y * 4 + bp_lane_y(lane);
    const int b0 = blockIdx.z * SB;
    float px, py;
    const bool in = bp_pixel(a, ix, iy, px, py);
    BpAcc<TS, NP> acc;
    acc.clear();
    if (__any_sync(0xffffffffu, in)) {
        bp_views<TS, NP, WEIGHTED, DEG, COVER>(acc, sino + blockIdx.z * group, plane, pairs, a, px,
                                               py, bp_share(a.V, g), bp_share(a.V, g + 1));
    }
    const size_t np = (size_t)a.nx * a.ny;
    float *out = img + (size_t)b0 * np + (size_t)iy * a.nx + ix;
    const bool store = ix < a.nx && iy < a.ny && g == 0;
#pragma unroll
    for (int q = 0; q < (SB + 3) / 4; ++q) {
        if (b0 + 4 * q >= batch) break;  // uniform
        float4 t;
        t.x = acc.value(4 * q);
        t.y = SB > 1 ? acc.value(SB > 1 ? 4 * q + 1 : 0) : 0.0f;
        t.z = SB > 2 ? acc.value(SB > 2 ? 4 * q + 2 : 0) : 0.0f;
        t.w = SB > 3 ? acc.value(SB > 3 ? 4 * q + 3 : 0) : 0.0f;
        __syncthreads();
        part[g][lane] = t;
        __syncthreads();
        if (g == 0) {
#pragma unroll
            for (int k = 1; k < kBpShares; ++k) {
                const float4 e = part[k][lane];
                t.x += e.x;
                t.y += e.y;
                t.z += e.z;
                t.w += e.w;
            }
        }
        if (store) {
            const float *tv = &t.x;
#pragma unroll
            for (int k = 0; k < (SB < 4 ? SB : 4); ++k)
                if (b0 + 4 * q + k < batch) out[(size_t)(4 * q + k) * np] = in ? tv[k] : 0.0f;
        }
    }
}

// Planes of four slices: [plane][V][C][4] from [batch][V][C] (zero past `batch`).
__global__ void __launch_bounds__(256)
    bp_planes_kernel(const float *__restrict__ sino, float4 *__restrict__ planes, size_t slice,
                     int batch) {
    const int b0 = 4 * blockIdx.y;
    for (size_t e = (size_t)blockIdx.x * 256 + threadIdx.x; e < slice;
         e += (size_t)gridDim.x * 256) {
        float v[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) v[s] = b0 + s < batch ? __ldg(sino + (b0 + s) * slice + e) : 0.0f;
        planes[blockIdx.y * slice + e] = make_float4(v[0], v[1], v[2], v[3]);
    }
}

// Transpose of bp_fan_kernel in scatter form (plans with texture weights, or
// without a workspace): each pixel-view scatters x * weight * (1-f, f)
// onto the two clamped detector taps with global atomics (L2 reductions).  A
// thread evaluates each pixel-view's geometry once for GSB slices.
// Atomics of one warp instruction that hit the same address serialise, so the
// 32 lanes of a warp always lie across the view's rays (where their columns
// differ): grid.z pairs a row pass (lanes along x, pixels of a thread 8 apart
// in y), which takes the views whose rays run along y, with a column pass
// (lanes along y) for the views whose rays run along x.  With one layout for
// all views, half of them put a warp's lanes along a ray onto a few columns
// (32 clinical slices: 15.6 -> 12.4 ms).  Adjacent lanes' columns are about
// one apart, so a lane adds its right neighbour's lower part into its own
// upper atomic when they share the address (12.4 -> 11.4 ms; 16-byte vector
// atomics covering both taps measured 24 ms).  (A shared-memory, fixed-point form
// with one block per view measured slower: every block then sweeps the
// whole image.)
template <bool WEIGHTED, int DEG, int GSB, bool TEX>
__global__ void __launch_bounds__(256)
    bp_fan_transpose_kernel(const float *__restrict__ img, float *__restrict__ sino,
                            const float2 *__restrict__ view_cs, BpArgs a, int batch) {
    // grid.z = 2 * slice groups: even z maps lanes along x and takes the views
    // whose rays run along y, odd z maps lanes along y and takes the others
    const bool colmode = blockIdx.z & 1;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int b0 = (blockIdx.z >> 1) * GSB;
    if (b0 >= batch) return;
    const int nsl = min(GSB, batch - b0);
    float px[kRowsPerThr], py[kRowsPerThr], xv[GSB][kRowsPerThr];
    bool nz[kRowsPerThr];
    bool any = false;
#pragma unroll
    for (int k = 0; k < kRowsPerThr; ++k) {
        // row mode: lane = x, the thread's pixels step 8 in y; column mode: swapped
        const int ix = colmode ? blockIdx.x * kTile + ty + 8 * k : blockIdx.x * kTile + tx;
        const int iy = colmode ? blockIdx.y * kTile + tx : blockIdx.y * kTile + ty + 8 * k;
        const double xd = (double)a.xmin + (double)a.dx * (ix + 0.5);
        const double yd = (double)a.ymin + (double)a.dy * (iy + 0.5);
        px[k] = (float)xd;
        py[k] = (float)yd;
        const bool in = ix < a.nx && iy < a.ny && (xd * xd + yd * yd <= a.fov_r2);
        nz[k] = false;
#pragma unroll
        for (int s = 0; s < GSB; ++s) {
            xv[s][k] = in && s < nsl
                           ? img[(size_t)(b0 + s) * a.nx * a.ny + (size_t)iy * a.nx + ix]
                           : 0.0f;
            nz[k] |= xv[s][k] != 0.0f;
        }
        any |= nz[k];
    }
    if (!__syncthreads_or(any)) return;
    for (int v = 0; v < a.V; ++v) {
        const float2 cs = __ldg(view_cs + v);
        // rays run along (c, s) = cs: row pass for |c| < |s|, column pass otherwise
        if ((fabsf(cs.x) >= fabsf(cs.y)) != colmode) continue;  // block-uniform
#pragma unroll
        for (int k = 0; k < kRowsPerThr; ++k) {
            if (!__any_sync(0xffffffffu, nz[k])) continue;  // warp-uniform
            const float U = fmaf(px[k], cs.x, fmaf(py[k], cs.y, a.R));
            const float t = fmaf(py[k], cs.x, -px[k] * cs.y);
            const float rU = __fdividef(1.0f, U);
            const float y = bp_column<DEG>(t * rU, a.ycoef, a.inv_dcol, a.pos_off);
            const bool ok = nz[k] && y > 0.5f && y < a.fC + 0.5f;
            int i;
            float f;
            split_pos(ok ? y : 1.0f, i, f);
            if constexpr (TEX) f = tex_weight(f);
            const int i0 = max(i - 1, 0), i1 = min(i, a.C - 1);
            const float w = WEIGHTED ? __fdividef(1.0f, fmaf(U, U, t * t)) : 1.0f;
            // the next lane's lower tap is usually this lane's upper one: this
            // lane adds the next lane's lower part there, and the next lane
            // skips that atomic
            const int lane = threadIdx.x;
            const int nb_i0 = __shfl_down_sync(0xffffffffu, ok ? i0 : -1, 1);
            const int pv_i1 = __shfl_up_sync(0xffffffffu, ok ? i1 : -2, 1);
            const bool take = ok && lane < 31 && nb_i0 == i1;
            const bool given = ok && lane > 0 && pv_i1 == i0;
#pragma unroll
            for (int s = 0; s < GSB; ++s) {
                const float val = ok ? xv[s][k] * w : 0.0f;
                const float lo = val * (1.0f - f), hi = val * f;
                const float nb_lo = __shfl_down_sync(0xffffffffu, lo, 1);
                const float up = take ? hi + nb_lo : hi;
                if (ok && s < nsl) {
                    float *row = sino + ((size_t)(b0 + s) * a.V + v) * a.C;
                    if (!given && lo != 0.0f) atomicAdd(row + i0, lo);
                    if (up != 0.0f) atomicAdd(row + i1, up);
                }
            }
        }
    }
}

struct BpLaunch {
    const ct_plan *p;
    BpArgs a;
    cudaStream_t s;
    int weighted;
};

// Slices of `nb` in groups of TS * NP (grid.z), planes `plane` bytes apart.
template <int TS, int NP>
void launch_bp(const BpLaunch &l, const void *sino, size_t plane, float *img, int nb) {
    const int groups = (nb + TS * NP - 1) / (TS * NP);
    const dim3 grid((l.a.nx + 7) / 8, (l.a.ny + 3) / 4, groups);
    auto go = [&](auto kern) {
        kern<<<grid, 256, 0, l.s>>>(static_cast<const char *>(sino), plane, NP * plane, img,
                                    reinterpret_cast<const float4 *>(l.p->d_view_pairs), l.a,
                                    nb);
    };
    const bool w = l.weighted != 0;
    if (l.p->bp_cover && l.p->atan_deg == 4 && !l.a.tex)
        w ? go(bp_fan_kernel<TS, NP, true, 4, true>) : go(bp_fan_kernel<TS, NP, false, 4, true>);
    else if (l.p->atan_deg != 0)
        w ? go(bp_fan_kernel<TS, NP, true, 8, false>) : go(bp_fan_kernel<TS, NP, false, 8, false>);
    else
        w ? go(bp_fan_kernel<TS, NP, true, 0, false>) : go(bp_fan_kernel<TS, NP, false, 0, false>);
    ct_count_launch();
}

template <bool W, int G, bool TEX>
void launch_bpt(int deg, dim3 grid, cudaStream_t s, const float *ip, float *sp, const float2 *vcs,
                const BpArgs &a, int nb) {
    dim3 block(kTile, 8, 1);
    if (deg == 4)
        bp_fan_transpose_kernel<W, 4, G, TEX><<<grid, block, 0, s>>>(ip, sp, vcs, a, nb);
    else if (deg == 8)
        bp_fan_transpose_kernel<W, 8, G, TEX><<<grid, block, 0, s>>>(ip, sp, vcs, a, nb);
    else
        bp_fan_transpose_kernel<W, 0, G, TEX><<<grid, block, 0, s>>>(ip, sp, vcs, a, nb);
}

template <int G>
void launch_bpt_any(bool w, bool tex, int deg, dim3 grid, cudaStream_t s, const float *ip,
                    float *sp, const float2 *vcs, const BpArgs &a, int nb) {
    if (w)
        (tex ? launch_bpt<true, G, true> : launch_bpt<true, G, false>)(deg, grid, s, ip, sp, vcs,
                                                                      a, nb);
    else
        (tex ? launch_bpt<false, G, true> : launch_bpt<false, G, false>)(deg, grid, s, ip, sp,
                                                                        vcs, a, nb);
}

}  // namespace

constexpr int kBpChunk = 64;  // slices per workspace chunk

// Batches of three or more read planes of four slices (ct_bp_fan, which has no
// workspace of the caller's, from four on).
size_t bp_fan_work_bytes(const ct_plan *p, int batch) {
    if (batch < 3) return 0;
    const size_t planes = ((batch < kBpChunk ? batch : kBpChunk) + 3) / 4;
    return sizeof(float4) * planes * p->g.n_views * p->g.n_cols;
}

int bp_fan(const ct_plan *p, const float *sino, float *img, int batch, int weighted, void *work,
           void *stream) {
    BpLaunch l{p, bp_args(p), (cudaStream_t)stream, weighted};
    const size_t slice = (size_t)l.a.V * l.a.C, plane = (size_t)l.a.nx * l.a.ny;
    if (batch < 3 || !work) {
        // the sinograms themselves, up to four slices per thread
        for (int b0 = 0; b0 < batch;) {
            const int left = batch - b0;
            int n;
            const float *sp = sino + (size_t)b0 * slice;
            float *ip = img + (size_t)b0 * plane;
            if (left >= 4) {
                n = left / 4 * 4 < 65535 * 4 ? left / 4 * 4 : 65535 * 4;
                launch_bp<1, 4>(l, sp, slice * sizeof(float), ip, n);
            } else if (left == 3) {
                n = 3;
                launch_bp<1, 3>(l, sp, slice * sizeof(float), ip, n);
            } else if (left == 2) {
                n = 2;
                launch_bp<1, 2>(l, sp, slice * sizeof(float), ip, n);
            } else {
                n = 1;
                launch_bp<1, 1>(l, sp, slice * sizeof(float), ip, n);
            }
            b0 += n;
        }
        return (int)cudaGetLastError();
    }
    float4 *planes = static_cast<float4 *>(work);
    for (int b0 = 0; b0 < batch; b0 += kBpChunk) {
        const int nb = batch - b0 < kBpChunk ? batch - b0 : kBpChunk;
        const size_t want = (slice + 255) / 256;
        bp_planes_kernel<<<dim3((unsigned)(want < 65535 ? want : 65535), (nb + 3) / 4), 256, 0,
                           l.s>>>(sino + (size_t)b0 * slice, planes, slice, nb);
        ct_count_launch();
        for (int k = 0; k < nb;) {
            const int left = nb - k;
            const float4 *src = planes + (size_t)(k / 4) * slice;
            float *ip = img + (size_t)(b0 + k) * plane;
            const size_t pb = slice * sizeof(float4);
            int n;
            if (left > 8) {
                n = left >= 16 ? left / 16 * 16 : left;
                if (left > 12)
                    launch_bp<4, 4>(l, src, pb, ip, n);
                else
                    launch_bp<4, 3>(l, src, pb, ip, n);
            } else if (left > 4) {
                n = left >= 8 ? left / 8 * 8 : left;
                launch_bp<4, 2>(l, src, pb, ip, n);
            } else {
                n = left;
                launch_bp<4, 1>(l, src, pb, ip, n);
            }
            k += n;
        }
    }
    return (int)cudaGetLastError();
}

size_t bp_fan_transpose_work_bytes(const ct_plan *p, int batch) {
    return bp_gather_work_bytes(p, batch);
}

// The gather form (bp_gather.cu) where the plan has its tables, the
// exact-weight interpolation and a workspace; otherwise the scatter below
// (texture-weight plans keep it: it repeats the forward's own column
// arithmetic, so the adjoint stays the exact transpose of those weights).
int bp_fan_transpose(const ct_plan *p, const float *img, float *sino, int batch, int weighted,
                     void *work, void *stream) {
    if (work && bp_gather_usable(p)) return bp_gather(p, img, sino, batch, weighted, work, stream);
    const BpArgs a = bp_args(p);
    const float2 *vcs = reinterpret_cast<const float2 *>(p->d_view_cs);
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaMemsetAsync(sino, 0, sizeof(float) * (size_t)batch * a.V * a.C, s);
    if (e != cudaSuccess) return (int)e;
    const int G = batch >= kBptSlices ? kBptSlices : 1;
    for (int b0 = 0; b0 < batch; b0 += 32767 * G) {
        const int nb = batch - b0 < 32767 * G ? batch - b0 : 32767 * G;
        dim3 grid((a.nx + kTile - 1) / kTile, (a.ny + kTile - 1) / kTile, 2 * ((nb + G - 1) / G));
        const float *ip = img + (size_t)b0 * a.nx * a.ny;
        float *sp = sino + (size_t)b0 * a.V * a.C;
        const bool tex = p->opts.texture_weights != 0;
        if (G == kBptSlices)
            launch_bpt_any<kBptSlices>(weighted != 0, tex, p->atan_deg, grid, s, ip, sp, vcs, a,
                                       nb);
        else
            launch_bpt_any<1>(weighted != 0, tex, p->atan_deg, grid, s, ip, sp, vcs, a, nb);
        ct_count_launch();
    }
    return (int)cudaGetLastError();
}

}  // namespace ctk
