// Ray-driven fan-beam forward projector (its transpose is in fp_adjoint.cu).
//
// Forward (replaces FP/transform.cu:103-146 and the per-view launch loop
// :162-169): all views and slices of a group in one launch.  Each launch first
// builds texel images (the padded image in both layouts, up to eight slices
// per texel), then fp_warp (fp_body.cuh) walks 32 adjacent rays of a view per
// warp, row by row, and adds every texel a ray touches once, with the sum of
// its samples' bilinear weights in closed form.  Output:
// p = 0.125*dx * sum_k bilinear_clamp(img, start + k*step), k < n.
//
// Bound: the issue slots for up to four slices (87% busy: the weights of a
// row are formed whatever the group), the L1 data path beyond (a warp's
// 32-byte loads take 8.4 of its cycles each; 81% busy with 16 slices).
// Clinical geometry (512^2, 984 x 888), against a walk that gathered four
// taps per cell from float4 quad images (us per call):
//   slices     1     2     4     5     8    13    16    32
//   before  1054  2036  1568  2618  2340  4958  4333  8476
//   now      657   715   824  1056  1060  1819  1824  3646
#include <cstdint>

#include "fp_body.cuh"

namespace ctk {
namespace {

// A block is one 32-channel group of one view, its four warps a quarter of the
// rows each (a small image's rays are too few to fill the GPU, and a large
// one's blocks end sooner): clinical geometry, against four adjacent views per
// block, each warp walking all rows: one slice 661 -> 645 us, sixteen 1955 ->
// 1834; 256^2 131 -> 114 us, 64^2 28 -> 15 us; two quarters per warp 640 us and
// 21.  Blocks run channel-group-major: the resident ones cover a few channel
// groups of every view, whose rays cross nearly the same texels.  (Blocks of one
// layout first: no faster.)
constexpr int kFpThreads = 32 * kFpParts;
constexpr int kFpChunk = 64;  // slices per texel-image workspace chunk
// Planes of eight slices per walk: the weights of a row are shared by 16
// slices.  Three or four planes hold 204 and 228 registers and measured
// slower (32 slices: 4.05 ms against two walks' 3.89, both without totals).
constexpr int kFpMaxPlanes = 2;
// Resident blocks per SM, swept on the clinical geometry: one slice 645 us with
// 9 (652 with 8, 674 with 10), two 713 with 10 (720 with 9), four 823 with 7
// (826 with 8, 836 with 9), eight 1059 with 7 (1064 with 6, 1092 with 5), sixteen
// 1834 with 4 (2188 with 3).
constexpr int fp_min_blocks(int ts, int np) {
    return ts == 1 ? 9 : ts == 2 ? 10 : ts == 4 ? 7 : np == 1 ? 7 : 4;
}

template <int TS>
__device__ __forceinline__ void store_texel(float *dst, const float *v) {
    if constexpr (TS == 1) {
        dst[0] = v[0];
    } else if constexpr (TS == 2) {
        *reinterpret_cast<float2 *>(dst) = make_float2(v[0], v[1]);
    } else {
#pragma unroll
        for (int k = 0; k < TS / 4; ++k)
            reinterpret_cast<float4 *>(dst)[k] =
                make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    }
}
// Texel images of slice groups of TS: blockIdx.z is group z (slices z TS ..,
// zero past `batch`), both layouts, from a 32 x 32 texel tile staged in shared
// memory so that both are read and written coalesced.
template <int TS>
__global__ void __launch_bounds__(256)
    build_texels_kernel(const float *__restrict__ img, float *__restrict__ tex, int nx, int ny,
                        int batch) {
    __shared__ float tile[TS][32][33];
    const int P = nx + 2;
    const int TX = blockIdx.x * 32, TY = blockIdx.y * 32, z = blockIdx.z;
    const size_t plane = (size_t)nx * ny, lay = (size_t)P * P * TS;
    float *t0 = tex + (size_t)z * 2 * lay, *t1 = t0 + lay;
    const int i = threadIdx.x;
    const int x = min(max(TX + i - 1, 0), nx - 1);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int j = threadIdx.y + 8 * r;
        const int y = min(max(TY + j - 1, 0), ny - 1);
        float v[TS];
#pragma unroll
        for (int k = 0; k < TS; ++k) {
            const int b = z * TS + k;
            v[k] = b < batch ? __ldg(img + (size_t)b * plane + (size_t)y * nx + x) : 0.0f;
            tile[k][j][i] = v[k];
        }
        if (TX + i < P && TY + j < P) store_texel<TS>(t0 + ((size_t)(TY + j) * P + TX + i) * TS, v);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int j = threadIdx.y + 8 * r;  // layout 1: row x = TX + j, column y = TY + i
        float v[TS];
#pragma unroll
        for (int k = 0; k < TS; ++k) v[k] = tile[k][i][j];
        if (TY + i < P && TX + j < P) store_texel<TS>(t1 + ((size_t)(TX + j) * P + TY + i) * TS, v);
    }
}

template <int TS, int NP>
__global__ void __launch_bounds__(kFpThreads, fp_min_blocks(TS, NP))
    fp_fan_kernel(const char *__restrict__ tex, float *__restrict__ sino,
                  const float4 *__restrict__ ray, const int *__restrict__ nsamp, int V, int C,
                  int wpv, int nx, float w, int batch) {
    __shared__ unsigned long long totals[TS > 1 ? TS * NP / 2 * kFpThreads : kFpThreads / 2];
    TexelImages im;
    im.layout = (size_t)(nx + 2) * (nx + 2) * TS * sizeof(float);
    im.plane = 2 * im.layout;
    im.base = tex;
    const int cg = blockIdx.x / V, v = blockIdx.x - cg * V;
    fp_warp<TS, NP>(im, sino, (size_t)V * C, ray, nsamp, V, C, wpv, nx, w, batch, v * wpv + cg,
                    totals, warp_index());
}

}  // namespace

// Slices per texel: the smallest group that holds the batch, planes of eight
// beyond four (a group's unused slices are zeros that are walked along: three
// slices as four take 856 us, where groups of two and one took 748 + 661).
int fp_texel_slices(int nb) { return nb >= 5 ? 8 : (nb >= 3 ? 4 : nb); }

size_t fp_fan_work_bytes(const ct_plan *p, int batch) {
    const size_t P = (size_t)p->g.nx + 2;
    const int chunk = batch < kFpChunk ? batch : kFpChunk;
    const int ts = fp_texel_slices(chunk);
    const size_t groups = ts ? (size_t)((chunk + ts - 1) / ts) : 0;
    // + 16 bytes to start the 32-byte texels on a 32-byte boundary
    return groups * ts * 2 * P * P * sizeof(float) + 16;
}

int fp_fan(const ct_plan *p, const float *img, float *sino, int batch, void *work,
           void *stream) {
    const int V = p->g.n_views, C = p->g.n_cols;
    const int nx = p->g.nx, ny = p->g.ny;
    const size_t plane = (size_t)nx * ny;
    const size_t n_rays = (size_t)V * C;
    const float4 *ray = reinterpret_cast<const float4 *>(p->d_ray);
    // 32-byte texels read by 32-byte loads (the workspace is 16-byte aligned)
    float *tex = reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(work) + 31) &
                                           ~(uintptr_t)31);
    cudaStream_t s = (cudaStream_t)stream;
    const int wpv = (C + 31) / 32;
    const int P = nx + 2;
    const size_t texels = 2 * (size_t)P * P;  // of one plane
    // chunks of at most kFpChunk slices share the workspace
    for (int c0 = 0; c0 < batch; c0 += kFpChunk) {
        const int nb = batch - c0 < kFpChunk ? batch - c0 : kFpChunk;
        const int ts = fp_texel_slices(nb), planes = (nb + ts - 1) / ts;
        const dim3 bgrid((P + 31) / 32, (P + 31) / 32, planes), bblock(32, 8);
        const float *src = img + (size_t)c0 * plane;
        auto build = [&](auto kern) { kern<<<bgrid, bblock, 0, s>>>(src, tex, nx, ny, nb); };
        ts == 8 ? build(build_texels_kernel<8>)
                : ts == 4 ? build(build_texels_kernel<4>)
                          : ts == 2 ? build(build_texels_kernel<2>) : build(build_texels_kernel<1>);
        ct_count_launch();
        for (int k = 0; k < planes;) {
            const int np = planes - k < kFpMaxPlanes ? planes - k : kFpMaxPlanes;
            const int b0 = c0 + k * ts, left = nb - k * ts;
            auto go = [&](auto kern) {
                kern<<<V * wpv, kFpThreads, 0, s>>>(
                    reinterpret_cast<const char *>(tex + (size_t)k * texels * ts),
                    sino + (size_t)b0 * n_rays, ray, p->d_nsamp, V, C, wpv, nx, p->fp_weight,
                    left);
            };
            if (ts == 1)
                go(fp_fan_kernel<1, 1>);
            else if (ts == 2)
                go(fp_fan_kernel<2, 1>);
            else if (ts == 4)
                go(fp_fan_kernel<4, 1>);
            else if (np == 1)
                go(fp_fan_kernel<8, 1>);
            else
                go(fp_fan_kernel<8, 2>);
            ct_count_launch();
            k += np;
        }
    }
    return (int)cudaGetLastError();
}

}  // namespace ctk
