// Exact transpose of the ray-driven projector (fp.cu) as a gather: no
// atomics, deterministic, one write per output value.
//
// The projector computes p[v,c] = w * sum_{k<n} B(x0 + k sx, y0 + k sy) with
// B the clamp-to-edge bilinear interpolation in texture coordinates (texel
// (i,j) centred at (i+1/2, j+1/2)) and (x0, y0, sx, sy, n) the ray table
// (FP/transform.cu:64-101, 119-144).  A sample in the cell between texel
// centres (ci+1/2 .. ci+3/2, cj+1/2 .. cj+3/2) gives its four corner texels
// the bilinear weights (1-fu)(1-fv), fu(1-fv), (1-fu)fv, fu fv, which are
// products of linear functions of the sample index inside the cell.
//
// Thread = one cell.  Per view it finds the few rays that can cross it, and
// for each computes the range of samples inside the cell (both neighbours of
// a cell boundary use the same threshold, so every sample lands in exactly
// one cell) and the four corner sums in closed form about the middle sample,
// times p[v,c] for up to 16 slices.  A second pass adds, per texel, the
// matching corner of its four cells.
//
// Bound: the issue slots for up to four slices (82% busy), load latency and
// the L1 data path with 16 (issue 48%, L1 72%).  Clinical geometry (512^2, 984 x
// 888), against groups of at least four slices whose loop formed the sample
// range by the step's sign and the corner sums from the first sample (us):
//   slices     1     2     4     5     8    13    16    32
//   before  2714  2695  2727  4773  3556  6141  4761  8529
//   now     1327  1521  1526  2001  2010  3024  3040  6084
// (Not kept: the next candidate's record loaded ahead, 1.84 ms for one slice;
// the record as two 16-byte loads, 3.41 ms for 16; the sinogram as planes of
// four slices, 3.11 ms; its load only after a hit, 1.42 and 3.01 ms.)
//
// Candidate rays of a view: the ray through the cell centre has fan angle
// gamma_p = atan(t/U) (the backprojector's geometry in texture units); a ray
// meets the cell only if its angle is within asin(h/L) of gamma_p, with
// h = (|cos th| + |sin th|)/2 the cell's half-width across the ray direction
// th (plus 1/L for the change of th across the range) and L the distance to
// the source.  Candidates are conservative: a ray that misses adds zero.
//
// The border cells ci = -1 and ci = nx-1 (likewise in v) extend to the FOV
// edge: the clamped taps put both of their corners on one texel, so all of
// the weight goes to that corner; they take their candidate rays from the
// angular range of their bounding box.
#include "fp_body.cuh"

namespace ctk {
namespace {

constexpr int kAdjThreads = 256;
constexpr int kAdjChunk = 64;  // slices per workspace chunk
// Warp groups of a block over the same cells, each with its share of the views:
// eight times the blocks of one group, so that a small image still fills the
// GPU and a large one ends without a long last wave (64^2, one slice: 111 ->
// 23 us; 512^2: four groups 1361 us, eight 1332).
constexpr int kAdjSplit = 8;
// Few views leave a share nothing to do, and adding the shares takes as long as 30 views
// of 16 slices: then a warp takes all views of its own patch.  512^2, 1 / 4 / 16 slices,
// us, eight shares -> one: 4 views 30 / 48 / 130 -> 17 / 28 / 62, 24 views 54 / 77 / 189
// -> 53 / 66 / 130, 32 views 64 / 85 / 203 -> 69 / 81 / 158; 256^2: 8 views 15 / 23 / 46 ->
// 17 / 23 / 35, 16 views 19 / 25 / 50 -> 25 / 33 / 48; 128^2: 8 views 16 / 17 / 21 -> 16 /
// 23 / 29.  A rule on the geometry alone, so that a slice gives the same bits in every batch.
inline bool adj_whole_views(const ct_plan *p) {
    return p->g.n_views <= 24 &&
           (long long)p->g.n_views * 8000 <= (long long)p->g.nx * p->g.ny;
}
// Resident blocks per SM (clinical geometry): one slice 1361 us with 5 (1391
// with 6, 1371 with 4), four 1538 with 4 (1646 with 5, 1690 with 3), eight
// 2033 with 4 (2168 with 3), sixteen 2969 with 2 (4630 with 1).
constexpr int adj_min_blocks(int sb) { return sb == 16 ? 2 : sb == 1 ? 5 : 4; }

struct CellArgs {
    int V, C, nx, ny;
    float coef[9];   // atan(z) = z * sum coef[k] z^(2k) on the FOV widened by 1.5 pixels
    float src;       // sid / dx (texture units)
    float fov;       // rfov / dx: the FOV disc is centred at (fov, fov)
    float left, inv_dcol;
    float chan_off;  // -left / dcol - 1/2: channel index = gamma / dcol + chan_off
    float skip_r2;   // (fov + 0.01)^2: cells whose nearest point is farther see no sample (all
                     // lie in the disc, within the rounding of a texture coordinate: 0.004
                     // at 32768 texels)
    int ring, ring_blocks;  // border cells, and their blocks (at the front of the grid)
    int px;          // interior blocks per row of blocks
};

template <int SB>
struct SinoVec {
    float v[SB];
    __device__ __forceinline__ void load(const float *__restrict__ p, bool ok) {
        if constexpr (SB == 1) {
            v[0] = CT_DLOAD(ok, p);
        } else {
#pragma unroll
            for (int q = 0; q < SB / 4; ++q) {
                const float4 t = CT_DLOAD(ok, reinterpret_cast<const float4 *>(p) + q);
                v[4 * q] = t.x;
                v[4 * q + 1] = t.y;
                v[4 * q + 2] = t.z;
                v[4 * q + 3] = t.w;
            }
        }
    }
};

// Corner sums of a cell for SB slices; slice pairs in f32x2 registers.
template <int SB>
struct Corner {
    static constexpr int NP = SB > 1 ? SB / 2 : 1;
    unsigned long long p[NP];
    float one;
    __device__ __forceinline__ void clear() {
        one = 0.0f;
#pragma unroll
        for (int s = 0; s < NP; ++s) p[s] = 0ull;
    }
    __device__ __forceinline__ void add(float w, const SinoVec<SB> &x) {
        if constexpr (SB == 1) {
            one = fmaf(w, x.v[0], one);
        } else {
            const unsigned long long ww = pack2(w, w);
#pragma unroll
            for (int s = 0; s < NP; ++s)
                p[s] = fma2(ww, pack2(x.v[2 * s], x.v[2 * s + 1]), p[s]);
        }
    }
    __device__ __forceinline__ float value(int s) const {
        if constexpr (SB == 1) return one;
        const float2 v = unpack2(p[s / 2]);
        return (s & 1) ? v.y : v.x;
    }
};

// [nb][V][C] -> [V][C][SB] (missing slices are zero): one (view, channel)
// holds its SB slices in consecutive floats.
template <int SB>
__global__ void __launch_bounds__(256)
    interleave_kernel(const float *__restrict__ sino, float *__restrict__ out, int nb,
                      size_t slice) {
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < slice;
         e += (size_t)gridDim.x * blockDim.x) {
        float v[SB];
#pragma unroll
        for (int s = 0; s < SB; ++s) v[s] = s < nb ? __ldg(sino + s * slice + e) : 0.0f;
        float4 *o = reinterpret_cast<float4 *>(out + e * SB);
#pragma unroll
        for (int q = 0; q < SB / 4; ++q)
            o[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    }
}

// The candidate channels [c0, c0 + n) of two views at once (f32x2 lanes: view
// v and v + 1) for an interior cell centred at (x, y) from the isocentre.
template <int DEG>
__device__ __forceinline__ void candidates2(float x, float y, const float4 &cs, const CellArgs &a,
                                            int c0[2], int n[2]) {
    const unsigned long long cx = pack2(cs.x, cs.z), cy = pack2(cs.y, cs.w);
    const unsigned long long x2 = pack2(x, x), y2 = pack2(y, y);
    const unsigned long long U2 = fma2(x2, cx, fma2(y2, cy, pack2(a.src, a.src)));
    const unsigned long long T2 = fma2(y2, cx, mul2(pack2(-x, -x), cy));
    const float2 U = unpack2(U2), T = unpack2(T2);
    unsigned long long g2;
    if constexpr (DEG == 0) {
        g2 = pack2(atanf(T.x / U.x), atanf(T.y / U.y));
    } else {
        const unsigned long long z =
            mul2(T2, pack2(__fdividef(1.0f, U.x), __fdividef(1.0f, U.y)));
        const unsigned long long s2 = mul2(z, z);
        unsigned long long p = pack2(a.coef[DEG], a.coef[DEG]);
#pragma unroll
        for (int k = DEG - 1; k >= 0; --k) p = fma2(p, s2, pack2(a.coef[k], a.coef[k]));
        g2 = mul2(z, p);
    }
    const unsigned long long inv = pack2(a.inv_dcol, a.inv_dcol);
    const unsigned long long cp = fma2(g2, inv, pack2(a.chan_off, a.chan_off));
    // half-width of the cell across the ray, plus the drift of its direction
    const float2 l2 = unpack2(fma2(U2, U2, mul2(T2, T2)));
    const unsigned long long rL = pack2(rsqrtf(l2.x), rsqrtf(l2.y));
    const unsigned long long mcx = pack2(-cs.x, -cs.z);
    const float2 e = unpack2(fma2(cy, T2, mul2(mcx, U2))), f = unpack2(fma2(cy, U2, mul2(cx, T2)));
    const unsigned long long h = pack2(0.5f * (fabsf(e.x) + fabsf(f.x)) + 1.0f,
                                       0.5f * (fabsf(e.y) + fabsf(f.y)) + 1.0f);
    // asin(h / L) <= z (1 + z^2), z = h / L; h is in units of 1 / rL
    const unsigned long long z = mul2(mul2(h, rL), rL);
    const unsigned long long zc = mul2(z, fma2(z, z, pack2(1.0f, 1.0f)));
    const float2 c = unpack2(cp), w = unpack2(fma2(zc, inv, pack2(0.01f, 0.01f)));
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float mid = k ? c.y : c.x, hw = k ? w.y : w.x;
        const float lo = ceil_magic(fminf(fmaxf(mid - hw, 0.0f), (float)a.C));
        const float hi = -ceil_magic(-fminf(fmaxf(mid + hw, -1.0f), (float)(a.C - 1)));
        c0[k] = __float_as_int(lo + kMagic) - kMagicInt;
        n[k] = __float_as_int(fmaxf(hi - lo + 1.0f, 0.0f) + kMagic) - kMagicInt;
    }
}

// The same for one view and a border cell, from its bounding box [u0, u1] x
// [v0, v1] (texture coordinates).
__device__ __forceinline__ void candidates_box(float u0, float u1, float v0, float v1, float2 cs,
                                               const CellArgs &a, int &c0, int &n) {
    float lo = INFINITY, hi = -INFINITY;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float x = (k & 1 ? u1 : u0) - a.fov, y = (k & 2 ? v1 : v0) - a.fov;
        const float U = fmaf(x, cs.x, fmaf(y, cs.y, a.src));
        const float T = fmaf(y, cs.x, -x * cs.y);
        const float q = (atanf(T / U) - a.left) * a.inv_dcol;
        lo = fminf(lo, q);
        hi = fmaxf(hi, q);
    }
    lo -= 0.5f + 0.01f;
    hi -= 0.5f - 0.01f;
    c0 = max(0, (int)ceilf(fmaxf(lo, -1.0f)));
    n = max(0, min(a.C - 1, (int)floorf(fminf(hi, (float)a.C))) - c0 + 1);
}

// One candidate ray of a cell [ulo, uhi) x [vlo, vhi): its samples in the
// cell, and their corner sums times the sinogram.  (a, b) is its record.
// BORDER: mu (mv) = 0 puts all of the weight at fraction bu (bv).
template <int SB, bool BORDER>
__device__ __forceinline__ void add_ray(const float4 &a, const float4 &b,
                                        const float *__restrict__ sino, bool ok,
                                        float ulo, float uhi, float vlo, float vhi, float mu,
                                        float bu, float mv, float bv, Corner<SB> w[4]) {
    // samples between the crossings of the cell's sides; both neighbours of a
    // side use the same threshold, so every sample lands in exactly one cell
    // (a zero step has 1/step = 1e30: all samples or none)
    const float tu0 = (ulo - a.x) * b.x, tu1 = (uhi - a.x) * b.x;
    const float tv0 = (vlo - a.y) * b.y, tv1 = (vhi - a.y) * b.y;
    const float lo = fmaxf(fmaxf(fminf(tu0, tu1), fminf(tv0, tv1)), 0.0f);
    const float hi = fminf(fminf(fmaxf(tu0, tu1), fmaxf(tv0, tv1)), b.z);
    SinoVec<SB> x;
    x.load(sino, ok);
    const float ka = ceil_magic(lo), cnt = ceil_magic(hi) - ka;
    if (!(cnt > 0.0f)) return;
    // fractions toward the upper corners at the middle sample, and the sums
    // of fu, fv and fu fv over the samples
    float su = a.z, sv = a.w, st = b.w;
    float fu = fmaf(ka, su, a.x) - ulo, fv = fmaf(ka, sv, a.y) - vlo;
    if constexpr (BORDER) {
        fu = mu != 0.0f ? fu : bu;
        fv = mv != 0.0f ? fv : bv;
        su *= mu;
        sv *= mv;
        st *= mu * mv;
    }
    const float h = fmaf(cnt, 0.5f, -0.5f);
    const float xh = fmaf(su, h, fu), yh = fmaf(sv, h, fv);
    const float F = cnt * xh, G = cnt * yh;
    const float P = fmaf(F, yh, cnt * st * fmaf(cnt, cnt, -1.0f));
    const float W01 = G - P;
    w[0].add((cnt - F) - W01, x);
    w[1].add(F - P, x);
    w[2].add(W01, x);
    w[3].add(P, x);
}

// A warp takes a patch of 4 x 8 cells (whose cells see more similar candidate
// counts than a 32-cell row's).  A block is eight warps, KS over the same patch,
// on 8 / KS patches: warp g of a patch takes the view pairs g, g + KS, ...  With
// KS > 1 the warps' sums are added in shared memory at the end, in order.  The
// first ring_blocks blocks take the border cells, 256 / KS each.
template <int SB, int DEG, int KS>
__global__ void __launch_bounds__(kAdjThreads, adj_min_blocks(SB))
    fp_adjoint_cells_kernel(const float *__restrict__ sino, float *__restrict__ corners,
                            const float4 *__restrict__ ray_rec,
                            const float2 *__restrict__ view_cs, CellArgs a, int nsl) {
    constexpr int CELLS = kAdjThreads / KS;
    const int NXC = a.nx + 1, NYC = a.ny + 1;
    const int group = threadIdx.x / CELLS, cell = threadIdx.x - group * CELLS;
    const bool border = (int)blockIdx.x < a.ring_blocks;  // block-uniform
    int ic, jc;
    bool inside;
    if (border) {
        // the rows jc = 0 and ny, then the columns ic = 0 and nx between them
        int e = blockIdx.x * CELLS + cell;
        inside = e < a.ring;
        if (e < 2 * NXC) {
            ic = e % NXC;
            jc = e / NXC * a.ny;
        } else {
            e -= 2 * NXC;
            jc = 1 + e % max(1, NYC - 2);
            ic = e / max(1, NYC - 2) * a.nx;
        }
    } else {
        const int blk = blockIdx.x - a.ring_blocks;
        const int by = blk / a.px, bx = blk - by * a.px;
        if constexpr (KS == 1) {  // the block's patches: four across, two down
            const int patch = cell >> 5, ln = cell & 31;
            ic = 1 + (4 * bx + (patch & 3)) * 4 + (ln & 3);
            jc = 1 + (2 * by + (patch >> 2)) * 8 + (ln >> 2);
        } else {
            ic = 1 + bx * 4 + (cell & 3);
            jc = 1 + by * 8 + (cell >> 2);
        }
        inside = ic < a.nx && jc < a.ny;
    }
    const int ci = ic - 1, cj = jc - 1;
    const bool xlo = ci == -1, xhi = ci == a.nx - 1, ylo = cj == -1, yhi = cj == a.ny - 1;
    const float ulo0 = (float)ci + 0.5f, vlo0 = (float)cj + 0.5f;
    // cell span [lo, hi) in texture coordinates: the border cells reach to the
    // FOV edge
    const float ulo = xlo ? -INFINITY : ulo0, uhi = xhi ? INFINITY : (float)ci + 1.5f;
    const float vlo = ylo ? -INFINITY : vlo0, vhi = yhi ? INFINITY : (float)cj + 1.5f;
    // the cell's nearest point to the isocentre
    const float nu = fmaxf(fmaxf(ulo - a.fov, a.fov - uhi), 0.0f);
    const float nv = fmaxf(fmaxf(vlo - a.fov, a.fov - vhi), 0.0f);
    const bool act = inside && nu * nu + nv * nv <= a.skip_r2;
    Corner<SB> w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k].clear();
    const bool block_act = __syncthreads_or(act);
    if (act && !border) {
        const float x = (float)ci + 1.0f - a.fov, y = (float)cj + 1.0f - a.fov;
        for (int v = 2 * group; v < a.V; v += 2 * KS) {
            // the last view of an odd number is paired with itself, without candidates
            const bool two = v + 1 < a.V;
            const float2 ca = __ldg(view_cs + v), cb = __ldg(view_cs + (two ? v + 1 : v));
            int c0[2], n[2];
            candidates2<DEG>(x, y, make_float4(ca.x, ca.y, cb.x, cb.y), a, c0, n);
            if (!two) n[1] = 0;
            // one loop over both views' candidates: a warp iterates the maximum
            // of its lanes' totals (32 clinical slices: one view per loop 10.0
            // against 8.4 ms, four or eight views 9.0 / 9.8 ms)
            const int ra = v * a.C + c0[0], rb = (v + 1) * a.C + c0[1] - n[0];
            const int tot = n[0] + n[1];
            for (int t = 0; t < tot; ++t) {
                const int r = t + (t < n[0] ? ra : rb);
                const bool ok = (unsigned)r < (unsigned)(a.V * a.C);
                float4 p, q;
                ldg_v8(ok, ray_rec + 2 * (size_t)r, p, q);
                add_ray<SB, false>(p, q, sino + (size_t)r * SB, ok, ulo, uhi, vlo, vhi, 1.0f,
                                   0.0f, 1.0f, 0.0f, w);
            }
        }
    } else if (act) {
        const float u0 = xlo ? -1.0f : ulo, u1 = xhi ? 2.0f * a.fov + 1.0f : uhi;
        const float v0 = ylo ? -1.0f : vlo, v1 = yhi ? 2.0f * a.fov + 1.0f : vhi;
        // all of the weight goes to the corner inside the image; a cell that is
        // both first and last (a one-texel axis) never occurs: it has two cells
        const float mu = xlo || xhi ? 0.0f : 1.0f, bu = xlo ? 1.0f : 0.0f;
        const float mv = ylo || yhi ? 0.0f : 1.0f, bv = ylo ? 1.0f : 0.0f;
        for (int v = group; v < a.V; v += KS) {
            int c0, n;
            candidates_box(u0, u1, v0, v1, __ldg(view_cs + v), a, c0, n);
            for (int t = 0; t < n; ++t) {
                const int r = v * a.C + c0 + t;
                const bool ok = (unsigned)r < (unsigned)(a.V * a.C);
                float4 p, q;
                ldg_v8(ok, ray_rec + 2 * (size_t)r, p, q);
                add_ray<SB, true>(p, q, sino + (size_t)r * SB, ok, ulo, uhi, vlo, vhi, mu, bu, mv, bv, w);
            }
        }
    }
    const size_t plane = (size_t)NXC * NYC, o = (size_t)jc * NXC + ic;
    if constexpr (KS == 1) {
        if (!inside) return;
#pragma unroll
        for (int s = 0; s < SB; ++s) {
            if (s >= nsl) break;  // uniform
#pragma unroll
            for (int k = 0; k < 4; ++k) corners[(size_t)(4 * s + k) * plane + o] = w[k].value(s);
        }
        return;
    }
    // the groups' sums, slice by slice
    __shared__ float4 part[KS][CELLS];
    if (!block_act) {
        if (inside && group == 0)
            for (int s = 0; s < nsl; ++s)
                for (int k = 0; k < 4; ++k) corners[(size_t)(4 * s + k) * plane + o] = 0.0f;
        return;
    }
#pragma unroll
    for (int s = 0; s < SB; ++s) {
        if (s >= nsl) break;  // uniform
        __syncthreads();
        part[group][cell] =
            make_float4(w[0].value(s), w[1].value(s), w[2].value(s), w[3].value(s));
        __syncthreads();
        if (inside && group == 0) {
            float4 t = part[0][cell];
#pragma unroll
            for (int g = 1; g < KS; ++g) {
                const float4 e = part[g][cell];
                t.x += e.x;
                t.y += e.y;
                t.z += e.z;
                t.w += e.w;
            }
            float *cb = corners + (size_t)4 * s * plane + o;
            cb[0] = t.x;
            cb[plane] = t.y;
            cb[2 * plane] = t.z;
            cb[3 * plane] = t.w;
        }
    }
}

// texel (i, j) = corner 00 of cell (i, j) + 10 of (i-1, j) + 01 of (i, j-1)
// + 11 of (i-1, j-1), times the projector weight
__global__ void __launch_bounds__(256)
    fp_adjoint_combine_kernel(const float *__restrict__ corners, float *__restrict__ img, int nx,
                              int ny, float w, int batch) {
    const int NXC = nx + 1, NYC = ny + 1;
    const size_t plane = (size_t)NXC * NYC;
    const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y;
    if (i >= nx || j >= ny) return;
    for (int b = blockIdx.z; b < batch; b += gridDim.z) {
        const float *cb = corners + (size_t)b * 4 * plane;
        const size_t o00 = (size_t)(j + 1) * NXC + (i + 1);  // cell (i, j)
        const float t = cb[o00] + cb[plane + o00 - 1] + cb[2 * plane + o00 - NXC] +
                        cb[3 * plane + o00 - NXC - 1];
        img[(size_t)b * nx * ny + (size_t)j * nx + i] = t * w;
    }
}

// Slices a group's kernel takes (unused ones are zeros): the smallest that holds
// the rest.
int adj_slices(int nb) { return nb > 8 ? 16 : nb > 4 ? 8 : nb > 1 ? 4 : 1; }

size_t corner_bytes(const ct_plan *p, int nb) {
    return (4 * (size_t)nb * (p->g.nx + 1) * (p->g.ny + 1) * sizeof(float) + 255) / 256 * 256;
}

template <int SB>
void launch_cells(int deg, int split, unsigned blocks, cudaStream_t s, const float *sino,
                  float *corners, const float4 *rec, const float2 *vcs, const CellArgs &a, int nsl) {
    auto go = [&](auto kern) {
        kern<<<blocks, kAdjThreads, 0, s>>>(sino, corners, rec, vcs, a, nsl);
    };
    // (a degree-4 fit is the degree-8 polynomial with zero high coefficients)
    if (split == 1)
        deg ? go(fp_adjoint_cells_kernel<SB, 8, 1>) : go(fp_adjoint_cells_kernel<SB, 0, 1>);
    else if (deg == 4)
        go(fp_adjoint_cells_kernel<SB, 4, kAdjSplit>);
    else if (deg == 8)
        go(fp_adjoint_cells_kernel<SB, 8, kAdjSplit>);
    else
        go(fp_adjoint_cells_kernel<SB, 0, kAdjSplit>);
}

template <int SB>
void launch_group(int sms, int deg, int split, unsigned blocks, cudaStream_t s, const float *sino,
                  float *inter, float *corners, const float4 *rec, const float2 *vcs,
                  const CellArgs &a, int nsl) {
    const size_t slice = (size_t)a.V * a.C;
    if constexpr (SB > 1) {
        const size_t want = (slice + 255) / 256, most = (size_t)sms * 16;
        interleave_kernel<SB><<<(unsigned)(want < most ? want : most), 256, 0, s>>>(
            sino, inter, nsl, slice);
        ct_count_launch();
        sino = inter;
    }
    launch_cells<SB>(deg, split, blocks, s, sino, corners, rec, vcs, a, nsl);
    ct_count_launch();
}

}  // namespace

size_t fp_fan_adjoint_work_bytes(const ct_plan *p, int batch) {
    const int chunk = batch < kAdjChunk ? batch : kAdjChunk;
    // corner sums of a chunk, then one group's interleaved sinogram
    const int sb = adj_slices(chunk);
    return corner_bytes(p, chunk) +
           (sb > 1 ? sizeof(float) * sb * (size_t)p->g.n_views * p->g.n_cols : 0);
}

int fp_fan_adjoint(const ct_plan *p, const float *sino, float *img, int batch, void *work,
                   void *stream) {
    CellArgs a;
    a.V = p->g.n_views;
    a.C = p->g.n_cols;
    a.nx = p->g.nx;
    a.ny = p->g.ny;
    const double dx = p->g.dx;
    a.src = (float)((double)p->g.sid / dx);
    const double fov = (double)p->g.rfov / dx;
    a.fov = (float)fov;
    a.left = p->g.left;
    a.inv_dcol = (float)(1.0 / (double)p->g.dcol);
    a.chan_off = (float)(-(double)p->g.left / (double)p->g.dcol - 0.5);
    a.skip_r2 = (float)((fov + 0.01) * (fov + 0.01));
    for (int k = 0; k < 9; ++k) a.coef[k] = p->gather_atan_coef[k];
    const int deg = p->gather_atan_deg;
    const float2 *vcs = reinterpret_cast<const float2 *>(p->d_view_cs);
    const float4 *rrec = reinterpret_cast<const float4 *>(p->d_ray_rec);
    cudaStream_t s = (cudaStream_t)stream;
    const size_t plane = (size_t)a.nx * a.ny, slice = (size_t)a.V * a.C;
    const size_t cplane = (size_t)(a.nx + 1) * (a.ny + 1);
    a.ring = 2 * (a.nx + 1) + 2 * (a.ny - 1);
    const int split = adj_whole_views(p) ? 1 : kAdjSplit;
    const int cells = kAdjThreads / split, bw = split == 1 ? 16 : 4, bh = cells / bw;
    a.ring_blocks = (a.ring + cells - 1) / cells;
    a.px = (a.nx - 1 + bw - 1) / bw;
    const unsigned blocks = (unsigned)(a.ring_blocks + a.px * ((a.ny - 1 + bh - 1) / bh));
    for (int b0 = 0; b0 < batch; b0 += kAdjChunk) {
        const int nb = batch - b0 < kAdjChunk ? batch - b0 : kAdjChunk;
        float *corners = static_cast<float *>(work);
        float *inter = reinterpret_cast<float *>(static_cast<char *>(work) + corner_bytes(p, nb));
        for (int k = 0; k < nb;) {
            const int sb = adj_slices(nb - k), nsl = nb - k < sb ? nb - k : sb;
            const float *sp = sino + (size_t)(b0 + k) * slice;
            float *cp = corners + (size_t)k * 4 * cplane;
            if (sb == 16)
                launch_group<16>(p->sms, deg, split, blocks, s, sp, inter, cp, rrec, vcs, a, nsl);
            else if (sb == 8)
                launch_group<8>(p->sms, deg, split, blocks, s, sp, inter, cp, rrec, vcs, a, nsl);
            else if (sb == 4)
                launch_group<4>(p->sms, deg, split, blocks, s, sp, inter, cp, rrec, vcs, a, nsl);
            else
                launch_group<1>(p->sms, deg, split, blocks, s, sp, inter, cp, rrec, vcs, a, nsl);
            k += nsl;
        }
        fp_adjoint_combine_kernel<<<dim3((a.nx + 31) / 32, (a.ny + 7) / 8, nb), dim3(32, 8), 0,
                                    s>>>(corners, img + b0 * plane, a.nx, a.ny, p->fp_weight, nb);
        ct_count_launch();
    }
    return (int)cudaGetLastError();
}

}  // namespace ctk
