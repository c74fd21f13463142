// Nonlocal projectors on the FP64 tensor cores (mma.sync.m8n8k4.f64): the gather-contraction
//   c[a,ch][s] = E_ch dV sum_p P_ch(p) psi_s(g(p))
// of real FP64 and of k-point states, and the scatter  H u_s(g) += sum_{a,ch} conj(P_ch(p)) c[a,ch][s]
// of k-point states (ProjectionPP, PseudoPotOperator.h:740-772; PseudoPotOperator_kpoint_v2.h:2581-2700).
//
// The grid is cut into bricks of 16 x 8 x 4 points = 64 blocks of 8 consecutive x. Every
// sphere that meets a block stores its 4 channels x 8 points there, zero outside the sphere
// (35 % more values than sphere points on the diamond cells), so that one m8n8k4 product is
//   project: 8 states x 4 points  *  4 points x (2 spheres x 4 channels)
//   scatter: 8 states x 4 channels  *  4 channels x 8 points
// with no index list: the operand of 8 states x 8 points is a 16-byte load per lane, shared by
// all spheres that cover the block, and both passes read the same table. A sphere's values in a
// brick take one of 8 slots of an item (pairs of spheres that cover the same blocks side by
// side); a brick with more spheres has more items.
//   k_brick_project  a thread block per (item, 64 states) keeps the item's table in shared
//                    memory, each warp sums 8 states over the brick in registers;
//   k_brick_reduce   a coefficient is the sum of its sphere's brick partials in list order,
//                    whatever the batch, so a state's result does not depend on its batch;
//   k_brick_scatter  a thread block per (brick, 64 states), the coefficients in registers, H u
//                    read and written once per item.
// FP32 states are widened as they are used: the sums and the coefficients are FP64 for both types.
//
// k-points: P(p) = table(p) exp(i g.u) at the unwrapped coordinate u = r + (image) L, so the
// phase is that of the grid point times one number per image. Re and im rows are rotated by
// the grid point's phase after the load (and back before the store), the image's phase multiplies
// the brick's partial sums: the table stays real and is the same for every k-point (a table of
// Bloch phases per k-point, as the kernels these replace read, is 14 MB for 8 atoms).
//
// Measured, projection (with its sums) / scatter: 64 complex128 states of 80^3 0.26 / 0.28 ms
// (atom by atom and point by point: 0.41 / 0.33), 64 k-points x 16 complex64 states of 40^3
// 0.42 / 0.39 (0.58 / 0.61); real FP64, 256 states of 80^3 0.36 ms against 0.49, 528 of 120^3 2.71
// against 3.71, where the atom-by-atom kernel reads psi 2.65 times from DRAM. Real states keep
// their scatter by pairs of points (0.44 ms; this form 0.68) and FP32 the atom-by-atom projection
// (0.31; 0.34): there the 64- and 32-byte pieces of a load limit the bricks.
//
// A state with a NaN or Inf at a point spreads it to every sphere that meets the point's block
// (0 * NaN), up to 7 points further in x than the sphere itself.
#include "nonlocal.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "stencil_common.cuh"

namespace qg {
namespace {

constexpr int kBx = 16, kBy = 8, kBz = 4;  // brick; block b of row y: x half b & 1, plane b >> 1
constexpr int kThreads = 256;              // 8 warps
constexpr int kSlots = 8;                  // channel groups of an item (4 pairs)
constexpr int kMaxTab = 160;               // table blocks (512 B) of an item: two thread blocks fit an SM
// Partial sums of one slice of the states (a state of the 64-atom 80^3 cell has 165 KB): past
// it the projection goes slice by slice, which changes no bit.
constexpr size_t kPartBytes = size_t(192) << 20;

typedef unsigned long long u64;

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

template <typename T> struct Pair;
template <> struct Pair<double> { using type = double2; };
template <> struct Pair<float> { using type = float2; };

// Two x-neighbours of one state, zero past the row's end (x = the first point's coordinate); kept
// in their own type until they are used, so that nothing waits for the load before that.
template <typename T, bool VEC>
__device__ __forceinline__ typename Pair<T>::type load_pair(const T* p, int x, int nx) {
    typename Pair<T>::type v;
    v.x = v.y = T(0);
    if constexpr (VEC) {  // nx is even
        if (x < nx) v = *reinterpret_cast<const typename Pair<T>::type*>(p);
    } else {
        if (x < nx) v.x = p[0];
        if (x + 1 < nx) v.y = p[1];
    }
    return v;
}

template <typename T, bool VEC>
__device__ __forceinline__ void store_pair(T* p, const double (&v)[2], int x, int nx) {
    if constexpr (VEC) {
        if (x < nx) {
            if constexpr (sizeof(T) == 8) *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
            else *reinterpret_cast<float2*>(p) = make_float2((float)v[0], (float)v[1]);
        }
    } else {
        if (x < nx) p[0] = T(v[0]);
        if (x + 1 < nx) p[1] = T(v[1]);
    }
}

struct BrickGeom {
    int nx, ny, nz, nbx, nby;
    const int* item_brick;   // brick of an item
    const int* item_pair;    // [nitems + 1] first partial-sum block (pair) of an item
    const int* item_cg;      // [nitems * 8] coefficient group of a slot, -1: none
    const int* item_img;     // [nitems * 8] periodic image of a slot
    const u64* wmask;        // [nitems * 8 rows] bit 8 b + slot: the slot covers block b
    const int* wtab;         // [nitems * 8 rows + 1] first table block (64 doubles) of the row
    const int* brick_item;   // [nbricks + 1] items of a brick
    const double* tab;       // [pair of slots in a block][8 columns][8 points]
};

// Phase of the two points of a lane in block b, from the axes' phases of one k-point.
struct LanePhase {
    double2 px[2][2], pyz;
    const double2* pz;
    __device__ __forceinline__ void init(const double2* ph, const BrickGeom& g, int x, int y, int z0) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 2; ++e) px[h][e] = ph[min(x + 8 * h + e, g.nx - 1)];
        pyz = ph[g.nx + min(y, g.ny - 1)];
        pz = ph + g.nx + g.ny + z0;
    }
    __device__ __forceinline__ static double2 mul(double2 a, double2 b) {
        return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
    }
    __device__ __forceinline__ void at(int b, double2 (&o)[2]) const {
        const double2 w = mul(pyz, pz[b >> 1]);
        o[0] = mul(px[b & 1][0], w);
        o[1] = mul(px[b & 1][1], w);
    }
};

// The item's table into shared memory, 16 bytes per thread and step; table_ready waits for it.
__device__ __forceinline__ void fetch_table(double* tb, const BrickGeom& g, int item) {
    const int w0 = g.wtab[item * 8], w1 = g.wtab[item * 8 + 8];
    const double* src = g.tab + (long long)w0 * 64;
    for (int i = threadIdx.x; i < (w1 - w0) * 32; i += kThreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(tb + 2 * i)),
                     "l"(src + 2 * i)
                     : "memory");
}
__device__ __forceinline__ void table_ready() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}

// A unit is 8 states, of several k-points where they follow one another (the phase is the lane's): one
// group of 8 rows (real) or two, re and im (complex). ROWS: the 8
// warps take one row of the brick each for one unit (few units: more warps per state);
// otherwise they take one unit each and walk the whole brick, the table in shared memory. Both
// add a row's blocks first and then the rows in order, so the sums are the same to the bit.
// Bound: the FP64 tensor pipe (65 % busy for real, 50 for complex128, 58 for complex64 states) and the
// 64-byte pieces of the loads (3.2 TB/s of psi at 64 real states of 80^3); D blocks of states are in flight per
// warp. Two blocks per SM leave 128 registers, where the complex forms that walk the whole brick spill 28 to 84
// bytes.
template <typename T, bool CPLX, bool VEC, bool ROWS, int D>
__global__ void __launch_bounds__(kThreads, 2)
    k_brick_project(const T* __restrict__ X, long long ldx, long long ldk, long long xim, int ns, int nrow,
                    int unit0, int nunit, const BrickGeom g, const double2* __restrict__ phase, int nphase,
                    double* __restrict__ part, long long prow) {
    constexpr int S = CPLX ? 2 : 1;
    extern __shared__ __align__(16) double tb[];
    __shared__ double red[ROWS ? 8 : 1][ROWS ? S * 4 * 64 : 1];
    allow_next();
    const int chunks = ROWS ? nunit : (nunit + 7) / 8;
    const int item = blockIdx.x / chunks, ch = blockIdx.x - item * chunks;
    const int brick = g.item_brick[item];
    const int bx = brick % g.nbx, by = (brick / g.nbx) % g.nby, bz = brick / (g.nbx * g.nby);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
    const int np = g.item_pair[item + 1] - g.item_pair[item];
    const int ul = ROWS ? ch : ch * 8 + w;            // unit of this warp within the launch
    const int u = unit0 + min(ul, nunit - 1);
    const int row_r = min(u * 8 + r, nrow - 1), k = row_r / ns, s = row_r - k * ns;  // this lane's state
    const int x = bx * kBx + 2 * q, y0 = by * kBy, z0 = bz * kBz;
    const long long plane = (long long)g.nx * g.ny;
    const T* base = X + (long long)k * ldk + (long long)s * ldx + (x + (long long)g.nx * y0 + plane * z0);
    const double2* ph = CPLX ? phase + (long long)k * nphase : nullptr;

    using P2 = typename Pair<T>::type;
    P2 a[D][S];
    auto fetch = [&](u64 m, int row, int b, P2 (&v)[S]) {
        if ((m >> (8 * b)) & 255) {
            const T* p = base + (long long)row * g.nx + (b & 1) * 8 + (b >> 1) * plane;
#pragma unroll
            for (int i = 0; i < S; ++i) v[i] = load_pair<T, VEC>(p + (i ? xim : 0), x + (b & 1) * 8, g.nx);
        }
    };
    const int row_a = ROWS ? w : 0, row_b = ROWS ? w + 1 : 8;
    u64 mn = g.wmask[item * 8 + row_a];
#pragma unroll
    for (int d = 0; d < D - 1; ++d) fetch(mn, row_a, d, a[d]);
    fetch_table(tb, g, item);
    table_ready();
    const double* tp = tb + (g.wtab[item * 8 + row_a] - g.wtab[item * 8]) * 64 + 2 * lane;

    double tot[S][4][2];
    LanePhase lp;
    for (int row = row_a; row < row_b; ++row) {
        const u64 m = mn;
        mn = row + 1 < row_b ? g.wmask[item * 8 + row + 1] : 0;
        if constexpr (CPLX) lp.init(ph, g, x, y0 + row, z0);
        double acc[S][4][2];
#pragma unroll
        for (int i = 0; i < S; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            if (b + D - 1 < 8) fetch(m, row, b + D - 1, a[(b + D - 1) % D]);
            else fetch(mn, row + 1, b + D - 1 - 8, a[(b + D - 1) % D]);
            const unsigned mb = (unsigned)(m >> (8 * b)) & 255u;
            if (mb) {
                double v[S][2];
#pragma unroll
                for (int i = 0; i < S; ++i) {
                    v[i][0] = (double)a[b % D][i].x;
                    v[i][1] = (double)a[b % D][i].y;
                }
                if constexpr (CPLX) {
                    double2 e2[2];
                    lp.at(b, e2);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const double re = v[0][e], im = v[S - 1][e];
                        v[0][e] = e2[e].x * re - e2[e].y * im;
                        v[S - 1][e] = e2[e].y * re + e2[e].x * im;
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (mb >> (2 * j) & 3) {
                        const double2 t = *reinterpret_cast<const double2*>(tp);
                        tp += 64;
#pragma unroll
                        for (int i = 0; i < S; ++i) {
                            dmma(acc[i][j], v[i][0], t.x);
                            dmma(acc[i][j], v[i][1], t.y);
                        }
                    }
            }
        }
        if constexpr (ROWS) {
#pragma unroll
            for (int i = 0; i < S; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    *reinterpret_cast<double2*>(&red[w][(j * S + i) * 64 + 2 * lane]) = make_double2(acc[i][j][0], acc[i][j][1]);
        } else {
#pragma unroll
            for (int i = 0; i < S; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int e = 0; e < 2; ++e) tot[i][j][e] = row == 0 ? acc[i][j][e] : tot[i][j][e] + acc[i][j][e];
        }
    }
    const long long pair0 = g.item_pair[item];
    if constexpr (ROWS) {
        __syncthreads();
        for (int t = threadIdx.x; t < S * np * 64; t += kThreads) {
            double v = red[0][t];
#pragma unroll
            for (int i = 1; i < 8; ++i) v += red[i][t];
            const int j = t / (S * 64), i = (t / 64) % S;
            part[((pair0 + j) * prow + ((long long)ul * S + i) * 8) * 8 + t % 64] = v;
        }
    } else if (ul < nunit) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < np) {
#pragma unroll
                for (int i = 0; i < S; ++i)
                    *reinterpret_cast<double2*>(&part[((pair0 + j) * prow + ((long long)ul * S + i) * 8) * 8 + 2 * lane]) =
                        make_double2(tot[i][j][0], tot[i][j][1]);
            }
    }
}

// One coefficient group x 8 states: the 8 warps add contiguous eighths of the group's partial
// sums, then warp 0's lanes add the eighths in order. refs: {2 * pair + half, image}.
template <bool CPLX>
__global__ void __launch_bounds__(kThreads)
    k_brick_reduce(const double* part, long long prow, const int* __restrict__ cg_off,
                   const int2* __restrict__ cg_ref, int ns, int nrow, int unit0, const double2* __restrict__ phase,
                   int nphase, int img0, const double* __restrict__ scale, double* __restrict__ coef, long long rows) {
    __shared__ double sm[8][2][32];
    allow_next();
    const int cg = blockIdx.x, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long u = unit0 + blockIdx.y;
    const int k = (int)min(u * 8 + (lane >> 2), (long long)nrow - 1) / ns;
    const int r0 = cg_off[cg], n = cg_off[cg + 1] - r0;
    const int b0 = r0 + n * w / 8, b1 = r0 + n * (w + 1) / 8;
    const long long row = (long long)blockIdx.y * (CPLX ? 16 : 8) + (lane >> 2);
    wait_previous();  // part through plain loads: the read-only path may be read ahead of this
    const double* p = part + row * 8 + (lane & 3);
    double re = 0.0, im = 0.0;
#pragma unroll 4
    for (int i = b0; i < b1; ++i) {
        const int2 ref = __ldg(&cg_ref[i]);
        const double* s = p + (long long)(ref.x >> 1) * prow * 8 + (ref.x & 1) * 4;
        if constexpr (CPLX) {
            const double2 ph = __ldg(&phase[(long long)k * nphase + img0 + ref.y]);
            const double vr = s[0], vi = s[64];
            re += ph.x * vr - ph.y * vi;
            im += ph.x * vi + ph.y * vr;
        } else {
            re += s[0];
        }
    }
    sm[w][0][lane] = re;
    if constexpr (CPLX) sm[w][1][lane] = im;
    __syncthreads();
    if (w < (CPLX ? 2 : 1)) {
        double v = sm[0][w][lane];
#pragma unroll
        for (int t = 1; t < 8; ++t) v += sm[t][w][lane];
        v *= scale[cg * 4 + (lane & 3)];
        if constexpr (CPLX) coef[(cg * rows + u * 16 + w * 8) * 4 + lane] = v;
        else coef[(cg * 4 + (lane & 3)) * rows + u * 8 + (lane >> 2)] = v;
    }
}

// k-point states; a unit's coefficients of an item's slots stay in registers while the brick's
// blocks stream by. Units and rows as in k_brick_project.
template <typename T, bool VEC, bool ROWS, int D>
__global__ void __launch_bounds__(kThreads, 2)
    k_brick_scatter(T* __restrict__ HX, long long ldx, long long ldk, long long xim, int ns, int nrow, int nunit,
                    const BrickGeom g, const double2* __restrict__ phase, int nphase, int img0,
                    const double* coef, long long rows) {
    extern __shared__ __align__(16) double tb[];
    const int chunks = ROWS ? nunit : (nunit + 7) / 8;
    const int brick = blockIdx.x / chunks, ch = blockIdx.x - brick * chunks;
    const int bx = brick % g.nbx, by = (brick / g.nbx) % g.nby, bz = brick / (g.nbx * g.nby);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
    const int ul = ROWS ? ch : ch * 8 + w;
    const int u = min(ul, nunit - 1);
    const int row_r = min(u * 8 + r, nrow - 1), k = row_r / ns, s = row_r - k * ns;  // this lane's state
    const bool live = ul * 8 + r < nrow;
    const int x = bx * kBx + 2 * q, y0 = by * kBy, z0 = bz * kBz;
    const long long plane = (long long)g.nx * g.ny;
    T* base = HX + (long long)k * ldk + (long long)s * ldx + (x + (long long)g.nx * y0 + plane * z0);
    const double2* ph = phase + (long long)k * nphase;
    const int row_a = ROWS ? w : 0, row_b = ROWS ? w + 1 : 8;
    using P2 = typename Pair<T>::type;
    // Few units, where latency counts: the table, which no kernel before this one writes, on its way before the
    // wait (one complex64 state of 41^3 29.6 -> 28.7 us a call; for many units behind the loads that are used
    // first, 64 complex128 states of 80^3 0.4 % faster so).
    const int first = g.brick_item[brick], last = g.brick_item[brick + 1];
    if (ROWS && first < last) fetch_table(tb, g, first);
    wait_previous();
    for (int item = first; item < last; ++item) {
        P2 hv[D][2];
        auto fetch = [&](u64 m, int row, int b, P2 (&v)[2]) {
            if ((m >> (8 * b)) & 255) {
                const T* p = base + (long long)row * g.nx + (b & 1) * 8 + (b >> 1) * plane;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    v[i].x = v[i].y = T(0);
                    if (live) v[i] = load_pair<T, VEC>(p + (i ? xim : 0), x + (b & 1) * 8, g.nx);
                }
            }
        };
        u64 mn = g.wmask[item * 8 + row_a];
#pragma unroll
        for (int d = 0; d < D - 1; ++d) fetch(mn, row_a, d, hv[d]);
        double A[kSlots][2];  // times the image's conjugate phase
#pragma unroll
        for (int j = 0; j < kSlots; ++j) {
            const int cg = g.item_cg[item * 8 + j];
            A[j][0] = A[j][1] = 0.0;
            if (cg >= 0) {
                const double* c = &coef[(cg * rows + u * 16) * 4 + lane];
                const double re = c[0], im = c[32];
                const double2 p = __ldg(&ph[img0 + g.item_img[item * 8 + j]]);
                A[j][0] = p.x * re + p.y * im;
                A[j][1] = p.x * im - p.y * re;
            }
        }
        if (!ROWS || item > first) fetch_table(tb, g, item);
        table_ready();
        const double* tp = tb + (g.wtab[item * 8 + row_a] - g.wtab[item * 8]) * 64 + q * 8 + r;
        LanePhase lp;
        for (int row = row_a; row < row_b; ++row) {
            const u64 m = mn;
            mn = row + 1 < row_b ? g.wmask[item * 8 + row + 1] : 0;
            lp.init(ph, g, x, y0 + row, z0);
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                if (b + D - 1 < 8) fetch(m, row, b + D - 1, hv[(b + D - 1) % D]);
                else fetch(mn, row + 1, b + D - 1 - 8, hv[(b + D - 1) % D]);
                const unsigned mb = (unsigned)(m >> (8 * b)) & 255u;
                if (mb) {
                    const P2(&v)[2] = hv[b % D];
                    double n[2][2] = {};
#pragma unroll
                    for (int j = 0; j < kSlots; j += 2)
                        if (mb >> j & 3) {
                            const double t0 = tp[0], t1 = tp[32];
                            tp += 64;
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                dmma(n[i], A[j][i], t0);
                                dmma(n[i], A[j + 1][i], t1);
                            }
                        }
                    T* p = base + (long long)row * g.nx + (b & 1) * 8 + (b >> 1) * plane;
                    double2 e2[2];
                    lp.at(b, e2);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const double re = n[0][e], im = n[1][e];
                        n[0][e] = (double)(e ? v[0].y : v[0].x) + (e2[e].x * re + e2[e].y * im);
                        n[1][e] = (double)(e ? v[1].y : v[1].x) + (e2[e].x * im - e2[e].y * re);
                    }
                    if (live) {
#pragma unroll
                        for (int i = 0; i < 2; ++i) store_pair<T, VEC>(p + (i ? xim : 0), n[i], x + (b & 1) * 8, g.nx);
                    }
                }
            }
        }
        __syncthreads();  // the table is read no more
    }
}

// k-vectors of a launch, as kernel arguments: no copy from pageable memory, nothing to wait for, and a stream
// capture takes the launch.
struct KVecs {
    static constexpr int n = 128;
    double v[3 * n];  // a = g * h per axis
};

// Phases of the axes' grid coordinates and of the images for one k-point per blockIdx.y.
__global__ void k_phase_tables(int nx, int ny, int nz, int nimg, const int* __restrict__ img, const KVecs kh,
                               double2* __restrict__ out) {
    const int n = nx + ny + nz + nimg;
    const double ax = kh.v[3 * blockIdx.y], ay = kh.v[3 * blockIdx.y + 1], az = kh.v[3 * blockIdx.y + 2];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double th;
        if (i < nx) th = ax * i;
        else if (i < nx + ny) th = ay * (i - nx);
        else if (i < nx + ny + nz) th = az * (i - nx - ny);
        else {
            const int* m = img + 3 * (i - nx - ny - nz);
            th = ax * nx * m[0] + ay * ny * m[1] + az * nz * m[2];
        }
        double s, c;
        sincos(th, &s, &c);
        out[(long long)blockIdx.y * n + i] = make_double2(c, s);
    }
}

BrickGeom geom(qg_hamiltonian h) {
    const BrickTables& b = h->pj.bricks;
    return {h->nx, h->ny, h->nz, b.nbx, b.nby, b.item_brick, b.item_pair, b.item_cg, b.item_img,
            b.wmask, b.wtab, b.brick_item, b.tab};
}

int phase_count(qg_hamiltonian h) { return h->nx + h->ny + h->nz + h->pj.bricks.nimg; }

// 16-byte (FP32: 8-byte) pairs of x-neighbours need even rows and even strides.
template <typename T>
bool pairs_ok(qg_hamiltonian h, const T* X, long long ldx, long long ldk) {
    return h->nx % 2 == 0 && ldx % 2 == 0 && ldk % 2 == 0 && (uintptr_t)X % (2 * sizeof(T)) == 0;
}

// The warps of a block take rows of the brick (and the block one unit of 8 states) where whole
// units per warp would leave warps or SMs without work.
bool by_rows(long long items, int units) { return units < 8 || items * ((units + 7) / 8) < 148; }

// Units of 8 states of one projection + reduction launch pair.
int slice_units(const BrickTables& b, bool cplx, int units) {
    const size_t unit_bytes = (size_t)b.npairs * (cplx ? 16 : 8) * 8 * sizeof(double);
    return (int)std::max<size_t>(1, std::min<size_t>({(size_t)units, kPartBytes / unit_bytes / 8 * 8, 65528}));
}

template <typename T, bool CPLX, bool VEC, bool ROWS>
int launch_project(qg_hamiltonian h, int nk, int ns, const T* X, long long ldx, long long ldk, const double2* phase,
                   const double* scale, double* coef, double* part, cudaStream_t st,
                   const std::function<int(bool)>& stencil) {
    constexpr int D = CPLX ? 4 : 8;
    const BrickTables& b = h->pj.bricks;
    const int nrow = nk * ns, units = (nrow + 7) / 8, most = slice_units(b, CPLX, units);
    auto kern = k_brick_project<T, CPLX, VEC, ROWS, D>;
    if (allow_max_dynamic_smem(kern) != cudaSuccess) return QG_ERR_CUDA;
    const int np = phase_count(h);
    for (int u0 = 0; u0 < units; u0 += most) {
        const int nu = std::min(most, units - u0);
        const long long prow = (long long)nu * (CPLX ? 16 : 8);
        kern<<<(unsigned)((long long)b.nitems * (ROWS ? nu : (nu + 7) / 8)), kThreads, (size_t)b.max_tab * 512, st>>>(
            X, ldx, ldk, h->N(), ns, nrow, u0, nu, geom(h), phase, np, part, prow);
        // one slice: the stencil runs beside the projection, in small calls of few units beside the sums as well, and
        // ends after them (16 complex64 states of 40^3 53.1 -> 48.1 us a call, 8 real ones of 64 atoms on 80^3 100.9 ->
        // 94.4; 64 complex64 states of 40^3, 8 units, 157 -> 169: blocks of the sums keep the stencil off their SMs)
        const bool beside = stencil && nu == units, small = ROWS && small_call((long long)nk * ns * h->N());
        if (beside && !small) QG_TRY(stencil(true));
        QG_CUDA_TRY(launch_kernel(beside && small_call((long long)nk * ns * h->N()), k_brick_reduce<CPLX>, dim3(b.ncg, nu), dim3(kThreads), 0, st, part, prow,
                                  b.cg_off, b.cg_ref, ns, nrow, u0, phase, np, h->nx + h->ny + h->nz, scale, coef,
                                  coef_rows(nrow, CPLX)));
        if (beside && small) QG_TRY(stencil(true));
    }
    if (stencil && units > most) QG_TRY(stencil(false));
    QG_CUDA_TRY(cudaGetLastError());
    return QG_OK;
}

template <typename T, bool VEC, bool ROWS>
int launch_scatter(qg_hamiltonian h, int nk, int ns, T* HX, long long ldx, long long ldk, const double2* phase,
                   const double* coef, bool early, cudaStream_t st) {
    const BrickTables& b = h->pj.bricks;
    const int nrow = nk * ns, units = (nrow + 7) / 8;
    auto kern = k_brick_scatter<T, VEC, ROWS, 4>;
    if (allow_max_dynamic_smem(kern) != cudaSuccess) return QG_ERR_CUDA;
    QG_CUDA_TRY(launch_kernel(
        early, kern, dim3((unsigned)((long long)b.nbricks * (ROWS ? units : (units + 7) / 8))), dim3(kThreads),
        (size_t)b.max_tab * 512, st, HX, ldx, ldk, h->N(), ns, nrow, units, geom(h), phase, phase_count(h), h->nx + h->ny + h->nz, coef,
        coef_rows(nrow, true)));
    return QG_OK;
}

template <typename V>
int upload(V** dst, const std::vector<V>& src) {
    *dst = nullptr;
    if (src.empty()) return QG_OK;
    QG_CUDA_TRY(cudaMalloc(dst, src.size() * sizeof(V)));
    QG_CUDA_TRY(cudaMemcpy(*dst, src.data(), src.size() * sizeof(V), cudaMemcpyHostToDevice));
    return QG_OK;
}

int floor_div(int a, int b) { return a >= 0 ? a / b : -((b - 1 - a) / b); }

}  // namespace

size_t coef_elems(qg_hamiltonian h, int nk, int ns, bool cplx) {
    return (size_t)h->pj.na * h->pj.nch * coef_rows(nk * ns, cplx);
}

size_t part_elems(qg_hamiltonian h, int nk, int ns, bool cplx) {
    const BrickTables& b = h->pj.bricks;
    if (b.nitems == 0 || ns <= 0) return 0;
    return (size_t)b.npairs * slice_units(b, cplx, (nk * ns + 7) / 8) * (cplx ? 16 : 8) * 8;
}

// By the cell alone, so that a state's bits never depend on its batch: cells of more than 16 atoms,
// whose spheres overlap in the atom-by-atom kernel's reads (64 atoms, 256 states: 0.36 against 0.49
// ms; 216 atoms, 528 states: 2.70 against 3.71). On the 8-atom cell with 16 states the
// atom-by-atom kernel is one launch of 9 us against 7 + 4.
bool bricks_for_real(const DevProjectors& pj) { return pj.na > 16; }

int brick_project_launches(qg_hamiltonian h, int ns) {
    const BrickTables& b = h->pj.bricks;
    if (b.nitems == 0 || ns <= 0) return 0;
    const int units = (ns + 7) / 8, most = slice_units(b, false, units);
    return 2 * ((units + most - 1) / most);
}

template <typename T>
int brick_project(qg_hamiltonian h, int nk, int ns, bool cplx, const T* X, long long ldx, long long ldk,
                  const double2* phase, const double* scale, double* coef, double* part, cudaStream_t st,
                  const std::function<int(bool)>& stencil) {
    const BrickTables& b = h->pj.bricks;
    if (nk <= 0 || ns <= 0) return QG_OK;
    if (b.nitems == 0) {  // every table value is zero
        QG_CUDA_TRY(cudaMemsetAsync(coef, 0, coef_elems(h, nk, ns, cplx) * sizeof(double), st));
        return stencil ? stencil(false) : QG_OK;
    }
    const bool rows = by_rows(b.nitems, slice_units(b, cplx, (nk * ns + 7) / 8));
    const bool vec = pairs_ok(h, X, ldx, ldk) && (!cplx || h->N() % 2 == 0);
#define QG_GO(C, V, R) return launch_project<T, C, V, R>(h, nk, ns, X, ldx, ldk, phase, scale, coef, part, st, stencil)
    if (cplx) {
        if (vec && rows) QG_GO(true, true, true);
        if (vec) QG_GO(true, true, false);
        if (rows) QG_GO(true, false, true);
        QG_GO(true, false, false);
    }
    if constexpr (sizeof(T) == 8) {
        if (vec && rows) QG_GO(false, true, true);
        if (vec) QG_GO(false, true, false);
        if (rows) QG_GO(false, false, true);
        QG_GO(false, false, false);
    }
#undef QG_GO
    return QG_ERR_UNSUPPORTED;
}

template <typename T>
int brick_scatter_z(qg_hamiltonian h, int nk, int ns, T* HX, long long ldx, long long ldk, const double2* phase,
                    const double* coef, bool early, cudaStream_t st) {
    const BrickTables& b = h->pj.bricks;
    if (b.nitems == 0 || nk <= 0 || ns <= 0) return QG_OK;
    const bool rows = by_rows(b.nbricks, (nk * ns + 7) / 8);
    const bool vec = pairs_ok(h, HX, ldx, ldk) && h->N() % 2 == 0;
#define QG_GO(V, R) return launch_scatter<T, V, R>(h, nk, ns, HX, ldx, ldk, phase, coef, early, st)
    if (vec && rows) QG_GO(true, true);
    if (vec) QG_GO(true, false);
    if (rows) QG_GO(false, true);
    QG_GO(false, false);
#undef QG_GO
}

template int brick_project<double>(qg_hamiltonian, int, int, bool, const double*, long long, long long, const double2*,
                                   const double*, double*, double*, cudaStream_t,
                                   const std::function<int(bool)>&);
template int brick_project<float>(qg_hamiltonian, int, int, bool, const float*, long long, long long, const double2*,
                                  const double*, double*, double*, cudaStream_t, const std::function<int(bool)>&);
template int brick_scatter_z<double>(qg_hamiltonian, int, int, double*, long long, long long, const double2*,
                                     const double*, bool, cudaStream_t);
template int brick_scatter_z<float>(qg_hamiltonian, int, int, float*, long long, long long, const double2*,
                                    const double*, bool, cudaStream_t);

int ensure_phases(qg_hamiltonian h, int nk, const double* kv, cudaStream_t st, const double2** out) {
    BrickTables& b = h->pj.bricks;
    *out = nullptr;
    if (b.nitems == 0) return QG_OK;
    const int n = phase_count(h);
    if (!((int)b.phase_k.size() == 3 * nk && std::equal(kv, kv + 3 * nk, b.phase_k.begin()))) {
        b.phase_k.clear();
        QG_TRY(b.phase.reserve((size_t)nk * n * sizeof(double2)));
        for (int k0 = 0; k0 < nk; k0 += KVecs::n) {
            const int m = std::min(KVecs::n, nk - k0);
            KVecs kh;
            for (int k = 0; k < m; ++k) {
                kh.v[3 * k] = kv[3 * (k0 + k)] * h->hx;
                kh.v[3 * k + 1] = kv[3 * (k0 + k) + 1] * h->hy;
                kh.v[3 * k + 2] = kv[3 * (k0 + k) + 2] * h->hz;
            }
            k_phase_tables<<<dim3((n + 127) / 128, m), 128, 0, st>>>(h->nx, h->ny, h->nz, b.nimg, b.img, kh,
                                                                     b.phase.as<double2>() + (size_t)k0 * n);
        }
        QG_CUDA_TRY(cudaGetLastError());
        b.phase_k.assign(kv, kv + 3 * nk);
    }
    *out = b.phase.as<double2>();
    return QG_OK;
}

void free_bricks(BrickTables& b) {
    cudaFree(b.item_brick); cudaFree(b.item_pair); cudaFree(b.item_cg); cudaFree(b.item_img); cudaFree(b.wmask);
    cudaFree(b.wtab); cudaFree(b.brick_item); cudaFree(b.tab); cudaFree(b.cg_off); cudaFree(b.cg_ref);
    cudaFree(b.img);
    b.phase.release();
    b = BrickTables();
}

BrickLists list_bricks(const int (&n)[3], const std::vector<int>& atom_off, const std::vector<int>& u,
                       const std::vector<std::vector<double>>& tabs) {
    BrickLists b;
    const int na = (int)atom_off.size() - 1, nch = (int)tabs.size(), ng = nch / 4;
    b.nbx = (n[0] + kBx - 1) / kBx;
    b.nby = (n[1] + kBy - 1) / kBy;
    const int nbz = (n[2] + kBz - 1) / kBz;
    b.nbricks = b.nbx * b.nby * nbz;
    b.ncg = na * ng;

    // one record per (atom, image, brick) in order of their first points, and the runs of points in one
    // block: points [p, p + len) of the atom at x0 .. of block blk in row w of the record's brick
    struct Rec {
        int atom, img, brick;
        u64 mask[8];  // bit 8 b of mask[w]: row w, block b
    };
    struct Run {
        int rec, p;
        unsigned char at, x0, len;  // at = 8 w + blk
    };
    std::vector<Rec> recs;
    std::vector<Run> runs;
    runs.reserve(u.size() / 12 + 16);
    std::vector<int> newest(b.nbricks, -1), before;  // records of a brick, the newest first
    for (int a = 0; a < na; ++a) {
        const int first = (int)recs.size();
        for (int p = atom_off[a]; p < atom_off[a + 1];) {
            const int* up = &u[3 * (size_t)p];
            int im[3], f[3];
            for (int d = 0; d < 3; ++d) {
                im[d] = floor_div(up[d], n[d]);
                f[d] = up[d] - im[d] * n[d];
            }
            const int most = std::min({8 - f[0] % 8, n[0] - f[0], atom_off[a + 1] - p});
            int len = 1;
            while (len < most && up[3 * len] == up[0] + len && up[3 * len + 1] == up[1] && up[3 * len + 2] == up[2]) ++len;
            int ii = 0;
            const int ni = (int)b.img.size() / 3;
            while (ii < ni && std::memcmp(&b.img[3 * ii], im, sizeof(im)) != 0) ++ii;
            if (ii == ni) b.img.insert(b.img.end(), im, im + 3);
            const int brick = f[0] / kBx + b.nbx * (f[1] / kBy + b.nby * (f[2] / kBz));
            int r = newest[brick];
            while (r >= first && recs[r].img != ii) r = before[r];
            if (r < first) {  // none of this atom
                r = (int)recs.size();
                recs.push_back({a, ii, brick, {}});
                before.push_back(newest[brick]);
                newest[brick] = r;
            }
            const int w = f[1] % kBy, blk = (f[2] % kBz) * 2 + (f[0] % kBx) / 8;
            recs[r].mask[w] |= u64(1) << (8 * blk);
            runs.push_back({r, p, (unsigned char)(8 * w + blk), (unsigned char)(f[0] % 8), (unsigned char)len});
            p += len;
        }
    }
    // records by brick (kept in atom order)
    std::vector<int> first(b.nbricks + 1, 0), order(recs.size());
    for (const Rec& r : recs) first[r.brick + 1]++;
    for (int i = 0; i < b.nbricks; ++i) first[i + 1] += first[i];
    {
        std::vector<int> fill(first.begin(), first.end() - 1);
        for (size_t i = 0; i < recs.size(); ++i) order[fill[recs[i].brick]++] = (int)i;
    }
    b.item_pair.push_back(0);
    b.brick_item.push_back(0);
    size_t ntab = 0;                                    // table blocks of two halves (pairs of groups)
    std::vector<int> half(recs.size() * ng * 64, -1);   // half of a record's channel group and block
    std::vector<std::vector<int2>> refs(b.ncg);
    auto shared = [](const Rec& p, const Rec& q) {
        int s = 0;
        for (int w = 0; w < 8; ++w) s += __builtin_popcountll(p.mask[w] & q.mask[w]);
        return s;
    };
    b.max_tab = 0;
    for (int br = 0; br < b.nbricks; ++br) {
        struct Cg { int rec, g; };
        std::vector<Cg> todo;
        for (int i = first[br]; i < first[br + 1]; ++i)
            for (int g = 0; g < ng; ++g) todo.push_back({order[i], g});
        // pairs of channel groups that cover the most blocks together, in record order
        std::vector<std::pair<Cg, Cg>> pairs;
        std::vector<char> used(todo.size(), 0);
        for (size_t i = 0; i < todo.size(); ++i) {
            if (used[i]) continue;
            int best = -1, most = 0;
            for (size_t j = i + 1; j < todo.size(); ++j) {
                if (used[j]) continue;
                const int s = shared(recs[todo[i].rec], recs[todo[j].rec]);
                if (s > most) {
                    most = s;
                    best = (int)j;
                }
            }
            if (best < 0) continue;
            used[i] = used[best] = 1;
            pairs.push_back({todo[i], todo[best]});
        }
        // groups that cover no block with another: two and two
        for (size_t i = 0, open = 0; i < todo.size(); ++i) {
            if (used[i]) continue;
            if (open) pairs.back().second = todo[i];
            else pairs.push_back({todo[i], Cg{-1, 0}});
            open = !open;
        }
        for (size_t p0 = 0, p1; p0 < pairs.size(); p0 = p1) {
            int blocks = 0;
            for (p1 = p0; p1 < pairs.size() && p1 < p0 + 4; ++p1) {
                int n = 0;
                for (int w = 0; w < 8; ++w) {
                    u64 m = recs[pairs[p1].first.rec].mask[w];
                    if (pairs[p1].second.rec >= 0) m |= recs[pairs[p1].second.rec].mask[w];
                    n += __builtin_popcountll(m);
                }
                if (p1 > p0 && blocks + n > kMaxTab) break;
                blocks += n;
            }
            b.max_tab = std::max(b.max_tab, blocks);
            const int item = (int)b.item_brick.size(), np = (int)(p1 - p0);
            Cg slot[kSlots];
            for (int j = 0; j < 4; ++j) {
                slot[2 * j] = j < np ? pairs[p0 + j].first : Cg{-1, 0};
                slot[2 * j + 1] = j < np ? pairs[p0 + j].second : Cg{-1, 0};
            }
            b.item_brick.push_back(br);
            for (int j = 0; j < kSlots; ++j) {
                const bool on = slot[j].rec >= 0;
                const int cg = on ? recs[slot[j].rec].atom * ng + slot[j].g : -1;
                b.item_cg.push_back(cg);
                b.item_img.push_back(on ? recs[slot[j].rec].img : 0);
                if (on) refs[cg].push_back(make_int2(2 * (b.item_pair[item] + j / 2) + (j & 1), recs[slot[j].rec].img));
            }
            for (int w = 0; w < 8; ++w) {
                u64 m = 0;
                for (int j = 0; j < kSlots; ++j)
                    if (slot[j].rec >= 0) m |= recs[slot[j].rec].mask[w] << j;
                b.wmask.push_back(m);
                b.wtab.push_back((int)ntab);
                for (int blk = 0; blk < 8; ++blk)
                    for (int j = 0; j < 4; ++j) {
                        if (!((m >> (8 * blk + 2 * j)) & 3)) continue;
                        for (int hf = 0; hf < 2; ++hf) {
                            const Cg& s = slot[2 * j + hf];
                            if (s.rec >= 0) half[((size_t)s.rec * ng + s.g) * 64 + 8 * w + blk] = (int)(2 * ntab) + hf;
                        }
                        ++ntab;
                    }
            }
            b.item_pair.push_back(b.item_pair[item] + np);
        }
        b.brick_item.push_back((int)b.item_brick.size());
    }
    b.wtab.push_back((int)ntab);
    // the values: 4 channels x 8 points per half
    b.tab.resize(ntab * 64, 0.0);
    for (const Run& r : runs)
        for (int g = 0; g < ng; ++g) {
            double* to = &b.tab[(size_t)half[((size_t)r.rec * ng + g) * 64 + r.at] * 32 + r.x0];
            for (int c = 0; c < 4; ++c) std::copy_n(&tabs[4 * g + c][r.p], r.len, to + 8 * c);
        }
    b.nitems = (int)b.item_brick.size();
    b.npairs = b.item_pair.back();
    b.nimg = (int)b.img.size() / 3;
    b.cg_off.push_back(0);
    for (const auto& v : refs) {
        b.cg_ref.insert(b.cg_ref.end(), v.begin(), v.end());
        b.cg_off.push_back((int)b.cg_ref.size());
    }
    return b;
}

int upload_bricks(qg_hamiltonian h, const BrickLists& l) {
    BrickTables& b = h->pj.bricks;
    b.nbx = l.nbx;
    b.nby = l.nby;
    b.nbricks = l.nbricks;
    b.nitems = l.nitems;
    b.npairs = l.npairs;
    b.max_tab = l.max_tab;
    b.ncg = l.ncg;
    b.nimg = l.nimg;
    QG_TRY(upload(&b.item_brick, l.item_brick));
    QG_TRY(upload(&b.item_pair, l.item_pair));
    QG_TRY(upload(&b.item_cg, l.item_cg));
    QG_TRY(upload(&b.item_img, l.item_img));
    QG_TRY(upload(&b.wmask, l.wmask));
    QG_TRY(upload(&b.wtab, l.wtab));
    QG_TRY(upload(&b.brick_item, l.brick_item));
    QG_TRY(upload(&b.tab, l.tab));
    QG_TRY(upload(&b.cg_off, l.cg_off));
    QG_TRY(upload(&b.cg_ref, l.cg_ref));
    QG_TRY(upload(&b.img, l.img));
    return QG_OK;
}

}  // namespace qg
