// FD stencil + local potential of complex k-point states,
//   H u = V u - 1/2 (Lap + 2i g.grad - g^2) u,
// on split complex rows {re[N], im[N]} (LaplasianKpoint{2nd,6th,8th}_halo_f,
// GridDifferenceKpoint2nd.h:19-92, 6th.h:19-107, 8th.h:18-122), sm_100a.
//
// Plane ring of tma_ring.cuh: a producer lane streams the re and im rows of a work item's planes
// (state, y tile of ty full x-rows, z slab) with bulk copies, the consumer warps release a stage when
// their reads of it are done, one persistent block per SM. Lanes 0-15 of a warp own the real parts of 16
// vectors of PX x-points in RPT adjacent rows, lanes 16-31 the imaginary parts of the same points: a
// thread keeps the 2R + 1 z-values of one part in registers, forms its Laplacian L and first
// derivative D, and the pair exchanges D by shuffle,  re: V re + L re - D im,  im: V im + L im + D re.
// With two rows a thread reads 18 vectors from shared memory for two outputs instead of 26.
//
// Bound: latency. 11 (FP64) or 15 (FP32) warps are what the z-windows leave room for; the FP64 pipe is
// 48 %, the issue slots 48 %, L1 45 % and L2 16 % busy. A thread with both parts of a point (two windows,
// 168 registers with spills, 10 warps) took 0.66 ms for 64 complex128 states of 80^3 and 1.22 ms for 64
// k-points x 16 complex64 states of 40^3; this one 0.44 and 0.62 ms (0.65 where it starts beside the projection's
// last blocks). One row per thread: 0.51 / 0.75.
// Every wait is bounded (QG_ERR_TIMEOUT in the device status word on expiry).
#include <algorithm>
#include <cstdint>

#include "qg_internal.h"
#include "stencil_common.cuh"
#include "tma_ring.cuh"

namespace qg {
namespace {

using namespace ring;

// Steps per unrolled body: the z-window then moves down by U registers. Rotating it by renaming over
// 2R + 1 steps (no moves, 86 KB of code) lost half the issue slots to instruction fetches.
constexpr int U = 2;
constexpr size_t kSmemKb = 224;
// Consumer threads: 11 warps of 168 registers (FP64), 15 of 128 (FP32).
template <typename T> constexpr int kConsumers = sizeof(T) == 8 ? 352 : 480;

constexpr int radius_of(int order) { return order == 2 ? 1 : (order == 8 ? 4 : 3); }

template <typename T> struct V16;
template <> struct V16<double> { using type = double2; };
template <> struct V16<float> { using type = float4; };

template <typename T, int PX>
union Vec {
    typename V16<T>::type v;
    T e[PX];
};

// First-derivative weights of an axis as multiples of the first ((672, -168, 32, -3), (45, -9, 1),
// 1): a k-point brings three numbers, not twelve.
template <int ORDER>
__device__ __forceinline__ constexpr double der_ratio(int i) {
    return ORDER == 8 ? (i == 0 ? 1.0 : i == 1 ? -168.0 / 672.0 : i == 2 ? 32.0 / 672.0 : -3.0 / 672.0)
                      : (i == 0 ? 1.0 : i == 1 ? -9.0 / 45.0 : 1.0 / 45.0);
}

// One pair of neighbours at distance i + 1 of an axis: lap += w (p + m), der += ratio (p - m).
template <typename T, int ORDER>
__device__ __forceinline__ void add_pair(T& lap, T& der, T p, T m, T w, int i) {
    lap += w * (p + m);
    der += T(der_ratio<ORDER>(i)) * (p - m);
}

// NXC > 0: the row length as a compile-time constant, which makes the y-neighbour offsets immediates of the
// shared-memory loads; the row lengths of the synthetic cells (40 points per 8-atom cell edge), as in the
// other ring kernels. Order 8, without / with: 256 complex64 states of 40^3 239 / 214 us, 64 of 80^3 433 / 350, 64
// complex128 states of 80^3 574 / 485, 16 of 120^3 523 / 439 (order 6: 193 / 190, -, 441 / 405). All other lengths run
// without.
template <typename T, int ORDER, int NXC, int RPT>
__global__ void __launch_bounds__(kConsumers<T> + 32, 1) k_stencil_kpoint(const HamArgs<T> a, const WorkGrid wg, int nst) {
    constexpr int PX = 16 / sizeof(T);
    constexpr int R = radius_of(ORDER);
    constexpr int NV = (R + PX - 1) / PX;
    using VT = typename V16<T>::type;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);
    uint64_t* empty = full + nst;
    volatile int* ctl = reinterpret_cast<volatile int*>(empty + nst);  // [0] abort, [1] last position issued
    T* ringp = reinterpret_cast<T*>(smem + kBarBytes);

    const int nx = NXC > 0 ? NXC : a.nx, ny = a.ny, nz = a.nz, ty = a.ty;
    const int comp_elems = (ty + 2 * R) * nx;
    const int stage_elems = 2 * comp_elems;
    const int tpr = nx / PX, nvec = tpr * (ty / RPT);
    const int t = threadIdx.x;
    const long long plane = (long long)nx * ny;

    allow_next();
    if (t == 0) {
        for (int i = 0; i < nst; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], (uint32_t)(blockDim.x >> 5) - 1);
        }
        ctl[0] = 0;
        ctl[1] = -1;
        fence_mbar_init();
    }
    __syncthreads();

    if (t < 32) {
        if (t == 0) produce_planes<T, R, 2>(a, wg, nst, nx, ringp, full, empty, ctl);
    } else {
        const int lane = t & 31;
        const int im = lane >> 4;
        const int vraw = ((t >> 5) - 1) * 16 + (lane & 15);
        const bool act = vraw < nvec;
        const int vec = act ? vraw : nvec - 1;  // the last warp's spare lanes repeat the last vector
        const int ix0 = (vec % tpr) * PX, ly = vec / tpr * RPT;
        const int own = im * comp_elems + (R + ly) * nx + ix0;
        int xoff[2 * NV];
#pragma unroll
        for (int v = 0; v < 2 * NV; ++v) {
            int xx = ix0 + (v < NV ? v - NV : v - NV + 1) * PX;
            xx += (xx < 0) ? nx : 0;
            xx -= (xx >= nx) ? nx : 0;
            xoff[v] = own - ix0 + xx;
        }
        int j = 0;         // stage of the next plane to come
        uint32_t ph = 0;
        int jz = 0;        // stage of the oldest plane not released
        auto release = [&] {
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[jz]);
            if (++jz == nst) jz = 0;
        };
        bool bad = false;
        for (int item = blockIdx.x; item < wg.items && !bad; item += gridDim.x) {
            const int slab = item % wg.nslab;
            const int tile = (item / wg.nslab) % wg.tiles;
            const int s = item / (wg.nslab * wg.tiles);
            const int zs = slab * wg.zslab;
            const int ze = min(nz, zs + wg.zslab);
            const long long col = ((long long)tile * ty + ly) * nx + ix0 + (long long)zs * plane;
            T c0 = a.c0, gx = a.dx[0], gy = a.dy[0], gz = a.dz[0];
            if (a.kco) {
                const T* kc = a.kco + (long long)(s / a.nsk) * 13;
                c0 = kc[0];
                gx = kc[1];
                gy = kc[5];
                gz = kc[9];
            }
            const T* vp = a.V + col;
            T* hxp = a.HX + state_offset(a, s, true) + col + (im ? a.hxim : 0);
            // q: planes z - R .. z + R of the own part, plane z - R + d in slot k + d at unrolled
            // step k; after U steps the window moves down by U
            Vec<T, PX> q[RPT][2 * R + U];
            bool w = true;
#pragma unroll
            for (int d = 0; d < 2 * R; ++d) {
                if (w && !mbar_wait(&full[j], ph)) w = false;
#pragma unroll
                for (int r = 0; r < RPT; ++r)
                    q[r][d].v = *reinterpret_cast<const VT*>(ringp + j * stage_elems + own + r * nx);
                if (++j == nst) { j = 0; ph ^= 1u; }
                if (d < R) release();  // planes zs - R .. zs - 1 live on in registers only
            }
            if (__any_sync(0xffffffffu, !w || ctl[0] != 0)) {
                bad = true;
                break;
            }
            for (int z = zs; z < ze && !bad;) {
#pragma unroll
                for (int k = 0; k < U; ++k) {
                    if (z >= ze) break;
                    Vec<T, PX> vnow[RPT];  // V of plane z: used last, so that the step hides its latency
#pragma unroll
                    for (int r = 0; r < RPT; ++r) vnow[r].v = __ldg(reinterpret_cast<const VT*>(vp + r * nx));
                    vp += plane;
                    const T* st = ringp + jz * stage_elems;
                    // axis by axis, outermost pair first
                    T lap[RPT][PX], der[RPT][PX];
#pragma unroll
                    for (int r = 0; r < RPT; ++r) {
                        T xv[(2 * NV + 1) * PX];
#pragma unroll
                        for (int v = 0; v < 2 * NV; ++v) {
                            Vec<T, PX> wv;
                            wv.v = *reinterpret_cast<const VT*>(st + xoff[v] + r * nx);
#pragma unroll
                            for (int e = 0; e < PX; ++e) xv[(v < NV ? v : v + 1) * PX + e] = wv.e[e];
                        }
#pragma unroll
                        for (int e = 0; e < PX; ++e) xv[NV * PX + e] = q[r][k + R].e[e];
#pragma unroll
                        for (int e = 0; e < PX; ++e) {
                            T l = T(0), g = T(0);
#pragma unroll
                            for (int i = R - 1; i >= 0; --i)
                                add_pair<T, ORDER>(l, g, xv[NV * PX + e + 1 + i], xv[NV * PX + e - 1 - i], a.cx[i], i);
                            lap[r][e] = c0 * q[r][k + R].e[e] + l;
                            der[r][e] = gx * g;
                        }
                    }
                    {
                        // rows above (lo) and below (hi) the thread's rows, one distance at a time
                        T l[RPT][PX], g[RPT][PX];
#pragma unroll
                        for (int r = 0; r < RPT; ++r)
#pragma unroll
                            for (int e = 0; e < PX; ++e) l[r][e] = g[r][e] = T(0);
                        auto row = [&](int dy) {
                            Vec<T, PX> v;
                            v.v = *reinterpret_cast<const VT*>(st + own + dy * nx);
                            return v;
                        };
                        Vec<T, PX> lo = row(-R), hi = row(RPT - 1 + R);
#pragma unroll
                        for (int i = R - 1; i >= 0; --i) {  // distance i + 1
                            Vec<T, PX> lo1 = i > 0 ? row(-i) : q[0][k + R];
                            Vec<T, PX> hi1 = i > 0 ? row(RPT - 1 + i) : q[RPT - 1][k + R];
#pragma unroll
                            for (int e = 0; e < PX; ++e) {
                                if constexpr (RPT == 1) {
                                    add_pair<T, ORDER>(l[0][e], g[0][e], hi.e[e], lo.e[e], a.cy[i], i);
                                } else {
                                    add_pair<T, ORDER>(l[0][e], g[0][e], hi1.e[e], lo.e[e], a.cy[i], i);
                                    add_pair<T, ORDER>(l[RPT - 1][e], g[RPT - 1][e], hi.e[e], lo1.e[e], a.cy[i], i);
                                }
                            }
                            lo = lo1;
                            hi = hi1;
                        }
#pragma unroll
                        for (int r = 0; r < RPT; ++r)
#pragma unroll
                            for (int e = 0; e < PX; ++e) {
                                lap[r][e] += l[r][e];
                                der[r][e] += gy * g[r][e];
                            }
                    }
                    release();  // plane z is no longer read
                    // plane z + R is waited for only now, behind the sums that do not need it
                    const bool ok = mbar_wait(&full[j], ph);
                    if (__any_sync(0xffffffffu, !ok)) {
                        bad = true;
                        break;
                    }
#pragma unroll
                    for (int r = 0; r < RPT; ++r)
                        q[r][k + 2 * R].v = *reinterpret_cast<const VT*>(ringp + j * stage_elems + own + r * nx);
                    if (++j == nst) { j = 0; ph ^= 1u; }
#pragma unroll
                    for (int r = 0; r < RPT; ++r)
#pragma unroll
                        for (int e = 0; e < PX; ++e) {
                            T l = T(0), g = T(0);
#pragma unroll
                            for (int i = R - 1; i >= 0; --i)
                                add_pair<T, ORDER>(l, g, q[r][k + R + 1 + i].e[e], q[r][k + R - 1 - i].e[e],
                                                   a.cz[i], i);
                            lap[r][e] += l;
                            der[r][e] += gz * g;
                        }
                    Vec<T, PX> out[RPT];
#pragma unroll
                    for (int r = 0; r < RPT; ++r)
#pragma unroll
                        for (int e = 0; e < PX; ++e) {
                            const T other = __shfl_xor_sync(0xffffffffu, im ? -der[r][e] : der[r][e], 16);
                            out[r].e[e] = (vnow[r].e[e] * q[r][k + R].e[e] + lap[r][e]) + other;
                        }
#pragma unroll
                    for (int r = 0; r < RPT; ++r)
                        if (act) *reinterpret_cast<VT*>(hxp + r * nx) = out[r].v;
                    hxp += plane;
                    ++z;
                }
#pragma unroll
                for (int r = 0; r < RPT; ++r)
#pragma unroll
                    for (int d = 0; d < 2 * R; ++d) q[r][d] = q[r][d + U];
            }
            if (bad) break;
            for (int d = 0; d < R; ++d) release();  // planes ze .. ze + R - 1
        }
        if (bad) {
            ctl[0] = 1;
            if (lane == 0) atomicExch(a.err, (int)QG_ERR_TIMEOUT);
        }
    }
    __syncthreads();
    if (t == 0 && ctl[0]) {
        const int last = ctl[1];
        for (int ps = max(0, last - nst + 1); ps <= last; ++ps) mbar_wait(&full[ps % nst], (uint32_t)(ps / nst) & 1u);
    }
    wait_previous();
}

// Ring stages of a tile of ty rows, -1: too few fit (R + 1 planes are held, 2 more in flight).
int stages(int R, int ty, int nx, size_t elem) {
    const size_t stage = (size_t)2 * (ty + 2 * R) * nx * elem;
    const int n = (int)std::min<size_t>(kMaxStages, (kSmemKb * 1024 - kBarBytes) / stage);
    return n >= R + 3 ? n : -1;
}

int max_slabs(int nz, int R) {
    int n = 1;
    while (nz / (2 * n) >= 2 * R) n *= 2;
    return n;
}

// Threads that own a tile.
int consumers(int nx, int ty, int px, int rpt) { return (nx / px * (ty / rpt) + 15) / 16 * 32; }

// Rows per tile, a divisor of ny: the largest that the consumers and the ring hold (the halo
// rows cost copies from L2), of those that still give every SM an item; else the smallest of R or more.
template <typename T>
int tile_rows(const HamArgs<T>& a, int order, int rpt) {
    constexpr int PX = 16 / sizeof(T);
    const int R = radius_of(order);
    int ty = 0;
    for (int t = 1; t <= a.ny; ++t) {
        if (a.ny % t != 0 || t % rpt != 0 || consumers(a.nx, t, PX, rpt) > kConsumers<T> || stages(R, t, a.nx, sizeof(T)) < 0) continue;
        if (ty < R || (long long)a.ns * (a.ny / t) * max_slabs(a.nz, R) >= sm_count()) ty = t;
    }
    return ty;
}

template <typename T, int ORDER, int RPT, int NXC = 0>
int launch_order(const HamArgs<T>& a, cudaStream_t st) {
    constexpr int PX = 16 / sizeof(T);
    constexpr int R = radius_of(ORDER);
    if constexpr (NXC == 0 && ORDER >= 6) {
        switch (a.nx) {
            case 40: return launch_order<T, ORDER, RPT, 40>(a, st);
            case 80: return launch_order<T, ORDER, RPT, 80>(a, st);
            case 120: return launch_order<T, ORDER, RPT, 120>(a, st);
            default: break;
        }
    }
    const int nst = stages(R, a.ty, a.nx, sizeof(T));
    const size_t smem = kBarBytes + (size_t)nst * 2 * (a.ty + 2 * R) * a.nx * sizeof(T);
    auto kern = k_stencil_kpoint<T, ORDER, NXC, RPT>;
    if (nst < 0 || allow_max_dynamic_smem(kern) != cudaSuccess) return QG_ERR_UNSUPPORTED;
    const int threads = 32 + consumers(a.nx, a.ty, PX, RPT);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem) != cudaSuccess || per_sm < 1)
        return QG_ERR_UNSUPPORTED;
    const int G0 = sm_count() * per_sm;
    WorkGrid wg;
    wg.tiles = a.ny / a.ty;
    // z slabs: enough items for about four per block, slabs of at least 2R planes
    const long long base = (long long)a.ns * wg.tiles;
    wg.nslab = 1;
    while (base * wg.nslab < 4LL * G0 && a.nz / (wg.nslab * 2) >= 2 * R) wg.nslab *= 2;
    wg.zslab = (a.nz + wg.nslab - 1) / wg.nslab;
    wg.nslab = (a.nz + wg.zslab - 1) / wg.zslab;
    wg.items = (int)(base * wg.nslab);
    QG_CUDA_TRY(launch_kernel(a.early, kern, dim3(std::min(G0, wg.items)), dim3(threads), smem, st, a, wg, nst));
    return QG_OK;
}

template <typename T, int RPT>
int launch_rows(const HamArgs<T>& a, int order, cudaStream_t st) {
    switch (order) {
        case 2: return launch_order<T, 2, RPT>(a, st);
        case 6: return launch_order<T, 6, RPT>(a, st);
        default: return launch_order<T, 8, RPT>(a, st);
    }
}

}  // namespace

template <typename T>
bool stencil_kpoint_ok(const HamArgs<T>& a, int order) {
    constexpr int PX = 16 / sizeof(T);
    if (order != 2 && order != 6 && order != 8) return false;
    const int R = radius_of(order);
    if ((a.xim % PX) || (a.hxim % PX) || a.nx % PX != 0 || ((uintptr_t)a.X % 16) || ((uintptr_t)a.HX % 16) ||
        ((uintptr_t)a.V % 16) || (a.ldx % PX) || (a.ldhx % PX) || !a.err || a.ny < 2 * R || a.nx < 2 * R)
        return false;
    return tile_rows(a, order, 1) > 0 || tile_rows(a, order, 2) > 0;
}

// Returns QG_ERR_UNSUPPORTED (launching nothing) when the shape or alignment does not fit.
template <typename T>
int launch_stencil_kpoint(const HamArgs<T>& a, int order, cudaStream_t st) {
    if (!stencil_kpoint_ok<T>(a, order)) return QG_ERR_UNSUPPORTED;
    HamArgs<T> b = a;
    b.ty = tile_rows(a, order, 2);
    if (b.ty > 0) return launch_rows<T, 2>(b, order, st);
    b.ty = tile_rows(a, order, 1);
    return launch_rows<T, 1>(b, order, st);
}

template bool stencil_kpoint_ok<double>(const HamArgs<double>&, int);
template bool stencil_kpoint_ok<float>(const HamArgs<float>&, int);
template int launch_stencil_kpoint<double>(const HamArgs<double>&, int, cudaStream_t);
template int launch_stencil_kpoint<float>(const HamArgs<float>&, int, cudaStream_t);

}  // namespace qg
