// 8th-order periodic FD gradient of real states (Gradient8th, GridGradient8th.h:19-235) for the
// nonlocal forces, the x and y derivatives as banded products on the FP64 tensor cores
// (mma.sync.m8n8k4.f64).
//
// A producer lane streams the planes of a work item (state, tile of ty rows, z slab) into a ring of
// shared-memory stages -- TMA boxes of whole rows (or of 8 ntx + 8 columns, with the 4 wrapped
// columns of a tile that reaches over an end of the row in a box of their own): the tile's rows, 4 rows above and 4 below -- and
// the consumer warps release a stage when its last reader has passed. A consumer warp owns 8 x 8
// points of the plane, lane (r, q) = (lane / 4, lane % 4) the points (y0 + r, x0 + 2 q) and its right
// neighbour -- the accumulator layout of m8n8k4. Per plane: 16 inputs of 8 outputs in four steps
// along x (band on the right) and along y (band on the left), the z difference from the 9 values of
// each point in registers, which rotate by renaming. Bound: DRAM, 8 bytes in and 24 out per point;
// 139 of 256 states of 80^3 take 0.49 ms (0.35 ms of bytes at the copy rate), against 4.0 ms for
// 24 neighbour loads per point from L1 (k_gradient8, which stays for the shapes TMA does not take).
// The same products in the Hamiltonian's stencil measured slower than its vector kernels (1.17
// against 0.55 ms real, 0.63 against 0.44 k-points): the FP64 tensor and vector instructions share
// one pipe, where 16 band products per axis and point cost more than 9 of 13 additions saved.
//
// Any ny >= 8 and nx, nz whose rows TMA takes (even nx, 16-byte state strides): a tile past the last
// row starts at ny - ty and leaves the rows of the tile before it to that one, columns past the last
// are not stored. A NaN or Inf reaches every output of the 8 x 8 tiles that read its point. Every
// wait is bounded (QG_ERR_TIMEOUT in the device status word on expiry).
#include <cuda.h>

#include <algorithm>
#include <cstdint>

#include "qg_internal.h"
#include "stencil_common.cuh"
#include "tc_common.cuh"
#include "tma_ring.cuh"

namespace qg {
namespace {

using namespace ring;

constexpr int R = 4;   // neighbours each side
constexpr int Q = 2 * R + 1;
constexpr int KB = 4;  // steps of 4 inputs: outputs 0 .. 7 take inputs -4 .. 11
constexpr int kHalo = 4;
constexpr int kThreads = 512;  // 15 consumer warps of at most 128 registers
constexpr size_t kSmemKb = 224;

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

// Sections of a stage, each on a 128-byte boundary: the 4 rows above the tile, the
// tile, the 4 rows below, the wrapped columns (elements).
struct Sections {
    int pitch, main, below, edge, size;
    __host__ __device__ Sections(int ty, int pitch_, bool split) : pitch(pitch_) {
        auto up = [](int n) { return (n + 15) / 16 * 16; };
        main = up(kHalo * pitch);
        below = main + up(ty * pitch);
        edge = below + up(kHalo * pitch);
        size = edge + (split ? up(kHalo * ty) : 0);
    }
    // row i of the tile, -4 <= i < ty + 4
    __device__ int row(int i, int ty) const {
        return i < 0 ? (i + kHalo) * pitch : (i < ty ? main + i * pitch : below + (i - ty) * pitch);
    }
};

struct GradMaps {
    CUtensorMap main, halo, edge;  // boxes {pitch, ty}, {pitch, 4}, {4, ty} of the states' planes
};

struct GradArgs {
    const double* X;
    long long ldx;
    const int* sidx;  // input state of an output state
    double* out;      // component c of state s at out + (c * ns + s) * N
    int ns, nx, ny, nz, ty;
    double s[3];      // 672 / (840 h) per axis
    int pitch;        // elements of a row in shared memory
    int ntx;          // x tiles of 8 of a block's tile
    int xsplit;       // tiles along x; 1: whole rows, stored from x = 0
    int nst;          // ring stages
    int* err;
    int stall;        // test hook: the producer issues nothing
};

__device__ __forceinline__ void tma_box(void* dst, const CUtensorMap* map, int x, int y, int z, int s, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(
            smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(x), "r"(y), "r"(z), "r"(s)
        : "memory");
}

// coefficient of neighbour d over that of neighbour 1
__device__ __forceinline__ double der(int d) {
    return d == 1 ? 1.0 : (d == 2 ? -168.0 / 672.0 : (d == 3 ? 32.0 / 672.0 : (d == 4 ? -3.0 / 672.0 : 0.0)));
}

__global__ void __launch_bounds__(kThreads, 1)
    k_gradient_mma(const __grid_constant__ GradMaps maps, const GradArgs a, const WorkGrid wg) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int nst = a.nst;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);
    uint64_t* empty = full + nst;
    volatile int* ctl = reinterpret_cast<volatile int*>(empty + nst);  // [0] abort, [1] last position issued
    double* ringp = reinterpret_cast<double*>(smem + kBarBytes);
    const int nx = a.nx, ny = a.ny, nz = a.nz, ty = a.ty;
    const bool split = a.xsplit > 1;
    const Sections sec(ty, a.pitch, split);
    const long long plane = (long long)nx * ny, N = plane * nz;
    const int t = threadIdx.x, lane = t & 31;

    if (t == 0) {
        for (int i = 0; i < nst; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], (uint32_t)(blockDim.x / 32 - 1));
        }
        ctl[0] = 0;
        ctl[1] = -1;
        fence_mbar_init();
    }
    __syncthreads();

    if (t < 32) {
        // ---------------- producer ----------------
        int pos = 0;
        for (int item = blockIdx.x; item < wg.items && t == 0 && !a.stall; item += gridDim.x) {
            const int slab = item % wg.nslab;
            const int tile = (item / wg.nslab) % wg.tiles;
            const int s = a.sidx[item / (wg.nslab * wg.tiles)];
            const int zs = slab * wg.zslab;
            const int ze = min(nz, zs + wg.zslab);
            const int y0 = min((tile / a.xsplit) * ty, ny - ty);
            const int xi = tile % a.xsplit, xa = split ? xi * 8 * a.ntx - kHalo : 0;
            const int above = wrap_idx(y0 - kHalo, ny), below = wrap_idx(y0 + ty, ny);
            // wrapped columns: the last 4 left of the first tile, the first 4 right of every tile whose halo ends
            // past the row (the last one, and the one before a last tile narrower than the halo)
            const int xe = !split ? -1 : (xi == 0 ? nx - kHalo : ((xi + 1) * 8 * a.ntx + kHalo > nx ? 0 : -1));
            // 4 halo rows that wrap inside come row by row
            const bool ra = above + kHalo > ny, rb = below + kHalo > ny;
            const int xl = max(xa, 0), xn = min(nx, xa + a.pitch) - xl;  // a row's columns inside the grid
            const uint32_t bytes = (uint32_t)(8 * (ty * a.pitch + kHalo * (ra ? xn : a.pitch) +
                                                   kHalo * (rb ? xn : a.pitch) + (xe >= 0 ? kHalo * ty : 0)));
            bool stop = false;
            for (int p = zs - R; p <= ze - 1 + R; ++p, ++pos) {
                const int j = pos % nst, n = pos / nst;
                if (ctl[0] != 0) stop = true;
                else if (n > 0 && !mbar_wait(&empty[j], (uint32_t)(n - 1) & 1u)) {
                    ctl[0] = 1;
                    atomicExch(a.err, (int)QG_ERR_TIMEOUT);
                    stop = true;
                }
                if (stop) break;
                const int z = wrap_idx(p, nz);
                double* dst = ringp + (size_t)j * sec.size;
                mbar_expect_tx(&full[j], bytes);
                tma_box(dst + sec.main, &maps.main, xa, y0, z, s, &full[j]);
                const double* src = a.X + (long long)s * a.ldx + (long long)z * plane + xl;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    double* to = dst + (h ? sec.below : 0);
                    const int yh = h ? below : above;
                    if (h ? rb : ra) {
                        for (int i = 0; i < kHalo; ++i)
                            bulk_g2s(to + i * a.pitch + (xl - xa), src + (long long)wrap_idx(yh + i, ny) * nx,
                                     (uint32_t)(xn * 8), &full[j]);
                    } else {
                        tma_box(to, &maps.halo, xa, yh, z, s, &full[j]);
                    }
                }
                if (xe >= 0) tma_box(dst + sec.edge, &maps.edge, xe, y0, z, s, &full[j]);
                ctl[1] = pos;
            }
            if (stop) break;
        }
    } else {
        // ---------------- consumers ----------------
        const int w = (t >> 5) - 1, r = lane >> 2, q = lane & 3;
        const int xt = w % a.ntx, row0 = 8 * (w / a.ntx);
        double bd[KB];  // band values of the lane: input 4 kk + q - 4 against output r
#pragma unroll
        for (int kk = 0; kk < KB; ++kk) {
            const int d = 4 * kk + q - kHalo - r;
            bd[kk] = d < 0 ? -der(-d) : der(d);
        }
        int pos = 0;
        bool bad = false;
        for (int item = blockIdx.x; item < wg.items && !bad; item += gridDim.x) {
            const int slab = item % wg.nslab;
            const int tile = (item / wg.nslab) % wg.tiles;
            const int s = item / (wg.nslab * wg.tiles);
            const int zs = slab * wg.zslab;
            const int ze = min(nz, zs + wg.zslab);
            const int iy = min((tile / a.xsplit) * ty, ny - ty) + row0 + r;
            const int xi = tile % a.xsplit, xs = xi * 8 * a.ntx;  // first column of the tile
            const int x0 = xs + 8 * xt, xp = x0 + 2 * q;          // the lane's points xp, xp + 1
            const bool live = xp < nx && iy >= (tile / a.xsplit) * ty;  // rows of the tile before are its own
            // shared-memory offsets; warps and lanes past the row's end work on other columns
            const int irow = sec.row(row0 + r, ty);
            const int own = irow + (split ? xp - xs + kHalo : (xp < nx ? xp : 0));
            int xo[KB], yo[KB];
#pragma unroll
            for (int kk = 0; kk < KB; ++kk) {
                const int x = x0 + 4 * kk + q - kHalo;
                if (!split) xo[kk] = irow + wrap_idx(x, nx);
                else if (x < 0) xo[kk] = sec.edge + (row0 + r) * kHalo + x + kHalo;
                else if (x >= nx) xo[kk] = sec.edge + (row0 + r) * kHalo + min(x - nx, kHalo - 1);
                else xo[kk] = irow + min(x - xs + kHalo, a.pitch - 1);
                yo[kk] = sec.row(row0 + 4 * kk - kHalo + q, ty) + (split ? x0 + r - xs + kHalo : (x0 + r < nx ? x0 + r : 0));
            }
            double win[Q][2];  // plane z - R + d in slot (k + d) % Q at unrolled step k
            int j = pos % nst;
            uint32_t ph = (uint32_t)(pos / nst) & 1u;
            bool ok = true;
            auto lds2 = [](double (&v)[2], const double* p) {
                const double2 u = *reinterpret_cast<const double2*>(p);
                v[0] = u.x;
                v[1] = u.y;
            };
#pragma unroll
            for (int d = 0; d < 2 * R; ++d) {
                if (ok && !mbar_wait(&full[j], ph)) ok = false;
                lds2(win[d], ringp + (size_t)j * sec.size + own);
                if (++j == nst) { j = 0; ph ^= 1u; }
            }
            if (!__all_sync(0xffffffffu, ok)) {
                bad = true;
                break;
            }
            int jz = pos % nst;
            if (lane == 0) {
                for (int d = 0, i = jz; d < R; ++d) {  // planes zs - R .. zs - 1 live on in registers only
                    mbar_arrive(&empty[i]);
                    if (++i == nst) i = 0;
                }
            }
            jz = (pos + R) % nst;
            int jp = j;  // stage of plane z + R
            uint32_t php = ph;
            double* op = a.out + (long long)s * N + (long long)iy * nx + xp;
            const long long comp = (long long)a.ns * N;
            for (int z = zs; z < ze && !bad;) {
#pragma unroll
                for (int k = 0; k < Q; ++k) {
                    if (z >= ze) break;
                    const bool got = mbar_wait(&full[jp], php);
                    if (!__all_sync(0xffffffffu, got)) {
                        bad = true;
                        break;
                    }
                    const double* stz = ringp + (size_t)jz * sec.size;
                    lds2(win[(k + 2 * R) % Q], ringp + (size_t)jp * sec.size + own);
                    double g[3][2] = {};
#pragma unroll
                    for (int kk = 0; kk < KB; ++kk) {
                        dmma(g[0], stz[xo[kk]], bd[kk]);
                        dmma(g[1], bd[kk], stz[yo[kk]]);
                    }
#pragma unroll
                    for (int e = 0; e < 2; ++e)
#pragma unroll
                        for (int d = R; d >= 1; --d)
                            g[2][e] += der(d) * (win[(k + R + d) % Q][e] - win[(k + R - d) % Q][e]);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&empty[jz]);  // plane z is no longer read
                    if (live) {
#pragma unroll
                        for (int c = 0; c < 3; ++c)
                            *reinterpret_cast<double2*>(op + c * comp + (long long)z * plane) =
                                make_double2(a.s[c] * g[c][0], a.s[c] * g[c][1]);
                    }
                    ++z;
                    if (++jz == nst) jz = 0;
                    if (++jp == nst) { jp = 0; php ^= 1u; }
                }
            }
            if (bad) break;
            __syncwarp();
            if (lane == 0)
                for (int d = 0; d < R; ++d) {  // planes ze .. ze + R - 1
                    mbar_arrive(&empty[jz]);
                    if (++jz == nst) jz = 0;
                }
            pos += ze - zs + 2 * R;
        }
        if (bad) {
            ctl[0] = 1;
            if (lane == 0) atomicExch(a.err, (int)QG_ERR_TIMEOUT);
        }
    }
    __syncthreads();
    if (t == 0 && ctl[0]) {
        // wind down: wait (bounded) for the fills still in flight
        const int last = ctl[1];
        for (int ps = max(0, last - nst + 1); ps <= last; ++ps) mbar_wait(&full[ps % nst], (uint32_t)(ps / nst) & 1u);
    }
}

// Tile of a block: among the shapes whose warps (one per 8 x 8 points) and ring fit, the one
// that copies and computes the fewest points per useful point; a copied point costs about half
// of a computed one.
bool plan(GradArgs& a) {
    const int nxt = (a.nx + 7) / 8, maxw = kThreads / 32 - 1;
    double least = 1e300;
    for (int split = 1; split <= nxt; ++split) {
        const int ntx = (nxt + split - 1) / split;
        if (ntx > maxw || (split > 1 && (nxt + ntx - 1) / ntx != split)) continue;
        if (split == 2 && 8 * ntx + kHalo > a.nx) continue;  // the first tile would wrap on both sides
        const int cols = split > 1 ? 8 * ntx + 2 * kHalo : a.nx;
        // row pitch in which the 8 rows x 4 inputs of an operand fall into different banks
        int pitch = (cols + 3) / 4 * 4;
        if (pitch % 8 != 4) pitch += 4;
        if (pitch > 256) continue;
        for (int nyw = 1; ntx * nyw <= maxw && 8 * nyw <= a.ny; ++nyw) {
            const int ty = 8 * nyw;
            const int nst = ring_stages(R, (size_t)Sections(ty, pitch, split > 1).size * 8, 3, kSmemKb);
            if (nst < 0) break;
            const double cost = (a.ny + ty - 1) / ty * split * (8.0 * ntx * ty + 0.5 * cols * (ty + 2 * kHalo));
            if (cost < least) {
                least = cost;
                a.ty = ty;
                a.pitch = pitch;
                a.ntx = ntx;
                a.xsplit = split;
                a.nst = nst;
            }
        }
    }
    return least < 1e300;
}

}  // namespace

int launch_gradient8(const double* X, long long ldx, int nin, const int* sidx, int ns, double* out, int nx, int ny, int nz,
                     const double* h, int* err, int stall, cudaStream_t st) {
    GradArgs a{X, ldx, sidx, out, ns, nx, ny, nz, 0, {}, 0, 0, 0, 0, err, stall};
    for (int d = 0; d < 3; ++d) a.s[d] = 672.0 / (840.0 * h[d]);
    tchost::EncodeTiledFn enc = tchost::encode_fn();
    if (!enc || nx % 2 || ldx % 2 || (uintptr_t)X % 16 || (uintptr_t)out % 16 || !plan(a)) return QG_ERR_UNSUPPORTED;
    GradMaps maps;
    const cuuint64_t dims[4] = {(cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz, (cuuint64_t)nin};
    const cuuint64_t strides[3] = {(cuuint64_t)nx * 8, (cuuint64_t)nx * ny * 8, (cuuint64_t)ldx * 8};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    auto encode = [&](CUtensorMap* map, int bx, int by) {
        const cuuint32_t box[4] = {(cuuint32_t)bx, (cuuint32_t)by, 1, 1};
        return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<double*>(X), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    if (!encode(&maps.main, a.pitch, a.ty) || !encode(&maps.halo, a.pitch, kHalo) || !encode(&maps.edge, kHalo, a.ty))
        return QG_ERR_UNSUPPORTED;
    if (allow_max_dynamic_smem(k_gradient_mma) != cudaSuccess) return QG_ERR_CUDA;
    const int G0 = sm_count();
    WorkGrid wg;
    wg.tiles = (ny + a.ty - 1) / a.ty * a.xsplit;
    // z slabs: the fewest plane steps of the busiest block; the 2R planes that only fill the
    // window cost about half a step each
    const long long base = (long long)ns * wg.tiles;
    double least = 1e300;
    wg.nslab = wg.zslab = 1;
    for (int n = 1; n <= std::max(1, nz / 4); ++n) {
        const int zs = (nz + n - 1) / n, slabs = (nz + zs - 1) / zs;
        const double cost = (double)((base * slabs + G0 - 1) / G0) * (zs + R);
        if (cost < 0.98 * least) {
            least = cost;
            wg.nslab = slabs;
            wg.zslab = zs;
        }
    }
    if (base * wg.nslab > 0x7fffffffLL) return QG_ERR_UNSUPPORTED;
    wg.items = (int)(base * wg.nslab);
    const size_t smem = kBarBytes + (size_t)a.nst * Sections(a.ty, a.pitch, a.xsplit > 1).size * 8;
    const int threads = 32 * (a.ntx * (a.ty / 8) + 1);
    k_gradient_mma<<<std::min(G0, wg.items), threads, smem, st>>>(maps, a, wg);
    QG_CUDA_TRY(cudaGetLastError());
    return QG_OK;
}

}  // namespace qg
