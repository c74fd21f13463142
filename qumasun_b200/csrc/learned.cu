// Learned LOBPCG preconditioner: a 4-layer periodic 3D convolutional network
//   in  = [r / rms(r), V / vscale]                         (2 channels)
//   h1  = relu(conv3(in)), h2 = relu(conv3(h1)), h3 = relu(conv3(h2))   (16 channels each)
//   out = conv3(h3)                                       (1 channel)
// applied as w = T r + rms(r) * out, T the kinetic preconditioner (precond.cu), so
// the network learns a correction to the plain preconditioner and an untrained
// (zero last layer) network leaves it unchanged. 3^3 kernels, circular padding
// (the grid is periodic), BF16 weights and activations, FP32 accumulation; about
// 15.1k multiply-adds per voxel, as the network the engine was specified with.
//
// Kernels (CUDA cores, one thread per voxel of an 8 x 8 x 4 tile):
//   k_conv_fwd     out[co][v] = b[co] + sum_ci sum_tap W[co][ci][tap] in[ci][v + off(tap)];
//                  the input tile (+ 1-voxel periodic halo) of one channel and that
//                  channel's weights, stored [tap][co], sit in shared memory;
// Backward pass on the tensor cores, FP32 gradients as three BF16 pieces (described below):
//   k_dgrad_mma    backward data of the 16 -> 16 layers (transposed convolution = convolution
//                  with transposed weights and flipped taps on a periodic grid) times the ReLU
//                  mask of the layer below; the 1 -> 16 step runs in k_conv_fwd;
//   k_wgrad_mma    dW[co][ci][tap] = sum_v dout[co][v] in[ci][v + off(tap)], tiles in turn per
//                  block, the blocks' sums added in a fixed order (deterministic);
//   k_adam         Adam on FP32 master weights, BF16 copies for the kernels.
// Forward pass on the tensor cores (the default where nx is a multiple of 8):
//   k_conv_tc      every layer as 27 tcgen05.mma per z plane over shared-memory halo
//                  planes (described below); k_conv_fwd then serves the backward pass and
//                  grids the tensor-core kernel does not take.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "qg_internal.h"
#include "tc_common.cuh"

namespace {

constexpr int TX = 8, TY = 8, TZ = 4;
constexpr int TV = TX * TY * TZ;  // voxels per tile
constexpr int HX = TX + 2, HY = TY + 2, HZ = TZ + 2;
constexpr int HV = HX * HY * HZ;
constexpr int kLayers = 4;
constexpr int kCin[kLayers] = {2, 16, 16, 16};
constexpr int kCout[kLayers] = {16, 16, 16, 1};

constexpr int wcount(int l) { return kCin[l] * kCout[l] * 27; }
constexpr int lsize(int l) { return wcount(l) + kCout[l]; }
constexpr int woff(int l) { return l == 0 ? 0 : woff(l - 1) + lsize(l - 1); }
constexpr int kParams = woff(kLayers);  // 15169

struct Grid {
    int nx, ny, nz;
    int tx, ty, tz;  // tiles per axis
    long long N;
};

__device__ __forceinline__ int wrapi(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

__device__ __forceinline__ int wrap_any(int i, int n) {
    i %= n;
    return i < 0 ? i + n : i;
}

__device__ __forceinline__ float ldf(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ float ldf(const float* p) { return *p; }
__device__ __forceinline__ void stf(__nv_bfloat16* p, float v) { *p = __float2bfloat16(v); }
__device__ __forceinline__ void stf(float* p, float v) { *p = v; }

// out (B x COUT x N) = conv(in (B x CIN x N)); W bf16 [COUT][CIN][27]; bias may be null.
// mask (B x COUT x N, may be null): out *= (mask > 0) (ReLU derivative of the layer below).
template <int CIN, int COUT, bool RELU, typename TI, typename TO>
__global__ void __launch_bounds__(TV) k_conv_fwd(const TI* __restrict__ in, const __nv_bfloat16* __restrict__ W,
                                                 const float* __restrict__ bias, TO* __restrict__ out,
                                                 const __nv_bfloat16* __restrict__ mask, Grid g) {
    __shared__ float tin[HV];
    __shared__ __align__(16) float w[27 * COUT];
    const int tile = blockIdx.x, b = blockIdx.y;
    const int bx = (tile % g.tx) * TX, by = ((tile / g.tx) % g.ty) * TY, bz = (tile / (g.tx * g.ty)) * TZ;
    const int t = threadIdx.x;
    const int lx = t % TX, ly = (t / TX) % TY, lz = t / (TX * TY);
    const int x = bx + lx, y = by + ly, z = bz + lz;
    const bool inside = x < g.nx && y < g.ny && z < g.nz;
    float acc[COUT];
#pragma unroll
    for (int c = 0; c < COUT; ++c) acc[c] = bias ? bias[c] : 0.f;
    const TI* inb = in + (long long)b * CIN * g.N;
    for (int ci = 0; ci < CIN; ++ci) {
        const TI* ic = inb + (long long)ci * g.N;
        for (int i = t; i < HV; i += TV) {
            const int hx = i % HX, hy = (i / HX) % HY, hz = i / (HX * HY);
            const int gx = wrapi(bx + hx - 1, g.nx), gy = wrapi(by + hy - 1, g.ny), gz = wrapi(bz + hz - 1, g.nz);
            tin[i] = ldf(ic + gx + (long long)g.nx * (gy + (long long)g.ny * gz));
        }
        for (int i = t; i < 27 * COUT; i += TV) {
            const int tap = i / COUT, co = i % COUT;
            w[i] = __bfloat162float(W[((long long)co * CIN + ci) * 27 + tap]);
        }
        __syncthreads();
#pragma unroll
        for (int tap = 0; tap < 27; ++tap) {
            const int dx = tap % 3, dy = (tap / 3) % 3, dz = tap / 9;
            const float xv = tin[(lx + dx) + HX * ((ly + dy) + HY * (lz + dz))];
            if constexpr (COUT % 4 == 0) {
#pragma unroll
                for (int c = 0; c < COUT; c += 4) {
                    const float4 wv = *reinterpret_cast<const float4*>(&w[tap * COUT + c]);
                    acc[c] += wv.x * xv;
                    acc[c + 1] += wv.y * xv;
                    acc[c + 2] += wv.z * xv;
                    acc[c + 3] += wv.w * xv;
                }
            } else {
#pragma unroll
                for (int c = 0; c < COUT; ++c) acc[c] += w[tap * COUT + c] * xv;
            }
        }
        __syncthreads();
    }
    if (!inside) return;
    const long long v = x + (long long)g.nx * (y + (long long)g.ny * z);
#pragma unroll
    for (int c = 0; c < COUT; ++c) {
        float o = acc[c];
        if (RELU) o = fmaxf(o, 0.f);
        const long long idx = ((long long)b * COUT + c) * g.N + v;
        if (mask && __bfloat162float(mask[idx]) <= 0.f) o = 0.f;
        stf(out + idx, o);
    }
}

// ---------------- backward pass on the tensor cores (mma.sync m16n8k16, BF16 in, FP32 sums)
// The FP32 gradients enter as three BF16 pieces (d = d1 + d2 + d3 to 2^-24 of d or 5e-41), the activations and
// weights are BF16 already, so the products are those of the FP32 kernels; the FP32 sums of a
// tile are added to the running sums with ordinary rounding. Bound: k_dgrad_mma the shared-memory reads of the
// operands (ldmatrix, 80 % of L1), k_wgrad_mma the tensor pipe (44 %) and, before it in every tile, the loads
// that stage the tile; one layer of 16 x 16 channels at 32 states of 40^3 is 14 G multiply-adds: 0.43
// and 0.35 ms.
// Operand tiles are [voxel][16 channels], 32 bytes a voxel; the two 16-byte halves of a voxel
// change places every 4 voxels, so the 8 rows of any ldmatrix fall into different banks.
__device__ __forceinline__ int half_at(int v, int h) { return (2 * v + (h ^ ((v >> 2) & 1))) * 8; }  // in elements

__device__ __forceinline__ void ldm4(uint32_t (&r)[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 8 channels of one voxel as three BF16 pieces into the half h of voxel v of each piece's tile.
__device__ __forceinline__ void put_pieces(__nv_bfloat16* tile, int piece_elems, int v, int h, const float (&d)[8]) {
    __align__(16) __nv_bfloat16 p[3][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        // finite values beyond the largest BF16 round towards zero, Inf is one piece (Inf - Inf is NaN)
        p[0][i] = fabsf(d[i]) > 3.38e38f ? __float2bfloat16_rz(d[i]) : __float2bfloat16(d[i]);
        const float r1 = isinf(d[i]) ? 0.f : d[i] - __bfloat162float(p[0][i]);
        p[1][i] = __float2bfloat16(r1);
        p[2][i] = __float2bfloat16(r1 - __bfloat162float(p[1][i]));
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
        *reinterpret_cast<uint4*>(tile + k * piece_elems + half_at(v, h)) = *reinterpret_cast<const uint4*>(p[k]);
}

constexpr int kWgThreads = 288;  // 9 warps, three taps each (dz = w / 3, dy = w % 3)

// Weight and bias gradients: dW[co][ci][tap] = sum_v dout[co][v] in[ci][v + off(tap)], the
// contraction over voxels as 16 ci x 16 voxels times 16 voxels x 8 co. A block walks the tiles
// blockIdx.x, + gridDim.x, ... and writes one set of partial sums: part[blk][co][ci * 27 + tap],
// then part[blk][COUT * CIN * 27 + co].
template <int CIN, int COUT>
__global__ void __launch_bounds__(kWgThreads) k_wgrad_mma(const __nv_bfloat16* __restrict__ in,
                                                          const float* __restrict__ dout, float* __restrict__ part,
                                                          Grid g, int ntile) {
    constexpr int NH = COUT > 8 ? 2 : 1;
    extern __shared__ __align__(16) __nv_bfloat16 wsm[];
    __nv_bfloat16* at = wsm;                 // [HV][16]
    __nv_bfloat16* dt = wsm + HV * 16;       // [3][TV][16]
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    const int tiles = g.tx * g.ty * g.tz;
    float sum[3][NH][4], bias[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) bias[i] = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int n = 0; n < NH; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[k][n][e] = 0.f;
    for (int it = blockIdx.x; it < ntile; it += gridDim.x) {
        const int b = it / tiles, tile = it - b * tiles;
        const int bx = (tile % g.tx) * TX, by = ((tile / g.tx) % g.ty) * TY, bz = (tile / (g.tx * g.ty)) * TZ;
        const __nv_bfloat16* inb = in + (long long)b * CIN * g.N;
        const float* db = dout + (long long)b * COUT * g.N;
        for (int i = t; i < 2 * HV; i += kWgThreads) {
            const int v = i >> 1, h = i & 1;
            const int hx = v % HX, hy = (v / HX) % HY, hz = v / (HX * HY);
            const long long at0 = wrap_any(bx + hx - 1, g.nx) +
                                  (long long)g.nx * (wrap_any(by + hy - 1, g.ny) + (long long)g.ny * wrap_any(bz + hz - 1, g.nz));
            __align__(16) __nv_bfloat16 c[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
                c[j] = h * 8 + j < CIN ? inb[(long long)(h * 8 + j) * g.N + at0] : __float2bfloat16(0.f);
            *reinterpret_cast<uint4*>(at + half_at(v, h)) = *reinterpret_cast<const uint4*>(c);
        }
        for (int i = t; i < 2 * TV; i += kWgThreads) {  // h = i & 1 = t & 1: one half per thread
            const int v = i >> 1, h = i & 1;
            const int x = bx + v % TX, y = by + (v / TX) % TY, z = bz + v / (TX * TY);
            const bool inside = x < g.nx && y < g.ny && z < g.nz;  // others contribute nothing
            const long long at0 = x + (long long)g.nx * (y + (long long)g.ny * z);
            float d[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                d[j] = inside && h * 8 + j < COUT ? db[(long long)(h * 8 + j) * g.N + at0] : 0.f;
                bias[j] += d[j];
            }
            put_pieces(dt, TV * 16, v, h, d);
        }
        __syncthreads();
        float acc[3][NH][4];
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int n = 0; n < NH; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[k][n][e] = 0.f;
        const int mi = lane >> 3, row = lane & 7;
        const int dz = w / 3, dy = w % 3;
        for (int k0 = 0; k0 < TV; k0 += 16) {  // rows of 8 voxels: (ly, lz) and (ly + 1, lz)
            const int ly = (k0 / TX) % TY, lz = k0 / (TX * TY);
            uint32_t bf[3][4];
#pragma unroll
            for (int p = 0; p < 3; ++p) ldm4t(bf[p], dt + p * TV * 16 + half_at(k0 + (mi & 1) * 8 + row, mi >> 1));
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
                uint32_t af[4];
                ldm4t(af, at + half_at(dx + row + HX * (ly + (mi >> 1) + dy + HY * (lz + dz)), mi & 1));
#pragma unroll
                for (int p = 0; p < 3; ++p)
#pragma unroll
                    for (int n = 0; n < NH; ++n) mma16816(acc[dx][n], af, bf[p][2 * n], bf[p][2 * n + 1]);
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int n = 0; n < NH; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) sum[k][n][e] += acc[k][n][e];
        __syncthreads();
    }
    float* pb = part + (long long)blockIdx.x * (COUT * CIN * 27 + COUT);
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int n = 0; n < NH; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int ci = (lane >> 2) + 8 * (e >> 1), co = 8 * n + 2 * (lane & 3) + (e & 1);
                if (ci < CIN && co < COUT) pb[(co * CIN + ci) * 27 + 3 * w + k] = sum[k][n][e];
            }
    float(*bsum)[8] = reinterpret_cast<float(*)[8]>(wsm);  // the tiles are read no more
#pragma unroll
    for (int j = 0; j < 8; ++j) bsum[t][j] = bias[j];
    __syncthreads();
    if (t < COUT) {
        float s = 0.f;
        for (int i = t >> 3; i < kWgThreads; i += 2) s += bsum[i][t & 7];
        pb[COUT * CIN * 27 + t] = s;
    }
}

// Backward data of a 16 -> 16 layer: out[c][v] = (mask > 0) sum_k sum_tap W[k][c][tap] din[k][v - off(tap)],
// 16 voxels x 16 k times 16 k x 8 c per tap; Wt as k_transpose_w writes it ([c][k][26 - tap], so
// that the sum reads din[v + off]). One block per tile, two groups of 16 voxels per warp.
constexpr int kDgSmem = (3 * HV * 16 + 27 * 256) * 2;
__global__ void __launch_bounds__(256) k_dgrad_mma(const float* __restrict__ din, const __nv_bfloat16* __restrict__ Wt,
                                                   float* __restrict__ out, const __nv_bfloat16* __restrict__ mask,
                                                   Grid g) {
    extern __shared__ __align__(16) __nv_bfloat16 wsm[];
    __nv_bfloat16* dt = wsm;                      // [3][HV][16]
    __nv_bfloat16* ws = wsm + 3 * HV * 16;        // [27][lane][n half][k half][2]
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    const int tile = blockIdx.x, b = blockIdx.y;
    const int bx = (tile % g.tx) * TX, by = ((tile / g.tx) % g.ty) * TY, bz = (tile / (g.tx * g.ty)) * TZ;
    const float* db = din + (long long)b * 16 * g.N;
    for (int i = t; i < 27 * 256; i += 256) {
        const int tap = i >> 8, l = (i >> 3) & 31, n = (i >> 2) & 1, kh = (i >> 1) & 1, e = i & 1;
        const int c = 8 * n + (l >> 2), k = 8 * kh + 2 * (l & 3) + e;
        ws[i] = Wt[(c * 16 + k) * 27 + tap];
    }
    for (int i = t; i < 2 * HV; i += 256) {
        const int v = i >> 1, h = i & 1;
        const int hx = v % HX, hy = (v / HX) % HY, hz = v / (HX * HY);
        const long long at0 = wrap_any(bx + hx - 1, g.nx) +
                              (long long)g.nx * (wrap_any(by + hy - 1, g.ny) + (long long)g.ny * wrap_any(bz + hz - 1, g.nz));
        float d[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) d[j] = db[(long long)(h * 8 + j) * g.N + at0];
        put_pieces(dt, HV * 16, v, h, d);
    }
    __syncthreads();
    const int mi = lane >> 3, row = lane & 7;
    float acc[2][2][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[m][n][e] = 0.f;
    // group m of the warp: voxel rows ly, ly + 1 of plane lz
    const int lz = w >> 1, ly0 = (w & 1) * 4;
#pragma unroll 1
    for (int tap = 0; tap < 27; ++tap) {
        const int dx = tap % 3, dy = (tap / 3) % 3, dz = tap / 9;
        const uint4 bw = *reinterpret_cast<const uint4*>(ws + tap * 256 + lane * 8);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const int v = dx + row + HX * (ly0 + 2 * m + (mi & 1) + dy + HY * (lz + dz));
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                uint32_t af[4];
                ldm4(af, dt + p * HV * 16 + half_at(v, mi >> 1));
                mma16816(acc[m][0], af, bw.x, bw.y);
                mma16816(acc[m][1], af, bw.z, bw.w);
            }
        }
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int x = bx + (lane >> 2), y = by + ly0 + 2 * m + (e >> 1), z = bz + lz;
                if (x >= g.nx || y >= g.ny || z >= g.nz) continue;
                const int c = 8 * n + 2 * (lane & 3) + (e & 1);
                const long long idx = ((long long)b * 16 + c) * g.N + x + (long long)g.nx * (y + (long long)g.ny * z);
                out[idx] = __bfloat162float(mask[idx]) <= 0.f ? 0.f : acc[m][n][e];
            }
}

// grad[i] = sum over blocks of part[blk][i]: 8 threads per value add contiguous eighths of the
// blocks in order, then the eighths are added in order.
__global__ void __launch_bounds__(256) k_reduce_parts(const float* __restrict__ part, int nblk, int n,
                                                      float* __restrict__ grad) {
    __shared__ float sm[8][32];
    const int l = threadIdx.x & 31, seg = threadIdx.x >> 5, i = blockIdx.x * 32 + l;
    float s = 0.f;
    if (i < n) {
        const int k1 = (int)((long long)nblk * (seg + 1) / 8);
#pragma unroll 4
        for (int k = (int)((long long)nblk * seg / 8); k < k1; ++k) s += part[(long long)k * n + i];
    }
    sm[seg][l] = s;
    __syncthreads();
    if (seg == 0 && i < n) {
        s = sm[0][l];
#pragma unroll
        for (int k = 1; k < 8; ++k) s += sm[k][l];
        grad[i] = s;
    }
}

// transposed, flipped weights of one layer: Wt[ci][co][26 - tap] = W[co][ci][tap]
__global__ void k_transpose_w(const __nv_bfloat16* __restrict__ W, int cin, int cout, __nv_bfloat16* __restrict__ Wt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cin * cout * 27) return;
    const int co = i / (cin * 27), ci = (i / 27) % cin, tap = i % 27;
    Wt[((long long)ci * cout + co) * 27 + (26 - tap)] = W[i];
}

__global__ void k_to_bf16(const float* __restrict__ src, int n, __nv_bfloat16* __restrict__ dst) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = __float2bfloat16(src[i]);
}

__global__ void k_adam(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                       const float* __restrict__ g, int n, float lr, float b1, float b2, float eps, float c1,
                       float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// rms[s] = sqrt(mean_i R[s][i]^2) (one block per state)
__global__ void k_rms(const double* __restrict__ R, long long ld, long long N, double* __restrict__ rms) {
    __shared__ double red[32];
    const double* r = R + (long long)blockIdx.x * ld;
    double s = 0.0;
    for (long long i = threadIdx.x; i < N; i += blockDim.x) s += r[i] * r[i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
        const double v = sqrt(tot / (double)N);
        rms[blockIdx.x] = v > 0.0 ? v : 1.0;
    }
}

// network input of state s: [R[s] / rms[s], V / vscale] as bf16 (B x 2 x N)
__global__ void k_make_input(const double* __restrict__ R, long long ld, const double* __restrict__ V, double vscale,
                             const double* __restrict__ rms, long long N, int B, __nv_bfloat16* __restrict__ in) {
    const long long total = (long long)B * N;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int s = (int)(e / N);
        const long long i = e - (long long)s * N;
        in[((long long)s * 2) * N + i] = __double2bfloat16(R[(long long)s * ld + i] / rms[s]);
        in[((long long)s * 2 + 1) * N + i] = __double2bfloat16(V[i] / vscale);
    }
}

// out[s][i] (+)= rms[s] * p[s][i]
__global__ void k_emit(const float* __restrict__ p, const double* __restrict__ rms, long long N, int B, double* __restrict__ out,
                       long long ldo, int accumulate) {
    const long long total = (long long)B * N;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int s = (int)(e / N);
        const long long i = e - (long long)s * N;
        const double v = rms[s] * (double)p[e];
        double* o = out + (long long)s * ldo + i;
        *o = accumulate ? *o + v : v;
    }
}

// MSE loss terms: dp = 2 (p - y/rms) / sum_s |y_s/rms_s|^2, lossv[e] = (p - t)^2, tnorm[e] = t^2
__global__ void k_loss(const float* __restrict__ p, const double* __restrict__ Y, long long ldy,
                       const double* __restrict__ rms, long long N, int B, float* __restrict__ dp,
                       double* __restrict__ acc2) {
    __shared__ double red[2][32];
    const long long total = (long long)B * N;
    double se = 0.0, st = 0.0;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int s = (int)(e / N);
        const long long i = e - (long long)s * N;
        const double tv = Y[(long long)s * ldy + i] / rms[s];
        const double d = (double)p[e] - tv;
        dp[e] = (float)(2.0 * d);
        se += d * d;
        st += tv * tv;
    }
    for (int o = 16; o > 0; o >>= 1) {
        se += __shfl_xor_sync(0xffffffffu, se, o);
        st += __shfl_xor_sync(0xffffffffu, st, o);
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = se;
        red[1][threadIdx.x >> 5] = st;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, bsum = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            a += red[0][w];
            bsum += red[1][w];
        }
        acc2[2 * blockIdx.x] = a;
        acc2[2 * blockIdx.x + 1] = bsum;
    }
}

__global__ void k_scale_f(float* __restrict__ x, long long n, const double* __restrict__ inv) {
    const float s = (float)inv[0];
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        x[i] *= s;
}


// ---------------------------------------------------------------------------
// The network layers on the 5th-generation tensor cores (sm_100a).
// One CTA (4 warps) owns a column block of CX x CY voxels of one state (two groups of 8
// x-voxels, each one M = 128 MMA with its own 16-column accumulator) and marches CZ
// planes in z. The input's halo planes (CX+2 x CY+2 voxels) sit in shared memory split
// into two 8-channel halves, each voxel's 8 channels one 16-byte row, so that operand A
// of one tap -- 128 voxels (x fastest) x 16 input channels -- is the canonical K-major
// layout without swizzle at a shifted start address: each run of 8 voxels along x is one
// core matrix (8 rows of 16 bytes), consecutive y rows are HXC * 16 bytes apart (SBO)
// and the second channel half one half-plane further (LBO). The 27 taps are then 27
// tcgen05.mma.kind::f16 (M 128, N 16, K 16, BF16 in, FP32 accumulator in TMEM) with no
// im2col copy; the weights sit as [tap][channel half][co][8 ci] (LBO 256 B, SBO 128 B).
// After the MMAs of plane z are committed the CTA loads halo plane z + 2 (ring of 4),
// then reads the accumulator back with tcgen05.ld (one TMEM lane per voxel), adds the
// bias, applies ReLU where the layer has one and stores (BF16 activations, FP32 for the
// last layer). Layers with fewer channels use the same 16 x 16 MMA: the missing input
// channels are zero in the halo, the missing outputs have zero weights and are not
// stored. Same periodic convolution as k_conv_fwd; the products are summed in a
// different order (per tap on the tensor cores).
using namespace qg::tc;

constexpr int CX = 16, CY = 16, CZ = 8;         // voxels of a CTA's column block; z planes per CTA
constexpr int kGroupsX = CX / 8;                // M = 128 groups (8 x-voxels x 16 y rows) per plane
constexpr int HXC = CX + 2, HYC = CY + 2;
constexpr int kHalfB = HXC * HYC * 16;          // one 8-channel half of a halo plane (5184 B)
constexpr int kSlotB = 2 * kHalfB;              // one halo plane
constexpr int kSlots = 4;
constexpr int kWB = 27 * 512;                   // weights, bf16 [tap][half][co][8]
// shared memory: the halo ring, the weights, the mbarrier and the TMEM address (54 KB;
// a tap's operand reaches at most the end of the ring)
constexpr int kConvTcSmem = kSlots * kSlotB + kWB + 64;
constexpr uint32_t kIdescConv = (1u << 4) | (1u << 7) | (1u << 10) | ((16u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ uint64_t desc_nosw(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr & 0x3FFFF) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

__device__ __forceinline__ void umma_conv(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(kIdescConv), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

// out (B x COUT x N) = act(conv(in (B x CIN x N)) + bias); W bf16 [COUT][CIN][27];
// CIN, COUT <= 16 (the MMA is always 16 x 16 per tap: missing input channels are zero
// in the halo, missing output channels have zero weights and are not stored). Grid:
// x = (x block, y block, z slab), y = state. Requires nx % 8 == 0; in a last x block of
// 8 voxels the second group computes on periodic copies and stores nothing.
template <int CIN, int COUT, bool RELU, typename TO>
__global__ void __launch_bounds__(128) k_conv_tc(const __nv_bfloat16* __restrict__ in,
                                                 const __nv_bfloat16* __restrict__ W,
                                                 const float* __restrict__ bias, TO* __restrict__ out,
                                                 Grid g, int tiles_y, int* err) {
    static_assert(CIN >= 1 && CIN <= 16 && COUT >= 1 && COUT <= 16, "16 x 16 channel MMA");
    extern __shared__ __align__(128) unsigned char csm[];
    unsigned char* halo = csm;
    unsigned char* wsm = csm + kSlots * kSlotB;
    uint64_t* bar = reinterpret_cast<uint64_t*>(wsm + kWB);
    volatile uint32_t* tslot = reinterpret_cast<volatile uint32_t*>(bar + 1);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int txb = (g.nx + CX - 1) / CX;
    int blk = blockIdx.x;
    const int xb = blk % txb;
    blk /= txb;
    const int yb = blk % tiles_y;
    const int zs = blk / tiles_y;
    const int b = blockIdx.y;
    const int x0 = xb * CX, y0 = yb * CY, z0 = zs * CZ, z1 = min(g.nz, z0 + CZ);

    if (t == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32((const void*)tslot)),
                     "r"(32)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // weights: element ((tap * 2 + h) * 16 + co) * 8 + j = W[co][h * 8 + j][tap] (zero past CIN, COUT)
    __nv_bfloat16* wb = reinterpret_cast<__nv_bfloat16*>(wsm);
    for (int i = t; i < 27 * 256; i += 128) {
        const int j = i & 7, co = (i >> 3) & 15, h = (i >> 7) & 1, tap = i >> 8, ci = h * 8 + j;
        wb[i] = (ci < CIN && co < COUT) ? W[(co * CIN + ci) * 27 + tap] : __float2bfloat16(0.f);
    }
    if constexpr (CIN < 16) {
        // the channels the input lacks stay zero in every halo plane
        for (int i = t; i < kSlots * kSlotB / 16; i += 128) reinterpret_cast<uint4*>(halo)[i] = make_uint4(0, 0, 0, 0);
        __syncthreads();
    }
    const __nv_bfloat16* inb = in + (long long)b * CIN * g.N;
    const int xl0 = wrap_any(x0 - 1, g.nx), xr0 = wrap_any(x0 + CX, g.nx);
    int xm[kGroupsX];  // start of each 8-voxel interior run (periodic past nx; multiples of 8)
#pragma unroll
    for (int q = 0; q < kGroupsX; ++q) xm[q] = wrap_any(x0 + 8 * q, g.nx);
    auto load_plane = [&](int z) {  // z in [-1, nz]: halo plane z into slot (z + 4) % 4
        const int zz = wrap_any(z, g.nz);
        unsigned char* dst = halo + ((z + 4) & 3) * kSlotB;
        // one (channel, y row) per step: each run of 8 interior voxels as one 16-byte load
        // (x0 and nx are multiples of 8), the two periodic edge voxels as single loads
        for (int e = t; e < CIN * HYC; e += 128) {
            // channels on consecutive lanes: 8 lanes fill one voxel's 16-byte row
            const int ci = e % CIN, yh = e / CIN;
            const long long row = (long long)ci * g.N + (long long)g.nx * (wrap_any(y0 + yh - 1, g.ny) + (long long)g.ny * zz);
            __nv_bfloat16 vals[HXC];
            vals[0] = inb[row + xl0];
            vals[HXC - 1] = inb[row + xr0];
#pragma unroll
            for (int q = 0; q < kGroupsX; ++q) {
                const uint4 mid = *reinterpret_cast<const uint4*>(inb + row + xm[q]);
                const __nv_bfloat16* mv = reinterpret_cast<const __nv_bfloat16*>(&mid);
#pragma unroll
                for (int i = 0; i < 8; ++i) vals[1 + 8 * q + i] = mv[i];
            }
            __nv_bfloat16* rowdst = reinterpret_cast<__nv_bfloat16*>(dst + (ci >> 3) * kHalfB + yh * HXC * 16) + (ci & 7);
#pragma unroll
            for (int xh = 0; xh < HXC; ++xh) rowdst[xh * 8] = vals[xh];
        }
    };
    load_plane(z0 - 1);
    load_plane(z0);
    load_plane(z0 + 1);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // thread stores -> tensor core reads
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    const uint32_t hbase = smem_u32(halo), wbase = smem_u32(wsm);
    float bs[COUT];
#pragma unroll
    for (int c = 0; c < COUT; ++c) bs[c] = bias[c];
    const int m = warp * 32 + lane, xl = m & 7, yl = m >> 3;
    uint32_t phase = 0;
    bool bad = false;
    for (int z = z0; z < z1; ++z) {
        if (t == 0) {
#pragma unroll 1
            for (int tap = 0; tap < 27; ++tap) {
                const int dx = tap % 3, dy = (tap / 3) % 3, dz = tap / 9;
                const uint64_t bd = desc_nosw(wbase + tap * 512, 256, 128);
#pragma unroll
                for (int q = 0; q < kGroupsX; ++q) {
                    const uint32_t a =
                        hbase + (uint32_t)((((z - 1 + dz) + 4) & 3) * kSlotB + (dy * HXC + dx + 8 * q) * 16);
                    umma_conv(tmem + (uint32_t)(16 * q), desc_nosw(a, kHalfB, HXC * 16), bd, tap ? 1u : 0u);
                }
            }
            umma_commit(bar);
        }
        if (z + 1 < z1) load_plane(z + 2);  // for plane z + 1 (the slot of plane z - 2, not read now)
        const bool ok = mbar_wait(bar, phase);
        if (__syncthreads_or(!ok)) {
            bad = true;
            break;
        }
        phase ^= 1u;
        tc_fence_after();
        const int y = y0 + yl;
#pragma unroll
        for (int q = 0; q < kGroupsX; ++q) {
            uint32_t r[16];
            tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(16 * q), r);
            tmem_wait_ld();
            const int x = x0 + 8 * q + xl;
            if (y < g.ny && x < g.nx) {
                const long long v = x + (long long)g.nx * (y + (long long)g.ny * z);
                TO* ob = out + (long long)b * COUT * g.N + v;
#pragma unroll
                for (int c = 0; c < COUT; ++c) {
                    float o = __uint_as_float(r[c]) + bs[c];
                    if (RELU) o = fmaxf(o, 0.f);
                    stf(ob + (long long)c * g.N, o);
                }
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    }
    if (bad) {
        if (t == 0) {
            atomicExch(err, (int)QG_ERR_TIMEOUT);
            mbar_wait(bar, phase);  // bounded: the MMAs in flight finish before TMEM is freed
        }
        __syncthreads();
    }
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(32) : "memory");
    }
}

bool conv_tc_ok(const Grid& g, int B) {
    if (g.nx % 8 != 0 || B > 65535) return false;
    const long long nblk = (long long)((g.nx + CX - 1) / CX) * ((g.ny + CY - 1) / CY) * ((g.nz + CZ - 1) / CZ);
    return nblk <= 0x7fffffffLL;
}

template <int CIN, int COUT, bool RELU, typename TO>
int launch_conv_tc(const __nv_bfloat16* in, const __nv_bfloat16* W, const float* bias, TO* out, const Grid& g, int B,
                   int* err, cudaStream_t st) {
    const int tiles_y = (g.ny + CY - 1) / CY;
    const long long nblk = (long long)((g.nx + CX - 1) / CX) * tiles_y * ((g.nz + CZ - 1) / CZ);
    QG_CUDA_TRY(cudaFuncSetAttribute(k_conv_tc<CIN, COUT, RELU, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     kConvTcSmem));
    k_conv_tc<CIN, COUT, RELU, TO><<<dim3((unsigned)nblk, B), 128, kConvTcSmem, st>>>(in, W, bias, out, g, tiles_y, err);
    QG_CUDA_TRY(cudaGetLastError());
    return QG_OK;
}
}  // namespace

struct qg_learned_s {
    qg_context ctx = nullptr;
    DevBuf master, adam_m, adam_v, grad, wbf, wtbf;  // params FP32 / BF16, transposed BF16 weights
    DevBuf act, dact, part, small, loss_acc;         // activations, gradients, partials, scratch
    int step = 0;
    bool tensor_cores = true;  // the forward layers on tcgen05 where the grid allows
};

namespace {

Grid make_grid(int nx, int ny, int nz) {
    Grid g;
    g.nx = nx; g.ny = ny; g.nz = nz;
    g.tx = (nx + TX - 1) / TX; g.ty = (ny + TY - 1) / TY; g.tz = (nz + TZ - 1) / TZ;
    g.N = (long long)nx * ny * nz;
    return g;
}

// forward through the 4 layers; keeps every layer's output in L->act:
//   act = [in (B x 2 x N) | h1 | h2 | h3 (B x 16 x N each), bf16] and p (B x N, float) after them
int forward(qg_learned L, const Grid& g, int B, cudaStream_t st, __nv_bfloat16** acts, float** pout) {
    const size_t N = (size_t)g.N;
    const size_t need = (size_t)B * N * (2 + 16 * 3) * sizeof(__nv_bfloat16) + (size_t)B * N * sizeof(float) + 256;
    QG_TRY(L->act.reserve(need));
    __nv_bfloat16* a0 = L->act.as<__nv_bfloat16>();
    __nv_bfloat16* a1 = a0 + (size_t)B * 2 * N;
    __nv_bfloat16* a2 = a1 + (size_t)B * 16 * N;
    __nv_bfloat16* a3 = a2 + (size_t)B * 16 * N;
    float* p = reinterpret_cast<float*>(a3 + (size_t)B * 16 * N);
    acts[0] = a0; acts[1] = a1; acts[2] = a2; acts[3] = a3;
    *pout = p;
    const __nv_bfloat16* W = L->wbf.as<__nv_bfloat16>();
    const float* P = L->master.as<float>();  // biases are read in FP32
    if (L->tensor_cores && conv_tc_ok(g, B)) {
        // every layer on tcgen05 (16 x 16 channel MMAs; layer 1 pads its 2 input channels,
        // layer 4 its 1 output channel)
        int* err = L->ctx->dev_status;
        QG_TRY((launch_conv_tc<2, 16, true>(a0, W + woff(0), P + woff(0) + wcount(0), a1, g, B, err, st)));
        QG_TRY((launch_conv_tc<16, 16, true>(a1, W + woff(1), P + woff(1) + wcount(1), a2, g, B, err, st)));
        QG_TRY((launch_conv_tc<16, 16, true>(a2, W + woff(2), P + woff(2) + wcount(2), a3, g, B, err, st)));
        QG_TRY((launch_conv_tc<16, 1, false>(a3, W + woff(3), P + woff(3) + wcount(3), p, g, B, err, st)));
        return QG_OK;
    }
    const dim3 grid(g.tx * g.ty * g.tz, B);
    k_conv_fwd<2, 16, true, __nv_bfloat16, __nv_bfloat16><<<grid, TV, 0, st>>>(a0, W + woff(0), P + woff(0) + wcount(0), a1, nullptr, g);
    k_conv_fwd<16, 16, true, __nv_bfloat16, __nv_bfloat16><<<grid, TV, 0, st>>>(a1, W + woff(1), P + woff(1) + wcount(1), a2, nullptr, g);
    k_conv_fwd<16, 16, true, __nv_bfloat16, __nv_bfloat16><<<grid, TV, 0, st>>>(a2, W + woff(2), P + woff(2) + wcount(2), a3, nullptr, g);
    k_conv_fwd<16, 1, false, __nv_bfloat16, float><<<grid, TV, 0, st>>>(a3, W + woff(3), P + woff(3) + wcount(3), p, nullptr, g);
    QG_CUDA_TRY(cudaGetLastError());
    return QG_OK;
}

int prepare_input(qg_learned L, const Grid& g, int B, const double* R, long long ldr, const double* V,
                  double vscale, cudaStream_t st, double** rms_out) {
    QG_TRY(L->small.reserve((size_t)(B + 8) * sizeof(double)));
    double* rms = L->small.as<double>();
    k_rms<<<B, 256, 0, st>>>(R, ldr, g.N, rms);
    const size_t N = (size_t)g.N;
    const size_t need = (size_t)B * N * (2 + 16 * 3) * sizeof(__nv_bfloat16) + (size_t)B * N * sizeof(float) + 256;
    QG_TRY(L->act.reserve(need));
    k_make_input<<<148 * 8, 256, 0, st>>>(R, ldr, V, vscale, rms, g.N, B, L->act.as<__nv_bfloat16>());
    QG_CUDA_TRY(cudaGetLastError());
    *rms_out = rms;
    return QG_OK;
}

int refresh_weights(qg_learned L, cudaStream_t st) {
    k_to_bf16<<<(kParams + 255) / 256, 256, 0, st>>>(L->master.as<float>(), kParams, L->wbf.as<__nv_bfloat16>());
    QG_CUDA_TRY(cudaGetLastError());
    return QG_OK;
}

// loss and parameter gradient (L->grad) of one batch; leaves the loss on the host
int loss_and_grad(qg_learned L, const Grid& g, int B, const double* R, long long ldr, const double* V, double vscale,
                  const double* Y, long long ldy, cudaStream_t st, double* loss) {
    double* rms = nullptr;
    QG_TRY(prepare_input(L, g, B, R, ldr, V, vscale, st, &rms));
    __nv_bfloat16* a[4];
    float* p = nullptr;
    QG_TRY(forward(L, g, B, st, a, &p));
    const size_t N = (size_t)g.N;
    // gradient buffers: dp (B x N) and two B x 16 x N float buffers
    QG_TRY(L->dact.reserve((size_t)B * N * (1 + 32) * sizeof(float)));
    float* dp = L->dact.as<float>();
    float* dA = dp + (size_t)B * N;
    float* dB = dA + (size_t)B * 16 * N;
    const int nlb = 148 * 4;
    QG_TRY(L->loss_acc.reserve((size_t)(2 * nlb + 4) * sizeof(double)));
    double* acc2 = L->loss_acc.as<double>();
    k_loss<<<nlb, 256, 0, st>>>(p, Y, ldy, rms, g.N, B, dp, acc2);
    std::vector<double> h(2 * nlb);
    QG_CUDA_TRY(cudaMemcpyAsync(h.data(), acc2, 2 * nlb * sizeof(double), cudaMemcpyDeviceToHost, st));
    QG_CUDA_TRY(cudaStreamSynchronize(st));
    double se = 0.0, stt = 0.0;
    for (int i = 0; i < nlb; ++i) {
        se += h[2 * i];
        stt += h[2 * i + 1];
    }
    const double inv = stt > 0.0 ? 1.0 / stt : 1.0;
    *loss = se * inv;
    // dp <- dp / sum |t|^2
    QG_CUDA_TRY(cudaMemcpyAsync(acc2 + 2 * nlb, &inv, sizeof(double), cudaMemcpyHostToDevice, st));
    k_scale_f<<<148 * 8, 256, 0, st>>>(dp, (long long)B * g.N, acc2 + 2 * nlb);

    const dim3 grid(g.tx * g.ty * g.tz, B);
    const long long ntile = (long long)grid.x * grid.y;
    if (ntile > 0x7fffffffLL) return QG_ERR_UNSUPPORTED;
    const int nblk = (int)std::min<long long>(ntile, 148 * 2);  // blocks of the weight gradients, tiles in turn
    const int maxl = 16 * 16 * 27 + 16;
    QG_TRY(L->part.reserve((size_t)nblk * maxl * sizeof(float)));
    float* part = L->part.as<float>();
    float* G = L->grad.as<float>();
    const __nv_bfloat16* Wt = L->wtbf.as<__nv_bfloat16>();
    const __nv_bfloat16* W = L->wbf.as<__nv_bfloat16>();
    for (int l = 0; l < kLayers; ++l)
        k_transpose_w<<<(wcount(l) + 255) / 256, 256, 0, st>>>(W + woff(l), kCin[l], kCout[l],
                                                                L->wtbf.as<__nv_bfloat16>() + woff(l));
    constexpr int kWgSmem = (HV + 3 * TV) * 32;
    static_assert(kWgSmem <= 48 * 1024, "no opt-in");
    auto reduce = [&](int l) { k_reduce_parts<<<(lsize(l) + 31) / 32, 256, 0, st>>>(part, nblk, lsize(l), G + woff(l)); };
    if (qg::allow_max_dynamic_smem(k_dgrad_mma) != cudaSuccess) return QG_ERR_CUDA;
    // layer 4 (16 -> 1, linear)
    k_wgrad_mma<16, 1><<<nblk, kWgThreads, kWgSmem, st>>>(a[3], dp, part, g, (int)ntile);
    reduce(3);
    k_conv_fwd<1, 16, false, float, float><<<grid, TV, 0, st>>>(dp, Wt + woff(3), nullptr, dA, a[3], g);
    // layer 3 (16 -> 16)
    k_wgrad_mma<16, 16><<<nblk, kWgThreads, kWgSmem, st>>>(a[2], dA, part, g, (int)ntile);
    reduce(2);
    k_dgrad_mma<<<grid, 256, kDgSmem, st>>>(dA, Wt + woff(2), dB, a[2], g);
    // layer 2 (16 -> 16)
    k_wgrad_mma<16, 16><<<nblk, kWgThreads, kWgSmem, st>>>(a[1], dB, part, g, (int)ntile);
    reduce(1);
    k_dgrad_mma<<<grid, 256, kDgSmem, st>>>(dB, Wt + woff(1), dA, a[1], g);
    // layer 1 (2 -> 16)
    k_wgrad_mma<2, 16><<<nblk, kWgThreads, kWgSmem, st>>>(a[0], dA, part, g, (int)ntile);
    reduce(0);
    QG_CUDA_TRY(cudaGetLastError());
    return QG_OK;
}

}  // namespace

extern "C" {

int qg_learned_num_params(void) { return kParams; }

int qg_hamiltonian_set_learned(qg_hamiltonian h, qg_learned nn, double vscale) {
    if (!h || (nn && (nn->ctx != h->ctx || !(vscale > 0)))) return QG_ERR_INVALID;
    h->learned = nn;
    h->learned_vscale = nn ? vscale : 1.0;
    return QG_OK;
}

int qg_learned_create(qg_context ctx, qg_learned* out) {
    if (!ctx || !out) return QG_ERR_INVALID;
    QG_CUDA_TRY(cudaSetDevice(ctx->device));
    qg_learned L = new qg_learned_s();
    L->ctx = ctx;
    const size_t pb = (size_t)kParams * sizeof(float);
    int rc = L->master.reserve(pb);
    if (rc == QG_OK) rc = L->adam_m.reserve(pb);
    if (rc == QG_OK) rc = L->adam_v.reserve(pb);
    if (rc == QG_OK) rc = L->grad.reserve(pb);
    if (rc == QG_OK) rc = L->wbf.reserve((size_t)kParams * sizeof(__nv_bfloat16));
    if (rc == QG_OK) rc = L->wtbf.reserve((size_t)kParams * sizeof(__nv_bfloat16));
    if (rc != QG_OK) {
        delete L;
        return rc;
    }
    cudaMemsetAsync(L->master.ptr, 0, pb, ctx->stream);
    cudaMemsetAsync(L->adam_m.ptr, 0, pb, ctx->stream);
    cudaMemsetAsync(L->adam_v.ptr, 0, pb, ctx->stream);
    refresh_weights(L, ctx->stream);
    ctx->live_hamiltonians++;
    *out = L;
    return QG_OK;
}

int qg_learned_destroy(qg_learned L) {
    if (!L) return QG_ERR_INVALID;
    cudaSetDevice(L->ctx->device);
    cudaStreamSynchronize(L->ctx->stream);
    for (DevBuf* b : {&L->master, &L->adam_m, &L->adam_v, &L->grad, &L->wbf, &L->wtbf, &L->act, &L->dact, &L->part,
                      &L->small, &L->loss_acc})
        b->release();
    L->ctx->live_hamiltonians--;
    delete L;
    return QG_OK;
}

int qg_learned_set_params(qg_learned L, const float* params, int n) {
    if (!L || !params || n != kParams) return QG_ERR_INVALID;
    QG_CUDA_TRY(cudaSetDevice(L->ctx->device));
    QG_CUDA_TRY(cudaMemcpyAsync(L->master.ptr, params, (size_t)n * sizeof(float), cudaMemcpyHostToDevice,
                                L->ctx->stream));
    QG_TRY(refresh_weights(L, L->ctx->stream));
    QG_CUDA_TRY(cudaStreamSynchronize(L->ctx->stream));
    return QG_OK;
}

int qg_learned_get_params(qg_learned L, float* params, int n) {
    if (!L || !params || n != kParams) return QG_ERR_INVALID;
    QG_CUDA_TRY(cudaSetDevice(L->ctx->device));
    QG_CUDA_TRY(cudaMemcpyAsync(params, L->master.ptr, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost,
                                L->ctx->stream));
    QG_CUDA_TRY(cudaStreamSynchronize(L->ctx->stream));
    return QG_OK;
}

int qg_learned_set_tensor_cores(qg_learned L, int on) {
    if (!L) return QG_ERR_INVALID;
    QG_CUDA_TRY(cudaStreamSynchronize(L->ctx->stream));
    L->tensor_cores = on != 0;
    return QG_OK;
}

int qg_learned_apply_d(qg_learned L, int nx, int ny, int nz, int ns, const double* R, long long ldr, const double* V,
                       double vscale, double* out, long long ldo, int accumulate) {
    if (!L || nx < 3 || ny < 3 || nz < 3 || ns <= 0 || !R || !V || !out || !(vscale > 0)) return QG_ERR_INVALID;
    const Grid g = make_grid(nx, ny, nz);
    if (ldr < g.N || ldo < g.N || ns > 65535) return QG_ERR_INVALID;
    QG_CUDA_TRY(cudaSetDevice(L->ctx->device));
    cudaStream_t st = L->ctx->stream;
    // states in chunks whose activations (50 bf16 channels + the float output per
    // voxel) stay within about 4 GB
    const long long per_state = g.N * (50 * 2 + 4);
    const int chunk = (int)std::max<long long>(1, std::min<long long>(ns, (4LL << 30) / per_state));
    for (int s0 = 0; s0 < ns; s0 += chunk) {
        const int B = std::min(chunk, ns - s0);
        double* rms = nullptr;
        QG_TRY(prepare_input(L, g, B, R + (long long)s0 * ldr, ldr, V, vscale, st, &rms));
        __nv_bfloat16* a[4];
        float* p = nullptr;
        QG_TRY(forward(L, g, B, st, a, &p));
        k_emit<<<148 * 8, 256, 0, st>>>(p, rms, g.N, B, out + (long long)s0 * ldo, ldo, accumulate);
    }
    QG_CUDA_TRY(cudaGetLastError());
    return QG_OK;
}

int qg_learned_gradient(qg_learned L, int nx, int ny, int nz, int ns, const double* R, long long ldr, const double* V,
                        double vscale, const double* Y, long long ldy, double* loss, float* grad_host) {
    if (!L || nx < 3 || ny < 3 || nz < 3 || ns <= 0 || !R || !V || !Y || !loss || !(vscale > 0))
        return QG_ERR_INVALID;
    const Grid g = make_grid(nx, ny, nz);
    if (ldr < g.N || ldy < g.N || ns > 65535) return QG_ERR_INVALID;
    QG_CUDA_TRY(cudaSetDevice(L->ctx->device));
    QG_TRY(loss_and_grad(L, g, ns, R, ldr, V, vscale, Y, ldy, L->ctx->stream, loss));
    if (grad_host) {
        QG_CUDA_TRY(cudaMemcpyAsync(grad_host, L->grad.ptr, (size_t)kParams * sizeof(float), cudaMemcpyDeviceToHost,
                                    L->ctx->stream));
        QG_CUDA_TRY(cudaStreamSynchronize(L->ctx->stream));
    }
    return QG_OK;
}

int qg_learned_train_step(qg_learned L, int nx, int ny, int nz, int ns, const double* R, long long ldr,
                          const double* V, double vscale, const double* Y, long long ldy, float lr, double* loss) {
    QG_TRY(qg_learned_gradient(L, nx, ny, nz, ns, R, ldr, V, vscale, Y, ldy, loss, nullptr));
    cudaStream_t st = L->ctx->stream;
    L->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - powf(b1, (float)L->step), c2 = 1.f - powf(b2, (float)L->step);
    k_adam<<<(kParams + 255) / 256, 256, 0, st>>>(L->master.as<float>(), L->adam_m.as<float>(), L->adam_v.as<float>(),
                                                  L->grad.as<float>(), kParams, lr, b1, b2, 1e-8f, c1, c2);
    QG_TRY(refresh_weights(L, st));
    return QG_OK;
}

}  // extern "C"
