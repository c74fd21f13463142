// Complex k-point Hamiltonian on the device (mHamiltonianMatrix_ddm of
// QUMASUN_KPOINT, qumasun_kpoint.matrix.h:25-50):
//   H_k u = V u + sum_atoms sum_k E_k sum_m conj(P_km) dV (P_km . u) - 1/2 (Lap + 2i g.grad - g^2) u,
//   P_km(r) = w_k(r) Y_lm(r) exp(i g.r) at the unwrapped image position of each cube point
//   (mCreateProjectorRadialOnBlock, PseudoPotOperator_kpoint_v2.h:287-420; ProjectionPP :2581-2700).
// States are split complex, one state = {re[N], im[N]} (lobpcg_z_multi_mpi.h:1005-1012).
// Launches for a block of states, as on the real path: the projection and the scatter on the
// tensor cores (nonlocal.cu: Bloch phases of the grid points and of the periodic images, the
// projector tables of the real path), and between them
//   k_stencil_kpoint  V u - 1/2 (Lap + 2i g.grad - g^2) u, both parts of a plane staged together
//                   (stencil_kpoint.cu); any other shape runs k_kpoint_plain
#include <algorithm>
#include <cmath>

#include "nonlocal.h"
#include "qg_internal.h"
#include "stencil_common.cuh"

namespace qg {
namespace {

// The per-k-point stencil coefficients of a launch, 32 k-points at a time.
struct KcoArgs {
    static constexpr int n = 32 * 13;
    double v[n];
};
template <typename T>
__global__ void k_store_kco(const KcoArgs args, int n, T* __restrict__ out) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) out[i] = T(args.v[i]);
}

// Any-shape fallback for V u - 1/2 (Lap + 2i g.grad - g^2) u at FD order 2, 6 or 8: one
// thread per (point, state), neighbours read from global memory with periodic wrap. The
// sums follow LaplasianKpoint{2nd,6th,8th}_halo_f (order 2: c0 p + cx (p+x + p-x) + ...;
// orders 6, 8: c0 p, then the x, y and z groups). Runs beside the projection as the ring kernels do.
template <typename T, int ORDER>
__global__ void __launch_bounds__(256) k_kpoint_plain(const HamArgs<T> a) {
    constexpr int R = ORDER == 2 ? 1 : (ORDER == 6 ? 3 : 4);
    const long long N = (long long)a.nx * a.ny * a.nz;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    allow_next();
    if (i >= N) return;
    const int s = blockIdx.y;
    const int ix = (int)(i % a.nx), iy = (int)((i / a.nx) % a.ny), iz = (int)(i / ((long long)a.nx * a.ny));
    T c0 = a.c0, dxc[4], dyc[4], dzc[4];
    for (int d = 0; d < 4; ++d) {
        dxc[d] = a.dx[d];
        dyc[d] = a.dy[d];
        dzc[d] = a.dz[d];
    }
    if (a.kco) {
        const T* kc = a.kco + (long long)(s / a.nsk) * 13;
        c0 = kc[0];
        for (int d = 0; d < 4; ++d) {
            dxc[d] = kc[1 + d];
            dyc[d] = kc[5 + d];
            dzc[d] = kc[9 + d];
        }
    }
    T lap[2], der[2], cen[2];
    for (int c = 0; c < 2; ++c) {
        const T* u = a.X + state_offset(a, s, false) + (c ? a.xim : 0);
        auto at = [&](int dx, int dy, int dz) {
            return u[wrap_idx(ix + dx, a.nx) + (long long)a.nx * (wrap_idx(iy + dy, a.ny) + (long long)a.ny * wrap_idx(iz + dz, a.nz))];
        };
        T xm[R], xp[R], ym[R], yp[R], zm[R], zp[R];
        for (int d = 1; d <= R; ++d) {
            xm[d - 1] = at(-d, 0, 0); xp[d - 1] = at(d, 0, 0);
            ym[d - 1] = at(0, -d, 0); yp[d - 1] = at(0, d, 0);
            zm[d - 1] = at(0, 0, -d); zp[d - 1] = at(0, 0, d);
        }
        cen[c] = u[i];
        T l, g;
        if constexpr (ORDER == 2) {
            l = c0 * cen[c] + a.cx[0] * (xp[0] + xm[0]) + a.cy[0] * (yp[0] + ym[0]) + a.cz[0] * (zp[0] + zm[0]);
            g = dxc[0] * (xp[0] - xm[0]);
            g += dyc[0] * (yp[0] - ym[0]);
            g += dzc[0] * (zp[0] - zm[0]);
        } else if constexpr (ORDER == 6) {
            l = c0 * cen[c];
            l += a.cx[2] * (xp[2] + xm[2]) + a.cx[1] * (xp[1] + xm[1]) + a.cx[0] * (xp[0] + xm[0]);
            l += a.cy[2] * (yp[2] + ym[2]) + a.cy[1] * (yp[1] + ym[1]) + a.cy[0] * (yp[0] + ym[0]);
            l += a.cz[2] * (zp[2] + zm[2]) + a.cz[1] * (zp[1] + zm[1]) + a.cz[0] * (zp[0] + zm[0]);
            g = dxc[2] * (xp[2] - xm[2]) + dxc[1] * (xp[1] - xm[1]) + dxc[0] * (xp[0] - xm[0]);
            g += dyc[2] * (yp[2] - ym[2]) + dyc[1] * (yp[1] - ym[1]) + dyc[0] * (yp[0] - ym[0]);
            g += dzc[2] * (zp[2] - zm[2]) + dzc[1] * (zp[1] - zm[1]) + dzc[0] * (zp[0] - zm[0]);
        } else {
            l = c0 * cen[c];
            l += a.cx[3] * (xp[3] + xm[3]) + a.cx[2] * (xp[2] + xm[2]) + a.cx[1] * (xp[1] + xm[1]) + a.cx[0] * (xp[0] + xm[0]);
            l += a.cy[3] * (yp[3] + ym[3]) + a.cy[2] * (yp[2] + ym[2]) + a.cy[1] * (yp[1] + ym[1]) + a.cy[0] * (yp[0] + ym[0]);
            l += a.cz[3] * (zp[3] + zm[3]) + a.cz[2] * (zp[2] + zm[2]) + a.cz[1] * (zp[1] + zm[1]) + a.cz[0] * (zp[0] + zm[0]);
            g = dxc[3] * (xp[3] - xm[3]) + dxc[2] * (xp[2] - xm[2]) + dxc[1] * (xp[1] - xm[1]) + dxc[0] * (xp[0] - xm[0]);
            g += dyc[3] * (yp[3] - ym[3]) + dyc[2] * (yp[2] - ym[2]) + dyc[1] * (yp[1] - ym[1]) + dyc[0] * (yp[0] - ym[0]);
            g += dzc[3] * (zp[3] - zm[3]) + dzc[2] * (zp[2] - zm[2]) + dzc[1] * (zp[1] - zm[1]) + dzc[0] * (zp[0] - zm[0]);
        }
        lap[c] = l;
        der[c] = g;
    }
    const T v = a.V[i];
    T* h = a.HX + state_offset(a, s, true) + i;
    h[0] = (v * cen[0] + lap[0]) - der[1];
    h[a.hxim] = (v * cen[1] + lap[1]) + der[0];
    wait_previous();
}

// c0 and the first-derivative coefficients of -1/2 (Lap + 2i g.grad - g^2) at FD order
// 2, 6 or 8, exactly as LaplasianKpoint{2nd,6th,8th}_halo_f form them
// (GridDifferenceKpoint2nd.h:19-35, 6th.h:19-47, 8th.h:18-50): out[0] = c0,
// out[1..4] = dx, [5..8] = dy, [9..12] = dz (first R entries of each used).
void kpoint_coefs(const qg_hamiltonian h, const double* g, double* out) {
    const double coefk = -0.5;
    const double hh[3] = {h->hx, h->hy, h->hz};
    const double gg = g[0] * g[0] + g[1] * g[1] + g[2] * g[2];
    if (h->order == 2)
        out[0] = -coefk * (2.0 / (hh[0] * hh[0]) + 2.0 / (hh[1] * hh[1]) + 2.0 / (hh[2] * hh[2])) - coefk * gg;
    else if (h->order == 6)
        out[0] = -245.0 * coefk *
                     (1.0 / (90.0 * hh[0] * hh[0]) + 1.0 / (90.0 * hh[1] * hh[1]) + 1.0 / (90.0 * hh[2] * hh[2])) -
                 coefk * gg;
    else
        out[0] = -14350.0 / 5040.0 * coefk * (1.0 / (hh[0] * hh[0]) + 1.0 / (hh[1] * hh[1]) + 1.0 / (hh[2] * hh[2])) -
                 coefk * gg;
    const double coef2 = coefk * 2.0;
    for (int d = 0; d < 3; ++d) {
        const bool on = std::fabs(g[d]) >= 1.0e-8;  // the reference's _ddm skips |g| < 1e-8
        double* o = out + 1 + 4 * d;
        o[0] = o[1] = o[2] = o[3] = 0.0;
        if (!on) continue;
        if (h->order == 2) {
            o[0] = coef2 * g[d] / (2.0 * hh[d]);
        } else if (h->order == 6) {
            o[0] = 45.0 * coef2 * g[d] / (60.0 * hh[d]);
            o[1] = -9.0 * coef2 * g[d] / (60.0 * hh[d]);
            o[2] = coef2 * g[d] / (60.0 * hh[d]);
        } else {
            o[0] = 672.0 * coef2 * g[d] / (840.0 * hh[d]);
            o[1] = -168.0 * coef2 * g[d] / (840.0 * hh[d]);
            o[2] = 32.0 * coef2 * g[d] / (840.0 * hh[d]);
            o[3] = -3.0 * coef2 * g[d] / (840.0 * hh[d]);
        }
    }
}

}  // namespace

template <typename T>
int apply_hamiltonian_zk(qg_hamiltonian h, int nk, const double* kv, int nsk, const T* X, long long ldx,
                         long long ldk, T* HX, long long ldhx, long long ldkh, double* scratch, cudaStream_t st,
                         PhaseTimer* pt) {
    if (h->order != 2 && h->order != 6 && h->order != 8) return QG_ERR_UNSUPPORTED;
    const DevProjectors& pj = h->pj;
    const long long N = h->N();
    HamArgs<T> a{};
    a.X = X; a.ldx = ldx; a.HX = HX; a.ldhx = ldhx; a.ns = nk * nsk;
    a.xim = N; a.hxim = N;
    if constexpr (sizeof(T) == 8) a.V = reinterpret_cast<const T*>(h->V_d);
    else a.V = reinterpret_cast<const T*>(h->V_f);
    a.nx = h->nx; a.ny = h->ny; a.nz = h->nz; a.ty = h->ty;
    a.err = h->ctx->dev_status;
    const double coefk = -0.5;
    const double hh[3] = {h->hx, h->hy, h->hz};
    T* cs[3] = {a.cx, a.cy, a.cz};
    for (int d = 0; d < 3; ++d) {
        if (h->order == 2) {
            cs[d][0] = T(coefk / (hh[d] * hh[d]));
        } else if (h->order == 6) {
            const double s = 90.0 * hh[d] * hh[d];
            cs[d][2] = T(coefk / s);
            cs[d][1] = T(-13.5 * coefk / s);
            cs[d][0] = T(135.0 * coefk / s);
        } else {
            const double s = 5040.0 * hh[d] * hh[d];
            cs[d][3] = T(-9.0 * coefk / s);
            cs[d][2] = T(128.0 * coefk / s);
            cs[d][1] = T(-1008.0 * coefk / s);
            cs[d][0] = T(8064.0 * coefk / s);
        }
    }
    std::vector<double> kc((size_t)13 * nk);
    for (int k = 0; k < nk; ++k) kpoint_coefs(h, kv + 3 * k, kc.data() + 13 * k);
    a.c0 = T(kc[0]);
    for (int d = 0; d < 4; ++d) {
        a.dx[d] = T(kc[1 + d]);
        a.dy[d] = T(kc[5 + d]);
        a.dz[d] = T(kc[9 + d]);
    }
    if (nk > 1) {
        QG_TRY(h->kco.reserve(kc.size() * sizeof(T)));
        // as kernel arguments: no copy from pageable memory and no synchronisation (12 us of a 62 us call)
        for (size_t at = 0; at < kc.size(); at += KcoArgs::n) {
            KcoArgs args;
            const int n = (int)std::min<size_t>(KcoArgs::n, kc.size() - at);
            std::copy_n(kc.begin() + at, n, args.v);
            k_store_kco<T><<<1, 256, 0, st>>>(args, n, h->kco.as<T>() + at);
        }
        a.kco = h->kco.as<T>();
        a.nsk = nsk;
        a.ldkx = ldk;
        a.ldkhx = ldkh;
    }
    const bool nonlocal = pj.na > 0 && pj.nch > 0;
    if (pt) pt->mark(0, st);
    const double2* phase = nullptr;
    constexpr int PX = 16 / sizeof(T);
    const bool plain = h->stencil_variant == 1 || !stencil_kpoint_ok<T>(a, h->order) || (nk > 1 && (ldk % PX || ldkh % PX));
    auto stencil = [&](bool early) -> int {
        if (plain) {
            dim3 g((unsigned)((N + 255) / 256), (unsigned)(nk * nsk));
            auto kern = h->order == 2 ? k_kpoint_plain<T, 2> : (h->order == 6 ? k_kpoint_plain<T, 6> : k_kpoint_plain<T, 8>);
            QG_CUDA_TRY(launch_kernel(early, kern, g, dim3(256), 0, st, a));
            return QG_OK;
        }
        a.early = early;
        return launch_stencil_kpoint<T>(a, h->order, st);
    };
    const bool together = nonlocal && !pt;  // events between the kernels would order them
    if (nonlocal) {
        QG_TRY(ensure_phases(h, nk, kv, st, &phase));
        QG_TRY(brick_project<T>(h, nk, nsk, true, X, ldx, ldk, phase, pj.ch_scale, scratch,
                                scratch + coef_elems(h, nk, nsk, true), st,
                                together ? std::function<int(bool)>(stencil) : std::function<int(bool)>()));
    }
    if (pt) pt->mark(1, st);
    if (!together) QG_TRY(stencil(false));
    if (pt) pt->mark(2, st);
    if (nonlocal) QG_TRY(brick_scatter_z<T>(h, nk, nsk, HX, ldhx, ldkh, phase, scratch, together && small_call((long long)nk * nsk * N), st));
    if (pt) pt->mark(-1, st);
    QG_CUDA_TRY(cudaGetLastError());
    return QG_OK;
}

template <typename T>
int apply_hamiltonian_z(qg_hamiltonian h, int ns, const T* X, long long ldx, T* HX, long long ldhx, double* scratch,
                        cudaStream_t st, PhaseTimer* pt) {
    const double kv[3] = {h->gx, h->gy, h->gz};
    return apply_hamiltonian_zk<T>(h, 1, kv, ns, X, ldx, 0, HX, ldhx, 0, scratch, st, pt);
}

template int apply_hamiltonian_zk<double>(qg_hamiltonian, int, const double*, int, const double*, long long,
                                          long long, double*, long long, long long, double*, cudaStream_t,
                                          PhaseTimer*);
template int apply_hamiltonian_zk<float>(qg_hamiltonian, int, const double*, int, const float*, long long, long long,
                                         float*, long long, long long, double*, cudaStream_t, PhaseTimer*);
template int apply_hamiltonian_z<double>(qg_hamiltonian, int, const double*, long long, double*, long long, double*,
                                         cudaStream_t, PhaseTimer*);
template int apply_hamiltonian_z<float>(qg_hamiltonian, int, const float*, long long, float*, long long, double*,
                                        cudaStream_t, PhaseTimer*);

}  // namespace qg

namespace {

template <typename T>
int apply_z_checked(qg_hamiltonian h, int ns, const T* X, long long ldx, T* HX, long long ldhx) {
    if (!h || ns < 0 || (ns > 0 && (!X || !HX))) return QG_ERR_INVALID;
    if (ns == 0) return QG_OK;
    const long long N = h->N();
    if (ldx < 2 * N || ldhx < 2 * N) return QG_ERR_INVALID;
    if (h->order != 2 && h->order != 6 && h->order != 8) return QG_ERR_UNSUPPORTED;
    QG_CUDA_TRY(cudaSetDevice(h->ctx->device));
    QG_TRY(h->coef.reserve(qg::kpoint_scratch(h, 1, ns)));
    double* coef = h->coef.as<double>();
    return qg::apply_hamiltonian_z<T>(h, ns, X, ldx, HX, ldhx, coef, h->ctx->stream);
}

template <typename T>
int apply_zk_checked(qg_hamiltonian h, int nk, const double* kvecs, int nsk, const T* X, long long ldx, long long ldk,
                     T* HX, long long ldhx, long long ldkh) {
    if (!h || nk <= 0 || nsk < 0 || !kvecs || (nsk > 0 && (!X || !HX))) return QG_ERR_INVALID;
    if (nsk == 0) return QG_OK;
    const long long N = h->N();
    if (ldx < 2 * N || ldhx < 2 * N) return QG_ERR_INVALID;
    if (nk > 1 && (ldk < (long long)nsk * ldx || ldkh < (long long)nsk * ldhx)) return QG_ERR_INVALID;
    if (h->order != 2 && h->order != 6 && h->order != 8) return QG_ERR_UNSUPPORTED;
    QG_CUDA_TRY(cudaSetDevice(h->ctx->device));
    QG_TRY(h->coef.reserve(qg::kpoint_scratch(h, nk, nsk)));
    double* coef = h->coef.as<double>();
    return qg::apply_hamiltonian_zk<T>(h, nk, kvecs, nsk, X, ldx, ldk, HX, ldhx, ldkh, coef, h->ctx->stream);
}

}  // namespace

extern "C" {

int qg_hamiltonian_apply_zk(qg_hamiltonian h, int nk, const double* kvecs, int nsk, const double* X, long long ldx,
                            long long ldk, double* HX, long long ldhx, long long ldkh) {
    return apply_zk_checked<double>(h, nk, kvecs, nsk, X, ldx, ldk, HX, ldhx, ldkh);
}

int qg_hamiltonian_apply_zkf(qg_hamiltonian h, int nk, const double* kvecs, int nsk, const float* X, long long ldx,
                             long long ldk, float* HX, long long ldhx, long long ldkh) {
    return apply_zk_checked<float>(h, nk, kvecs, nsk, X, ldx, ldk, HX, ldhx, ldkh);
}

int qg_hamiltonian_apply_zf(qg_hamiltonian h, int ns, const float* X, long long ldx, float* HX, long long ldhx) {
    return apply_z_checked<float>(h, ns, X, ldx, HX, ldhx);
}

int qg_hamiltonian_apply_z(qg_hamiltonian h, int ns, const double* X, long long ldx, double* HX, long long ldhx) {
    return apply_z_checked(h, ns, X, ldx, HX, ldhx);
}

int qg_hamiltonian_apply_timed_z(qg_hamiltonian h, int ns, const double* X, long long ldx, double* HX,
                                 long long ldhx, float* ms_phases) {
    if (!h || ns <= 0 || !X || !HX || !ms_phases) return QG_ERR_INVALID;
    const long long N = h->N();
    if (ldx < 2 * N || ldhx < 2 * N) return QG_ERR_INVALID;
    if (h->order != 2 && h->order != 6 && h->order != 8) return QG_ERR_UNSUPPORTED;
    QG_CUDA_TRY(cudaSetDevice(h->ctx->device));
    QG_TRY(h->coef.reserve(qg::kpoint_scratch(h, 1, ns)));
    double* coef = h->coef.as<double>();
    qg::PhaseTimer pt;
    QG_TRY(qg::apply_hamiltonian_z(h, ns, X, ldx, HX, ldhx, coef, h->ctx->stream, &pt));
    pt.totals(ms_phases);
    QG_CUDA_TRY(cudaGetLastError());
    return QG_OK;
}

int qg_hamiltonian_apply_host_z(qg_hamiltonian h, int ns, const double* X, double* HX) {
    if (!h || ns < 0 || (ns > 0 && (!X || !HX))) return QG_ERR_INVALID;
    if (ns == 0) return QG_OK;
    const long long N2 = 2 * h->N();
    return qg::host_pipelined_apply(h, ns, N2, X, HX, [&](int nc, const double* xd, double* hd) {
        return apply_z_checked(h, nc, xd, N2, hd, N2);
    });
}

}  // extern "C"
