// Definitions shared by the stencil kernels (hamiltonian.cu, stencil_tma.cu).
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace qg {

// Overlap of the kernels of an operator application (programmatic dependent launch). The projection
// and the stencil read the same states and write different buffers: the projection lets the next kernel
// of its stream start as soon as its own last blocks have (allow_next), the stencil starts beside it and ends
// only after it (wait_previous, last thing), so that whatever follows the stencil follows both. In small calls the
// kernels after the stencil start early too, read their tables and then wait (wait_previous): large calls
// lose by that, blocks that come onto an SM beside the stencil's keep its shared-memory split and little
// L1 (256 states of 80^3: the scatter 0.65 ms instead of 0.44). 16 states of 40^3: 36.9 us per call one
// after another, 31.0 so; one complex64 state of 40^3 41.1 with the brick projection before the stencil, 34.9
// with the stencil beside it, 30.5 beside its sums too; 64 states of 80^3 399 and 389 (256: the same within the
// noise).
__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// elems points of all states together: up to here (32 MB of FP64) the launches weigh.
constexpr bool small_call(long long elems) { return elems <= (4LL << 20); }

// Launch; early: may start while the kernel before it in the stream still runs (which must call
// allow_next, and this one wait_previous).
template <typename... P, typename... A>
cudaError_t launch_kernel(bool early, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, P(std::forward<A>(args))...);
}

template <typename T>
struct HamArgs {
    const T* X;
    long long ldx;
    T* HX;
    long long ldhx;
    int ns;
    const T* V;
    int nx, ny, nz;
    int ty;
    int zslab;
    T c0;
    T cx[4], cy[4], cz[4];
    int* err;        // device status word: nonzero after a bounded wait gave up
    int stall;       // test hook: the ring kernels' producer issues nothing, so the
                     // consumers' bounded waits run out (QG_ERR_TIMEOUT)
    // complex (k-point) states: the imaginary part of a state starts xim (hxim)
    // elements after its real part; dx/dy/dz are the 8th-order first-derivative
    // coefficients 2*coef*g/(840h)*(672, -168, 32, -3) per axis (zero for an
    // axis whose |g| < 1e-8), c0 then carries the -coef*|g|^2 term
    long long xim, hxim;
    T dx[4], dy[4], dz[4];
    // several k-points in one launch: states are grouped by k, nsk per k;
    // state s of k-point k starts at X + k*ldkx + s*ldx (HX + k*ldkhx + s*ldhx), and
    // kco[k*13 + {0, 1..4, 5..8, 9..12}] replaces c0, dx, dy, dz (nsk = 0: one k-point)
    int nsk;
    long long ldkx, ldkhx;
    const T* kco;
    bool early;      // host: launch beside the projection before it (launch_kernel)
};

// first element of global state index s (k-point major when several k-points share a launch)
template <typename T>
__device__ __forceinline__ long long state_offset(const HamArgs<T>& a, int s, bool out) {
    if (a.nsk <= 0) return (long long)s * (out ? a.ldhx : a.ldx);
    const int k = s / a.nsk, sl = s - k * a.nsk;
    return out ? (long long)k * a.ldkhx + (long long)sl * a.ldhx : (long long)k * a.ldkx + (long long)sl * a.ldx;
}

__device__ __forceinline__ int wrap_idx(int i, int n) {
    i %= n;
    return i < 0 ? i + n : i;
}


// Real states, one plane and row per consumer step (stencil_tma.cu).
template <typename T>
int launch_stencil_tma(const HamArgs<T>& a, int order, cudaStream_t st);
// True when launch_stencil_tma accepts this shape and alignment.
template <typename T>
bool stencil_tma_ok(const HamArgs<T>& a, int order);
// Real states, two output planes per consumer step (stencil_pair.cu).
template <typename T>
int launch_stencil_pair(const HamArgs<T>& a, int order, cudaStream_t st);
template <typename T>
bool stencil_pair_ok(const HamArgs<T>& a, int order);
// Real states, two grid rows per consumer thread, V streamed through the ring (vring) or
// read one plane ahead from global memory (stencil_rows.cu).
template <typename T>
int launch_stencil_rows(const HamArgs<T>& a, int order, cudaStream_t st, bool vring = true);
template <typename T>
bool stencil_rows_ok(const HamArgs<T>& a, int order, bool vring = true);

// Complex k-point states of orders 2, 6 and 8 (stencil_kpoint.cu).
template <typename T>
int launch_stencil_kpoint(const HamArgs<T>& a, int order, cudaStream_t st);
template <typename T>
bool stencil_kpoint_ok(const HamArgs<T>& a, int order);

// 8th-order periodic FD gradient of the listed real states (sidx, DEVICE) of the nin at X (gradient.cu):
// component d of state s at out + (d * ns + s) * N (Gradient8th, GridGradient8th.h:19-235).
// QG_ERR_UNSUPPORTED where TMA does not take the rows. err, stall: as in HamArgs.
int launch_gradient8(const double* X, long long ldx, int nin, const int* sidx, int ns, double* out, int nx, int ny, int nz,
                     const double* h, int* err, int stall, cudaStream_t st);

}  // namespace qg
