// Nonlocal projectors as FP64 tensor-core contractions over bricks of the grid (nonlocal.cu).
#pragma once
#include <functional>
#include <vector>

#include "qg_internal.h"

namespace qg {

// The lists of BrickTables (qg_internal.h) on the host.
struct BrickLists {
    int nbx, nby, nbricks, nitems, npairs, max_tab, ncg, nimg;
    std::vector<int> item_brick, item_pair, item_cg, item_img, wtab, brick_item, cg_off, img;
    std::vector<unsigned long long> wmask;
    std::vector<double> tab;
    std::vector<int2> cg_ref;
};
// From the sphere points of one geometry on a grid of n points per axis: atom a owns the points
// [atom_off[a], atom_off[a+1]), u = 3 unwrapped grid coordinates per point (rows of
// consecutive x one after another), tabs[ch][p] the channel values. No CUDA call.
BrickLists list_bricks(const int (&n)[3], const std::vector<int>& atom_off, const std::vector<int>& u,
                       const std::vector<std::vector<double>>& tabs);
int upload_bricks(qg_hamiltonian h, const BrickLists& l);
void free_bricks(BrickTables& b);

// Rows of projector coefficients: the count of states (of all k-points) rounded up to 16 (real), or
// {re, im} in alternating groups of 8 (complex).
inline long long coef_rows(int ns, bool cplx) { return cplx ? 16LL * ((ns + 7) / 8) : coef_ld(ns); }

// Doubles of the coefficients of nk x ns states, and of the bricks' partial sums of one slice of
// them; an operator application takes both as one scratch, the coefficients first.
size_t coef_elems(qg_hamiltonian h, int nk, int ns, bool cplx);
size_t part_elems(qg_hamiltonian h, int nk, int ns, bool cplx);
// Whether real FP64 states are projected brick by brick (see the rule at its definition).
bool bricks_for_real(const DevProjectors& pj);
// The same for real states of type T under the operator's blocking: FP32 states and a forced split of the atoms
// go atom by atom, straight into the coefficients.
template <typename T>
bool real_by_bricks(qg_hamiltonian h) {
    return sizeof(T) == sizeof(double) && h->proj_parts == 0 && bricks_for_real(h->pj);
}
// Bytes of scratch of an application to real states of type T, and to nk x ns k-point states.
template <typename T>
size_t real_scratch(qg_hamiltonian h, int ns) {
    return real_by_bricks<T>(h) ? (coef_elems(h, 1, ns, false) + part_elems(h, 1, ns, false)) * sizeof(double)
                                : coef_scratch_elems(h, ns) * sizeof(T);
}
inline size_t kpoint_scratch(qg_hamiltonian h, int nk, int ns) {
    return (coef_elems(h, nk, ns, true) + part_elems(h, nk, ns, true)) * sizeof(double);
}
// Kernels brick_project launches for ns real states.
int brick_project_launches(qg_hamiltonian h, int ns);

// Real: coef[(atom * nch + ch) * coef_ld(ns) + s] = scale[atom * nch + ch] * sum_p P(p) psi_s(p).
// Complex: coef[(cg * coef_rows + row) * 4 + c], cg = atom * (nch / 4) + channel group;
// phase: the tables of ensure_phases (real states: nullptr). stencil (may be empty) launches a kernel that reads
// X and touches neither coef nor part: beside the projection where it can (early, see launch_kernel).
template <typename T>
int brick_project(qg_hamiltonian h, int nk, int ns, bool cplx, const T* X, long long ldx, long long ldk,
                  const double2* phase, const double* scale, double* coef, double* part, cudaStream_t st,
                  const std::function<int(bool early)>& stencil = {});
// HX += sum over spheres and channels conj(P) coef, complex states.
template <typename T>
int brick_scatter_z(qg_hamiltonian h, int nk, int ns, T* HX, long long ldx, long long ldk, const double2* phase,
                    const double* coef, bool early, cudaStream_t st);

// Bloch phases exp(i g.r) of nk k-vectors (HOST, 3 each): per k-point nx + ny + nz values of
// the axes, then one per periodic image; rebuilt when the k-vectors change.
int ensure_phases(qg_hamiltonian h, int nk, const double* kv, cudaStream_t st, const double2** out);

}  // namespace qg
