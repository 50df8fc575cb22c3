// modal.h -- modal stencil kernels of linear constant-coefficient scalar operators (modal.cu).
#pragma once
#include "dg_kernel.cuh"
#include "dg_registry.h"

namespace bosss {

enum { VARIANT_MODAL = 3 };   // beside KernelVariant: one entry per (phys, D, K, mode), any rule

// The modal kernel integrates exactly what the quadrature does: it applies when the form is
// linear with constant coefficients (nu2 = 0) and the rule with Q nodes per direction is exact
// for it. The integrands have degree 2K per direction (boundary data: K + 2 <= 2Q - 1), so
// Q >= K + 1 suffices; a lower rule has a quadrature error that belongs to the result and
// keeps the quadrature kernels.
inline bool modal_applies(int phys, const PhysParams& ph, int K, int Q) {
    return (phys == PHYS_TRANSPORT || phys == PHYS_SIP) && !(ph.has_sip && ph.nu2 != 0.0) && Q >= K + 1;
}

// launch entry of a mode (launch null: no instance)
KernelEntry modal_entry(int phys, int D, int K, int mode);

// ---- batches: instances of one degree in one launch, one tile per CTA
struct ModalTile {
    int b[3];        // tile extent in memory order (slow, middle, fast); 2D: middle = 1
    int t[3];        // tiles per memory direction
    int s0, planes;  // first plane of the slowest direction and number of planes that hold the launch's cells
    int ncell;       // b[0] * b[1] * b[2]
};
struct ModalItem {
    int inst, tile;
};
// tile extents for the cells [cbeg, cend) of a grid; `shared`: the launch holds other grids too,
// so that this one need not spread over the whole chip
ModalTile modal_tiling(const EvalArgs& a, int D, int K, bool shared = false);

}  // namespace bosss
