// The projector products of Nonlocal::act in FP64 for small blocks, one k-point or a batch, on FP64 tensor instructions.
#pragma once
#include <cuda_runtime.h>

#include "common.h"

namespace b200 {

// One k-point: vkb (nkb x npw, pitch npwx), its D-folded form, psi and H psi (nb x npw, pitch ld).
struct ProjEntry {
    const double2 *vkb, *vkbd;
    const double2* psi;
    double2* hpsi;
    int npw, npwx;
};
constexpr int kMaxProjBatch = 128;

// Partial sums and tile counters of becp (one H|psi> at a time per workspace).
struct ProjWorkspace {
    DeviceArray<double2> part;
    DeviceArray<unsigned> count;
};

// becp (nk blocks of nkb x nb, column b at b * nkb) = vkb^H psi
void proj_becp(const ProjEntry* e, int nk, int nkb, int nb, int ld, double2* becp, ProjWorkspace& w, cudaStream_t s);
// H psi += vkbd becp
void proj_add(const ProjEntry* e, int nk, int nkb, int nb, int ld, const double2* becp, cudaStream_t s);
// where these beat a library GEMM per product and k-point: one k-point or a batch of nk; a spinor block of nb bands
bool proj_small(int nkb, int nb, int npw, int nk);
bool proj_small_spinor(int nkb, int nb, int npw);
// where these beat the int8 emulation (gemm_oz.cu); npol = 2: spinors
bool proj_beats_int8(int nkb, int nb, int npw, int npol);

}  // namespace b200
