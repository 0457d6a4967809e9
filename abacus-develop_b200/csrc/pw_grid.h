// Device-resident plane-wave grid: FFT plans, stick maps and per-k sphere maps.
//
// Layouts in HBM (one pool, one GPU):
//  * psi / hpsi: band b at psi + b*ld, G in the order of the basis (ABACUS's
//    igl2isz_k order: sticks by ixy = x*ny + y, z ascending from the bottom).
//  * stick buffer (fused H|psi>): per band nz planes of nst sticks,
//    element (band, z, s) at band*nz*nst + z*nst + s.  A z-plane is contiguous,
//    so the plane pass reads and writes whole planes with coalesced accesses.
//  * r box (drop-in transforms): ABACUS's order r = (ix*ny + iy)*nz + iz.
//  * V_eff for the fused path: transposed once to (z, y, x) so a plane row is
//    contiguous.
#pragma once
#include <cuda_runtime.h>

#include <memory>
#include <vector>

#include "common.h"
#include "fft_core.cuh"
#include "line_plan.h"
#include "pw_basis.h"

namespace b200 {

// One FFT axis: plan plus twiddles in both precisions.
struct FftAxis {
    FftPlan1D plan{};
    std::vector<double2> h_tw64;
    DeviceArray<double2> tw64;
    DeviceArray<float2> tw32;
    DeviceArray<double2> rt64;  // the n roots W_n^j = exp(-2 pi i j / n), j < n (line transforms)
    DeviceArray<float2> rt32;
    void build(int n);  // host plan + twiddles
    void upload();
};

// Sphere -> stick maps for one k-point.
struct KMap {
    int npw = 0;
    std::vector<int> h_gofs, h_gpk, h_glist;
    std::vector<double> h_precond;
    DeviceArray<int> gofs;   // nst+1 offsets of each stick's entries in the sorted list
    DeviceArray<int> gpk;    // packed (stick << 10) | z per sorted entry
    DeviceArray<int> glist;  // G index (position in psi) per sorted entry
    DeviceArray<int> ig2ixyz;
    DeviceArray<double> gk2;
    DeviceArray<float> gk2f;
    DeviceArray<double> precond;  // Davidson preconditioner 1 + g2 + sqrt(1 + (g2-1)^2)
    DeviceArray<double> gkcar;    // k+G cartesian (npw x 3, units of tpiba): PW_Basis_K::getgpluskcar
    std::vector<int2> h_sd;       // stick descriptors of the line transforms (StickMapView::sd)
    DeviceArray<int2> sd;
};

// Index maps handed to kernels by value.
struct StickMapView {
    int nst, nz;
    const int* gofs;
    const int* gpk;
    const int* glist;
    const int2* sd;  // per stick (line transforms): first position in psi, first z | count << 16
};
struct PlaneMapView {
    int nst, nxc;
    const int* xc;    // per stick: compact x-column index
    const int* sy;    // per stick: y
    const int* xpos;  // per compact column: x
    // line transforms: the sticks of column c are those of y in [0, cd.y) and [cd.z, cd.w), from stick cd.x on;
    // the occupied x are [0, xm) and [xh, nx), x >= xh in column x - xoff
    const int4* cd;
    int xm, xh, xoff;
};

// A launch shape of the plane pass on the line transforms: nw warps a CTA, L rows a warp at a time, `ctas` CTAs
// resident on an SM, `work` the instructions of the busiest warp (estimate).
struct PlaneShape {
    int nw = 0, L = 0, ctas = 0;
    double work = 0;
    size_t smem = 0;
};
// The line transforms of a grid; [0]: FP64, [1]: FP32.  ok: every edge factors, and the occupied x, the y of each
// column and the z of each stick are runs (a sphere's always are).  shapes[precision][npol - 1]: candidates, empty
// where a plane does not fit in shared memory.
struct LinePlan {
    bool ok = false;
    LineGeom x[2], y[2], z[2];
    LineGeom xbox[2], ybox[2];  // x and y lines whose threads are neighbours in the line index (box_lines.cu)
    int xm = 0, xh = 0, xoff = 0;
    std::vector<PlaneShape> shapes[2][2];
};

struct PWGrid {
    PWBasisK basis;
    int nx = 0, ny = 0, nz = 0, nst = 0, nxc = 0;
    FftAxis ax, ay, az;
    DeviceArray<int> st_xc, st_y, xpos, st_ixy;
    std::vector<int> h_xpos, h_xc, h_sy, h_sixy;
    std::vector<int> h_smap;  // per compact column c and y < ny: the stick at (xpos[c], y), or -1 (nxc x ny)
    std::vector<KMap> kmaps;
    LinePlan lines;
    std::vector<int4> h_cdesc;
    DeviceArray<int4> cdesc;
    bool on_device = false;
    // launch shape of the plane pass on the line transforms, per precision (0, 1: the estimate's best, v: its v-th)
    int plane_variant64 = 0, plane_variant32 = 0;

    void build(const PWBasisK& b);  // host-side plans and maps only (no GPU needed)
    void ensure_device();           // uploads plans and maps on first device use
    StickMapView stick_view(int ik) const {
        const KMap& k = kmaps[ik];
        return StickMapView{nst, nz, k.gofs.ptr, k.gpk.ptr, k.glist.ptr, k.sd.ptr};
    }
    PlaneMapView plane_view() const {
        return PlaneMapView{nst, nxc, st_xc.ptr, st_y.ptr, xpos.ptr, cdesc.ptr, lines.xm, lines.xh, lines.xoff};
    }
    long nxyz() const { return long(nx) * ny * nz; }
};

// Shared-memory footprint helpers (bytes) for the launch shapes used by the kernels.
constexpr int kStickTile = 16;   // sticks per CTA in the z passes
constexpr int kPlaneCols = 8;    // y-FFT column chunk in the plane pass
constexpr int kPlaneRows = 8;    // x-FFT row chunk in the plane pass
constexpr int kBoxTile = 16;     // z-columns per CTA in the box x/y passes
inline int odd_ld(int n) { return n | 1; }
size_t zpass_smem(const PWGrid& g, size_t elem);
size_t plane_smem(const PWGrid& g, size_t elem);

// ---- launchers (fft_kernels.cu); all asynchronous on `s` ----
// Fused local part of H|psi> for nb bands (one chunk): hpsi = Ekin psi + V_loc psi (accumulate==0 zeroes padding).
template <typename T, typename R>
void launch_hpsi_local(const PWGrid& g, int ik, const R* veff_zyx, int nb, int ld, const T* psi,
                       T* hpsi, T* stickbuf, double tpiba2, int accumulate, cudaStream_t s);
// k-point batch: one entry per k (its stick maps, psi / hpsi with leading dimension ld, npwk, gk2 in the
// precision of the call); passed by value so a launch needs no device-side argument buffer.
constexpr int kMaxKBatch = 128;
struct KBatchEntry {
    StickMapView sm;
    const void* psi;
    void* hpsi;
    int ld, npw;
    const void* gk2;
};
struct KBatchArgs {
    KBatchEntry e[kMaxKBatch];
};
// The line transforms of grid g (host; fills g.lines and the run descriptors of columns and sticks).
void build_line_plan(PWGrid& g);
// The three passes on the line transforms (fft_lines.cu); false (nothing launched) where g.lines does not hold or a
// plane does not fit in shared memory.
bool lines_supported(const PWGrid& g, size_t elem, int npol);
template <typename T, typename R>
bool launch_hpsi_local_lines(const PWGrid& g, int ik, const R* veff_zyx, int nb, int ld, const T* psi, T* hpsi,
                             T* stickbuf, double tpiba2, int accumulate, cudaStream_t s);
template <typename T, typename R>
bool launch_hpsi_local_kbatch_lines(const PWGrid& g, const KBatchArgs& args, int nk, int nb, const R* veff_zyx,
                                    T* stickbuf, int chunk, double tpiba2, cudaStream_t s);
template <typename T, typename R>
bool launch_hpsi_local_nc_lines(const PWGrid& g, int ik, const R* veff4_zyx, int ncols, int ld, const T* psi, T* hpsi,
                                T* stickbuf, double tpiba2, cudaStream_t s);
// Drop-in transforms (PW_Basis_K::recip_to_real / real_to_recip on the GPU), one band.
// the local part of H|psi> for npol = 2 (Veff::act's spinor branch, veff_pw.cpp:73-104, with Ekinetic::act on both
// components): ncols spinor columns (band b's components at columns 2b, 2b+1, pitch ld), the four V_eff
// components in (z, y, x) order; stickbuf holds ncols stick sets, rbuf ncols real-space boxes
template <typename T, typename R>
void launch_hpsi_local_nc(const PWGrid& g, int ik, const R* veff4_zyx, int ncols, int ld, const T* psi, T* hpsi,
                          T* stickbuf, T* rbuf, double tpiba2, cudaStream_t s);
template <typename T>
void launch_recip_to_real(const PWGrid& g, int ik, const T* in, T* out, T* aux, int add, double factor, cudaStream_t s);
template <typename T>
void launch_real_to_recip(const PWGrid& g, int ik, const T* in, T* out, T* aux, int add, double factor, cudaStream_t s);
// both on the line transforms (box_lines.cu); false (nothing launched) where they do not hold
template <typename T>
bool launch_box_lines(const PWGrid& g, int ik, bool inverse, const T* in, T* out, T* aux, int add, double factor,
                      cudaStream_t s);
// V_eff (ABACUS r order) -> (z, y, x) transposed copy, in precision R.
template <typename R>
void launch_transpose_veff(const PWGrid& g, const double* veff, R* out, cudaStream_t s);
// psi -> rho on the line transforms (where lines_supported): rho_shape chooses the launch for chunks of up to nbc
// bands; bands [b0, b0 + nbc) of psi go through the inverse z pass into sb, then w_chunk[b] |psi_b(r)|^2 is summed into
// shape.nsplit partial grids ws in (z, y, x) order (first = 1 overwrites them); launch_rho_reduce adds them to rho
struct RhoShape {
    PlaneShape plane;
    int nsplit = 0;
    bool sums = false;  // a CTA's sums in shared memory
};
RhoShape rho_shape(const PWGrid& g, size_t elem, int nbc);
// the most partial grids rho_shape chooses for up to nbc bands (kRhoPartBytes of them where more than one)
constexpr size_t kRhoPartBytes = size_t(128) << 20;
int rho_splits_most(const PWGrid& g, size_t elem, int nbc);
template <typename T, typename R>
void launch_rho_chunk(const PWGrid& g, const RhoShape& shape, int ik, int b0, int nbc, int ld, const T* psi,
                      const double* w_chunk, T* sb, R* ws, int first, cudaStream_t s);
template <typename R> void launch_rho_reduce(const PWGrid& g, int nsplit, const R* ws, R* rho, cudaStream_t s);
// Stick buffer of a band chunk of the local passes.  One launch over many bands has fewer partly filled waves: 160
// bands at 96^3 in FP64 run 1.35 ms in one chunk of 428 MB, 1.47 ms in chunks of 48 MB (which do not stay in L2
// either way), 480 bands at 128^3 in FP32 5.27 ms at 512 MB, 5.20 at 1.6 GB, 5.68 at 48 MB.
constexpr size_t kStickBytes = size_t(512) << 20;
// Number of plane-pass launch shapes the autotuner may choose from (1 .. kPlaneVariants)
constexpr int kPlaneVariants = 5;

}  // namespace b200
