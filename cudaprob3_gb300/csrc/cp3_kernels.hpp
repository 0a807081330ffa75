// cp3_kernels.hpp -- launch wrappers of the kernels (host-callable, no CUDA types beyond
// cudaStream_t), shared by the C ABI and the batched driver.
#pragma once

#include <cuda_runtime.h>

#include "cp3_types.h"

namespace cp3 {

// Fields of one (density class, energy) entry of the mixed eigen table.
constexpr int kMixFields = 12;  // u1 (3), u2 (3) real unit eigenvectors; omega_1, omega_2 in
                                // turns per km, double-float as (hi1, hi2, lo1, lo2); 2 unused
                                // (one 48-byte entry per (class, energy))

inline int pad_energies(int ne) { return (ne + 31) / 32 * 32; }

// The mixed eigen table over (class, energy): real eigenvectors and double-float phase rates.
cudaError_t launch_table_mixed(const OscParams& p, const double* energies, int ne,
                               const double* cls_rho, int ncls, float* table, cudaStream_t s);
// The same from float pairs (hi, lo) split on the host: no FP64 instruction on the device.
cudaError_t launch_table_mixed(const OscParams& p, const float2* energies, int ne,
                               const float2* cls_rho, int ncls, float* table, cudaStream_t s);

// The table of the fixed-point FP64 bins (cp3_fixed.cuh), table_fx_words(ncls, ne) word pairs.
size_t table_fx_words(int ncls, int ne);
cudaError_t launch_table_fx(const OscParams& p, const double* energies, int ne,
                            const double* cls_rho, int ncls, int2* table, cudaStream_t s);

// Loads the mixed table kernel (the double-input instance) and the mixed per-bin kernel
// into the current device's context, as their first launch would.  With lazy module
// loading that first load may allocate device memory; a caller that must not allocate
// later (cp3_atmos_mixed_noalloc) calls these once, at set-up.
cudaError_t preload_table_mixed();
cudaError_t preload_atmos_mixed();

// Production-height averaging inputs of the FP64 kernels (n_bins == 0: fixed height).
struct AvgArrays {
    const double* prob = nullptr;  // [2][3][nc][n_bins][ne]: consecutive energies are contiguous
    const double* mid = nullptr;   // [nc][n_bins] mid path-length shift of each bin, km (0 where the
                                   // air segment has zero length)
    const double* wid = nullptr;   // [nc][n_bins] bin width, km (0 likewise)
    const signed char* scale = nullptr;  // [2][3][nc][ne] fx_weight_scale, where one is not zero
    int n_bins = 0;
};

// Cosine rows [begin, end) of a result (end < 0: through the last row).  early: the launch
// follows its table's with nothing in between, and may be scheduled while that one runs.
struct RowRange {
    int begin = 0, end = -1;
    bool early = false;
};

#ifdef __CUDACC__
// Programmatic dependent launch: a table's launch lets the bins' be scheduled as soon as all its
// blocks run (launch_dependents); the bins stage what the table does not hold and wait for its
// end before they read it (wait_for_previous; no wait where the launch was an ordinary one).
// They read it with __ldca: its lines are written during their own grid's life, which the
// read-only path does not allow for.  A call, before and after: FP64 PREM-4 400 x 400 40.2 and
// 35.7 us, PREM-12 307 x 811 73 and 68, quadratic 500 x 500 75 and 68 (its bins need the air's
// table only once their chain of layers is done); mixed PREM-4 200 x 200 to host memory 37 and 34.
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... Params, class... Args>
void launch_early(bool early, void (*kernel)(Params...), dim3 grid, int block, cudaStream_t s, Args... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3(block);
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = early ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, Params(args)...);  // the error is read with cudaGetLastError
}
#endif

// Atmospheric bins of an n_cosines-row result ([9][n_cosines][ne]), rows rr only.  The
// trajectory of row i is segments seg_off[i]..seg_off[i+1]-1 (air, then shells inwards); the
// table class of a row's segment l is l itself (class 0 the air, class l shell l-1, as
// build_trajectories numbers them), so no class array is read.
// FP64 bins from the fixed-point table, constant densities and a fixed production height.
// Bins whose table entries or phases are out of its range take the FP64 path, from the class
// densities.
cudaError_t launch_atmos_fx(const OscParams& p, const double* energies, int ne, const int2* table,
                            const double* cls_rho, int ncls, const int* seg_off,
                            const double* seg_len, int n_cosines, double* out, cudaStream_t s,
                            RowRange rr = RowRange{});
cudaError_t launch_atmos_mixed(const OscParams& p, const float* table, int ne,
                               const int* seg_off, const float2* seg_len, int n_cosines,
                               float* out, cudaStream_t s,
                               RowRange rr = RowRange{});

// Production-height averaging inputs of the mixed kernels (float, from AvgArrays on the host).
struct AvgMixed {
    const float* prob = nullptr;  // [2][3][nc][n_bins][ne]
    const float2* hm = nullptr;   // [nc][n_bins] mid shift of each bin, km, float pair (0 where the
                                  // air segment has zero length)
    const float* hw = nullptr;    // [nc][n_bins] bin width, km (0 likewise)
    int nb = 0, type = 0;
};

// Mixed atmospheric bins with production-height averaging.
cudaError_t launch_atmos_mixed_avg(const OscParams& p, const float* table, int ne,
                                   const int* seg_off, const float2* seg_len, int n_cosines,
                                   const AvgMixed& av, float* out, cudaStream_t s,
                                   RowRange rr = RowRange{});

// Mixed averaged bins with the quadratic density model (per-segment eigen-solve).
cudaError_t launch_atmos_mixed_inline_avg(const OscParams& p, const double* energies, int ne,
                                          const int* seg_off, const float2* seg_len,
                                          const double* seg_rho, int n_cosines,
                                          const AvgMixed& av, float* out, cudaStream_t s,
                                          RowRange rr = RowRange{});

// Atmospheric bins whose layers are solved in place.  FP64: quadratic densities (rho per
// segment) with the fixed-point table of the air alone (launch_table_fx, one class), and
// production-height averaging (avg.n_bins > 0), for quadratic densities as that (ncls = 0), for
// constant ones from the table of ncls classes (rho per class); mixed: quadratic densities.
cudaError_t launch_atmos_fx_inline(const OscParams& p, const double* energies, int ne,
                                   const int2* table, const int* seg_off, const double* seg_len, const double* rho,
                                   int ncls, int n_cosines, const AvgArrays& avg, double* out,
                                   cudaStream_t s, RowRange rr = RowRange{});
cudaError_t launch_atmos_mixed_inline(const OscParams& p, const double* energies, int ne,
                                      const int* seg_off, const float2* seg_len,
                                      const double* seg_rho, int n_cosines, float* out,
                                      cudaStream_t s, RowRange rr = RowRange{});

// The weights' scales [2][3][nc][ne] (fx_weight_scale); *any is set where one is not zero.
cudaError_t launch_weight_scales(const double* prob, int nc, int n_bins, int ne, signed char* scale,
                                 int* any, cudaStream_t s);
// n matrices [rows][cols] of doubles, each transposed to [cols][rows], as floats or doubles.
cudaError_t launch_weights_transpose(const double* src, int rows, long long cols, int n, void* dst,
                                     bool to_float, cudaStream_t s);

// out[i] = (x[i] rounded to float, the remainder rounded to float), on the device.
cudaError_t launch_split_pairs(const double* x, int n, float2* out, cudaStream_t s);

// One channel plane [nc][ne] (float or double) transposed to [ne][nc] doubles.
cudaError_t launch_plane_transpose(const void* src, bool is_float, int nc, int ne, double* dst,
                                   cudaStream_t s);

// Beam bins: rho_e = rho * 0.5 (electron density), L in km.
cudaError_t launch_beam_f64(const OscParams& p, const double* energies, int ne, double rho_e,
                            double L_km, double* out, cudaStream_t s);
cudaError_t launch_beam_mixed(const OscParams& p, const float2* energies, int ne, double rho_e,
                              double L_km, float* out, cudaStream_t s);

}  // namespace cp3
