// cp3_tables.cu -- eigen work: the per-(density class, energy) tables of the atmospheric
// kernels and the FP64 beam kernel.
//
// This translation unit is compiled with -fmad=false: where two levels nearly meet, its FP64
// arithmetic is the reference's (physics.hpp getMfast) in the reference's order, and keeping
// multiply and add separately rounded reproduces the reference's x86 results to the last
// bits where the eigen-system is ill-conditioned.
#include <algorithm>

#include "cp3_device.cuh"
#include "cp3_f64.cuh"
#include "cp3_fixed.cuh"
#include "cp3_mixed.cuh"
#include "cp3_kernels.hpp"

namespace cp3 {

namespace {

constexpr int kTableBlock = 128;

// The table of the fixed-point FP64 bins (cp3_fixed.cuh): for each class the rotation to the
// next class's eigenbasis and the phase rates, and once per energy the flavour rows and the
// vacuum coefficients.  A block is 32 energies by a run of kFxRun classes, one class a warp;
// the extra warp solves the class after the run, for the last rotation.  59 shells x 2000
// energies take 21 us (130 with the FP64 formulas), PREM-4 x 400 energies 11 us (31): one wave,
// its latency.
constexpr int kFxRun = 8;

__global__ void __launch_bounds__(32 * (kFxRun + 1))
    table_fx_kernel(const __grid_constant__ OscParams p, const double* __restrict__ energies,
                    int ne, int ne_pad, const double* __restrict__ cls_rho, int ncls,
                    int2* __restrict__ table) {
    __shared__ int2 s_u[kFxRun + 1][9][32];
    launch_dependents();
    const int lane = threadIdx.x & 31, wv = threadIdx.x >> 5;
    const int ie = blockIdx.x * 32 + lane, c = blockIdx.y * kFxRun + wv;
    const bool on = c < ncls && ie < ne;
    FxClass k;
    if (on) {
        fx_solve(&p, energies[ie], cls_rho[c], k);
#pragma unroll
        for (int f = 0; f < 9; f++) s_u[wv][f][lane] = make_int2(k.U[f / 3][f % 3].h, k.U[f / 3][f % 3].l);
        int2* ext = table + (size_t)ncls * kFxFields * ne_pad + ie;
        if (c < 2) {
            fx row[9];
            fx_rows(k.U, p.w, row);
#pragma unroll
            for (int f = 0; f < 9; f++)
                ext[(size_t)((c == 0 ? kFxV0 : kFxV1) + f) * ne_pad] = make_int2(row[f].h, row[f].l);
            if (c == 0) {
                fx v[13];
                fx_coefficients(row, v);
#pragma unroll
                for (int f = 0; f < 13; f++) ext[(size_t)(kFxVac + f) * ne_pad] = make_int2(v[f].h, v[f].l);
                if (ncls == 1) {
#pragma unroll
                    for (int f = 0; f < 9; f++) ext[(size_t)(kFxV1 + f) * ne_pad] = s_u[wv][f][lane];
                }
            }
        }
    }
    __syncthreads();
    if (!on || wv == kFxRun) return;  // (with fewer classes than a run there is no class after it)
    int2* t = table + (size_t)c * kFxFields * ne_pad + ie;
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const long long b = fx_bits(k.rate[q]);
        t[(size_t)(kFxRates + q) * ne_pad] = make_int2((int)b, (int)(b >> 32));
    }
    if (c + 1 == ncls) return;
    fx B[3][3], R[3][3];
#pragma unroll
    for (int f = 0; f < 9; f++) B[f / 3][f % 3] = fx_of(s_u[wv + 1][f][lane]);
    fx_rotation(B, k.U, R);
#pragma unroll
    for (int f = 0; f < 9; f++) t[(size_t)f * ne_pad] = make_int2(R[f / 3][f % 3].h, R[f / 3][f % 3].l);
}

// Mixed table: real unit eigenvectors u1, u2 of H0 + V e0 e0^T (P_k = u_k u_k^T) and the
// phase rates omega_k = 2.534 (m_k - m_0) / E as float pairs (rotated_eigen_vectors: FP32
// roots refined in double-float; FP64 only where two roots nearly coincide).  One 48-byte
// entry per (class c, energy e) at table[(c * ne_pad + e) * 12]: u1, u2, omega_1 hi/lo,
// omega_2 hi/lo, 2 unused -- three 16-byte words a thread reads with vector loads.
// Real = double (split on the device) or float2 (pairs split on the host: no FP64 at all).
template <class Real>
__global__ void __launch_bounds__(kTableBlock)
    table_mixed_kernel(const __grid_constant__ OscParams p, const Real* __restrict__ energies,
                       int ne, int ne_pad, const Real* __restrict__ cls_rho,
                       float* __restrict__ table) {
    launch_dependents();
    const int ie = blockIdx.x * kTableBlock + threadIdx.x;
    const int c = blockIdx.y;
    if (ie >= ne) return;
    float u[2][3], om[2][2];
    rotated_eigen_vectors(&p, to_df(energies[ie]), to_df(cls_rho[c]), u, om);
    store_table_entry(table + ((size_t)c * ne_pad + ie) * kMixFields, u, om);
}

// physics::calculate_beam (physics.hpp:1153-1260), one thread per energy; result [9][ne]: the
// fixed-point layer of the energy (fx_solve) and the one-layer expansion of its probabilities.
// 1e5 energies: 20.3 us (135 us in FP64 arithmetic, 582 FP64 instructions an energy).
__device__ const TrigTable g_trig = make_trig_table();

// A phase out of the fixed-point range: the FP64 formulas.
__device__ __noinline__ void beam_out_of_range(const OscParams* p, double E, double rho_e, double L,
                                               double* out, size_t plane) {
    Layer64 f;
    double dmv[3], arg[3];
    rotated_layer_f64(p, E, rho_e, f.u, dmv);
    layer64_phases(dmv, L, E, 1.0 / E, f, arg);
    layer_store64(layer_coefficients64(f.u, p->w), f.z, out, plane);
}

__global__ void __launch_bounds__(kTableBlock)
    beam_f64_kernel(const __grid_constant__ OscParams p, const double* __restrict__ energies,
                    int ne, double rho_e, double L, double* __restrict__ out) {
    __shared__ longlong2 s_trig[kTrigSize];
    for (int i = threadIdx.x; i < kTrigSize; i += kTableBlock)
        s_trig[i] = make_longlong2(g_trig.cs[i][0], g_trig.cs[i][1]);
    __syncthreads();
    const int ie = blockIdx.x * kTableBlock + threadIdx.x;
    if (ie >= ne) return;
    FxClass k;
    fx_solve(&p, energies[ie], rho_e, k);
    unsigned int bad = 0;
    cfx e[2];
#pragma unroll
    for (int q = 0; q < 2; q++) e[q] = fx_unit(fx_angle(k.rate[q], L, bad), s_trig);
    if ((bad >> 20) != 0) {
        beam_out_of_range(&p, energies[ie], rho_e, L, out + ie, (size_t)ne);
        return;
    }
    fx row[9], v[13];
    fx_rows(k.U, p.w, row);
    fx_coefficients(row, v);
    long long P[4];
    fx_one_layer(v, e, P);
    fx_store(P, out + ie, (size_t)ne);
}

}  // namespace

size_t table_fx_words(int ncls, int ne) {
    return ((size_t)ncls * kFxFields + kFxExtra) * pad_energies(ne);
}

cudaError_t launch_table_fx(const OscParams& p, const double* energies, int ne,
                            const double* cls_rho, int ncls, int2* table, cudaStream_t s) {
    if (ne <= 0 || ncls <= 0) return cudaSuccess;
    dim3 grid((ne + 31) / 32, (ncls + kFxRun - 1) / kFxRun);
    table_fx_kernel<<<grid, 32 * (std::min(ncls, kFxRun) + 1), 0, s>>>(p, energies, ne, pad_energies(ne),
                                                                       cls_rho, ncls, table);
    return cudaGetLastError();
}

template <class Real>
static cudaError_t table_mixed(const OscParams& p, const Real* energies, int ne,
                               const Real* cls_rho, int ncls, float* table, cudaStream_t s) {
    if (ne <= 0 || ncls <= 0) return cudaSuccess;
    dim3 grid((ne + kTableBlock - 1) / kTableBlock, ncls);
    table_mixed_kernel<Real><<<grid, kTableBlock, 0, s>>>(p, energies, ne, pad_energies(ne), cls_rho, table);
    return cudaGetLastError();
}

cudaError_t launch_table_mixed(const OscParams& p, const double* energies, int ne,
                               const double* cls_rho, int ncls, float* table, cudaStream_t s) {
    return table_mixed(p, energies, ne, cls_rho, ncls, table, s);
}

cudaError_t launch_table_mixed(const OscParams& p, const float2* energies, int ne,
                               const float2* cls_rho, int ncls, float* table, cudaStream_t s) {
    return table_mixed(p, energies, ne, cls_rho, ncls, table, s);
}

cudaError_t preload_table_mixed() {
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, table_mixed_kernel<double>);
}

cudaError_t launch_beam_f64(const OscParams& p, const double* energies, int ne, double rho_e,
                            double L_km, double* out, cudaStream_t s) {
    if (ne <= 0) return cudaSuccess;
    beam_f64_kernel<<<(ne + kTableBlock - 1) / kTableBlock, kTableBlock, 0, s>>>(p, energies, ne,
                                                                                rho_e, L_km, out);
    return cudaGetLastError();
}

}  // namespace cp3
