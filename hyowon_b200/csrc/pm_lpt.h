// pm_lpt.h -- device 1LPT initial conditions (internal, see pm_lpt.cu).
#pragma once

#include <cuda_runtime.h>

namespace hyowon {

// Transform plans and work arrays of the 1LPT map and its adjoint on one lattice
// side; made on first use, freed with the object (or by release()).
struct LptWork {
    int N = 0;
    void* block = nullptr;      // one allocation: the arrays below and cuFFT's own
    double2* delta = nullptr;   // half spectra
    double2* work = nullptr;
    double* real = nullptr;
    int r2c = 0, c2r = 0;       // cufftHandle
    bool plans = false;
    // 0, 6 (CUDA / cuFFT) or 7 (allocation); *err names the failure.
    int require(int n_side, cudaStream_t s, const char** err);
    void release();
    LptWork() = default;
    LptWork(const LptWork&) = delete;
    LptWork& operator=(const LptWork&) = delete;
    ~LptWork() { release(); }
};

// Writes positions / momenta of the N^3 lattice particles (index (iN+j)N+k)
// into d_pos[3] / d_mom[3]. d_noise (N^3 doubles, device) may be overwritten.
// Returns 0, 6 (CUDA / cuFFT) or 7 (allocation); *err names the failure.
int lpt_ics_device(LptWork& w, int N, double L, const double* d_noise, const double* d_xs,
                   const double* d_ys, const double* d_y2, int n_nodes, double pf,
                   double* const d_pos[3], double* const d_mom[3], unsigned int* d_status,
                   cudaStream_t s, const char** err);

// Vector-Jacobian product of the displacement map w.r.t. the noise: given the
// per-particle cotangents g_d (lattice order, N^3 each), writes
// d_grad = sum_d B_d^T g_d = -sum_d B_d g_d (B_d is antisymmetric).
int lpt_adjoint_device(LptWork& w, int N, double L, double* const d_g[3], const double* d_xs,
                       const double* d_ys, const double* d_y2, int n_nodes, double* d_grad,
                       cudaStream_t s, const char** err);

}  // namespace hyowon
