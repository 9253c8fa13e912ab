// pm_lpt.h -- device 1LPT initial conditions (internal, see pm_lpt.cu).
#pragma once

#include <cuda_runtime.h>

namespace hyowon {

// Transform plans and work arrays of the 1LPT map and its adjoint on one lattice
// side. The arrays are the caller's (place()), or a block of their own that is made
// on first use and freed with the object or by release().
struct LptWork {
    int N = 0;
    size_t bytes = 0;           // what the arrays below and cuFFT's own take
    size_t spectrum = 0, mesh = 0;   // of which a half spectrum and the mesh
    double2* delta = nullptr;   // half spectra
    double2* work = nullptr;
    double* real = nullptr;
    int r2c = 0, c2r = 0;       // cufftHandle
    bool plans = false;
    void* block = nullptr;      // the block of its own, if any
    // Plans for n_side, and `bytes`. 0 or 6 (cuFFT); *err names the failure.
    int plan(int n_side, const char** err);
    // Puts the arrays into `bytes` bytes of the caller's, 256-byte aligned, used by the
    // calls below until they return; null takes them out again.
    void place(void* at);
    // plan(), with a block of its own unless the arrays are placed. 0, 6 or 7 (allocation).
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
