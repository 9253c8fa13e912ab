// pm_adjoint.cu -- the differentiation form: gradient of a density-field loss
// with respect to the initial white noise, through 1LPT and the KDK PM step.
//
// Forward model (positions binary64 in both precisions; momenta, forces,
// meshes and FFTs in Real = double or float):
//   x0, p0 = 1LPT(w);  a_k = F(x_k)
//   p' = p_k + K1_k a_k;  x_{k+1} = wrap(x_k + D_k p');  p_{k+1} = p' + K2_k a_{k+1}
//   F(x) = gather_-grad( A deposit(x) ),  A = (1/dx^3) c2r(G(k) r2c(.))/N^3
//   L = 1/2 sum_c (delta_c - t_c)^2,  delta_c = M_c / Mbar - 1 on the PM mesh.
//
// Reverse pass ("reverse leapfrog"): KDK is time reversible, so the state of
// step k is reconstructed from step k+1 (x_k = x_{k+1} - D p', p' = p_{k+1} -
// K2 a_{k+1}, p_k = p' - K1 a_k) with one force solve per step; the stored
// (x, p) checkpoints every `ckpt_every` steps replace the reconstruction and
// bound its round-off drift. Cotangents (binary64):
//   lx += VJP_F(x_{k+1}; (K2_k + K1_{k+1}) lp)   (the two kicks that use
//         a_{k+1} share one VJP)
//   lp += D_k lx
// and a final VJP_F(x_0; K1_0 lp). The force VJP for a per-particle cotangent v:
//   u_d = CIC scatter of v_d            (transpose of the interpolation)
//   s   = sum_d D_d u_d                 (transpose of -grad: centred divergence)
//   psi = A s                           (A is real, even, hence symmetric)
//   d(v.F)/dx_j = sum_c dW_jc/dx_j (m psi_c + v_j . g_c),  g = -grad(phi(x))
// with the CIC weight derivative of the particle's own base cell (the one-sided
// convention of src/mesh/mass_assignment_directional.cpp:133-166). The
// 1LPT adjoint is dL/dw = -sum_d B_d (lx_d + pf lp_d) (pm_lpt.cu).
#include <cuda_runtime.h>
#include <cufft.h>

#include <cmath>
#include <cstring>
#include <exception>
#include <new>
#include <string>
#include <vector>

#include "hyowon_adjoint.h"
#include "hyowon_pm.h"
#include "pm_common.cuh"
#include "pm_lpt.h"
#include "pm_adjoint.h"
#include "pm_poisson.h"

namespace hyowon::adj {

namespace {

constexpr int kT = 256;
inline unsigned nb(uint64_t n) { return static_cast<unsigned>((n + kT - 1) / kT); }

template <typename R>
struct FFTTypes;
template <>
struct FFTTypes<double> {
    using C = double2;
    static constexpr cufftType R2C = CUFFT_D2Z;
    static constexpr cufftType C2R = CUFFT_Z2D;
    static cufftResult fwd(cufftHandle p, double* in, double2* out) {
        return cufftExecD2Z(p, in, reinterpret_cast<cufftDoubleComplex*>(out));
    }
    static cufftResult inv(cufftHandle p, double2* in, double* out) {
        return cufftExecZ2D(p, reinterpret_cast<cufftDoubleComplex*>(in), out);
    }
};
template <>
struct FFTTypes<float> {
    using C = float2;
    static constexpr cufftType R2C = CUFFT_R2C;
    static constexpr cufftType C2R = CUFFT_C2R;
    static cufftResult fwd(cufftHandle p, float* in, float2* out) {
        return cufftExecR2C(p, in, reinterpret_cast<cufftComplex*>(out));
    }
    static cufftResult inv(cufftHandle p, float2* in, float* out) {
        return cufftExecC2R(p, reinterpret_cast<cufftComplex*>(in), out);
    }
};

struct Corner {
    int ix, iy, iz;
    double fx, fy, fz;
};

__device__ __forceinline__ bool corner_of(double x, double y, double z, const Axis& a, Corner& c) {
    return cic_coord_f64(x, a, c.ix, c.fx) & cic_coord_f64(y, a, c.iy, c.fy)
        & cic_coord_f64(z, a, c.iz, c.fz);
}

__device__ __forceinline__ size_t cidx(int x, int y, int z, int N) {
    return (static_cast<size_t>(x) * N + y) * N + z;
}

__device__ __forceinline__ int up(int i, int N) { return i + 1 == N ? 0 : i + 1; }
__device__ __forceinline__ int dn(int i, int N) { return i == 0 ? N - 1 : i - 1; }

// Adds m * w to the 8 corner cells of a particle.
template <typename R>
__device__ __forceinline__ void deposit_corners(const Corner& c, R m, int N, R* __restrict__ mesh) {
    const R wx[2] = {R(1) - R(c.fx), R(c.fx)}, wy[2] = {R(1) - R(c.fy), R(c.fy)},
            wz[2] = {R(1) - R(c.fz), R(c.fz)};
    const int gx[2] = {c.ix, up(c.ix, N)}, gy[2] = {c.iy, up(c.iy, N)}, gz[2] = {c.iz, up(c.iz, N)};
    for (int u = 0; u < 2; ++u)
        for (int v = 0; v < 2; ++v)
            for (int w = 0; w < 2; ++w)
                atomicAdd(&mesh[cidx(gx[u], gy[v], gz[w], N)], m * wx[u] * wy[v] * wz[w]);
}

template <typename R>
__global__ void k_deposit(uint32_t n, const double* __restrict__ x, const double* __restrict__ y,
                          const double* __restrict__ z, R m, Axis a, R* __restrict__ mesh,
                          unsigned int* status) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Corner c;
    if (!corner_of(x[i], y[i], z[i], a, c)) {
        raise_status(status, ST_CELL_ESCAPE);
        return;
    }
    deposit_corners(c, m, a.N, mesh);
}

// Three-component CIC scatter (transpose of the interpolation) of the force
// cotangent coef * l. Particles
// stay in lattice order, so consecutive lanes usually hold z-neighbours in the
// same (x, y) cell column: when lane l+1's lower z cells are lane l's upper z
// cells, lane l hands its upper-z weights to lane l+1, which adds them to its
// own before the atomics (half the atomics for a matched pair; the sum is
// the same up to the order of additions, which atomics leave open anyway).
template <typename R>
__global__ void k_scatter3(uint32_t n, const double* __restrict__ x, const double* __restrict__ y,
                           const double* __restrict__ z, const double* __restrict__ l0,
                           const double* __restrict__ l1, const double* __restrict__ l2,
                           double coef, Axis a, R* __restrict__ u0, R* __restrict__ u1,
                           R* __restrict__ u2) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int N = a.N;
    Corner c{};
    const bool ok = i < n && corner_of(x[i], y[i], z[i], a, c);
    // contributions lo[u][v][d] (z cell iz) and hi[u][v][d] (z cell iz + 1)
    R lo[2][2][3], hi[2][2][3];
    int gx[2] = {0, 0}, gy[2] = {0, 0}, gz[2] = {0, 0};
    if (ok) {
        const R wx[2] = {R(1) - R(c.fx), R(c.fx)}, wy[2] = {R(1) - R(c.fy), R(c.fy)},
                wz[2] = {R(1) - R(c.fz), R(c.fz)};
        gx[0] = c.ix; gx[1] = up(c.ix, N);
        gy[0] = c.iy; gy[1] = up(c.iy, N);
        gz[0] = c.iz; gz[1] = up(c.iz, N);
        const R av[3] = {static_cast<R>(coef * l0[i]), static_cast<R>(coef * l1[i]),
                         static_cast<R>(coef * l2[i])};
        for (int u = 0; u < 2; ++u)
            for (int v = 0; v < 2; ++v)
                for (int d = 0; d < 3; ++d) {
                    lo[u][v][d] = wx[u] * wy[v] * wz[0] * av[d];
                    hi[u][v][d] = wx[u] * wy[v] * wz[1] * av[d];
                }
    } else {
        for (int u = 0; u < 2; ++u)
            for (int v = 0; v < 2; ++v)
                for (int d = 0; d < 3; ++d) lo[u][v][d] = hi[u][v][d] = R(0);
    }
    // the cell column and upper z cell of the lane below
    const int col = ok ? c.ix * N + c.iy : -1;
    const int col_below = __shfl_up_sync(0xffffffffu, col, 1);
    const int ztop_below = __shfl_up_sync(0xffffffffu, gz[1], 1);
    const bool take = lane > 0 && ok && col_below == col && ztop_below == gz[0];
    for (int u = 0; u < 2; ++u)
        for (int v = 0; v < 2; ++v)
            for (int d = 0; d < 3; ++d) {
                const R h = __shfl_up_sync(0xffffffffu, hi[u][v][d], 1);
                if (take) lo[u][v][d] += h;
            }
    // whether the lane above took this lane's upper weights
    const bool given = __shfl_down_sync(0xffffffffu, take ? 1 : 0, 1) != 0 && lane < 31;
    if (!ok) return;
    for (int u = 0; u < 2; ++u)
        for (int v = 0; v < 2; ++v) {
            const size_t k0 = cidx(gx[u], gy[v], gz[0], N);
            atomicAdd(&u0[k0], lo[u][v][0]);
            atomicAdd(&u1[k0], lo[u][v][1]);
            atomicAdd(&u2[k0], lo[u][v][2]);
            if (!given) {
                const size_t k1 = cidx(gx[u], gy[v], gz[1], N);
                atomicAdd(&u0[k1], hi[u][v][0]);
                atomicAdd(&u1[k1], hi[u][v][1]);
                atomicAdd(&u2[k1], hi[u][v][2]);
            }
        }
}

// s = sum_d (u_d[c+e_d] - u_d[c-e_d]) / (2 dx); one block per row (y, x), so that no
// thread divides a 64-bit cell number by N (18.6 us of a 128^3 mesh, whose four
// arrays take 10).
template <typename R>
__global__ void k_divergence(int N, const R* __restrict__ u0, const R* __restrict__ u1,
                             const R* __restrict__ u2, R inv_two_dx, R* __restrict__ s) {
    const int y = blockIdx.x, x = blockIdx.y;
    const size_t row = cidx(x, y, 0, N);
    const R* const xp = u0 + cidx(up(x, N), y, 0, N);
    const R* const xm = u0 + cidx(dn(x, N), y, 0, N);
    const R* const yp = u1 + cidx(x, up(y, N), 0, N);
    const R* const ym = u1 + cidx(x, dn(y, N), 0, N);
    const R* const zr = u2 + row;
    for (int z = threadIdx.x; z < N; z += blockDim.x)
        s[row + z] = ((xp[z] - xm[z]) + (yp[z] - ym[z]) + (zr[up(z, N)] - zr[dn(z, N)])) * inv_two_dx;
}

template <typename R, typename C>
__global__ void k_green(int N, C* __restrict__ modes, const R* __restrict__ lap, R c) {
    const int Hz = N / 2 + 1;
    const uint64_t total = static_cast<uint64_t>(N) * N * Hz;
    const uint64_t idx = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    if (idx == 0) {
        modes[0].x = R(0);
        modes[0].y = R(0);
        return;
    }
    const int iz = static_cast<int>(idx % Hz);
    const uint64_t t = idx / Hz;
    const int iy = static_cast<int>(t % N);
    const int ix = static_cast<int>(t / N);
    const R f = c / (lap[ix] + lap[iy] + lap[iz]);
    C v = modes[idx];
    v.x *= f;
    v.y *= f;
    modes[idx] = v;
}

// Loads the 4x4x4 stencil footprint of a particle's 8 corners and returns the
// centred-difference force g = -grad(phi) at each corner.
template <typename R>
__device__ __forceinline__ void corner_forces(const R* __restrict__ phi, const Corner& c, int N,
                                              R inv_two_dx, R g[2][2][2][3]) {
    const int xs[4] = {dn(c.ix, N), c.ix, up(c.ix, N), up(up(c.ix, N), N)};
    const int ys[4] = {dn(c.iy, N), c.iy, up(c.iy, N), up(up(c.iy, N), N)};
    const int zs[4] = {dn(c.iz, N), c.iz, up(c.iz, N), up(up(c.iz, N), N)};
    for (int u = 0; u < 2; ++u)
        for (int v = 0; v < 2; ++v)
            for (int w = 0; w < 2; ++w) {
                const int X = u + 1, Y = v + 1, Z = w + 1;
                g[u][v][w][0] = -(phi[cidx(xs[X + 1], ys[Y], zs[Z], N)] - phi[cidx(xs[X - 1], ys[Y], zs[Z], N)]) * inv_two_dx;
                g[u][v][w][1] = -(phi[cidx(xs[X], ys[Y + 1], zs[Z], N)] - phi[cidx(xs[X], ys[Y - 1], zs[Z], N)]) * inv_two_dx;
                g[u][v][w][2] = -(phi[cidx(xs[X], ys[Y], zs[Z + 1], N)] - phi[cidx(xs[X], ys[Y], zs[Z - 1], N)]) * inv_two_dx;
            }
}

// CIC-interpolated centred-gradient force at one position; false (nothing
// written) where the cell assignment fails.
template <typename R>
__device__ __forceinline__ bool force_at(double px, double py, double pz, const R* __restrict__ phi,
                                         const Axis& a, R inv_two_dx, R& s0, R& s1, R& s2) {
    Corner c;
    if (!corner_of(px, py, pz, a, c)) return false;
    R g[2][2][2][3];
    corner_forces(phi, c, a.N, inv_two_dx, g);
    const R wx[2] = {R(1) - R(c.fx), R(c.fx)}, wy[2] = {R(1) - R(c.fy), R(c.fy)},
            wz[2] = {R(1) - R(c.fz), R(c.fz)};
    s0 = s1 = s2 = 0;
    for (int u = 0; u < 2; ++u)
        for (int v = 0; v < 2; ++v)
            for (int w = 0; w < 2; ++w) {
                const R W = wx[u] * wy[v] * wz[w];
                s0 += W * g[u][v][w][0];
                s1 += W * g[u][v][w][1];
                s2 += W * g[u][v][w][2];
            }
    return true;
}

// One forward step of a particle at x_j, whose potential is known: a = F(x_j), the
// closing kick K2 of the step before (K2 = 0 at the start), the state to the
// checkpoint arrays when given, then, when `more`, the opening kick K1, the drift
// and the deposit at x_{j+1} into the zeroed `mesh`; else a to the acceleration
// arrays. One pass over the particles in place of force, two kicks, drift, deposit
// and the checkpoint's copies, each of which re-read what the last wrote: the
// forward pass of 16 steps at 128^3 takes 3.67 ms (4.56), of 8 steps at 48^3 on a
// 96^3 mesh in FP32 0.62 (0.81). The loads of the stencil bound it.
template <typename R>
struct Checkpoint {
    double* x[3];
    R* p[3];
};
template <typename R>
__global__ void __launch_bounds__(kT)
k_advance(uint32_t n, double* __restrict__ x0, double* __restrict__ x1, double* __restrict__ x2,
          R* __restrict__ p0, R* __restrict__ p1, R* __restrict__ p2, const R* __restrict__ phi,
          Axis a, R inv_two_dx, R K2, Checkpoint<R> save, int more, R K1, double D, R m,
          R* __restrict__ mesh, R* __restrict__ ax, R* __restrict__ ay, R* __restrict__ az,
          unsigned int* status) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = x0[i], y = x1[i], z = x2[i];
    R q0 = p0[i], q1 = p1[i], q2 = p2[i];
    R s0, s1, s2;
    if (!force_at(x, y, z, phi, a, inv_two_dx, s0, s1, s2)) return;   // raised by the deposit
    q0 += K2 * s0;
    q1 += K2 * s1;
    q2 += K2 * s2;
    if (save.x[0]) {
        save.x[0][i] = x;
        save.x[1][i] = y;
        save.x[2][i] = z;
        save.p[0][i] = q0;
        save.p[1][i] = q1;
        save.p[2][i] = q2;
    }
    if (!more) {
        ax[i] = s0;
        ay[i] = s1;
        az[i] = s2;
        p0[i] = q0;
        p1[i] = q1;
        p2[i] = q2;
        return;
    }
    q0 += K1 * s0;
    q1 += K1 * s1;
    q2 += K1 * s2;
    const double nx = wrap_f64(x + D * static_cast<double>(q0), a.L);
    const double ny = wrap_f64(y + D * static_cast<double>(q1), a.L);
    const double nz = wrap_f64(z + D * static_cast<double>(q2), a.L);
    x0[i] = nx;
    x1[i] = ny;
    x2[i] = nz;
    p0[i] = q0;
    p1[i] = q1;
    p2[i] = q2;
    Corner c;
    if (!corner_of(nx, ny, nz, a, c)) {
        raise_status(status, ST_CELL_ESCAPE);
        return;
    }
    deposit_corners(c, m, a.N, mesh);
}

// lp += D lx (the drift's transpose) and p += K a (a kick), one pass.
template <typename R>
__global__ void k_axpy3_kick(uint32_t n, double D, const double* __restrict__ x0,
                             const double* __restrict__ x1, const double* __restrict__ x2,
                             double* __restrict__ y0, double* __restrict__ y1,
                             double* __restrict__ y2, R* __restrict__ p0, R* __restrict__ p1,
                             R* __restrict__ p2, const R* __restrict__ a0,
                             const R* __restrict__ a1, const R* __restrict__ a2, R K) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    y0[i] += D * x0[i];
    y1[i] += D * x1[i];
    y2[i] += D * x2[i];
    p0[i] += K * a0[i];
    p1[i] += K * a1[i];
    p2[i] += K * a2[i];
}

template <typename R>
__global__ void k_force(uint32_t n, const double* __restrict__ x, const double* __restrict__ y,
                        const double* __restrict__ z, const R* __restrict__ phi, Axis a,
                        R inv_two_dx, R* __restrict__ ax, R* __restrict__ ay, R* __restrict__ az) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Corner c;
    if (!corner_of(x[i], y[i], z[i], a, c)) return;
    R g[2][2][2][3];
    corner_forces(phi, c, a.N, inv_two_dx, g);
    const R wx[2] = {R(1) - R(c.fx), R(c.fx)}, wy[2] = {R(1) - R(c.fy), R(c.fy)},
            wz[2] = {R(1) - R(c.fz), R(c.fz)};
    R s0 = 0, s1 = 0, s2 = 0;
    for (int u = 0; u < 2; ++u)
        for (int v = 0; v < 2; ++v)
            for (int w = 0; w < 2; ++w) {
                const R W = wx[u] * wy[v] * wz[w];
                s0 += W * g[u][v][w][0];
                s1 += W * g[u][v][w][1];
                s2 += W * g[u][v][w][2];
            }
    ax[i] = s0;
    ay[i] = s1;
    az[i] = s2;
}

// d(v.F)/dx of one particle: sum_c dW_c/dx (mpsi psi_c + v . g_c); phi may be null
// (v = 0).
template <typename R>
__device__ __forceinline__ void force_vjp(const Corner& c, int N, const R* __restrict__ psi, R mpsi,
                                          const R* __restrict__ phi, const R (&vv)[3],
                                          R inv_two_dx, R& s0, R& s1, R& s2) {
    R g[2][2][2][3];
    const bool with_v = phi != nullptr;
    if (with_v) corner_forces(phi, c, N, inv_two_dx, g);
    const R inv_dx = R(2) * inv_two_dx;
    const R wx[2] = {R(1) - R(c.fx), R(c.fx)}, wy[2] = {R(1) - R(c.fy), R(c.fy)},
            wz[2] = {R(1) - R(c.fz), R(c.fz)};
    const R dw[2] = {-inv_dx, inv_dx};
    const int gx[2] = {c.ix, up(c.ix, N)}, gy[2] = {c.iy, up(c.iy, N)}, gz[2] = {c.iz, up(c.iz, N)};
    s0 = s1 = s2 = 0;
    for (int u = 0; u < 2; ++u)
        for (int v = 0; v < 2; ++v)
            for (int w = 0; w < 2; ++w) {
                R h = mpsi * psi[cidx(gx[u], gy[v], gz[w], N)];
                if (with_v) h += vv[0] * g[u][v][w][0] + vv[1] * g[u][v][w][1] + vv[2] * g[u][v][w][2];
                s0 += dw[u] * wy[v] * wz[w] * h;
                s1 += wx[u] * dw[v] * wz[w] * h;
                s2 += wx[u] * wy[v] * dw[w] * h;
            }
}

// lx += d(v.F)/dx with v = coef * lp (phi null: the density loss alone).
template <typename R>
__global__ void k_vjp_gather(uint32_t n, const double* __restrict__ x, const double* __restrict__ y,
                             const double* __restrict__ z, const R* __restrict__ psi, R mpsi,
                             const R* __restrict__ phi, double coef, const double* __restrict__ l0,
                             const double* __restrict__ l1, const double* __restrict__ l2, Axis a,
                             R inv_two_dx, double* __restrict__ o0, double* __restrict__ o1,
                             double* __restrict__ o2) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Corner c;
    if (!corner_of(x[i], y[i], z[i], a, c)) return;
    R vv[3] = {R(0), R(0), R(0)};
    if (phi) {
        vv[0] = static_cast<R>(coef * l0[i]);
        vv[1] = static_cast<R>(coef * l1[i]);
        vv[2] = static_cast<R>(coef * l2[i]);
    }
    R s0, s1, s2;
    force_vjp(c, a.N, psi, mpsi, phi, vv, inv_two_dx, s0, s1, s2);
    o0[i] += static_cast<double>(s0);
    o1[i] += static_cast<double>(s1);
    o2[i] += static_cast<double>(s2);
}

// One reverse step of a particle from x_{j+1} to x_j where the forward pass kept
// both potentials: lx += d(v.F)/dx at x_{j+1} (v = coef lp), lp += D lx, the kick
// K2 undone, then either the checkpointed state or the drift D undone, a = F(x_j)
// from its potential, and the kick K1 undone. One pass in place of the gather, the
// axpy / kick and the un-step or the checkpoint's copies and force; with the
// scatter's and the gather's cotangents formed in place the reverse pass of the same
// runs takes 7.33 ms (8.56) and 0.91 (1.06).
template <typename R>
__global__ void __launch_bounds__(kT)
k_reverse(uint32_t n, double* __restrict__ x0, double* __restrict__ x1, double* __restrict__ x2,
          R* __restrict__ p0, R* __restrict__ p1, R* __restrict__ p2, R* __restrict__ ax,
          R* __restrict__ ay, R* __restrict__ az, const R* __restrict__ psi, R mpsi,
          const R* __restrict__ phi_next, const R* __restrict__ phi, double coef, double D, R K1,
          R K2, Checkpoint<R> from, Axis a, R inv_two_dx, double* __restrict__ lx0,
          double* __restrict__ lx1, double* __restrict__ lx2, double* __restrict__ lp0,
          double* __restrict__ lp1, double* __restrict__ lp2) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = x0[i], y = x1[i], z = x2[i];
    const double k0 = lp0[i], k1 = lp1[i], k2 = lp2[i];
    double g0 = lx0[i], g1 = lx1[i], g2 = lx2[i];
    {
        Corner c;
        if (corner_of(x, y, z, a, c)) {
            const R vv[3] = {static_cast<R>(coef * k0), static_cast<R>(coef * k1),
                             static_cast<R>(coef * k2)};
            R s0, s1, s2;
            force_vjp(c, a.N, psi, mpsi, phi_next, vv, inv_two_dx, s0, s1, s2);
            g0 += static_cast<double>(s0);
            g1 += static_cast<double>(s1);
            g2 += static_cast<double>(s2);
            lx0[i] = g0;
            lx1[i] = g1;
            lx2[i] = g2;
        }
    }
    lp0[i] = k0 + D * g0;
    lp1[i] = k1 + D * g1;
    lp2[i] = k2 + D * g2;
    double nx, ny, nz;
    R q0, q1, q2;
    if (from.x[0]) {
        nx = from.x[0][i];
        ny = from.x[1][i];
        nz = from.x[2][i];
        q0 = from.p[0][i];
        q1 = from.p[1][i];
        q2 = from.p[2][i];
    } else {
        q0 = p0[i] - K2 * ax[i];
        q1 = p1[i] - K2 * ay[i];
        q2 = p2[i] - K2 * az[i];
        nx = wrap_f64(x - D * static_cast<double>(q0), a.L);
        ny = wrap_f64(y - D * static_cast<double>(q1), a.L);
        nz = wrap_f64(z - D * static_cast<double>(q2), a.L);
    }
    x0[i] = nx;
    x1[i] = ny;
    x2[i] = nz;
    R s0, s1, s2;
    if (force_at(nx, ny, nz, phi, a, inv_two_dx, s0, s1, s2)) {
        ax[i] = s0;
        ay[i] = s1;
        az[i] = s2;
        if (!from.x[0]) {
            q0 -= K1 * s0;
            q1 -= K1 * s1;
            q2 -= K1 * s2;
        }
    }
    p0[i] = q0;
    p1[i] = q1;
    p2[i] = q2;
}

template <typename R>
__global__ void k_kick(uint32_t n, R* __restrict__ p0, R* __restrict__ p1, R* __restrict__ p2,
                       const R* __restrict__ a0, const R* __restrict__ a1,
                       const R* __restrict__ a2, R K) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    p0[i] += K * a0[i];
    p1[i] += K * a1[i];
    p2[i] += K * a2[i];
}

template <typename R>
__global__ void k_drift(uint32_t n, double* __restrict__ x0, double* __restrict__ x1,
                        double* __restrict__ x2, const R* __restrict__ p0, const R* __restrict__ p1,
                        const R* __restrict__ p2, double D, double L) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    x0[i] = wrap_f64(x0[i] + D * static_cast<double>(p0[i]), L);
    x1[i] = wrap_f64(x1[i] + D * static_cast<double>(p1[i]), L);
    x2[i] = wrap_f64(x2[i] + D * static_cast<double>(p2[i]), L);
}

__global__ void k_axpy3(uint32_t n, double a, const double* __restrict__ x0,
                        const double* __restrict__ x1, const double* __restrict__ x2,
                        double* __restrict__ y0, double* __restrict__ y1, double* __restrict__ y2) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    y0[i] += a * x0[i];
    y1[i] += a * x1[i];
    y2[i] += a * x2[i];
}

template <typename R>
__global__ void k_from_double(uint32_t n, const double* __restrict__ in, R* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = static_cast<R>(in[i]);
}

// delta = M / Mbar - 1; residual field r = (delta - t) * m / Mbar; loss += 1/2 (delta-t)^2
template <typename R>
__global__ void k_loss(uint64_t cells, const R* __restrict__ mesh, const double* __restrict__ target,
                       double inv_mbar, double m_over_mbar, R* __restrict__ field,
                       double* __restrict__ delta_out, double* loss) {
    double local = 0.0;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < cells;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const double delta = static_cast<double>(mesh[i]) * inv_mbar - 1.0;
        if (delta_out) delta_out[i] = delta;
        const double r = target ? delta - target[i] : 0.0;
        local += 0.5 * r * r;
        if (field) field[i] = static_cast<R>(r * m_over_mbar);
    }
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, local);
}

struct Fail {
    int code;
    std::string msg;
};

#define ACK(call)                                                              \
    do {                                                                       \
        cudaError_t e_ = (call);                                               \
        if (e_ != cudaSuccess) throw Fail{e_ == cudaErrorMemoryAllocation ? 7 : 6, \
                                          std::string(#call) + ": " + cudaGetErrorString(e_)}; \
    } while (0)
#define AFFT(call)                                                            \
    do {                                                                      \
        if ((call) != CUFFT_SUCCESS) throw Fail{6, std::string(#call)};       \
    } while (0)

// One device block that a run's work arrays are carved from (256-byte aligned),
// kept between the runs of an engine: some sixty cudaMalloc / cudaFree pairs a
// call took four fifths of a 128^3 gradient's 55 ms.
class Arena {
public:
    template <typename Layout>
    size_t count(Layout&& layout) {   // bytes that layout()'s arrays take
        base_ = nullptr;
        off_ = 0;
        layout();
        return off_;
    }
    template <typename Layout>
    void plan(Layout&& layout) {   // runs layout() twice: to count, then to place
        count(layout);
        if (off_ > cap_) {
            release();
            ACK(cudaMalloc(&block_, off_));
            cap_ = off_;
        }
        base_ = static_cast<char*>(block_);
        off_ = 0;
        layout();
    }
    template <typename T>
    T* take(size_t count) {
        const size_t at = off_;
        off_ += ((count ? count : 1) * sizeof(T) + 255) & ~static_cast<size_t>(255);
        return base_ ? reinterpret_cast<T*>(base_ + at) : nullptr;
    }
    size_t capacity() const { return cap_; }
    // Where the next array goes; reach() makes the layout at least that long.
    size_t offset() const { return off_; }
    void* at(size_t offset) const { return base_ ? base_ + offset : nullptr; }
    void reach(size_t offset) { off_ = off_ > offset ? off_ : (offset + 255) & ~static_cast<size_t>(255); }
    void release() {
        cudaFree(block_);
        block_ = nullptr;
        cap_ = 0;
    }
    Arena() = default;
    Arena(const Arena&) = delete;
    Arena& operator=(const Arena&) = delete;
    ~Arena() { release(); }

private:
    void* block_ = nullptr;
    char* base_ = nullptr;
    size_t cap_ = 0, off_ = 0;
};

struct PlanHandle {
    cufftHandle h = 0;
    bool made = false;
    cufftResult create() {
        const cufftResult r = cufftCreate(&h);
        made = r == CUFFT_SUCCESS;
        return r;
    }
    PlanHandle() = default;
    PlanHandle(const PlanHandle&) = delete;
    PlanHandle& operator=(const PlanHandle&) = delete;
    ~PlanHandle() {
        if (made) cufftDestroy(h);
    }
};

struct Events {
    cudaEvent_t e[3] = {};
    Events() { for (auto& v : e) cudaEventCreate(&v); }
    ~Events() { for (auto& v : e) cudaEventDestroy(v); }
};

template <typename R>
class Engine {
public:
    using C = typename FFTTypes<R>::C;

    Engine(const VjpConfig& cfg, cudaStream_t s) : cfg_(cfg), s_(s) {
        N_ = static_cast<int>(cfg.mesh_size);
        n_ = static_cast<uint32_t>(cfg.n_side * cfg.n_side * cfg.n_side);
        cells_ = static_cast<uint64_t>(N_) * N_ * N_;
        half_ = static_cast<uint64_t>(N_) * N_ * (N_ / 2 + 1);
        axis_.L = cfg.box_size;
        axis_.dx = cfg.box_size / static_cast<double>(N_);
        axis_.upper = std::nextafter(static_cast<double>(N_), 0.0);
        axis_.N = N_;
        inv_two_dx_ = static_cast<R>(1.0 / (2.0 * axis_.dx));
        const double pi = 3.14159265358979323846;
        const double G = 6.67430e-11 * (1e10 * 1.98847e30) / (3.085677581491367e22 * 1000.0 * 1000.0);
        const double dx = axis_.dx;
        // Mass mesh in mass units; A = (4 pi G / dx^3) / N^3 G(k) with the
        // 1/N^3 of the inverse transform folded in (mean removed at k = 0).
        c_green_ = static_cast<R>(4.0 * pi * G / (dx * dx * dx) / static_cast<double>(cells_));
        std::vector<R> lap(N_);
        for (int i = 0; i < N_; ++i) {
            const long long mode = i <= N_ / 2 ? i : static_cast<long long>(i) - N_;
            const double sn = std::sin(pi * static_cast<double>(mode) / N_);
            lap[i] = static_cast<R>(-4.0 / (dx * dx) * sn * sn);
        }
        four_pi_G_ = 4.0 * pi * G;
        scale_ = 1.0 / (dx * dx * dx) / static_cast<double>(cells_);
        five_ = poisson::supported(N_);
        size_t fft_bytes = 0, modes = half_;
        if (five_) {
            modes = sizeof(R) == 8 ? poisson::modes_elements_f64(N_) : poisson::modes_elements_f32(N_);
        } else {
            AFFT(r2c_.create());
            AFFT(c2r_.create());
            cufftSetAutoAllocation(r2c_.h, 0);
            cufftSetAutoAllocation(c2r_.h, 0);
            size_t w1 = 0, w2 = 0;
            AFFT(cufftMakePlan3d(r2c_.h, N_, N_, N_, FFTTypes<R>::R2C, &w1));
            AFFT(cufftMakePlan3d(c2r_.h, N_, N_, N_, FFTTypes<R>::C2R, &w2));
            fft_bytes = w1 > w2 ? w1 : w2;
        }
        char* ws = nullptr;
        fixed_.plan([&] {
            lap_ = fixed_.template take<R>(N_);
            tw_ = fixed_.template take<C>(N_);
            c_green_dev_ = fixed_.template take<R>(1);
            status_ = fixed_.template take<unsigned int>(1);
            ws = fixed_.template take<char>(fft_bytes);
            modes_ = fixed_.template take<C>(modes);
            mesh_ = fixed_.template take<R>(cells_);
            phi_own_ = fixed_.template take<R>(cells_);
            for (int a = 0; a < 3; ++a) {
                x_[a] = fixed_.template take<double>(n_);
                p_[a] = fixed_.template take<R>(n_);
                acc_[a] = fixed_.template take<R>(n_);
            }
        });
        phi_ = phi_own_;
        ACK(cudaMemcpy(lap_, lap.data(), sizeof(R) * N_, cudaMemcpyHostToDevice));
        if (five_) {
            // the production five-pass solve: own transforms with the Green's
            // multiply fused into the x pass (chunked half spectrum)
            const char* perr = nullptr;
            plan_ = poisson::create_plan(N_, sizeof(R) == 4, modes_, &perr);
            if (!plan_) throw Fail{HYOWON_ECUDA, perr ? perr : "five-pass plan"};
            std::vector<double> t(2 * static_cast<size_t>(N_));
            poisson::twiddles(N_, t.data());
            std::vector<C> tc(N_);
            for (int i = 0; i < N_; ++i) {
                tc[i].x = static_cast<R>(t[2 * i]);
                tc[i].y = static_cast<R>(t[2 * i + 1]);
            }
            ACK(cudaMemcpy(tw_, tc.data(), sizeof(C) * N_, cudaMemcpyHostToDevice));
            ACK(cudaMemcpy(c_green_dev_, &c_green_, sizeof(R), cudaMemcpyHostToDevice));
        } else {
            cufftSetWorkArea(r2c_.h, ws);
            cufftSetWorkArea(c2r_.h, ws);
            cufftSetStream(r2c_.h, s_);
            cufftSetStream(c2r_.h, s_);
        }
    }

    // A later call with the same geometry (box, mesh, lattice, form) reuses the
    // engine: its plans and work arrays; the rest of the configuration (P(k)
    // table, schedule, masses, checkpoints) is the call's own.
    bool same_geometry(const VjpConfig& c) const {
        return c.box_size == cfg_.box_size && c.mesh_size == cfg_.mesh_size
            && c.n_side == cfg_.n_side && c.precision == cfg_.precision;
    }
    void set_config(const VjpConfig& c, size_t potential_limit) {
        cfg_ = c;
        potential_limit_ = potential_limit;
    }

    // Gives the work arrays of a run back; the next run takes them again.
    void trim() {
        cudaStreamSynchronize(s_);
        lpt_.release();
        arena_.release();
    }

    ~Engine() {
        poisson::destroy_plan(plan_);
    }

    // acc = F(x); phi_ = potential at x, in the engine's own mesh.
    void force() {
        phi_ = phi_own_;
        ACK(cudaMemsetAsync(mesh_, 0, sizeof(R) * cells_, s_));
        k_deposit<R><<<nb(n_), kT, 0, s_>>>(n_, x_[0], x_[1], x_[2], static_cast<R>(cfg_.particle_mass),
                                            axis_, mesh_, status_);
        apply_green(mesh_, phi_);
        k_force<R><<<nb(n_), kT, 0, s_>>>(n_, x_[0], x_[1], x_[2], phi_, axis_, inv_two_dx_, acc_[0],
                                          acc_[1], acc_[2]);
        ++solves_;
    }

    // out = A in: r2c, Green's function (k = 0 zeroed), c2r with 1/N^3. On
    // power-of-two meshes the production five-pass solve (Green's multiply
    // inside the x pass; A is self-adjoint, so the adjoint uses it as is);
    // elsewhere cuFFT with a separate multiply.
    void apply_green(R* in, R* out) {
        if (five_) {
            int k = 0;
            if constexpr (sizeof(R) == 8) {
                // no mass check here: the source is a mass mesh or a divergence
                const poisson::GreenF64 g{lap_, nullptr, four_pi_G_, scale_, 0, 0.0, INFINITY,
                                          status_};
                k = poisson::forward_f64(plan_, N_, in, modes_, tw_, status_, s_) < 0
                        || poisson::green_f64(plan_, N_, modes_, tw_, g, s_) < 0
                        || poisson::inverse_f64(plan_, N_, modes_, out, tw_, status_, s_) < 0;
            } else {
                const poisson::GreenF32 g{lap_, nullptr, 0, c_green_dev_};
                k = poisson::forward_f32(plan_, N_, in, modes_, tw_, status_, s_) < 0
                        || poisson::green_f32(plan_, N_, modes_, tw_, g, status_, s_) < 0
                        || poisson::inverse_f32(plan_, N_, modes_, out, tw_, status_, s_) < 0;
            }
            if (k) throw Fail{HYOWON_ECUDA, "potential solve launch failed"};
            return;
        }
        AFFT(FFTTypes<R>::fwd(r2c_.h, in, modes_));
        k_green<R, C><<<nb(half_), kT, 0, s_>>>(N_, modes_, lap_, c_green_);
        AFFT(FFTTypes<R>::inv(c2r_.h, modes_, out));
    }

    void kick(double K) {
        k_kick<R><<<nb(n_), kT, 0, s_>>>(n_, p_[0], p_[1], p_[2], acc_[0], acc_[1], acc_[2],
                                         static_cast<R>(K));
    }

    void drift(double D) {
        k_drift<R><<<nb(n_), kT, 0, s_>>>(n_, x_[0], x_[1], x_[2], p_[0], p_[1], p_[2], D, cfg_.box_size);
    }

    // psi = A div(scatter(coef * lp)): the mesh half of VJP_F at x.
    void vjp_mesh(double coef, double* const lp[3], R* const u[3], R* psi) {
        // the three meshes lie one after the other
        ACK(cudaMemsetAsync(u[0], 0, sizeof(R) * static_cast<size_t>(u[2] - u[0] + cells_), s_));
        k_scatter3<R><<<nb(n_), kT, 0, s_>>>(n_, x_[0], x_[1], x_[2], lp[0], lp[1], lp[2], coef, axis_,
                                             u[0], u[1], u[2]);
        const int row_threads = N_ >= kT ? kT : (N_ + 31) / 32 * 32;
        k_divergence<R><<<dim3(N_, N_), row_threads, 0, s_>>>(N_, u[0], u[1], u[2], inv_two_dx_, mesh_);
        apply_green(mesh_, psi);
        ++vjps_;
    }

    // lx += VJP_F(x; coef * lp)
    void vjp(double coef, double* const lx[3], double* const lp[3], R* const u[3], R* psi) {
        vjp_mesh(coef, lp, u, psi);
        k_vjp_gather<R><<<nb(n_), kT, 0, s_>>>(n_, x_[0], x_[1], x_[2], psi,
                                               static_cast<R>(cfg_.particle_mass), phi_, coef, lp[0],
                                               lp[1], lp[2], axis_, inv_two_dx_, lx[0], lx[1], lx[2]);
    }

    void run(const double* noise, const double* target, double* loss_out, double* grad_out,
             double* delta_out, double* timings) {
        const uint64_t S = cfg_.n_steps;
        const uint64_t k = cfg_.ckpt_every > 0 ? cfg_.ckpt_every : 1;
        solves_ = vjps_ = 0;
        Events ev;
        const cudaEvent_t e0 = ev.e[0], e1 = ev.e[1], e2 = ev.e[2];
        ACK(cudaMemsetAsync(status_, 0, sizeof(unsigned int), s_));
        const bool want_grad = grad_out && target;
        const uint64_t n_ckpt = (S + k - 1) / k + 1;
        // Potentials start on 256-byte boundaries, as cuFFT's vector loads need.
        const uint64_t phi_stride = (cells_ + 63) / 64 * 64;
        double *d_noise = nullptr, *tab = nullptr, *d_loss = nullptr, *d_delta = nullptr,
               *d_target = nullptr, *grad = nullptr;
        double *pd[3], *lx[3] = {}, *lp[3] = {};
        R *u[3] = {}, *psi = nullptr, *field = nullptr, *kept_block = nullptr;
        std::vector<double*> cx(3 * n_ckpt);
        std::vector<R*> cp(3 * n_ckpt);
        const char* err = nullptr;
        if (const int rc = lpt_.plan(static_cast<int>(cfg_.n_side), &err))
            throw Fail{rc, err ? err : "LPT failed"};
        void* lpt_at = nullptr;
        bool keep = false;
        auto layout = [&] {
            d_noise = arena_.template take<double>(n_);
            tab = arena_.template take<double>(3 * cfg_.n_nodes);
            for (int a = 0; a < 3; ++a) pd[a] = arena_.template take<double>(n_);
            // The 1LPT map runs before the first checkpoint is written and its adjoint
            // after the last is read: their arrays take the checkpoints' place.
            const size_t first = arena_.offset();
            lpt_at = arena_.at(first);
            for (uint64_t c = 0; c < 3 * n_ckpt; ++c) {
                cx[c] = arena_.template take<double>(n_);
                cp[c] = arena_.template take<R>(n_);
            }
            arena_.reach(first + lpt_.bytes);
            if (want_grad) {
                for (int a = 0; a < 3; ++a) {
                    lx[a] = arena_.template take<double>(n_);
                    lp[a] = arena_.template take<double>(n_);
                }
                for (int a = 0; a < 3; ++a) u[a] = arena_.template take<R>(cells_);
                psi = arena_.template take<R>(cells_);
                grad = arena_.template take<double>(n_);
            }
            d_loss = arena_.template take<double>(1);
            if (delta_out) d_delta = arena_.template take<double>(cells_);
            if (target) d_target = arena_.template take<double>(cells_);
            field = arena_.template take<R>(cells_);
            if (keep) kept_block = arena_.template take<R>((S + 1) * phi_stride);
        };
        // The potential of every forward state (S + 1 meshes) is kept when
        // device memory allows: the reverse pass then re-derives each state's
        // force by one gather instead of a deposit and a Green's-function
        // solve. Particle states stay checkpointed every k steps either way.
        if (want_grad) {
            const size_t rest = arena_.count(layout);
            size_t free_b = 0, total_b = 0;
            const size_t need = (S + 1) * phi_stride * sizeof(R);
            keep = need <= potential_limit_ && cudaMemGetInfo(&free_b, &total_b) == cudaSuccess
                && rest <= free_b + arena_.capacity()
                && need + (size_t(1) << 30) < (free_b + arena_.capacity() - rest) / 2;
        }
        arena_.plan(layout);
        lpt_.place(lpt_at);
        // A block of more than 1/32 of the device's memory is given back.
        struct GiveBack {
            Engine& e;
            ~GiveBack() {
                size_t free_b = 0, total_b = 0;
                e.lpt_.place(nullptr);
                if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess
                    || e.arena_.capacity() > total_b / 32)
                    e.trim();
            }
        } give_back{*this};
        std::vector<R*> kept;
        if (keep)
            for (uint64_t j = 0; j <= S; ++j) kept.push_back(kept_block + j * phi_stride);
        auto keep_of = [&](uint64_t j) { return kept.empty() ? nullptr : kept[j]; };
        auto checkpoint = [&](uint64_t c) {
            Checkpoint<R> k;
            for (int a = 0; a < 3; ++a) {
                k.x[a] = cx[3 * c + a];
                k.p[a] = cp[3 * c + a];
            }
            return k;
        };
        auto restore = [&](uint64_t c) {
            for (int a = 0; a < 3; ++a) {
                ACK(cudaMemcpyAsync(x_[a], cx[3 * c + a], sizeof(double) * n_, cudaMemcpyDeviceToDevice, s_));
                ACK(cudaMemcpyAsync(p_[a], cp[3 * c + a], sizeof(R) * n_, cudaMemcpyDeviceToDevice, s_));
            }
        };
        // ---- 1LPT ---------------------------------------------------------
        ACK(cudaMemcpyAsync(d_noise, noise, sizeof(double) * n_, cudaMemcpyHostToDevice, s_));
        ACK(cudaMemcpyAsync(tab, cfg_.ln_k, sizeof(double) * cfg_.n_nodes, cudaMemcpyHostToDevice, s_));
        ACK(cudaMemcpyAsync(tab + cfg_.n_nodes, cfg_.ln_p, sizeof(double) * cfg_.n_nodes, cudaMemcpyHostToDevice, s_));
        ACK(cudaMemcpyAsync(tab + 2 * cfg_.n_nodes, cfg_.ln_p_y2, sizeof(double) * cfg_.n_nodes, cudaMemcpyHostToDevice, s_));
        if (target)
            ACK(cudaMemcpyAsync(d_target, target, sizeof(double) * cells_, cudaMemcpyHostToDevice, s_));
        const int lrc = lpt_ics_device(lpt_, static_cast<int>(cfg_.n_side), cfg_.box_size, d_noise, tab,
                                       tab + cfg_.n_nodes, tab + 2 * cfg_.n_nodes,
                                       static_cast<int>(cfg_.n_nodes), cfg_.momentum_factor, x_, pd,
                                       status_, s_, &err);
        if (lrc) throw Fail{lrc, err ? err : "LPT failed"};
        for (int a = 0; a < 3; ++a) k_from_double<R><<<nb(n_), kT, 0, s_>>>(n_, pd[a], p_[a]);
        // ---- forward with checkpoints -------------------------------------
        // Timed: the KDK forward from the 1LPT state, the loss, and the reverse
        // KDK pass (the 1LPT map and its adjoint, one FFT set each, are setup).
        cudaEventRecord(e0, s_);
        ACK(cudaMemsetAsync(mesh_, 0, sizeof(R) * cells_, s_));
        k_deposit<R><<<nb(n_), kT, 0, s_>>>(n_, x_[0], x_[1], x_[2], static_cast<R>(cfg_.particle_mass),
                                            axis_, mesh_, status_);
        for (uint64_t j = 0; j <= S; ++j) {
            // potential of state j from its deposit, then the step to state j + 1
            phi_ = keep_of(j) ? keep_of(j) : phi_own_;
            apply_green(mesh_, phi_);
            ++solves_;
            if (j < S) ACK(cudaMemsetAsync(mesh_, 0, sizeof(R) * cells_, s_));
            k_advance<R><<<nb(n_), kT, 0, s_>>>(
                n_, x_[0], x_[1], x_[2], p_[0], p_[1], p_[2], phi_, axis_, inv_two_dx_,
                static_cast<R>(j > 0 ? cfg_.K2[j - 1] : 0.0),
                j % k == 0 && j < S ? checkpoint(j / k) : Checkpoint<R>{}, j < S ? 1 : 0,
                static_cast<R>(j < S ? cfg_.K1[j] : 0.0), j < S ? cfg_.D[j] : 0.0,
                static_cast<R>(cfg_.particle_mass), mesh_, acc_[0], acc_[1], acc_[2], status_);
        }
        // ---- loss on the final CIC density ----------------------------------
        const double mbar = cfg_.particle_mass * static_cast<double>(n_) / static_cast<double>(cells_);
        ACK(cudaMemsetAsync(d_loss, 0, sizeof(double), s_));
        // mesh_ still holds the deposit of the last state: the solve reads it only
        k_loss<R><<<1184, kT, 0, s_>>>(cells_, mesh_, d_target, 1.0 / mbar, cfg_.particle_mass / mbar,
                                       field, d_delta, d_loss);
        ACK(cudaMemcpyAsync(loss_out, d_loss, sizeof(double), cudaMemcpyDeviceToHost, s_));
        if (delta_out)
            ACK(cudaMemcpyAsync(delta_out, d_delta, sizeof(double) * cells_, cudaMemcpyDeviceToHost, s_));
        cudaEventRecord(e1, s_);
        if (want_grad) {
            // ---- reverse leapfrog ---------------------------------------------
            for (int a = 0; a < 3; ++a) {
                ACK(cudaMemsetAsync(lx[a], 0, sizeof(double) * n_, s_));
                ACK(cudaMemsetAsync(lp[a], 0, sizeof(double) * n_, s_));
            }
            // dL/dx_S: deposit transpose with the weight derivative.
            k_vjp_gather<R><<<nb(n_), kT, 0, s_>>>(n_, x_[0], x_[1], x_[2], field, R(1), nullptr, 0.0,
                                                   nullptr, nullptr, nullptr, axis_, inv_two_dx_,
                                                   lx[0], lx[1], lx[2]);
            for (uint64_t jj = S; jj-- > 0;) {
                const double coef = cfg_.K2[jj] + (jj + 1 < S ? cfg_.K1[jj + 1] : 0.0);
                if (!kept.empty()) {
                    vjp_mesh(coef, lp, u, psi);   // at x_{jj+1}
                    k_reverse<R><<<nb(n_), kT, 0, s_>>>(
                        n_, x_[0], x_[1], x_[2], p_[0], p_[1], p_[2], acc_[0], acc_[1], acc_[2], psi,
                        static_cast<R>(cfg_.particle_mass), kept[jj + 1], kept[jj], coef, cfg_.D[jj],
                        static_cast<R>(cfg_.K1[jj]), static_cast<R>(cfg_.K2[jj]),
                        jj % k == 0 ? checkpoint(jj / k) : Checkpoint<R>{}, axis_, inv_two_dx_, lx[0],
                        lx[1], lx[2], lp[0], lp[1], lp[2]);
                    phi_ = kept[jj];
                    continue;
                }
                vjp(coef, lx, lp, u, psi);  // at x_{jj+1} with phi_{jj+1}
                // lp += D lx; reconstruct state jj: p' = p_{jj+1} - K2 a_{jj+1}
                k_axpy3_kick<R><<<nb(n_), kT, 0, s_>>>(n_, cfg_.D[jj], lx[0], lx[1], lx[2], lp[0],
                                                       lp[1], lp[2], p_[0], p_[1], p_[2], acc_[0],
                                                       acc_[1], acc_[2], static_cast<R>(-cfg_.K2[jj]));
                if (jj % k == 0) {
                    restore(jj / k);
                    force();
                } else {
                    drift(-cfg_.D[jj]);
                    force();
                    kick(-cfg_.K1[jj]);
                }
            }
            vjp(cfg_.K1[0], lx, lp, u, psi);  // at x_0
            cudaEventRecord(e2, s_);
            // ---- 1LPT adjoint: g_d = lx_d + pf lp_d -----------------------------
            k_axpy3<<<nb(n_), kT, 0, s_>>>(n_, cfg_.momentum_factor, lp[0], lp[1], lp[2], lx[0],
                                           lx[1], lx[2]);
            const int arc = lpt_adjoint_device(lpt_, static_cast<int>(cfg_.n_side), cfg_.box_size, lx, tab,
                                               tab + cfg_.n_nodes, tab + 2 * cfg_.n_nodes,
                                               static_cast<int>(cfg_.n_nodes), grad, s_, &err);
            if (arc) throw Fail{arc, err ? err : "LPT adjoint failed"};
            ACK(cudaMemcpyAsync(grad_out, grad, sizeof(double) * n_, cudaMemcpyDeviceToHost, s_));
        } else {
            cudaEventRecord(e2, s_);
        }
        ACK(cudaStreamSynchronize(s_));
        unsigned int st = 0;
        ACK(cudaMemcpy(&st, status_, sizeof(unsigned int), cudaMemcpyDeviceToHost));
        if (timings) {
            float t1 = 0.f, t2 = 0.f;
            cudaEventElapsedTime(&t1, e0, e1);
            cudaEventElapsedTime(&t2, e1, e2);
            timings[0] = t1;
            timings[1] = t2;
            timings[2] = static_cast<double>(solves_);
            timings[3] = static_cast<double>(vjps_);
        }
        if (st) throw Fail{HYOWON_ELOGIC, "a position left the mesh domain"};
    }

private:
    VjpConfig cfg_;
    cudaStream_t s_;
    int N_ = 0;
    uint32_t n_ = 0;
    uint64_t cells_ = 0, half_ = 0;
    Axis axis_{};
    R inv_two_dx_ = 0, c_green_ = 0;
    R* lap_ = nullptr;
    PlanHandle r2c_, c2r_;
    bool five_ = false;               // power-of-two mesh: five-pass solve
    poisson::Plan* plan_ = nullptr;
    C* tw_ = nullptr;
    R* c_green_dev_ = nullptr;
    double four_pi_G_ = 0.0, scale_ = 0.0;
    R* mesh_ = nullptr;
    R* phi_own_ = nullptr;
    R* phi_ = nullptr;
    C* modes_ = nullptr;
    unsigned int* status_ = nullptr;
    double* x_[3] = {};
    R* p_[3] = {};
    R* acc_[3] = {};
    uint64_t solves_ = 0, vjps_ = 0;
    size_t potential_limit_ = SIZE_MAX;
    Arena fixed_;       // what the engine keeps: meshes, spectrum, particle state
    Arena arena_;       // a run's work arrays
    LptWork lpt_;
};

thread_local std::string g_adj_err;

}  // namespace

// Engines kept by a PM handle between its VJP calls.
struct Cache {
    Engine<double>* e64 = nullptr;
    Engine<float>* e32 = nullptr;
    size_t potential_limit = SIZE_MAX;
    ~Cache() {
        delete e64;
        delete e32;
    }
};

void destroy_cache(Cache* c) { delete c; }

void trim_cache(Cache* c) {
    if (!c) return;
    if (c->e64) c->e64->trim();
    if (c->e32) c->e32->trim();
}

int limit_potentials(Cache** c, size_t bytes) {
    if (!*c) *c = new (std::nothrow) Cache();
    if (!*c) return HYOWON_ENOMEM;
    (*c)->potential_limit = bytes;
    return HYOWON_OK;
}

int run_cached(Cache** cache, const VjpConfig& cfg, cudaStream_t s, const double* noise,
               const double* target_delta, double* loss, double* grad_noise,
               double* final_delta, double* timings, std::string* err) {
    try {
        if (!*cache) *cache = new Cache();
        Cache* c = *cache;
        if (cfg.precision == HYOWON_FP64) {
            if (c->e64 && !c->e64->same_geometry(cfg)) {
                delete c->e64;
                c->e64 = nullptr;
            }
            if (!c->e64) c->e64 = new Engine<double>(cfg, s);
            c->e64->set_config(cfg, c->potential_limit);
            c->e64->run(noise, target_delta, loss, grad_noise, final_delta, timings);
        } else {
            if (c->e32 && !c->e32->same_geometry(cfg)) {
                delete c->e32;
                c->e32 = nullptr;
            }
            if (!c->e32) c->e32 = new Engine<float>(cfg, s);
            c->e32->set_config(cfg, c->potential_limit);
            c->e32->run(noise, target_delta, loss, grad_noise, final_delta, timings);
        }
    } catch (const Fail& f) {
        if (err) *err = f.msg;
        return f.code;
    } catch (const std::exception& e) {   // bad_alloc, length_error
        if (err) *err = std::string("out of host memory: ") + e.what();
        return HYOWON_ENOMEM;
    }
    return HYOWON_OK;
}

}  // namespace hyowon::adj

extern "C" {

const char* hyowon_vjp_last_error(void) { return hyowon::adj::g_adj_err.c_str(); }

int hyowon_vjp_1lpt_pm(const hyowon_vjp_config* cfg, const double* noise,
                       const double* target_delta, double* loss, double* grad_noise,
                       double* final_delta, double* timings) {
    using namespace hyowon::adj;
    g_adj_err.clear();
    if (!cfg || !noise || !loss) {
        g_adj_err = "config, noise and loss must be non-null";
        return HYOWON_EINVAL;
    }
    if (cfg->n_side < 2 || cfg->mesh_size < 2 || cfg->n_steps < 1 || !cfg->K1 || !cfg->D || !cfg->K2
        || cfg->n_nodes < 2 || !cfg->ln_k || !cfg->ln_p || !cfg->ln_p_y2
        || !(cfg->particle_mass > 0.0) || !(cfg->box_size > 0.0)
        || (cfg->precision != HYOWON_FP64 && cfg->precision != HYOWON_FP32_FIXED)) {
        g_adj_err = "invalid VJP configuration";
        return HYOWON_EINVAL;
    }
    if (grad_noise && !target_delta) {
        g_adj_err = "the gradient needs a target density";
        return HYOWON_EINVAL;
    }
    cudaStream_t s = nullptr;
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) {
        g_adj_err = "stream creation failed";
        return HYOWON_ECUDA;
    }
    int rc = HYOWON_OK;
    try {
        if (cfg->precision == HYOWON_FP64) {
            Engine<double> e(*cfg, s);
            e.run(noise, target_delta, loss, grad_noise, final_delta, timings);
        } else {
            Engine<float> e(*cfg, s);
            e.run(noise, target_delta, loss, grad_noise, final_delta, timings);
        }
    } catch (const Fail& f) {
        g_adj_err = f.msg;
        rc = f.code;
    } catch (const std::exception& e) {   // bad_alloc, length_error
        g_adj_err = std::string("out of host memory: ") + e.what();
        rc = HYOWON_ENOMEM;
    }
    cudaStreamDestroy(s);
    return rc;
}

}  // extern "C"
