// pm_tree.cu -- TreePM short-range force: Hilbert-ordered octree + warp-cooperative
// walk (include/hyowon_treepm.h).
//
// Build:
//   1. 63-bit Hilbert index per source (21 bits per axis). Its leading 3 l bits are
//      those of the level-l octree cell, so a cell's sources are consecutive, as
//      they are in the reference's octant order (src/gravity/octree.cpp:336-357),
//      and neighbours along the curve share a face at every level: a group of
//      consecutive targets has a box a fifth smaller per side than in Morton order;
//   2. stable LSD radix sort of (key, index), 8 passes of 8 bits;
//   3. node extraction in one sweep: a node at level l is a maximal run of equal
//      key >> 3(21-l) whose parent run holds >= 2 sources; runs holding one
//      source (or level 21) are leaves, so every leaf holds one source unless
//      sources coincide at 2^-21 L. The levels at which source i starts a node
//      follow from the digits it shares with its two neighbours alone; per-tile
//      level counts and one scan number the nodes level by level;
//   4. node mass and COM from exact 64-bit prefix sums of 2^-40 L fixed-point
//      coordinates (no summation-order error).
// Walk: one warp per group of G targets (G of 1, 4, 8 or 16, neighbours in key
// order). The 32 lanes classify 32 nodes at a time against the group's bounding
// box: dropped for every target, opened for every target, a monopole for every
// target, or undecided, in which case each target decides for itself in
// binary64. Sources and accepted monopoles collect in a shared-memory list that
// every target then filters by distance and sums. Each target's set of exact
// pairs and monopoles is the one of the reference's per-target walk. Stack depth
// and iterations are bounded; overflow is an error status, never an unbounded
// loop.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <exception>
#include <limits>
#include <new>
#include <string>
#include <utility>
#include <vector>

#include "hyowon_pm.h"
#include "hyowon_treepm.h"
#include "pm_common.cuh"
#include "pm_kernels.h"
#include "pm_tree.h"

namespace hyowon::tree {

namespace {

constexpr int kT = 256;
constexpr int kBits = 21;
// Per-warp stack of unopened child runs. Above kStackWide entries one run is
// popped at a time, so the stack stays within kStackWide + 31 + 7 * 21 + 8 entries.
constexpr int kStack = 320;
constexpr int kStackWide = 128;
constexpr unsigned kMaxIter = 1u << 24;

inline unsigned nb(uint64_t n, int t = kT) { return static_cast<unsigned>((n + t - 1) / t); }

struct Node {
    double cx, cy, cz, half;       // geometric cube
    double mx, my, mz, mass;       // centre of mass, mass
    unsigned long long prefix;     // key >> 3(21-level)
    uint32_t start, end;           // sorted source range
    uint32_t first_child, n_child; // children in the node array
    uint32_t level, leaf;
    double open2;                  // (2 half / theta + |COM - centre|_1)^2, set after the build
};

__device__ __forceinline__ unsigned long long spread3(unsigned v) {
    unsigned long long x = v & 0x1fffffu;
    x = (x | (x << 32)) & 0x1f00000000ffffull;
    x = (x | (x << 16)) & 0x1f0000ff0000ffull;
    x = (x | (x << 8)) & 0x100f00f00f00f00full;
    x = (x | (x << 4)) & 0x10c30c30c30c30c3ull;
    x = (x | (x << 2)) & 0x1249249249249249ull;
    return x;
}

__device__ __forceinline__ unsigned quant(double w, double L) {
    double t = floor(w / L * 2097152.0);
    t = t < 0.0 ? 0.0 : (t > 2097151.0 ? 2097151.0 : t);
    return static_cast<unsigned>(t);
}

// Hilbert index of a cell of the 2^21 lattice, by the bitwise transform of
// J. Skilling, "Programming the Hilbert curve", AIP Conf. Proc. 707, 381 (2004): the
// axes' bits are exchanged or inverted below each set or cleared bit from the top
// down, then Gray-coded; bit triples read in order give the index.
__device__ __forceinline__ unsigned long long hilbert_key(unsigned x, unsigned y, unsigned z) {
#pragma unroll 1
    for (unsigned q = 1u << (kBits - 1); q > 1u; q >>= 1) {
        const unsigned low = q - 1u;
        if (x & q) x ^= low;
        unsigned t = (x ^ y) & low;
        if (y & q) {
            x ^= low;
        } else {
            x ^= t;
            y ^= t;
        }
        t = (x ^ z) & low;
        if (z & q) {
            x ^= low;
        } else {
            x ^= t;
            z ^= t;
        }
    }
    y ^= x;
    z ^= y;
    unsigned t = 0;
#pragma unroll 1
    for (unsigned q = 1u << (kBits - 1); q > 1u; q >>= 1)
        if (z & q) t ^= q - 1u;
    return (spread3(x ^ t) << 2) | (spread3(y ^ t) << 1) | spread3(z ^ t);
}

__global__ void k_keys(uint32_t n, const double* __restrict__ x, const double* __restrict__ y,
                       const double* __restrict__ z, double L, double* __restrict__ wx,
                       double* __restrict__ wy, double* __restrict__ wz,
                       unsigned long long* __restrict__ key, uint32_t* __restrict__ val,
                       unsigned int* status) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a = wrap_f64(x[i], L), b = wrap_f64(y[i], L), c = wrap_f64(z[i], L);
    if (!(a >= 0.0 && a < L && b >= 0.0 && b < L && c >= 0.0 && c < L)) {
        raise_status(status, ST_NONFINITE_INPUT);
    }
    wx[i] = a;
    wy[i] = b;
    wz[i] = c;
    key[i] = hilbert_key(quant(a, L), quant(b, L), quant(c, L));
    val[i] = i;
}

// ---- stable LSD radix sort, 8-bit digits --------------------------------
constexpr int kTile = 4096;  // keys per tile (256 threads x 16 rounds)

__global__ void k_tile_hist(uint32_t n, const unsigned long long* __restrict__ key, int shift,
                            uint32_t n_tiles, uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kTile;
    for (int r = 0; r < kTile / kT; ++r) {
        const uint64_t i = base + r * kT + threadIdx.x;
        if (i < n) atomicAdd(&h[(key[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[static_cast<uint64_t>(threadIdx.x) * n_tiles + blockIdx.x] = h[threadIdx.x];
}

__global__ void k_tile_scatter(uint32_t n, const unsigned long long* __restrict__ key,
                               const uint32_t* __restrict__ val, int shift, uint32_t n_tiles,
                               const uint32_t* __restrict__ offs,
                               unsigned long long* __restrict__ key_out,
                               uint32_t* __restrict__ val_out) {
    __shared__ uint32_t run[256];        // keys of each digit already placed by this tile
    __shared__ uint32_t wcount[8][256];  // per-warp digit counts of the current round
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    run[threadIdx.x] = offs[static_cast<uint64_t>(threadIdx.x) * n_tiles + blockIdx.x];
    const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kTile;
    for (int r = 0; r < kTile / kT; ++r) {
        for (int w = 0; w < 8; ++w) wcount[w][threadIdx.x] = 0;
        __syncthreads();
        const uint64_t i = base + r * kT + threadIdx.x;
        const bool ok = i < n;
        const unsigned long long k = ok ? key[i] : 0ull;
        const unsigned d = ok ? static_cast<unsigned>((k >> shift) & 255u) : 256u;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const unsigned rank = __popc(peers & ((1u << lane) - 1u));
        if (ok && rank == 0) wcount[warp][d] = __popc(peers);
        __syncthreads();
        if (ok) {
            uint32_t before = run[d] + rank;
            for (int w = 0; w < warp; ++w) before += wcount[w][d];
            key_out[before] = k;
            val_out[before] = val[i];
        }
        __syncthreads();
        uint32_t tot = 0;
        for (int w = 0; w < 8; ++w) tot += wcount[w][threadIdx.x];
        run[threadIdx.x] += tot;
        __syncthreads();
    }
}

// ---- 64-bit exclusive scan (fixed-point COM prefix sums) ------------------
__global__ void k_scan64_block(const unsigned long long* __restrict__ in,
                               unsigned long long* __restrict__ out, uint64_t n,
                               unsigned long long* __restrict__ sums) {
    __shared__ unsigned long long wt[32];
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * 1024 + threadIdx.x;
    const unsigned long long v = i < n ? in[i] : 0ull;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) wt[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        unsigned long long w = wt[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        wt[lane] = w;
    }
    __syncthreads();
    const unsigned long long ex = inc - v + (warp ? wt[warp - 1] : 0ull);
    if (i < n) out[i] = ex;
    if (threadIdx.x == 1023 && sums) sums[blockIdx.x] = ex + v;
}

__global__ void k_scan64_add(unsigned long long* __restrict__ out, uint64_t n,
                             const unsigned long long* __restrict__ add) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) out[i] += add[i / 1024];
}

// ---- node extraction -------------------------------------------------------
__global__ void k_gather_sorted(uint32_t n, const uint32_t* __restrict__ val,
                                const double* __restrict__ wx, const double* __restrict__ wy,
                                const double* __restrict__ wz, double L, double* __restrict__ sx,
                                double* __restrict__ sy, double* __restrict__ sz,
                                unsigned long long* __restrict__ qx, unsigned long long* __restrict__ qy,
                                unsigned long long* __restrict__ qz, uint32_t* __restrict__ inv) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > n) return;
    if (i == n) {  // sentinel for the inclusive end of the prefix sums
        qx[n] = qy[n] = qz[n] = 0ull;
        return;
    }
    const uint32_t j = val[i];
    sx[i] = wx[j];
    sy[i] = wy[j];
    sz[i] = wz[j];
    const double s = 1099511627776.0 / L;  // 2^40 / L
    qx[i] = static_cast<unsigned long long>(llrint(wx[j] * s));
    qy[i] = static_cast<unsigned long long>(llrint(wy[j] * s));
    qz[i] = static_cast<unsigned long long>(llrint(wz[j] * s));
    inv[j] = i;
}

__global__ void k_target_slots(uint32_t nt, const uint32_t* __restrict__ targets,
                               const uint32_t* __restrict__ inv, uint32_t* __restrict__ at) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nt) at[i] = inv[targets[i]];
}

// Octal digits that keys a and b share from the top: their level-l cells are equal
// for l up to it (21: equal keys).
__device__ __forceinline__ int shared_digits(unsigned long long a, unsigned long long b) {
    const unsigned long long x = a ^ b;
    return x == 0 ? kBits : kBits - 1 - (63 - __clzll(x)) / 3;
}

// Levels at which source i starts a node: from the first digit it does not share
// with source i-1 to one past the last it shares with either neighbour (the cell
// above then holds two sources), empty for a repeated key.
__device__ __forceinline__ void node_levels(uint32_t i, uint32_t n,
                                            const unsigned long long* __restrict__ key, int& lo,
                                            int& hi, int& next) {
    const unsigned long long k = key[i];
    const int prev = i > 0 ? shared_digits(key[i - 1], k) : -1;
    next = i + 1 < n ? shared_digits(k, key[i + 1]) : -1;
    lo = prev + 1;
    const int m = prev > next ? prev : next;
    hi = m + 1 < kBits ? m + 1 : kBits;
}

constexpr int kLevels = kBits + 1;

// Nodes of each level that the sources of one tile (a block of kT) start.
__global__ void __launch_bounds__(kT)
k_level_counts(uint32_t n, const unsigned long long* __restrict__ key, uint32_t n_tiles,
               uint32_t* __restrict__ hist) {
    __shared__ uint32_t count[kLevels];
    if (threadIdx.x < kLevels) count[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t i = blockIdx.x * kT + threadIdx.x;
    int lo = 1, hi = 0, next;
    if (i < n) node_levels(i, n, key, lo, hi, next);
    for (int l = __reduce_min_sync(0xffffffffu, lo), top = __reduce_max_sync(0xffffffffu, hi);
         l <= top; ++l) {
        const unsigned m = __ballot_sync(0xffffffffu, l >= lo && l <= hi);
        if ((threadIdx.x & 31) == 0 && m) atomicAdd(&count[l], static_cast<uint32_t>(__popc(m)));
    }
    __syncthreads();
    if (threadIdx.x < kLevels)
        hist[static_cast<uint64_t>(threadIdx.x) * n_tiles + blockIdx.x] = count[threadIdx.x];
    if (blockIdx.x == 0 && threadIdx.x == 0) hist[static_cast<uint64_t>(kLevels) * n_tiles] = 0;
}

// End of the level's run that source i belongs to, searched from `from` (a source
// of that run): doubling steps, then bisection.
__device__ __forceinline__ uint32_t run_end(uint32_t n, const unsigned long long* __restrict__ key,
                                            unsigned long long prefix, int shift, uint32_t from) {
    uint32_t in = from, step = 1;
    while (in + step < n && (key[in + step] >> shift) == prefix) {
        in += step;
        step <<= 1;
    }
    uint32_t out = n - in > step ? in + step : n;   // first source known to lie outside
    while (out - in > 1) {
        const uint32_t mid = in + (out - in) / 2;
        if ((key[mid] >> shift) == prefix) in = mid;
        else out = mid;
    }
    return out;
}

// The nodes that the sources of one tile start, numbered level by level and, within
// a level, in source order (offs: the scanned counts). Deepest level first, so
// that a node's first child, which starts at the same source, is already
// numbered. Replaces a level-by-level build of 22 sweeps over the sources with two
// host reads each; the whole build, keys and
// sort with it, took 2.1 -> 0.42 ms for 30,000 sources, 4.1 -> 1.6 for 2.1M with masses
// and 18.4 -> 9.1 for 16.8M.
__global__ void __launch_bounds__(kT)
k_emit_nodes(uint32_t n, const unsigned long long* __restrict__ key, uint32_t n_tiles,
             const uint32_t* __restrict__ offs, double L, const double* __restrict__ sx,
             const double* __restrict__ sy, const double* __restrict__ sz,
             const unsigned long long* __restrict__ qx, const unsigned long long* __restrict__ qy,
             const unsigned long long* __restrict__ qz, double m, Node* __restrict__ nodes) {
    __shared__ uint32_t base[kT / 32][kLevels];   // first number of each warp's nodes
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t i = blockIdx.x * kT + threadIdx.x;
    int lo = 1, hi = 0, next = -1;
    if (i < n) node_levels(i, n, key, lo, hi, next);
    const int first = __reduce_min_sync(0xffffffffu, lo);
    const int last = __reduce_max_sync(0xffffffffu, hi);
    if (lane < kLevels) base[warp][lane] = 0;
    __syncwarp();
    for (int l = first; l <= last; ++l) {
        const unsigned b = __ballot_sync(0xffffffffu, l >= lo && l <= hi);
        if (lane == 0) base[warp][l] = __popc(b);
    }
    __syncthreads();
    if (threadIdx.x < kLevels) {
        uint32_t at = offs[static_cast<uint64_t>(threadIdx.x) * n_tiles + blockIdx.x];
        for (int w = 0; w < kT / 32; ++w) {
            const uint32_t c = base[w][threadIdx.x];
            base[w][threadIdx.x] = at;
            at += c;
        }
    }
    __syncthreads();
    const unsigned long long k = i < n ? key[i] : 0ull;
    const unsigned ux = i < n ? quant(sx[i], L) : 0u, uy = i < n ? quant(sy[i], L) : 0u,
                   uz = i < n ? quant(sz[i], L) : 0u;
    uint32_t child = 0xffffffffu, end = i + 1;
    for (int l = last; l >= first; --l) {
        const bool mine = l >= lo && l <= hi;
        const unsigned b = __ballot_sync(0xffffffffu, mine);
        if (!mine) continue;
        const uint32_t idx = base[warp][l] + __popc(b & ((1u << lane) - 1u));
        const int shift = 3 * (kBits - l);
        Node nd;
        nd.prefix = k >> shift;
        if (l <= next) end = run_end(n, key, nd.prefix, shift, end - 1);
        const uint32_t cnt = end - i;
        nd.leaf = (cnt == 1 || l == kBits) ? 1u : 0u;
        // cube: the level-l cell of the source's lattice coordinates
        const unsigned cxi = ux >> (kBits - l), cyi = uy >> (kBits - l), czi = uz >> (kBits - l);
        const double side = L / static_cast<double>(1ull << l);
        nd.half = 0.5 * side;
        nd.cx = (cxi + 0.5) * side;
        nd.cy = (cyi + 0.5) * side;
        nd.cz = (czi + 0.5) * side;
        const double inv = 1.0 / (static_cast<double>(cnt) * (1099511627776.0 / L));
        nd.mx = static_cast<double>(qx[end] - qx[i]) * inv;
        nd.my = static_cast<double>(qy[end] - qy[i]) * inv;
        nd.mz = static_cast<double>(qz[end] - qz[i]) * inv;
        nd.mass = m * cnt;
        nd.start = i;
        nd.end = end;
        nd.level = l;
        nd.first_child = 0xffffffffu;
        nd.n_child = 0;
        nd.open2 = 0.0;
        if (!nd.leaf) {
            nd.first_child = child;
            const int below = shift - 3;
            uint32_t kids = 0;
            if (cnt <= 16) {
                unsigned long long was = ~0ull;
                for (uint32_t j = i; j < end; ++j) {
                    const unsigned long long p = key[j] >> below;
                    kids += p != was ? 1u : 0u;
                    was = p;
                }
            } else {
                for (uint32_t j = i; j < end; ++kids) j = run_end(end, key, key[j] >> below, below, j);
            }
            nd.n_child = kids;
        }
        nodes[idx] = nd;
        child = idx;
    }
}

// ---- pair force -----------------------------------------------------------
// (r^2+eps^2)^(-3/2) - (1 - M_S(q)) / r^3 with M_S = erfc(q/2) + q/sqrt(pi) e^{-q^2/4}.
// For q < 0.05 the long-range part uses its series
//   (1 - M_S(q)) / r^3 = (1/sqrt(pi)) (1/6 - q^2/40 + q^4/448 - q^6/6912 + ...) / r_s^3
// (1 - M_S cancels there); otherwise (r^2+eps^2)^(-3/2) - 1/r^3 is formed as
// expm1(-1.5 log1p(eps^2/r^2)) / r^3 so no large terms cancel.
template <typename R>
__device__ __forceinline__ R short_factor_impl(R r2, R eps2, R inv_rs, R inv_rs3) {
    const R r = sqrt(r2);
    const R q = r * inv_rs;
    const R isp = R(0.5641895835477563);
    if (q < R(0.05)) {
        const R q2 = q * q;
        const R longf = isp * (R(1.0 / 6.0) + q2 * (R(-1.0 / 40.0)
                                                    + q2 * (R(1.0 / 448.0) - q2 * R(1.0 / 6912.0))))
            * inv_rs3;
        const R s = r2 + eps2;
        return R(1) / (s * sqrt(s)) - longf;
    }
    const R ms = erfc(R(0.5) * q) + q * isp * exp(R(-0.25) * q * q);
    const R ir = R(1) / r;
    return (expm1(R(-1.5) * log1p(eps2 / r2)) + ms) * ir * ir * ir;
}

__device__ __forceinline__ double min_image(double d, double L) {
    const double h = 0.5 * L;
    if (d >= h) d -= L;
    else if (d < -h) d += L;
    return d;
}

struct WalkParams {
    double L, r_cut, eps, r_s, G, m;
};

constexpr unsigned kCounters = 64;   // pairs of walk statistics counters

// Box coordinates as 32-bit fractions of L: differences wrap like the box does,
// so the signed difference is the minimum image.
__device__ __forceinline__ uint32_t box_fraction(double v, double L) {
    return __double2uint_rz(v * (4294967296.0 / L));   // saturates
}

// What the group tests of the walk read of a node, once after the build, in
// three 16-byte arrays that the lanes of a warp read as short runs (the children
// of a node are consecutive):
//   ga  cube centre and half side, in 2^-32 L (both exact)
//   gm  centre of mass in 2^-32 L, and the square of the opening distance in
//       the same unit (float bits)
//   gc  first child, children | leaf << 8, source range start and count
// The monopole criterion's target-independent side is open2: a node is accepted
// when its COM distance squared exceeds (2 half / theta + off)^2 with off the L1
// offset of the COM from the cube centre.
__global__ void k_walk_nodes(uint32_t n_nodes, double theta, double L, Node* __restrict__ nodes,
                             uint4* __restrict__ ga, uint4* __restrict__ gm,
                             uint4* __restrict__ gc) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_nodes) return;
    Node& nd = nodes[i];
    const double off = fabs(nd.mx - nd.cx) + fabs(nd.my - nd.cy) + fabs(nd.mz - nd.cz);
    const double need = 2.0 * nd.half / theta + off;
    nd.open2 = need * need;
    const double unit = 4294967296.0 / L;
    const float need_u = static_cast<float>(need * unit);
    ga[i] = make_uint4(box_fraction(nd.cx, L), box_fraction(nd.cy, L), box_fraction(nd.cz, L),
                       0x80000000u >> nd.level);
    gm[i] = make_uint4(box_fraction(nd.mx, L), box_fraction(nd.my, L), box_fraction(nd.mz, L),
                       __float_as_uint(need_u * need_u));
    gc[i] = make_uint4(nd.first_child, nd.n_child | (nd.leaf << 8), nd.start, nd.end - nd.start);
}

// The pair factor as A^3 F(u), A = (r^2 + eps^2)^(-1/2), u = 1/A, with
//   F(u) = 1 - u^3 h(u^2 - eps^2),
// h the long-range part (1 - M_S(q)) / r^3, an entire function of r^2: F is entire in
// u, softening included, and one polynomial in v = b - k u serves the whole cutoff
// sphere (v = 0 at the cutoff, 2 at r = 0; fit_poly, below): no branch, no error
// function, no exponential. F falls to M_S(4.5) = 0.0175 and further, so a
// polynomial for h, and A^3 - h formed from it, loses the outer pairs (5e-14 of them at
// 4.5 r_s, 5e-12 at 6). Here the first two coefficients are those of the expansion
// about the cutoff, where F is smallest, and the rest of the sum carries a factor v^2
// there; u enters with its rounding error (amplified 9 times by F at 4.5 r_s)
// restored. One rsqrt and DEG + 13 multiply-adds replace the erfc, exp, expm1,
// log1p, sqrt and division of short_factor_impl, which remains for cutoffs of so
// many r_s, or softenings so large, that no polynomial of these degrees reaches its
// accuracy (DEG = 0). Largest error of F over the sphere at 4.5 r_s: 1.0e-15 in
// binary64 (the closed form 7e-16), 2.8e-8 in the precision form (FP32 closed form
// 1.2e-6).
//
// The precision form takes A^3 - h, h of degree kDegFp32 in r^2, while that stays within
// half an FP32 rounding of the factor (up to 4.5 r_s): seven operations fewer, 5% of a
// walk of 16.8M sources.
constexpr int kDegFp32 = 12, kDegLow = 22, kDegMid = 28, kDegHigh = 36;
struct PairPoly {
    double k, half_k, b;        // v = b - k u; degree kDegFp32: tau = k r^2 - 1
    double c[kDegHigh + 1];     // c[0] + v (c[1] + v S(1 - v)), S's monomials from c[2];
                                // degree kDegFp32: h's monomials in tau
};

// h at r^2.
__host__ __device__ __forceinline__ double long_part(double r2, const PairPoly& pp) {
    const double tau = fma(r2, pp.k, -1.0);
    const double t2 = tau * tau;
    double even = pp.c[kDegFp32], odd = pp.c[kDegFp32 - 1];
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int k = kDegFp32 - 2; k >= 0; k -= 2) {
        even = fma(even, t2, pp.c[k]);
        if (k > 0) odd = fma(odd, t2, pp.c[k - 1]);
    }
    return fma(odd, tau, even);
}

// F at u = s a, s = r^2 + eps^2 and a its reciprocal square root.
template <int DEG, bool EXACT_U>
__host__ __device__ __forceinline__ double pair_poly(double s, double a, const PairPoly& pp) {
    const double u = s * a;
    double v = fma(-u, pp.k, pp.b);
    if constexpr (EXACT_U) v = fma(-pp.half_k * a, fma(-u, u, s), v);
    const double tau = 1.0 - v;
    const double t2 = tau * tau;
    double even = pp.c[DEG], odd = pp.c[DEG - 1];   // DEG is even
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int k = DEG - 2; k >= 2; k -= 2) {
        even = fma(even, t2, pp.c[k]);
        if (k > 2) odd = fma(odd, t2, pp.c[k - 1]);
    }
    return fma(fma(fma(odd, tau, even), v, pp.c[1]), v, pp.c[0]);
}

template <typename R, int DEG>
__device__ __forceinline__ double pair_factor(double r2, double eps2, double inv_rs,
                                              const PairPoly& pp) {
    if constexpr (DEG == 0) {
        const R irs = static_cast<R>(inv_rs);
        return static_cast<double>(short_factor_impl<R>(static_cast<R>(r2), static_cast<R>(eps2),
                                                        irs, irs * irs * irs));
    } else {
        const double s = r2 + eps2;
        double a;
        if constexpr (sizeof(R) == 8) {
            a = rsqrt(s);
        } else {
            // the FP32 reciprocal square root and one Newton step: 2e-14
            a = static_cast<double>(rsqrtf(static_cast<float>(s)));
            a = a * (1.5 - 0.5 * s * a * a);
        }
        if constexpr (DEG == kDegFp32) return a * a * a - long_part(r2, pp);
        else return a * a * a * pair_poly<DEG, sizeof(R) == 8>(s, a, pp);
    }
}

// Targets: sorted slots tslot[t] (null: target t is sorted slot t, every
// source). Output of target t goes to index out_idx[t] (null: t), written, or
// added to what is there when `add`. Source masses: sorted sm[] (null: P.m).
//
// One warp per block and group of G targets; lane l works for target l % G and
// takes every (32 / G)-th list entry. What bounds it: instruction issue, shared
// between the pair factors (FP64), the distance filter and the node tests. A walk
// with one lane per target ran with 11 of 32 lanes active, and each lane
// classified every node its warp reached in binary64; here a node costs one lane a
// few integer and FP32 operations for the whole group.
// Registers for 24 warps per SM (80; 8 to 44 bytes of spill in the closed form and at
// degree 36, none in the others); caps for 28 and 20 measured 34.2 / 33.6 / 34.8 ms on
// 2.1M clustered sources at G = 16. Shared memory holds 23 of these one-warp
// blocks per SM at G = 16 and 17 at G = 1, 4 and 8.
constexpr int kWalkWarps = 24;
template <int G>
struct WalkShape {
    static_assert(G >= 1 && G <= 16, "lane and mask layout");
    static constexpr int S = 32 / G;                  // lanes per target
    static constexpr int cap = S < 4 ? 32 * S : 128;  // list entries, >= 32
    static constexpr int per_lane = cap / S;          // one bit each of a 32-bit word
    static_assert(per_lane <= 32 && cap >= 32, "list layout");
};

template <typename R, int DEG, int G>
__global__ void __launch_bounds__(32, kWalkWarps)
k_walk(uint32_t n_targets, const uint32_t* __restrict__ tslot, const double* __restrict__ sx,
       const double* __restrict__ sy, const double* __restrict__ sz,
       const double* __restrict__ sm, const unsigned long long* __restrict__ skey,
       const Node* __restrict__ nodes, const uint4* __restrict__ ga,
       const uint4* __restrict__ gm, const uint4* __restrict__ gc, uint32_t n_nodes, WalkParams P,
       const PairPoly pp, const uint32_t* __restrict__ out_idx, int add, double* __restrict__ ax,
       double* __restrict__ ay, double* __restrict__ az,
       unsigned long long* __restrict__ counters, unsigned int* status) {
    using Shape = WalkShape<G>;
    constexpr int S = Shape::S, CAP = Shape::cap, PER = Shape::per_lane;
    constexpr uint32_t kGroup = (1u << G) - 1u;
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ double ex[CAP], ey[CAP], ez[CAP], ew[CAP];  // entry position (the group's image), G m
    __shared__ float4 erel[CAP];              // (position - group centre) / r_cut, target mask
    __shared__ float4 ucell[32], ucom[32];    // undecided nodes: cube centre, half; COM, opening
    __shared__ uint32_t unode[32], umask[32], uaccept[32], uopen[32];
    __shared__ uint32_t gfirst[32], gsource[32], gnode[32], gmono[32], gopen[32];
    __shared__ uint32_t run_first[kStack], run_count[kStack], run_mask[kStack];
    const int lane = threadIdx.x;
    const int t = lane % G, sub = lane / G;
    const unsigned below = (1u << lane) - 1u;
    const uint32_t t0 = blockIdx.x * G;
    const uint32_t n_here = n_targets - t0 < G ? n_targets - t0 : G;
    const bool valid = static_cast<uint32_t>(t) < n_here;
    const uint32_t ti = t0 + (valid ? t : 0u);
    const uint32_t slot = tslot ? tslot[ti] : ti;
    const double tx = sx[slot], ty = sy[slot], tz = sz[slot];

    // The group's bounding box in 2^-32 L: centre, and half sides with slack for
    // the rounding of positions and centres of mass to that unit. safe: every
    // source within r_cut of a target lies in the image nearest to the centre.
    // inner: in the image it is stored in.
    uint32_t gcu[3], ge[3];
    double ctr[3];
    bool safe = true, inner = true;
    const float unit_rc = static_cast<float>(P.r_cut * (4294967296.0 / P.L));
    const float inv_unit = 1.f / unit_rc;
    const double inv_rc = 1.0 / P.r_cut;
    float er[3], e_max = 0.f;   // half sides over r_cut
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const uint32_t u = box_fraction(a == 0 ? tx : (a == 1 ? ty : tz), P.L);
        const uint32_t lo = __reduce_min_sync(kAll, u), hi = __reduce_max_sync(kAll, u);
        gcu[a] = lo + (hi - lo) / 2;
        ge[a] = (hi - lo) / 2 + 4u;
        ctr[a] = gcu[a] * (P.L / 4294967296.0);
        const float span = unit_rc * 1.000001f + 2.f * static_cast<float>(ge[a]);
        safe = safe && span < 2147483000.f;
        inner = inner && static_cast<float>(lo) > unit_rc * 1.00001f + 1024.f
            && static_cast<float>(hi) < 4294966000.f - unit_rc * 1.00001f;
        er[a] = static_cast<float>(ge[a]) * inv_unit;
        e_max = fmaxf(e_max, er[a]);
    }
    inner = inner && safe;
    const float rc2 = unit_rc * unit_rc;
    const float rc2_hi = rc2 * 1.00001f, rc2_lo = rc2 * 0.99999f;
    // slack of FP32 coordinates relative to the centre, in units of r_cut
    // (magnitudes up to 2 + 2 e / r_cut, and 4 units of 2^-32 L)
    const float slack = 4e-7f * (2.f + 2.f * e_max) + 4.f * inv_unit;
    const float cut_hi = (1.f + 2.f * slack) * (1.f + 2.f * slack);
    const float cut_lo = (1.f - 2.f * slack) * (1.f - 2.f * slack);
    const float frx = static_cast<float>((tx - ctr[0]) * inv_rc);
    const float fry = static_cast<float>((ty - ctr[1]) * inv_rc);
    const float frz = static_cast<float>((tz - ctr[2]) * inv_rc);
    const double eps2 = P.eps * P.eps, inv_rs = 1.0 / P.r_s, rcut2 = P.r_cut * P.r_cut;

    const float reach2 = safe ? cut_hi : __int_as_float(0x7f800000);   // unsafe: no filter
    const uint32_t tbit = 1u << t;

    double fx = 0.0, fy = 0.0, fz = 0.0;
    uint32_t visits = 0, pairs = 0;
    int count = 0;   // entries in the list

    // Every target sums the listed entries: a distance filter into one bit per
    // entry, then the pair factor over the set bits.
    auto flush = [&]() {
        __syncwarp();
        // stale entries of a part-filled list belong to nobody
        for (int e = count + lane; e < CAP; e += 32) erel[e].w = 0.f;
        __syncwarp();
        uint32_t bits = 0;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const float4 c = erel[k * S + sub];
            const float dx = c.x - frx, dy = c.y - fry, dz = c.z - frz;
            if (dx * dx + dy * dy + dz * dz < reach2 && (__float_as_uint(c.w) & tbit)) bits |= 1u << k;
        }
        while (bits) {
            const int e = (__ffs(bits) - 1) * S + sub;
            bits &= bits - 1;
            double dx = ex[e] - tx, dy = ey[e] - ty, dz = ez[e] - tz;
            if (!safe) {
                dx = min_image(dx, P.L);
                dy = min_image(dy, P.L);
                dz = min_image(dz, P.L);
            }
            const double r2 = dx * dx + dy * dy + dz * dz;
            if (r2 < rcut2 && r2 != 0.0) {   // 0: the target itself
                const double f = pair_factor<R, DEG>(r2, eps2, inv_rs, pp) * ew[e];
                fx += f * dx;
                fy += f * dy;
                fz += f * dz;
                ++pairs;
            }
        }
        __syncwarp();
        count = 0;
    };

    if (lane == 0) {
        run_first[0] = 0;
        run_count[0] = 1;
        run_mask[0] = (1u << n_here) - 1u;
    }
    int sp = 1;
    __syncwarp();
    unsigned iter = 0;
    while (sp > 0) {
        if (++iter > kMaxIter) {
            if (lane == 0) raise_status(status, ST_CAPACITY);
            break;
        }
        // Pop child runs from the top, as many as give at most 32 nodes.
        uint32_t pop_first = 0, pop_n = 0, pop_mask = 0;
        if (lane < sp && (lane == 0 || sp <= kStackWide)) {
            pop_first = run_first[sp - 1 - lane];
            pop_n = run_count[sp - 1 - lane];
            pop_mask = run_mask[sp - 1 - lane];
        }
        uint32_t inc = pop_n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(kAll, inc, o);
            if (lane >= o) inc += v;
        }
        const uint32_t exc = inc - pop_n;
        const bool taken = pop_n > 0 && inc <= 32u;
        const int runs = __popc(__ballot_sync(kAll, taken));
        const unsigned starts = __reduce_or_sync(kAll, taken ? 1u << exc : 0u);
        const uint32_t total = __shfl_sync(kAll, inc, runs - 1);
        const int from = __popc(starts & (below | (1u << lane))) - 1;
        const uint32_t ni = __shfl_sync(kAll, pop_first - exc, from) + static_cast<uint32_t>(lane);
        uint32_t mask = __shfl_sync(kAll, pop_mask, from);
        const bool active = static_cast<uint32_t>(lane) < total;
        sp -= runs;
        if (runs == 0 || __any_sync(kAll, active && ni >= n_nodes)) {
            if (lane == 0) raise_status(status, ST_CELL_ESCAPE);
            break;
        }
        __syncwarp();

        // Classify node ni for the whole group. am: targets that take its
        // monopole; om: targets that need its children (a leaf's sources).
        uint32_t am = 0, om = 0;
        uint4 link = make_uint4(0, 0, 0, 0);
        bool undecided = false;
        float4 cell, com;
        if (active) {
            visits += __popc(mask);
            const uint4 a = ga[ni];
            link = gc[ni];
            const uint32_t h = a.w;
            const int d[3] = {static_cast<int>(a.x - gcu[0]), static_cast<int>(a.y - gcu[1]),
                              static_cast<int>(a.z - gcu[2])};
            if (h >= 0x40000000u) {
                om = mask;   // a quarter of the box or more: always opened
            } else {
                float near2 = 0.f, lo2 = 0.f, far2 = 0.f;
                bool apart = false;
                const float hf = static_cast<float>(h);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const uint32_t D = static_cast<uint32_t>(abs(d[k]));
                    const uint32_t low = D > ge[k] ? D - ge[k] : 0u;
                    const uint32_t gap = low > h ? low - h : 0u;
                    apart = apart || gap > 8u;
                    const float g = static_cast<float>(gap), l = static_cast<float>(low) + hf,
                                f = static_cast<float>(D) + static_cast<float>(ge[k]) + hf;
                    near2 += g * g;
                    lo2 += l * l;
                    far2 += f * f;
                }
                if (near2 < rc2_hi) {   // else outside every target's cutoff sphere
                    const bool leaf = (link.y >> 8) != 0;
                    om = mask;          // a leaf, or a node inside nobody's sphere
                    if (!leaf && lo2 < rc2_hi) {
                        const uint4 m = gm[ni];
                        const float open2 = __uint_as_float(m.w);
                        const int c[3] = {static_cast<int>(m.x - gcu[0]),
                                          static_cast<int>(m.y - gcu[1]),
                                          static_cast<int>(m.z - gcu[2])};
                        float min2 = 0.f, max2 = 0.f;
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            const uint32_t M = static_cast<uint32_t>(abs(c[k]));
                            const float l = static_cast<float>(M > ge[k] ? M - ge[k] : 0u);
                            const float f = static_cast<float>(M) + static_cast<float>(ge[k]);
                            min2 += l * l;
                            max2 += f * f;
                        }
                        if (open2 < rc2_hi && max2 > open2 * 0.99999f) {
                            om = 0;
                            if (apart && far2 < rc2_lo && min2 > open2 * 1.00001f) {
                                am = mask;
                            } else {
                                undecided = true;
                                cell = make_float4(d[0] * inv_unit, d[1] * inv_unit,
                                                   d[2] * inv_unit, hf * inv_unit);
                                com = make_float4(c[0] * inv_unit, c[1] * inv_unit,
                                                  c[2] * inv_unit, sqrtf(open2) * inv_unit);
                            }
                        }
                    }
                }
            }
        }

        // Undecided nodes, S at a time: each target applies the criterion itself,
        // in FP32 relative to the group's centre where that settles it, else with
        // the reference's binary64 expressions.
        const unsigned todo = __ballot_sync(kAll, undecided);
        if (todo) {
            const int n_todo = __popc(todo), at = __popc(todo & below);
            if (undecided) {
                ucell[at] = cell;
                ucom[at] = com;
                unode[at] = ni;
                umask[at] = mask;
            }
            __syncwarp();
            for (int b = 0; b < n_todo; b += S) {
                const int u = b + sub;
                bool accept = false, open = false;
                if (u < n_todo && ((umask[u] >> t) & 1u)) {
                    const float4 c = ucell[u], m = ucom[u];
                    const float dx = fabsf(c.x - frx), dy = fabsf(c.y - fry),
                                dz = fabsf(c.z - frz);
                    const float nx = fmaxf(dx - c.w, 0.f), ny = fmaxf(dy - c.w, 0.f),
                                nz = fmaxf(dz - c.w, 0.f);
                    const float gx = dx + c.w, gy = dy + c.w, gz = dz + c.w;
                    const float far2 = gx * gx + gy * gy + gz * gz;
                    const float mx = m.x - frx, my = m.y - fry, mz = m.z - frz;
                    const float r2 = mx * mx + my * my + mz * mz;
                    const float hi = m.w * 1.000001f + 2.f * slack;
                    const float lo = fmaxf(m.w * 0.999999f - 2.f * slack, 0.f);
                    const bool apart = fmaxf(nx, fmaxf(ny, nz)) > 2.f * slack;
                    // opening a node just outside the cutoff changes nothing: the
                    // sources below it are rejected by their own distances
                    open = nx * nx + ny * ny + nz * nz < cut_hi;
                    const bool maybe = !safe || (open && far2 < cut_hi && r2 > lo * lo);
                    accept = safe && maybe && apart && far2 < cut_lo && r2 > hi * hi;
                    if (maybe && !accept) {
                        const Node& nd = nodes[unode[u]];
                        const double dcx = fabs(min_image(nd.cx - tx, P.L)),
                                     dcy = fabs(min_image(nd.cy - ty, P.L)),
                                     dcz = fabs(min_image(nd.cz - tz, P.L));
                        const double h = nd.half;
                        const double qx = fmax(dcx - h, 0.0), qy = fmax(dcy - h, 0.0),
                                     qz = fmax(dcz - h, 0.0);
                        const double sx2 = dcx + h, sy2 = dcy + h, sz2 = dcz + h;
                        open = qx * qx + qy * qy + qz * qz < rcut2;
                        const int shift = 3 * (kBits - static_cast<int>(nd.level));
                        const bool contains = shift >= 64 || (skey[slot] >> shift) == nd.prefix;
                        if (open && !contains && sx2 * sx2 + sy2 * sy2 + sz2 * sz2 < rcut2) {
                            const double ox = min_image(nd.mx - tx, P.L),
                                         oy = min_image(nd.my - ty, P.L),
                                         oz = min_image(nd.mz - tz, P.L);
                            accept = ox * ox + oy * oy + oz * oz > nd.open2;
                        }
                    }
                    open = open && !accept;
                }
                const unsigned acc = __ballot_sync(kAll, accept), opn = __ballot_sync(kAll, open);
                if (t == 0 && u < n_todo) {
                    uaccept[u] = (acc >> (sub * G)) & kGroup;
                    uopen[u] = (opn >> (sub * G)) & kGroup;
                }
            }
            __syncwarp();
            if (undecided) {
                am = uaccept[at];
                om = uopen[at];
            }
            __syncwarp();
        }

        // Push the opened nodes' children; when every child holds one source,
        // and for a leaf, the sources join the list instead.
        const uint32_t n_child = link.y & 0xffu;
        const bool direct = om != 0 && ((link.y >> 8) != 0 || n_child == link.w);
        const bool push = om != 0 && !direct;
        const unsigned pushes = __ballot_sync(kAll, push);
        if (sp + __popc(pushes) > kStack || __any_sync(kAll, push && n_child > 8u)) {
            if (lane == 0) raise_status(status, n_child > 8u ? ST_CELL_ESCAPE : ST_CAPACITY);
            break;
        }
        if (push) {
            const int at = sp + __popc(pushes & below);
            run_first[at] = link.x;
            run_count[at] = n_child;
            run_mask[at] = om;
        }
        sp += __popc(pushes);

        // The list items of this step (a monopole and / or a source range per
        // lane), numbered across the warp and taken 32 at a time, one per lane.
        const uint32_t mono = am != 0 ? 1u : 0u;
        const uint32_t items = mono + (direct ? link.w : 0u);
        const unsigned givers = __ballot_sync(kAll, items != 0);
        if (givers) {
            uint32_t upto = items;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(kAll, upto, o);
                if (lane >= o) upto += v;
            }
            const uint32_t n_items = __shfl_sync(kAll, upto, 31), first = upto - items;
            if (items) {
                const int at = __popc(givers & below);
                gfirst[at] = first + mono;           // number of the first source
                gsource[at] = link.z;
                gnode[at] = ni;
                gmono[at] = am;
                gopen[at] = om;
            }
            __syncwarp();
            int before = 0;   // givers that start before the 32 items at hand
            for (uint32_t base = 0; base < n_items; base += 32) {
                const bool here = items && first >= base && first < base + 32;
                const unsigned starts_here = __reduce_or_sync(kAll, here ? 1u << (first - base) : 0u);
                const uint32_t i = base + static_cast<uint32_t>(lane);
                bool have = i < n_items;
                double x = 0.0, y = 0.0, z = 0.0, w = 0.0;
                float rx = 0.f, ry = 0.f, rz = 0.f;
                uint32_t who = 0;
                if (have) {
                    const int g = before + __popc(starts_here & (below | (1u << lane))) - 1;
                    const uint32_t f = gfirst[g];
                    if (i < f) {
                        const Node& nd = nodes[gnode[g]];
                        x = nd.mx;
                        y = nd.my;
                        z = nd.mz;
                        w = P.G * nd.mass;
                        who = gmono[g];
                    } else {
                        const uint32_t j = gsource[g] + (i - f);
                        x = sx[j];
                        y = sy[j];
                        z = sz[j];
                        w = P.G * (sm ? sm[j] : P.m);
                        who = gopen[g];
                    }
                    if (safe && !inner) {   // the image nearest to the centre
                        const double half = 0.5 * P.L;
                        if (x - ctr[0] > half) x -= P.L;
                        else if (x - ctr[0] < -half) x += P.L;
                        if (y - ctr[1] > half) y -= P.L;
                        else if (y - ctr[1] < -half) y += P.L;
                        if (z - ctr[2] > half) z -= P.L;
                        else if (z - ctr[2] < -half) z += P.L;
                    }
                    rx = static_cast<float>((x - ctr[0]) * inv_rc);
                    ry = static_cast<float>((y - ctr[1]) * inv_rc);
                    rz = static_cast<float>((z - ctr[2]) * inv_rc);
                    if (safe) {   // within reach of the group's box
                        const float qx = fmaxf(fabsf(rx) - er[0], 0.f),
                                    qy = fmaxf(fabsf(ry) - er[1], 0.f),
                                    qz = fmaxf(fabsf(rz) - er[2], 0.f);
                        have = qx * qx + qy * qy + qz * qz < cut_hi;
                    }
                }
                before += __popc(starts_here);
                const unsigned all = __ballot_sync(kAll, have);
                const int more = __popc(all);
                if (count + more > CAP) flush();
                if (have) {
                    const int e = count + __popc(all & below);
                    ex[e] = x;
                    ey[e] = y;
                    ez[e] = z;
                    ew[e] = w;
                    erel[e] = make_float4(rx, ry, rz, __uint_as_float(who));
                }
                count += more;
            }
        }
        __syncwarp();
    }
    if (count) flush();
#pragma unroll
    for (int o = G; o < 32; o <<= 1) {   // the lanes of one target
        fx += __shfl_xor_sync(kAll, fx, o);
        fy += __shfl_xor_sync(kAll, fy, o);
        fz += __shfl_xor_sync(kAll, fz, o);
    }
    if (valid && sub == 0) {
        const uint32_t o = out_idx ? out_idx[ti] : ti;
        if (add) {
            ax[o] += fx;
            ay[o] += fy;
            az[o] += fz;
        } else {
            ax[o] = fx;
            ay[o] = fy;
            az[o] = fz;
        }
    }
    // walk statistics: one atomic per warp, spread over kCounters pairs
    const unsigned all_visits = __reduce_add_sync(kAll, visits);
    const unsigned all_pairs = __reduce_add_sync(kAll, pairs);
    if (lane == 0) {
        unsigned long long* c = counters + 2 * (blockIdx.x % kCounters);
        atomicAdd(&c[0], static_cast<unsigned long long>(all_visits));
        atomicAdd(&c[1], static_cast<unsigned long long>(all_pairs));
    }
}

// h r_s^3 at r^2 = t r_s^2, t <= 4: the alternating series, terms falling from the first.
long double long_part_series(long double t) {
    const long double isp = 0.564189583547756286948079451560772586L;
    long double term = 1.0L / 4.0L, sum = 0.0L;   // t^k / (4^(k+1) (k+1)!)
    for (int k = 0; k < 30; ++k) {
        sum += (k & 1 ? -term : term) * 2.0L * (k + 1) / (2 * k + 3);
        term *= t / (4.0L * (k + 2));
    }
    return isp * sum;
}

long double shape_fraction(long double t) {   // M_S
    const long double isp = 0.564189583547756286948079451560772586L, q = std::sqrt(t);
    return std::erfc(0.5L * q) + q * isp * std::exp(-0.25L * t);
}

// F(u), the pair factor times s^(3/2), at r^2 = t r_s^2 and softening e r_s: below
// t = 4 (M_S > 0.5) as 1 - u^3 h, beyond as in short_factor_impl, which keeps the
// relative accuracy of a small F.
long double pair_shape(long double t, long double e) {
    const long double s = t + e * e, u3 = s * std::sqrt(s);
    if (t <= 4.0L) return 1.0L - u3 * long_part_series(t);
    return u3 / (t * std::sqrt(t)) * (std::expm1(-1.5L * std::log1p(e * e / t)) + shape_fraction(t));
}

constexpr long double kPiL = 3.141592653589793238462643383279502884L;

// Chebyshev interpolation, in monomials of tau, of the values y[i] at the N nodes
// tau_i = cos(pi (i + 1/2) / N).
template <int N>
void interpolate(const long double (&y)[N], long double (&mono)[N]) {
    long double wave[4 * N], ta[N] = {}, tb[N] = {};
    for (int i = 0; i < 4 * N; ++i) wave[i] = std::cos(kPiL * i / (2 * N));
    for (int i = 0; i < N; ++i) mono[i] = 0.0L;
    ta[0] = 1.0L;
    tb[1] = 1.0L;
    for (int j = 0; j < N; ++j) {
        long double s = 0.0L;
        for (int i = 0; i < N; ++i) s += y[i] * wave[j * (2 * i + 1) % (4 * N)];
        s *= (j ? 2.0L : 1.0L) / N;
        for (int i = 0; i < N; ++i) mono[i] += s * ta[i];
        // T_j in monomials by the recurrence T_{j+1} = 2 tau T_j - T_{j-1}
        for (int i = N - 1; i >= 0; --i) {
            const long double old = tb[i];
            tb[i] = (i ? 2.0L * tb[i - 1] : 0.0L) - ta[i];
            ta[i] = old;
        }
    }
}

// Whether the polynomial gives F within `want` of itself at 96 distances from the
// cutoff inwards.
template <int DEG, bool EXACT_U>
bool close_to_shape(double ratio, double eps, double r_s, double want, const PairPoly& pp) {
    for (int i = 0; i < 96; ++i) {
        const double r = ratio * r_s * (1.0 - (i + 0.01) / 96.0);
        const double r2 = r * r, s = r2 + eps * eps, root = std::sqrt(s);
        const long double f = pair_shape(static_cast<long double>(r2) / r_s / r_s,
                                         static_cast<long double>(eps) / r_s);
        const long double p = DEG == kDegFp32 ? 1.0 - s * root * long_part(r2, pp)
                                              : pair_poly<DEG, EXACT_U>(s, 1.0 / root, pp);
        if (!(std::fabs(p - f) <= want * std::fabs(f))) return false;
    }
    return true;
}

// The polynomial of degree DEG for a cutoff of `ratio` r_s: in v, two steps of division
// by v taken off, or (degree kDegFp32) that of h; false when it is not within `want`.
template <int DEG, bool EXACT_U>
bool fit_poly(double ratio, double eps, double r_s, double want, PairPoly* out) {
    constexpr int n = DEG + 1;
    const long double e = static_cast<long double>(eps) / r_s;
    const long double t_max = static_cast<long double>(ratio) * ratio * (1.0L + 1e-9L);
    const long double u_max = std::sqrt(t_max + e * e), width = t_max / (u_max + e);
    out->k = static_cast<double>(DEG == kDegFp32 ? 2.0L / (t_max * r_s * r_s) : 2.0L / (width * r_s));
    out->half_k = 0.5 * out->k;
    out->b = static_cast<double>(2.0L * u_max / width);
    if (!std::isfinite(out->k) || !std::isfinite(out->b)) return false;
    long double y[n], mono[n];
    for (int i = 0; i < n; ++i) {
        const long double tau = std::cos(kPiL * (i + 0.5L) / n);
        if (DEG == kDegFp32) {
            const long double t = 0.5L * t_max * (tau + 1.0L);
            const long double h = t <= 4.0L ? long_part_series(t)
                                            : (1.0L - shape_fraction(t)) / (t * std::sqrt(t));
            y[i] = h / (static_cast<long double>(r_s) * r_s * r_s);
        } else {   // u / r_s by the rounded k and b
            const long double u = (static_cast<long double>(out->b) - 1.0L + tau)
                / (static_cast<long double>(out->k) * r_s);
            y[i] = pair_shape((u - e) * (u + e), e);
        }
    }
    interpolate(y, mono);
    for (int step = 0; step < 2 && DEG != kDegFp32; ++step) {   // remainder, then quotient
        for (int i = n - 2; i >= step; --i) mono[i] += mono[i + 1];
    }
    for (int i = 0; i < n; ++i)
        out->c[i] = static_cast<double>(i == 1 && DEG != kDegFp32 ? -mono[i] : mono[i]);
    return close_to_shape<DEG, EXACT_U>(ratio, eps, r_s, want, *out);
}

// What the walk evaluates the pair factor by: the lowest degree whose F is within
// nine roundings in binary64 (a few ulp, as short_factor_impl) or half an FP32
// rounding of itself; 0: short_factor_impl. At a softening of r_s / 37, r_cut = 4.5 r_s
// takes 28 and 12, and short_factor_impl serves binary64 from 6.1 r_s on, where F is
// 3e-4, or from where softening makes F cross zero (5 r_s at eps = 0.3 r_s); the
// precision form from 9.5 r_s on at most.
struct PairForm {
    int degree = 0;
    PairPoly poly{};
};
constexpr double kWant64 = 2e-15, kWant32 = 6e-8;

PairForm pair_form(const hyowon_treepm_params& P) {
    PairForm f;
    PairPoly* const pp = &f.poly;
    const double ratio = P.cutoff / P.split_scale;
    if (!(ratio < 10.0)) return f;
    if (P.precision == HYOWON_FP64) {
        if (fit_poly<kDegLow, true>(ratio, P.softening, P.split_scale, kWant64, pp)) f.degree = kDegLow;
        else if (fit_poly<kDegMid, true>(ratio, P.softening, P.split_scale, kWant64, pp)) f.degree = kDegMid;
        else if (fit_poly<kDegHigh, true>(ratio, P.softening, P.split_scale, kWant64, pp)) f.degree = kDegHigh;
    } else {
        if (fit_poly<kDegFp32, false>(ratio, P.softening, P.split_scale, kWant32, pp)) f.degree = kDegFp32;
        else if (fit_poly<kDegLow, false>(ratio, P.softening, P.split_scale, kWant32, pp)) f.degree = kDegLow;
        else if (fit_poly<kDegHigh, false>(ratio, P.softening, P.split_scale, kWant32, pp)) f.degree = kDegHigh;
    }
    return f;
}

// Per-particle masses: node mass and centre of mass summed bottom-up, one
// level at a time from the deepest (leaves from their sources in sorted order,
// internal nodes from their children in child order: a fixed order, so the
// moments are the same bits run to run). A massless node keeps its cube centre.
__global__ void k_gather_masses(uint32_t n, const uint32_t* __restrict__ val,
                                const double* __restrict__ mass, double* __restrict__ sm) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) sm[i] = mass[val[i]];
}

__global__ void k_moments(uint32_t begin, uint32_t end, const double* __restrict__ sx,
                          const double* __restrict__ sy, const double* __restrict__ sz,
                          const double* __restrict__ sm, Node* __restrict__ nodes) {
    const uint32_t k = begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= end) return;
    Node& nd = nodes[k];
    double M = 0.0, X = 0.0, Y = 0.0, Z = 0.0;
    if (nd.leaf) {
        for (uint32_t i = nd.start; i < nd.end; ++i) {
            const double m = sm[i];
            M += m;
            X += m * sx[i];
            Y += m * sy[i];
            Z += m * sz[i];
        }
    } else {
        for (uint32_t c = 0; c < nd.n_child; ++c) {
            const Node& ch = nodes[nd.first_child + c];
            M += ch.mass;
            X += ch.mass * ch.mx;
            Y += ch.mass * ch.my;
            Z += ch.mass * ch.mz;
        }
    }
    nd.mass = M;
    if (M > 0.0) {
        nd.mx = X / M;
        nd.my = Y / M;
        nd.mz = Z / M;
    } else {
        nd.mx = nd.cx;
        nd.my = nd.cy;
        nd.mz = nd.cz;
    }
}

struct Fail {
    int code;
    std::string msg;
};

#define TCK(call)                                                                           \
    do {                                                                                    \
        cudaError_t e_ = (call);                                                            \
        if (e_ != cudaSuccess) throw Fail{e_ == cudaErrorMemoryAllocation ? HYOWON_ENOMEM  \
                                                                         : HYOWON_ECUDA,    \
                                          std::string(#call) + ": " + cudaGetErrorString(e_)}; \
    } while (0)

}  // namespace

// Device scratch kept between calls: one block that the buffers of a call are
// carved from (256-byte aligned), so that repeated solves allocate nothing.
// A call that needs more than it holds takes the rest from cudaMalloc and
// records the total, and the next call regrows the block to that size.
//
// The node arrays' size is known only within the call, and a clustering run's tree
// grows from step to step (1.39 n nodes near a lattice, 1.46 n clustered): they are
// carved for `nodes` nodes, at least 2 n and a fourth more than any tree that went
// beyond that had. Sized exactly, a larger tree cost its solve 36 ms and the next 7
// (4.1M sources, whose build takes 2.0). Where memory is too short, exactly.
struct Workspace {
    void* base = nullptr;
    size_t cap = 0;
    size_t want = 0;
    uint32_t nodes = 0;
    bool exact = false;
    uint64_t allocations = 0;   // cudaMalloc calls made for it
};

uint64_t workspace_allocations(const Workspace* ws) { return ws ? ws->allocations : 0; }

Workspace* create_workspace() { return new (std::nothrow) Workspace(); }

void destroy_workspace(Workspace* ws) {
    if (!ws) return;
    if (ws->base) cudaFree(ws->base);
    delete ws;
}

namespace {

struct Mem {
    Workspace* ws;
    size_t off = 0;
    std::vector<void*> p;   // buffers beyond the workspace, freed with this
    explicit Mem(Workspace* w = nullptr) : ws(w) {
        if (ws && ws->want > ws->cap) {
            // the previous call finished its work before returning
            if (ws->base) cudaFree(ws->base);
            ws->base = nullptr;
            ws->cap = 0;
            if (!allocate(&ws->base, ws->want)) {
                // buffer by buffer instead, and without room for a larger tree
                ws->want = 0;
                ws->exact = true;
                return;
            }
            ws->cap = ws->want;
        }
    }
    // Nodes that the node arrays of a tree of n_nodes on n sources are carved for.
    uint32_t node_room(uint32_t n, uint32_t n_nodes) {
        if (!ws || ws->exact) return n_nodes;
        if (n_nodes > ws->nodes || n > ws->nodes / 2) {
            const uint64_t room = std::max<uint64_t>(2ull * n, n_nodes + n_nodes / 4ull);
            ws->nodes = static_cast<uint32_t>(std::min<uint64_t>(room, 0xFFFFFFF0ull));
        }
        return std::max(ws->nodes, n_nodes);
    }
    bool allocate(void** q, size_t bytes) {
        if (ws) ++ws->allocations;
        const cudaError_t e = cudaMalloc(q, bytes);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            return false;
        }
        TCK(e);
        return true;
    }
    // `count` elements, or at least `least` where memory is short.
    template <typename T>
    T* get_room(size_t count, size_t least) {
        const size_t at = off;
        try {
            return get<T>(count);
        } catch (const Fail& f) {
            if (f.code != HYOWON_ENOMEM || count <= least) throw;
        }
        ws->exact = true;
        off = at;
        return get<T>(least);
    }
    template <typename T>
    T* get(size_t count) {
        const size_t bytes = (((count ? count : 1) * sizeof(T)) + 255) & ~static_cast<size_t>(255);
        if (ws) {
            const size_t at = off;
            off += bytes;
            if (off <= ws->cap) return reinterpret_cast<T*>(static_cast<char*>(ws->base) + at);
        }
        void* q = nullptr;
        if (!allocate(&q, bytes)) throw Fail{HYOWON_ENOMEM, "octree work arrays could not be allocated"};
        p.push_back(q);
        return static_cast<T*>(q);
    }
    ~Mem() {
        if (ws && off > ws->want) ws->want = off;
        for (void* q : p) cudaFree(q);
    }
};

void scan64(Mem& mem, const unsigned long long* in, unsigned long long* out, uint64_t n,
            cudaStream_t s) {
    const uint64_t blocks = (n + 1023) / 1024;
    if (blocks == 1) {
        k_scan64_block<<<1, 1024, 0, s>>>(in, out, n, nullptr);
        return;
    }
    unsigned long long* sums = mem.get<unsigned long long>(blocks);
    unsigned long long* sums_ex = mem.get<unsigned long long>(blocks);
    k_scan64_block<<<static_cast<unsigned>(blocks), 1024, 0, s>>>(in, out, n, sums);
    scan64(mem, sums, sums_ex, blocks, s);
    k_scan64_add<<<nb(n), kT, 0, s>>>(out, n, sums_ex);
}

struct WalkArgs {
    uint32_t nt;
    const uint32_t* tslot;
    const double *sx, *sy, *sz, *sm;
    const unsigned long long* skey;
    const Node* nodes;
    const uint4 *ga, *gm, *gc;
    uint32_t n_nodes;
    WalkParams W;
    const uint32_t* out_idx;
    int add;
    double *ax, *ay, *az;
    unsigned long long* counters;
    unsigned int* status;
};

template <typename R, int DEG, int G>
void launch_walk_as(const WalkArgs& A, const PairPoly& pp, cudaStream_t s) {
    const unsigned blocks = static_cast<unsigned>((static_cast<uint64_t>(A.nt) + G - 1) / G);
    k_walk<R, DEG, G><<<blocks, 32, 0, s>>>(A.nt, A.tslot, A.sx, A.sy, A.sz, A.sm, A.skey, A.nodes,
                                             A.ga, A.gm, A.gc, A.n_nodes, A.W, pp, A.out_idx, A.add,
                                             A.ax, A.ay, A.az, A.counters, A.status);
}

template <typename R, int DEG>
void launch_walk_deg(const WalkArgs& A, const PairPoly& pp, int group, cudaStream_t s) {
    switch (group) {
        case 1: launch_walk_as<R, DEG, 1>(A, pp, s); break;
        case 4: launch_walk_as<R, DEG, 4>(A, pp, s); break;
        case 8: launch_walk_as<R, DEG, 8>(A, pp, s); break;
        default: launch_walk_as<R, DEG, 16>(A, pp, s); break;
    }
}

template <typename R>
void launch_walk(const WalkArgs& A, const PairForm& form, int group, cudaStream_t s) {
    switch (form.degree) {
        case kDegFp32:
            if constexpr (sizeof(R) == 4) launch_walk_deg<R, kDegFp32>(A, form.poly, group, s);
            break;
        case kDegLow: launch_walk_deg<R, kDegLow>(A, form.poly, group, s); break;
        case kDegMid:
            if constexpr (sizeof(R) == 8) launch_walk_deg<R, kDegMid>(A, form.poly, group, s);
            break;
        case kDegHigh: launch_walk_deg<R, kDegHigh>(A, form.poly, group, s); break;
        default: launch_walk_deg<R, 0>(A, form.poly, group, s);
    }
}

// Targets a warp takes. A larger group shares the node tests among more targets
// but has a larger box, so more undecided nodes and rejected pairs, and fewer
// warps. Measured walk ms at G = 4 / 8 / 16 (clustered sources, every source a
// target; binary64 with the pair factor at degree 20, 26.6 instead of 25.4 at 28):
// 30,000: 0.87 / 0.96 / 1.36; 262,144: 4.7 / 4.0 / 4.9; 2.1M: 39 / 30 / 25;
// 16.8M: 290 / 213 / 166 (in Morton order 25 to 30% more: 4.9, 32 and 191 at the
// chosen G; one lane per target: 15, 48, 168 and 696). Targets that are a sample of
// the sources lie further apart: of 2.1M sources, 4,096 targets take 0.66 ms at
// G = 1 (1.6 at 4; 48 with one lane per target), 524,288 12 at G = 4, 10.4 at 8 and
// 10.3 at 16 (23 at 1, 82 with one lane per target).
int walk_group(uint32_t n, uint32_t nt) {
    if (nt < n / 8 + 1) return 1;
    if (nt < 100000) return 4;
    return nt < 1000000 || nt < n / 2 + 1 ? 8 : 16;
}

thread_local std::string g_err;

}  // namespace

// Builds the octree of the n device sources (x, y, z; masses or, when null,
// P.particle_mass) and walks the targets on stream s: with host_targets the
// nt listed source indices, results written to ax/ay/az[target] in list order;
// without (nt = n), every source in key order, results added to
// ax/ay/az[source]. Output arrays are device memory. Device work is ordered on
// s; the call returns after it has finished.
int run(const hyowon_treepm_params& P, uint32_t n, const double* x, const double* y,
        const double* z, const double* masses, const uint32_t* host_targets, uint32_t nt,
        double* ax, double* ay, double* az, cudaStream_t s, double* stats,
        Workspace* ws = nullptr) {
    Mem mem(ws);
    struct Events {
        cudaEvent_t e[4] = {};
        Events() { for (auto& v : e) cudaEventCreate(&v); }
        ~Events() { for (auto& v : e) cudaEventDestroy(v); }
    } ev;
    unsigned int* status = mem.get<unsigned int>(1);
    TCK(cudaMemsetAsync(status, 0, sizeof(unsigned int), s));
    double* wx = mem.get<double>(n);
    double* wy = mem.get<double>(n);
    double* wz = mem.get<double>(n);
    unsigned long long* key[2] = {mem.get<unsigned long long>(n), mem.get<unsigned long long>(n)};
    uint32_t* val[2] = {mem.get<uint32_t>(n), mem.get<uint32_t>(n)};
    cudaEventRecord(ev.e[0], s);
    k_keys<<<nb(n), kT, 0, s>>>(n, x, y, z, P.box_size, wx, wy, wz, key[0], val[0], status);
    // radix sort
    const uint32_t n_tiles = static_cast<uint32_t>((n + kTile - 1) / kTile);
    uint32_t* hist = mem.get<uint32_t>(256ull * n_tiles + 1);
    uint32_t* offs = mem.get<uint32_t>(256ull * n_tiles + 1);
    uint32_t* scan_tmp = mem.get<uint32_t>(scan_tmp_elements(256u * n_tiles + 1));
    int cur = 0;
    for (int pass = 0; pass < 8; ++pass) {
        const int shift = 8 * pass;
        k_tile_hist<<<n_tiles, kT, 0, s>>>(n, key[cur], shift, n_tiles, hist);
        launch_exclusive_scan(hist, offs, 256u * n_tiles, scan_tmp, s);
        k_tile_scatter<<<n_tiles, kT, 0, s>>>(n, key[cur], val[cur], shift, n_tiles, offs,
                                               key[1 - cur], val[1 - cur]);
        cur = 1 - cur;
    }
    const unsigned long long* skey = key[cur];
    const uint32_t* sval = val[cur];
    double* sx = mem.get<double>(n);
    double* sy = mem.get<double>(n);
    double* sz = mem.get<double>(n);
    unsigned long long* q[3];
    unsigned long long* pq[3];
    for (int a = 0; a < 3; ++a) {
        q[a] = mem.get<unsigned long long>(n + 1);
        pq[a] = mem.get<unsigned long long>(n + 1);
    }
    uint32_t* inv = mem.get<uint32_t>(n);
    k_gather_sorted<<<nb(n + 1), kT, 0, s>>>(n, sval, wx, wy, wz, P.box_size, sx, sy, sz, q[0],
                                             q[1], q[2], inv);
    for (int a = 0; a < 3; ++a) scan64(mem, q[a], pq[a], n + 1, s);
    double* sm = nullptr;
    if (masses) {
        sm = mem.get<double>(n);
        k_gather_masses<<<nb(n), kT, 0, s>>>(n, sval, masses, sm);
    }
    // nodes: how many of each level, then all in one sweep
    const uint32_t n_node_tiles = nb(n);
    const uint32_t n_counts = kLevels * n_node_tiles + 1;
    uint32_t* level_hist = mem.get<uint32_t>(n_counts);
    uint32_t* level_offs = mem.get<uint32_t>(n_counts);
    uint32_t* level_tmp = mem.get<uint32_t>(scan_tmp_elements(n_counts));
    k_level_counts<<<n_node_tiles, kT, 0, s>>>(n, skey, n_node_tiles, level_hist);
    launch_exclusive_scan(level_hist, level_offs, n_counts, level_tmp, s);
    const PairForm form = pair_form(P);   // while the device sorts and counts
    uint32_t level_begin[kLevels + 1];   // the last entry: the number of nodes
    TCK(cudaMemcpy2DAsync(level_begin, sizeof(uint32_t), level_offs,
                          sizeof(uint32_t) * n_node_tiles, sizeof(uint32_t), kLevels + 1,
                          cudaMemcpyDeviceToHost, s));
    TCK(cudaStreamSynchronize(s));
    // A level has at most n nodes, so the differences are its counts even where the
    // 32-bit running total wrapped; only a total that needs more bits is refused.
    uint64_t total = 0;
    int depth = 0;
    for (int l = 0; l < kLevels; ++l) {
        const uint32_t here = level_begin[l + 1] - level_begin[l];
        total += here;
        if (here) depth = l;
    }
    if (total > 0xFFFFFFF0ull) throw Fail{HYOWON_ERUNTIME, "octree of more than 2^32-16 nodes"};
    const uint32_t node_base = static_cast<uint32_t>(total);
    const uint32_t room = mem.node_room(n, node_base);
    Node* nodes = mem.get_room<Node>(room, node_base);
    k_emit_nodes<<<n_node_tiles, kT, 0, s>>>(n, skey, n_node_tiles, level_offs, P.box_size, sx, sy,
                                             sz, pq[0], pq[1], pq[2], P.particle_mass, nodes);
    if (sm) {
        for (int l = depth; l >= 0; --l) {
            const uint32_t b = level_begin[l], e = level_begin[l + 1];
            k_moments<<<nb(e - b), kT, 0, s>>>(b, e, sx, sy, sz, sm, nodes);
        }
    }
    uint4* ga = mem.get_room<uint4>(room, node_base);
    uint4* gm = mem.get_room<uint4>(room, node_base);
    uint4* gc = mem.get_room<uint4>(room, node_base);
    k_walk_nodes<<<nb(node_base), kT, 0, s>>>(node_base, P.theta, P.box_size, nodes, ga, gm, gc);
    cudaEventRecord(ev.e[1], s);
    const uint32_t* dslots = nullptr;
    const uint32_t* out_idx = nullptr;
    if (host_targets) {
        // targets in key order for warp coherence; results land in list order
        for (uint32_t i = 0; i < nt; ++i)
            if (host_targets[i] >= n) throw Fail{HYOWON_EINVAL, "target index out of range"};
        uint32_t* d_targets = mem.get<uint32_t>(nt);
        uint32_t* d_at = mem.get<uint32_t>(nt);
        TCK(cudaMemcpyAsync(d_targets, host_targets, sizeof(uint32_t) * nt, cudaMemcpyHostToDevice, s));
        k_target_slots<<<nb(nt), kT, 0, s>>>(nt, d_targets, inv, d_at);
        std::vector<uint32_t> at(nt), slots(nt), dest(nt);
        TCK(cudaMemcpyAsync(at.data(), d_at, sizeof(uint32_t) * nt, cudaMemcpyDeviceToHost, s));
        TCK(cudaStreamSynchronize(s));
        std::vector<std::pair<uint32_t, uint32_t>> order(nt);
        for (uint32_t i = 0; i < nt; ++i) order[i] = {at[i], i};
        std::sort(order.begin(), order.end());
        for (uint32_t i = 0; i < nt; ++i) {
            slots[i] = order[i].first;
            dest[i] = order[i].second;
        }
        uint32_t* d_slots = mem.get<uint32_t>(nt);
        uint32_t* d_dest = mem.get<uint32_t>(nt);
        TCK(cudaMemcpyAsync(d_slots, slots.data(), sizeof(uint32_t) * nt, cudaMemcpyHostToDevice, s));
        TCK(cudaMemcpyAsync(d_dest, dest.data(), sizeof(uint32_t) * nt, cudaMemcpyHostToDevice, s));
        TCK(cudaStreamSynchronize(s));
        dslots = d_slots;
        out_idx = d_dest;
    } else {
        out_idx = sval;   // sorted slot t holds source sval[t]
    }
    unsigned long long* counters = mem.get<unsigned long long>(2 * kCounters);
    TCK(cudaMemsetAsync(counters, 0, 2 * kCounters * sizeof(unsigned long long), s));
    const double G = 6.67430e-11 * (1e10 * 1.98847e30) / (3.085677581491367e22 * 1000.0 * 1000.0);
    const WalkParams W{P.box_size, P.cutoff, P.softening, P.split_scale, G, P.particle_mass};
    const WalkArgs A{nt, dslots, sx, sy, sz, sm, skey, nodes, ga, gm, gc, node_base, W,
                     out_idx, host_targets ? 0 : 1, ax, ay, az, counters, status};
    const int group = walk_group(n, nt);
    cudaEventRecord(ev.e[2], s);
    if (P.precision == HYOWON_FP64) launch_walk<double>(A, form, group, s);
    else launch_walk<float>(A, form, group, s);
    TCK(cudaPeekAtLastError());
    cudaEventRecord(ev.e[3], s);
    unsigned long long cnt[2] = {0, 0}, cnt_all[2 * kCounters];
    unsigned int st = 0;
    TCK(cudaMemcpyAsync(cnt_all, counters, sizeof(cnt_all), cudaMemcpyDeviceToHost, s));
    TCK(cudaMemcpyAsync(&st, status, sizeof(st), cudaMemcpyDeviceToHost, s));
    TCK(cudaStreamSynchronize(s));
    for (unsigned i = 0; i < 2 * kCounters; ++i) cnt[i & 1] += cnt_all[i];
    if (stats) {
        float tb = 0.f, tw = 0.f;
        cudaEventElapsedTime(&tb, ev.e[0], ev.e[1]);
        cudaEventElapsedTime(&tw, ev.e[2], ev.e[3]);
        stats[0] = node_base;
        stats[1] = depth;
        stats[2] = nt ? static_cast<double>(cnt[0]) / nt : 0.0;
        stats[3] = nt ? static_cast<double>(cnt[1]) / nt : 0.0;
        stats[4] = tb;
        stats[5] = tw;
    }
    if (st & ST_NONFINITE_INPUT) throw Fail{HYOWON_EINVAL, "source positions must be finite"};
    if (st & ST_CAPACITY) throw Fail{HYOWON_ERUNTIME, "tree walk exceeded its stack or iteration bound"};
    if (st & ST_CELL_ESCAPE) throw Fail{HYOWON_ELOGIC, "octree child link out of range"};
    return HYOWON_OK;
}

int short_forces(const hyowon_treepm_params& P, uint32_t n, const double* hx, const double* hy,
                 const double* hz, uint32_t nt, const uint32_t* htargets, double* hax,
                 double* hay, double* haz, double* stats) {
    cudaStream_t s = nullptr;
    TCK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct StreamGuard {
        cudaStream_t s;
        ~StreamGuard() { cudaStreamDestroy(s); }
    } guard{s};
    Mem mem;
    double* x = mem.get<double>(n);
    double* y = mem.get<double>(n);
    double* z = mem.get<double>(n);
    TCK(cudaMemcpyAsync(x, hx, sizeof(double) * n, cudaMemcpyHostToDevice, s));
    TCK(cudaMemcpyAsync(y, hy, sizeof(double) * n, cudaMemcpyHostToDevice, s));
    TCK(cudaMemcpyAsync(z, hz, sizeof(double) * n, cudaMemcpyHostToDevice, s));
    double* oax = mem.get<double>(nt);
    double* oay = mem.get<double>(nt);
    double* oaz = mem.get<double>(nt);
    run(P, n, x, y, z, nullptr, htargets, nt, oax, oay, oaz, s, stats);
    TCK(cudaMemcpyAsync(hax, oax, sizeof(double) * nt, cudaMemcpyDeviceToHost, s));
    TCK(cudaMemcpyAsync(hay, oay, sizeof(double) * nt, cudaMemcpyDeviceToHost, s));
    TCK(cudaMemcpyAsync(haz, oaz, sizeof(double) * nt, cudaMemcpyDeviceToHost, s));
    TCK(cudaStreamSynchronize(s));
    return HYOWON_OK;
}

int device_short_forces(const hyowon_treepm_params& P, uint32_t n, const double* x,
                        const double* y, const double* z, const double* masses, double* ax,
                        double* ay, double* az, cudaStream_t s, double* stats, std::string* err,
                        Workspace* ws) {
    try {
        return run(P, n, x, y, z, masses, nullptr, n, ax, ay, az, s, stats, ws);
    } catch (const Fail& f) {
        if (err) *err = f.msg;
        return f.code;
    } catch (const std::exception& e) {   // bad_alloc, length_error
        if (err) *err = std::string("out of host memory: ") + e.what();
        return HYOWON_ENOMEM;
    }
}

}  // namespace hyowon::tree

extern "C" {

const char* hyowon_treepm_last_error(void) { return hyowon::tree::g_err.c_str(); }

int hyowon_treepm_short_forces(const hyowon_treepm_params* params, uint64_t n, const double* x,
                               const double* y, const double* z, uint64_t n_targets,
                               const uint32_t* targets, double* ax, double* ay, double* az,
                               double* stats) {
    using namespace hyowon::tree;
    g_err.clear();
    if (!params || !x || !y || !z || !targets || !ax || !ay || !az || n < 2 || n > 0xFFFFFFF0ull
        || n_targets == 0 || n_targets > n) {
        g_err = "invalid TreePM short-range arguments";
        return HYOWON_EINVAL;
    }
    const hyowon_treepm_params& P = *params;
    if (!(P.box_size > 0.0) || !(P.split_scale > 0.0) || !(P.cutoff > 0.0)
        || !(P.cutoff < 0.5 * P.box_size) || !(P.softening > 0.0) || !(P.theta > 0.0)
        || !(P.particle_mass > 0.0)
        || (P.precision != HYOWON_FP64 && P.precision != HYOWON_FP32_FIXED)) {
        g_err = "TreePM parameters must be finite positive with r_cut < L/2";
        return HYOWON_EINVAL;
    }
    try {
        return short_forces(P, static_cast<uint32_t>(n), x, y, z,
                            static_cast<uint32_t>(n_targets), targets, ax, ay, az, stats);
    } catch (const Fail& f) {
        g_err = f.msg;
        return f.code;
    } catch (const std::exception& e) {   // bad_alloc, length_error
        g_err = std::string("out of host memory: ") + e.what();
        return HYOWON_ENOMEM;
    }
}

}  // extern "C"
