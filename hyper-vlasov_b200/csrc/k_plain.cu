// Plain-path kernels: one kernel per reference routine, in the reference's
// operation order.  This translation unit is compiled with --fmad=false so
// that a*b+c stays two rounded operations, as in the reference built with
// -ffp-contract=off; with identical inputs the HV_F64 results of deposit
// (sorted mode), FDM, merge, SOR, gather and push are bit-identical to it.
#include <algorithm>
#include <cmath>

#include <cub/device/device_radix_sort.cuh>

#include "grid_sync.cuh"
#include "hv_internal.h"

namespace hv {
namespace {

constexpr int kBlock = 256;

// Integer cell coordinate and fractional offset of one axis,
// distribute_volumetric_particles_cic (include/tools.hpp:50-60).
template <typename T>
struct Axis {
    T c;  // (n/2) (x/d_max + 1)
};

template <typename T>
__device__ __forceinline__ T cell_coord(T pos, T dmax, int n) {
    return (n / T(2.0)) * (pos / dmax + T(1.0));
}

template <typename T>
__device__ __forceinline__ bool in_grid(T cx, T cy, T cz, int nx, int ny, int nz) {
    // a NaN coordinate is outside: converted to an index it would be any
    return cx >= T(0.0) && cy >= T(0.0) && cz >= T(0.0) && cx < nx && cy < ny && cz < nz;
}

// ---- CIC deposit, atomic (include/tools.hpp:35-96) -----------------------
template <typename T>
__global__ void k_deposit_atomic(Geom g, int protons, int total, const T *__restrict__ x,
                                 const T *__restrict__ y, const T *__restrict__ z, T *rho) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    T cx = cell_coord<T>(x[i], T(g.dmx), nx);
    T cy = cell_coord<T>(y[i], T(g.dmy), ny);
    T cz = cell_coord<T>(z[i], T(g.dmz), nz);
    if (!in_grid<T>(cx, cy, cz, nx, ny, nz)) return;
    int x0 = (int)cx, y0 = (int)cy, z0 = (int)cz;
    int x1 = x0 + 1, y1 = y0 + 1, z1 = z0 + 1;
    T d_x = cx - x0, d_y = cy - y0, d_z = cz - z0;
    T t_x = T(1.0) - d_x, t_y = T(1.0) - d_y, t_z = T(1.0) - d_z;
    long long off = (i < protons) ? 0 : g.G;
    long long sy = nz, sx = (long long)ny * nz;
    T *b = rho + off;
    atomicAdd(b + x0 * sx + y0 * sy + z0, t_x * t_y * t_z);
    if (x1 < nx) atomicAdd(b + x1 * sx + y0 * sy + z0, d_x * t_y * t_z);
    if (y1 < ny) atomicAdd(b + x0 * sx + y1 * sy + z0, t_x * d_y * t_z);
    if (x1 < nx && y1 < ny) atomicAdd(b + x1 * sx + y1 * sy + z0, d_x * d_y * t_z);
    if (z1 < nz) atomicAdd(b + x0 * sx + y0 * sy + z1, t_x * t_y * d_z);
    if (x1 < nx && z1 < nz) atomicAdd(b + x1 * sx + y0 * sy + z1, d_x * t_y * d_z);
    if (y1 < ny && z1 < nz) atomicAdd(b + x0 * sx + y1 * sy + z1, t_x * d_y * d_z);
    if (x1 < nx && y1 < ny && z1 < nz) atomicAdd(b + x1 * sx + y1 * sy + z1, d_x * d_y * d_z);
}

// ---- CIC deposit, sorted / deterministic ---------------------------------
// Key of a particle = species * G + linear cell (x0, y0, z0); particles outside
// the grid get key 2G and sort last.
template <typename T>
__global__ void k_cell_keys(Geom g, int protons, int total, const T *__restrict__ x,
                            const T *__restrict__ y, const T *__restrict__ z, unsigned int *keys,
                            int *vals) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    T cx = cell_coord<T>(x[i], T(g.dmx), g.nx);
    T cy = cell_coord<T>(y[i], T(g.dmy), g.ny);
    T cz = cell_coord<T>(z[i], T(g.dmz), g.nz);
    unsigned int key;
    if (!in_grid<T>(cx, cy, cz, g.nx, g.ny, g.nz)) {
        key = (unsigned int)(2 * g.G);
    } else {
        long long cell = ((long long)(int)cx * g.ny + (int)cy) * g.nz + (int)cz;
        key = (unsigned int)(cell + ((i < protons) ? 0 : g.G));
    }
    keys[i] = key;
    vals[i] = i;
}

// A sorted particle: its fractional offsets in the cell, and the index of the
// next particle of its cell (kNoParticle: it is the last).
constexpr int kNoParticle = 0x7fffffff;
template <typename T>
struct Entry;
template <>
struct __align__(16) Entry<float> {
    float d[3];
    int next;
};
template <>
struct __align__(16) Entry<double> {
    double d[3];
    int next, pad;
};

// The arrays behind the entries.
template <typename T>
struct SortedParticles {
    const T *x, *y, *z;
    const unsigned int *keys;  // ascending
    const int *idx;            // particle of each place
    int total;
};

template <typename T>
__device__ __forceinline__ Entry<T> entry_of(const Geom &g, const SortedParticles<T> &p, int s, unsigned int key, int i) {
    const T cx = cell_coord<T>(p.x[i], T(g.dmx), g.nx);
    const T cy = cell_coord<T>(p.y[i], T(g.dmy), g.ny);
    const T cz = cell_coord<T>(p.z[i], T(g.dmz), g.nz);
    Entry<T> e;
    e.d[0] = cx - (int)cx;
    e.d[1] = cy - (int)cy;
    e.d[2] = cz - (int)cz;
    e.next = s + 1 == p.total || p.keys[s + 1] != key ? kNoParticle : p.idx[s + 1];
    return e;
}

// Entries in sorted order (ent null: none are kept), and every occupied cell's
// first place (cell_start is -1 for the others; a search per cell cost 63 us at
// 128^3).
template <typename T>
__global__ void k_deposit_entries(Geom g, SortedParticles<T> p, int *cell_start, Entry<T> *ent) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= p.total) return;
    const unsigned int key = p.keys[s];
    if ((long long)key >= 2 * g.G) return;
    if (ent) ent[s] = entry_of<T>(g, p, s, key, p.idx[s]);
    if (s == 0 || p.keys[s - 1] != key) cell_start[key] = s;
}

// One thread per node: merges the particle lists of the (up to) eight cells
// that touch the node, in increasing particle index, and sums their CIC
// weights sequentially from 0 -- the order of a single-threaded run of the
// reference's deposit loop (include/tools.hpp:46-95).  One entry a turn for
// every lane, whatever list it comes from: a loop that follows one list while
// it stays the smallest takes fewer turns per node, but its lanes leave it at
// different turns and wait for each other.  The heads are in registers, the
// places in shared memory ([list][thread]: no bank conflicts), and an entry
// brings its successor's index, so that a turn waits for memory once.  A head
// is a key, index times eight plus list, and the keys are kept sorted: the
// popped one's successor moves to its place by minima and maxima alone.
// K: 32 bits where every index fits (kMaxIndex32), else 64.
// Block: nodes along z; grid: (z blocks, y, x of both species).  Bound by the
// instructions of a turn times a node's ~100 entries.  208Pb 2.08 M / 128^3 in
// float: 102 us; 133 with the smallest of eight unsorted heads searched each
// turn, 232 following one list while it is the smallest; blocks of 64 or 32
// threads 8 or 20 % slower.  40Ca, 4,000 in double: 24-34 us, latency.
constexpr int kMaxIndex32 = (1 << 29) - 2;  // its key is below kNoParticle's, 0xfffffff8

// kKept: the entries are in memory; else each is formed when its turn comes,
// from arrays in the callers' order (the same bits, more loads).
template <typename T, typename K, bool kKept>
__global__ void __launch_bounds__(128) k_deposit_merge(Geom g, const Entry<T> *__restrict__ ent,
                                                       const int *__restrict__ cell_start,
                                                       const int *__restrict__ sorted_idx, SortedParticles<T> part,
                                                       T *rho) {
    __shared__ int s_pos[8][128];
    const int iz = blockIdx.x * blockDim.x + threadIdx.x, iy = blockIdx.y, tid = threadIdx.x;
    const int sp = blockIdx.z >= (unsigned)g.nx ? 1 : 0, ix = blockIdx.z - sp * g.nx;
    const long long s_off = sp ? g.G : 0;
    const int lane = tid & 31;
    constexpr K none = (K)kNoParticle << 3;
    K head[8];  // ascending
#pragma unroll
    for (int l = 0; l < 8; l++) head[l] = none | 7;
    // x takes its place among head[1..7], and head[0] is dropped
    auto replace_first = [&](K x) {
#pragma unroll
        for (int l = 0; l < 7; l++) {
            head[l] = min(head[l + 1], x);
            x = max(head[l + 1], x);
        }
        head[7] = x;
    };
    int first[8];
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int dx = r >> 1, dy = r & 1, cx = ix - dx, cy = iy - dy;
        const long long row = s_off + ((long long)cx * g.ny + cy) * g.nz;
        int here = -1, below = -1;
        if (cx >= 0 && cy >= 0) {
            if (iz < g.nz) here = __ldg(cell_start + row + iz);
            if (lane == 0 && iz > 0 && iz <= g.nz) below = __ldg(cell_start + row + iz - 1);
        }
        const int up = __shfl_up_sync(0xffffffffu, here, 1);
        if (lane) below = up;
        first[2 * r] = here;
        first[2 * r + 1] = below;
    }
    if (iz >= g.nz) return;
    int lists = 0;
#pragma unroll
    for (int l = 0; l < 8; l++) {
        s_pos[l][tid] = first[l];
        first[l] = first[l] >= 0 ? __ldg(sorted_idx + first[l]) : kNoParticle;
        lists += first[l] != kNoParticle;
    }
    if (lists) {
        // what leaves at the end is always `none`
#pragma unroll
        for (int l = 0; l < 8; l++) {
            K x = (K)first[l] << 3 | l;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const K lo = min(head[q], x);
                x = max(head[q], x);
                head[q] = lo;
            }
        }
    }
    T acc = T(0.0);
    while (head[0] < none) {
        const int best = (int)(head[0] & 7);
        const int p = s_pos[best][tid];
        Entry<T> e;
        if constexpr (kKept) e = ent[p];
        else e = entry_of<T>(g, part, p, part.keys[p], sorted_idx[p]);
        s_pos[best][tid] = p + 1;
        replace_first((K)e.next << 3 | best);
        // node = cell + corner; corner bit 1 means the "1" side (weight d)
        const T wx = (best & 4) ? e.d[0] : T(1.0) - e.d[0];
        const T wy = (best & 2) ? e.d[1] : T(1.0) - e.d[1];
        const T wz = (best & 1) ? e.d[2] : T(1.0) - e.d[2];
        acc += wx * wy * wz;
    }
    rho[s_off + ((long long)ix * g.ny + iy) * g.nz + iz] = acc;
}

// ---- smoothing (include/physics.hpp:202-234) -----------------------------
template <typename T>
__global__ void k_smooth_direct(Geom g, int ntaps, int lx, int ly, int lz, const int *__restrict__ taps,
                                const T *__restrict__ w, T term, const T *__restrict__ src, T *dst) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * g.G) return;
    const long long off = i >= g.G ? g.G : 0;
    const long long node = i - off;
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const int iz = (int)(node % nz), iy = (int)((node / nz) % ny), ix = (int)(node / ((long long)ny * nz));
    const T *s = src + off;
    T rho_f = T(0.0);
    const bool interior = ix >= lx && ix < nx - lx && iy >= ly && iy < ny - ly && iz >= lz && iz < nz - lz;
    if (interior) {
        for (int t = 0; t < ntaps; t++) {
            int p = __ldg(taps + t);
            int a = (p >> 20) - 512, b = ((p >> 10) & 1023) - 512, c = (p & 1023) - 512;
            long long j = node + ((long long)a * ny + b) * nz + c;
            rho_f += s[j] * __ldg(w + t);
        }
    } else {
        for (int t = 0; t < ntaps; t++) {
            int p = __ldg(taps + t);
            int a = (p >> 20) - 512, b = ((p >> 10) & 1023) - 512, c = (p & 1023) - 512;
            int jx = ix + a, jy = iy + b, jz = iz + c;
            if (jx < 0 || jx >= nx || jy < 0 || jy >= ny || jz < 0 || jz >= nz) continue;
            rho_f += s[((long long)jx * ny + jy) * nz + jz] * __ldg(w + t);
        }
    }
    dst[i] = rho_f * term;  // physics.hpp:229-232
}

// The same sums, in the same order, four consecutive z per thread: the source
// rows that a block's outputs reach at one x offset are staged in shared
// memory with zeros outside the grid (adding w * 0 changes no sum), and along
// a run of taps a thread's four source values shift through registers, one new
// load a tap.  Stored by z mod 4, so that consecutive threads read consecutive
// words.  A tap then costs a thread two shared loads and eight operations
// instead of four times two global loads, the index arithmetic and two
// operations: 64^3 in double, half-width 4, 533 -> 95 us.
constexpr int kRowThreads = 128;
struct RowTile {
    int qz, ty, pitch, words, wmax;  // quads of a z row, y rows of a block, words of a quarter row, of a slab, weights
};

template <typename T>
__global__ void __launch_bounds__(kRowThreads) k_smooth_rows(Geom g, RowTile rt, int lx, int ly, int lz, int runs,
                                                             const int *__restrict__ tab, const T *__restrict__ w,
                                                             T term, const T *__restrict__ src, T *dst) {
    extern __shared__ __align__(16) unsigned char row_smem[];
    T *rows = reinterpret_cast<T *>(row_smem), *ws = rows + rt.words;
    const int nx = g.nx, ny = g.ny, nz = g.nz, tid = threadIdx.x;
    const int ix = blockIdx.y, y0 = blockIdx.x * rt.ty, nrows = rt.ty + 2 * ly, width = nz + 2 * lz;
    const T *s = src + (blockIdx.z ? g.G : 0);
    const int4 *run = reinterpret_cast<const int4 *>(tab);
    const int *slab = tab + 4 * runs;
    const int r = tid / rt.qz, q = tid - r * rt.qz;
    const bool mine = r < rt.ty && y0 + r < ny;
    T acc0 = T(0), acc1 = T(0), acc2 = T(0), acc3 = T(0);
    for (int a = -lx; a <= lx; a++) {
        const int r0 = slab[a + lx], r1 = slab[a + lx + 1], jx = ix + a;
        if (r0 == r1 || jx < 0 || jx >= nx) continue;
        const int t0 = run[r0].w, t1 = run[r1 - 1].w + run[r1 - 1].z;
        __syncthreads();
        for (int e = tid; e < t1 - t0; e += kRowThreads) ws[e] = w[t0 + e];
        int some = 0;
        for (int e = tid; e < nrows * width; e += kRowThreads) {
            const int rr = e / width, zz = e - rr * width, jy = y0 - ly + rr, jz = zz - lz;
            const bool in = jy >= 0 && jy < ny && jz >= 0 && jz < nz;
            const T v = in ? s[((long long)jx * ny + jy) * nz + jz] : T(0);
            some |= v != T(0);
            rows[(rr * 4 + (zz & 3)) * rt.pitch + (zz >> 2)] = v;
        }
        // rows without density add w * 0 to every sum
        if (!__syncthreads_or(some) || !mine) continue;
        for (int k = r0; k < r1; k++) {
            const int4 v = run[k];
            const T *row = rows + (r + ly + v.x) * 4 * rt.pitch + q;
            const T *wk = ws + v.w - t0;
            int z = v.y + lz;  // padded position of the first tap for z = 4 q
            auto at = [&](int p) { return row[(p & 3) * rt.pitch + (p >> 2)]; };
            T v0 = at(z), v1 = at(z + 1), v2 = at(z + 2);
            for (int t = 0; t < v.z; t++) {
                const T v3 = at(z + 3 + t), wt = wk[t];
                acc0 += v0 * wt;
                acc1 += v1 * wt;
                acc2 += v2 * wt;
                acc3 += v3 * wt;
                v0 = v1;
                v1 = v2;
                v2 = v3;
            }
        }
    }
    if (!mine) return;
    T *d = dst + (blockIdx.z ? g.G : 0) + ((long long)ix * ny + y0 + r) * nz + 4 * q;
    const T out[4] = {acc0, acc1, acc2, acc3};
    for (int u = 0; u < 4; u++)
        if (4 * q + u < nz) d[u] = out[u] * term;  // physics.hpp:229-232
}

// ---- Skyrme (include/physics.hpp:272-281, physics_formulas.hpp:70-77) ------
template <typename T>
__device__ __forceinline__ T skyrme_u(T A, T B, T C, T gamma, T rho_p, T rho_n, T tau) {
    T rho = rho_p + rho_n;
    T t = rho / T(0.16);
    return A * t + B * pow(t, gamma) + T(2.0) * tau * C * ((rho_n - rho_p) / T(0.16));
}

template <typename T>
__global__ void k_skyrme(long long G, T A, T B, T C, T gamma, const T *__restrict__ rho, T *U) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= G) return;
    T rp = rho[i], rn = rho[i + G];
    U[i] = skyrme_u<T>(A, B, C, gamma, rp, rn, T(-1.0));
    U[i + G] = skyrme_u<T>(A, B, C, gamma, rp, rn, T(+1.0));
}

// ---- Coulomb boundary (include/tools.hpp:283-300) -------------------------
template <typename T>
__device__ __forceinline__ T node_pos(T dmax, int i, int n) {
    return dmax * (T(2.0) * (T)i / (T)n - T(1.0));
}

template <typename T, typename A>  // A: arithmetic type of the monopole
__global__ void k_boundary(Geom g, int Z, T *phi) {
    long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= g.G) return;
    const int nz = g.nz, ny = g.ny, nx = g.nx;
    const int k = (int)(id % nz), j = (int)((id / nz) % ny), i = (int)(id / ((long long)ny * nz));
    if (!(i == 0 || j == 0 || k == 0 || i == nx - 1 || j == ny - 1 || k == nz - 1)) return;
    A v0 = node_pos<A>(A(g.dmx), i, nx), v1 = node_pos<A>(A(g.dmy), j, ny), v2 = node_pos<A>(A(g.dmz), k, nz);
    A r = sqrt(v0 * v0 + v1 * v1 + v2 * v2);
    phi[id] = (T)(A(1.44) * Z / r);
}

// ---- red-black SOR (include/physics.hpp:99-157) ---------------------------
// One cooperative launch per solve; the stopping rule is tested after every
// iteration, as the reference's loop does, but on the device and one half
// sweep late.  A black update has its node's final neighbours at hand, so it
// forms the node's residual too; a red node's residual of iteration t needs
// the black values of t, which the red half sweep of t + 1 reads anyway.  The
// test of iteration t therefore runs while the black half sweep of t + 1
// does; when t met the rule, both half sweeps of t + 1 are taken back from the
// values they saved.  An iteration is two half sweeps and two grid barriers;
// the arithmetic of every kept value is the reference's.
//
// Bound by the latency of a half sweep (operands from L2, three divisions) and
// of the barrier.  A step of the plain double path, mostly this solve: 208Pb
// 64^3 15.4 -> 4.0 ms, 40Ca 32^3 2.6 -> 0.56 ms (five launches, a serial sum
// and a synchronisation an iteration before).
constexpr int kSorBlock = 1024;

template <typename T>
struct PlainSor {
    int nx, ny, nz, half, count;  // count: colour points, (nx - 2)(ny - 2) half
    T omega, inv_dx2, hx2, hy2, hz2, src_c, tol_t;
    T rx, ry, rz;                 // reciprocals of hx2, hy2, hz2
    double ix2, iy2, iz2, diag, bsrc, tol;
    int criterion, max_iter, nblocks;
    long long max_spin;
    T *phi, *saved;
    const T *rho;
    double *partials;             // [nblocks][2]
    unsigned *bar;
    int *status;                  // [0] error, [1] iterations, [2] 1 converged, 2 not finite
    double *metric;
};

template <typename T>
__device__ __forceinline__ T nan_max(T a, T b) {
    return (b > a || b != b) ? b : a;
}

// sx / hx2 + sy / hy2 + sz / hz2 + src as the reference rounds it.  kDiv 0:
// divisions; 1: the h2 are powers of two; 2: from the rounded reciprocals, by
// Markstein's theorem (Markstein 1990): a quotient within an ulp plus the exact
// remainder's correction is the rounded quotient (two corrections: the first
// product may be two ulps off).  The remainders are exact unless they underflow,
// for quotients of 2^-929 and more; smaller ones, an ulp off at most, leave a
// sum of 2^-700 or more as it is, since each addition that they could sway has
// terms within 2^54 of each other.  A smaller sum, and one that is not finite,
// is formed anew with divisions.  An iteration of 32^3 at h = 0.9 fm / 64^3 at
// 0.45: divisions 6.6 / 9.5 us, this form 6.4 / 9.25 (6.1 / 9.15 without the
// test of the sum).  The divisions are a call where the loop has the registers
// for one (kCall, the grid's form), in line in the cluster's.
template <typename T>
__device__ __forceinline__ T corrected(T v, T h, T y) {
    T q = v * y;
    q = fma(fma(-h, q, v), y, q);
    return fma(fma(-h, q, v), y, q);
}
__device__ __forceinline__ bool small_or_not_finite(double t) {
    return (unsigned)(__double2hiint(t) & 0x7fffffff) - 0x14300000u >= 0x7ff00000u - 0x14300000u;
}
__device__ __forceinline__ bool small_or_not_finite(float) { return true; }
template <typename T>
__device__ __noinline__ T divided_sum(T sx, T hx2, T sy, T hy2, T sz, T hz2, T src) {
    return sx / hx2 + sy / hy2 + sz / hz2 + src;
}

template <int kDiv, bool kCall, typename T>
__device__ __forceinline__ T stencil_sum(const PlainSor<T> &a, T sx, T sy, T sz, T src) {
    if constexpr (kDiv == 1) return sx * a.rx + sy * a.ry + sz * a.rz + src;
    if constexpr (kDiv == 2) {
        const T t = corrected(sx, a.hx2, a.rx) + corrected(sy, a.hy2, a.ry) + corrected(sz, a.hz2, a.rz) + src;
        if (__builtin_expect(!small_or_not_finite(t), 1)) return t;
        if constexpr (kCall) return divided_sum(sx, a.hx2, sy, a.hy2, sz, a.hz2, src);
    }
    return sx / a.hx2 + sy / a.hy2 + sz / a.hz2 + src;
}

// Node of colour point t, or -1 (the last point of a short line).
template <typename T>
__device__ __forceinline__ int colour_node(const PlainSor<T> &a, int color, int t) {
    const int l = t / a.half, kk = t - l * a.half, li = l / (a.ny - 2);
    const int j = 1 + l - li * (a.ny - 2), i = 1 + li;
    const int k = 1 + ((i + j + 1 + color) & 1) + 2 * kk;
    return k < a.nz - 1 ? (i * a.ny + j) * a.nz + k : -1;
}

template <typename T, int kDiv>
__global__ void __launch_bounds__(kSorBlock, 1) k_sor_plain(PlainSor<T> a) {
    __shared__ int s_stop;
    __shared__ double s_metric;
    __shared__ T s_max[kSorBlock / 32];
    const int tid = threadIdx.x, b = blockIdx.x, stride = a.nblocks * kSorBlock, first = b * kSorBlock + tid;
    const int sx = a.ny * a.nz, sy = a.nz;
    const bool rel = a.criterion == HV_SOR_REL_RESIDUAL;
    // the first point of each colour, decoded once (most grids: the only one)
    const int node0[2] = {first < a.count ? colour_node(a, 0, first) : -1,
                          first < a.count ? colour_node(a, 1, first) : -1};
    double rr = 0.0, bb = 0.0;
    T diff = T(0);

    auto sweep = [&](int color, bool sources) {
        for (int t = first; t < a.count; t += stride) {
            const int id = t == first ? node0[color] : colour_node(a, color, t);
            if (id < 0) continue;
            const T r = __ldg(a.rho + id);
            const T xp = __ldcg(a.phi + id + sx), xm = __ldcg(a.phi + id - sx);
            const T yp = __ldcg(a.phi + id + sy), ym = __ldcg(a.phi + id - sy);
            const T zp = __ldcg(a.phi + id + 1), zm = __ldcg(a.phi + id - 1);
            const T old = __ldcg(a.phi + id);
            const T star = stencil_sum<kDiv, true>(a, xp + xm, yp + ym, zp + zm, a.src_c * r) * a.inv_dx2;
            const T nv = (T(1.0) - a.omega) * old + a.omega * star;
            a.saved[id] = old;
            __stcg(a.phi + id, nv);
            if (rel) {
                // b + lap_h phi in double: of the iterate before at a red node,
                // of this one at a black node
                const double bv = a.bsrc * (double)r;
                const double lap = ((double)xp + (double)xm) * a.ix2 + ((double)yp + (double)ym) * a.iy2 +
                                   ((double)zp + (double)zm) * a.iz2 - a.diag * (double)(color ? nv : old);
                const double res = bv + lap;
                rr += res * res;
                if (sources) bb += bv * bv;
            } else {
                diff = nan_max(diff, (T)fabs(nv - old));
            }
        }
    };
    auto take_back = [&](int color) {
        for (int t = first; t < a.count; t += stride) {
            const int id = t == first ? node0[color] : colour_node(a, color, t);
            if (id >= 0) a.phi[id] = a.saved[id];
        }
    };
    // warp 0: the test of iteration `t` from the blocks' partial results
    auto test = [&](int t) {
        double u = 0.0, v = 0.0;
        for (int q = tid; q < a.nblocks; q += 32) {
            const double p = __ldcg(a.partials + 2 * q);
            if (rel) {
                u += p;
                v += __ldcg(a.partials + 2 * q + 1);
            } else {
                u = nan_max(u, p);
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const double p = __shfl_xor_sync(0xffffffffu, u, o), q = __shfl_xor_sync(0xffffffffu, v, o);
            u = rel ? u + p : nan_max(u, p);
            v += q;
        }
        if (tid == 0) {
            const double m = !rel ? u : v > 0.0 ? sqrt(u / v) : sqrt(u);
            const bool ok = rel ? m <= a.tol : (T)m < a.tol_t;
            s_metric = m;
            s_stop = m != m ? 2 : ok ? 1 : t >= a.max_iter ? 3 : 0;
        }
    };

    unsigned target = 0;  // the host zeroes the barrier before each launch
    int it = 0;
    while (true) {
        it++;
        if (!rel && it > 1 && tid < 32) test(it - 1);
        // rr still holds the black nodes' residual of iteration it - 1
        if (!rel) diff = T(0);
        sweep(0, it == 1);
        if (rel) {
            double u = rr, v = bb;
            block_sum2(u, v);
            if (tid == 0) {
                a.partials[2 * b] = u;
                a.partials[2 * b + 1] = v;
            }
            rr = 0.0;
        } else if (it > 1) {
            __syncthreads();
            if (s_stop) {
                take_back(0);
                break;
            }
        }
        if (!epoch_barrier(a.bar, target, a.nblocks, a.status, a.max_spin)) return;
        if (rel && it > 1 && tid < 32) test(it - 1);
        sweep(1, it == 1);
        if (rel) {
            __syncthreads();
            if (it > 1 && s_stop) {
                take_back(0);
                take_back(1);
                break;
            }
        } else {
            T m = diff;
            for (int o = 16; o > 0; o >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, o));
            if ((tid & 31) == 0) s_max[tid >> 5] = m;
            __syncthreads();
            if (tid == 0) {
                for (int w = 1; w < kSorBlock / 32; w++) m = nan_max(m, s_max[w]);
                a.partials[2 * b] = (double)m;
            }
        }
        if (!epoch_barrier(a.bar, target, a.nblocks, a.status, a.max_spin)) return;
    }
    if (b == 0 && tid == 0) {
        a.status[1] = it - 1;
        a.status[2] = s_stop == 3 ? 0 : s_stop;
        a.metric[0] = s_metric;
    }
}

// ---- the same solve in one thread-block cluster ------------------------------
// For small grids (sor_cluster_launch): each block of the cluster holds P x planes for the whole solve, in
// colour-split rows, and reads its neighbours' face planes through distributed
// shared memory.  The half sweeps then wait for the cluster's hardware barrier
// instead of a grid barrier through L2, at the price of fewer double units.
// Same order of operations, same values.  40Ca 32^3: 6.7 -> 4.5 us an iteration.
constexpr int kClusterThreads = 1024, kSorRanks = 16;
constexpr size_t kSorClusterSmem = 220 * 1024;  // planes of one block; its static arrays take 1.5 KB

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned at_rank(const void *p, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ double ld_cluster(unsigned p, double) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ float ld_cluster(unsigned p, float) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_cluster(unsigned p, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(p), "d"(v) : "memory");
}

template <typename T, int kDiv>
__global__ void __launch_bounds__(kClusterThreads, 1) k_sor_cluster(PlainSor<T> a, int ranks, int P) {
    extern __shared__ __align__(16) unsigned char cluster_smem[];
    __shared__ int s_stop;
    __shared__ double s_metric, s_mine[2], s_part[16][2];
    __shared__ T s_max[kClusterThreads / 32];
    T *s = reinterpret_cast<T *>(cluster_smem);
    const int tid = threadIdx.x, rank = (int)cluster_rank();
    const int nx = a.nx, ny = a.ny, nz = a.nz, nz2 = (nz + 1) / 2, rows = ny - 2, plane = ny * 2 * nz2;
    const int x0 = 1 + rank * P, np = max(0, min(P, nx - 1 - x0));
    const bool rel = a.criterion == HV_SOR_REL_RESIDUAL;
    const int count = np * rows * a.half;
    for (int e = tid; e < np * ny * nz; e += kClusterThreads) {
        const int r = e / nz, k = e - r * nz, p = r / ny, j = r - p * ny;
        s[r * 2 * nz2 + ((x0 + p + j + k) & 1) * nz2 + (k >> 1)] = a.phi[(size_t)x0 * ny * nz + e];
    }
    // the neighbours' face planes: a block's memory, or the grid's face
    const unsigned below = rank > 0 ? at_rank(s + (P - 1) * plane, rank - 1) : 0u;
    const unsigned above = rank + 1 < ranks ? at_rank(s, rank + 1) : 0u;
    // points t = tid, tid + stride, ...: (p, j, kk) advances by fixed steps
    const int dkk = kClusterThreads % a.half, dl = kClusterThreads / a.half, dj = dl % rows, dp = dl / rows;
    const int l0 = tid / a.half, kk0 = tid - l0 * a.half, p0 = l0 / rows, j0 = l0 - p0 * rows;
    double rr = 0.0, bb = 0.0;
    T diff = T(0);
    cluster_barrier();

    auto points = [&](int color, auto body) {
        int p = p0, j = j0, kk = kk0;
        for (int t = tid; t < count; t += kClusterThreads) {
            const int i = x0 + p, y = j + 1, k = 1 + ((i + y + 1 + color) & 1) + 2 * kk;
            if (k < nz - 1) body(p, i, y, k, ((p * ny + y) * 2 + color) * nz2 + (k >> 1));
            kk += dkk;
            j += dj;
            p += dp;
            if (kk >= a.half) {
                kk -= a.half;
                j++;
            }
            if (j >= rows) {
                j -= rows;
                p++;
            }
        }
    };
    auto sweep = [&](int color, bool sources) {
        points(color, [&](int p, int i, int y, int k, int own) {
            const int id = (i * ny + y) * nz + k;
            const T r = __ldg(a.rho + id);
            const int kh = k >> 1, other = (y * 2 + (color ^ 1)) * nz2, row = p * plane + other;
            const T xm = p > 0 ? s[row - plane + kh] : i > 1 ? ld_cluster(below + (other + kh) * (int)sizeof(T), T(0))
                                                              : __ldg(a.phi + id - ny * nz);
            const T xp = p + 1 < np ? s[row + plane + kh]
                         : i < nx - 2 ? ld_cluster(above + (other + kh) * (int)sizeof(T), T(0))
                                      : __ldg(a.phi + id + ny * nz);
            const T yp = s[row + 2 * nz2 + kh], ym = s[row - 2 * nz2 + kh];
            const T zp = s[row + ((k + 1) >> 1)], zm = s[row + ((k - 1) >> 1)];
            const T old = s[own];
            const T star = stencil_sum<kDiv, false>(a, xp + xm, yp + ym, zp + zm, a.src_c * r) * a.inv_dx2;
            const T nv = (T(1.0) - a.omega) * old + a.omega * star;
            a.saved[id] = old;
            s[own] = nv;
            if (rel) {
                const double bv = a.bsrc * (double)r;
                const double lap = ((double)xp + (double)xm) * a.ix2 + ((double)yp + (double)ym) * a.iy2 +
                                   ((double)zp + (double)zm) * a.iz2 - a.diag * (double)(color ? nv : old);
                const double res = bv + lap;
                rr += res * res;
                if (sources) bb += bv * bv;
            } else {
                diff = nan_max(diff, (T)fabs(nv - old));
            }
        });
    };
    auto take_back = [&](int color) {
        points(color, [&](int, int i, int y, int k, int own) { s[own] = a.saved[(i * ny + y) * nz + k]; });
    };
    // every block gets every block's partial results
    auto share = [&](double u, double v) {
        if (tid == 0) {
            s_mine[0] = u;
            s_mine[1] = v;
        }
        __syncthreads();
        if (tid < ranks) {
            const unsigned to = at_rank(s_part[rank], tid);
            st_cluster(to, s_mine[0]);
            st_cluster(to + 8, s_mine[1]);
        }
    };
    auto test = [&](int t) {
        if (tid == 0) {
            double u = 0.0, v = 0.0;
            for (int q = 0; q < ranks; q++) {
                u = rel ? u + s_part[q][0] : nan_max(u, s_part[q][0]);
                v += s_part[q][1];
            }
            const double m = !rel ? u : v > 0.0 ? sqrt(u / v) : sqrt(u);
            const bool ok = rel ? m <= a.tol : (T)m < a.tol_t;
            s_metric = m;
            s_stop = m != m ? 2 : ok ? 1 : t >= a.max_iter ? 3 : 0;
        }
    };

    int it = 0;
    while (true) {
        it++;
        if (!rel && it > 1) test(it - 1);
        if (!rel) diff = T(0);
        sweep(0, it == 1);
        if (rel) {
            double u = rr, v = bb;
            block_sum2(u, v);
            share(u, v);
            rr = 0.0;
        } else if (it > 1) {
            __syncthreads();
            if (s_stop) {
                take_back(0);
                break;
            }
        }
        cluster_barrier();
        if (rel && it > 1) test(it - 1);
        sweep(1, it == 1);
        if (rel) {
            __syncthreads();
            if (it > 1 && s_stop) {
                take_back(0);
                take_back(1);
                break;
            }
        } else {
            T m = diff;
            for (int o = 16; o > 0; o >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, o));
            if ((tid & 31) == 0) s_max[tid >> 5] = m;
            __syncthreads();
            if (tid == 0)
                for (int w = 1; w < kClusterThreads / 32; w++) m = nan_max(m, s_max[w]);
            share((double)m, 0.0);
        }
        cluster_barrier();
    }
    // no block leaves while another may still read its planes
    cluster_barrier();
    for (int e = tid; e < np * rows * (nz - 2); e += kClusterThreads) {
        const int r = e / (nz - 2), k = 1 + e - r * (nz - 2), p = r / rows, j = 1 + r - p * rows;
        a.phi[(size_t)((x0 + p) * ny + j) * nz + k] = s[((p * ny + j) * 2 + ((x0 + p + j + k) & 1)) * nz2 + (k >> 1)];
    }
    if (rank == 0 && tid == 0) {
        a.status[1] = it - 1;
        a.status[2] = s_stop == 3 ? 0 : s_stop;
        a.metric[0] = s_metric;
    }
}

// Sums `width`-wide rows of partials (nblocks rows) in fixed order.
// The rows come to shared memory first, all loads at once: the sums' serial
// chain then waits for additions, not for memory (18 us before, 3 after).
constexpr int kSumRows = 1024;
__global__ void k_sum_partials(const double *__restrict__ partials, int nblocks, int width,
                               double *out) {
    __shared__ double sh[kSumRows * 6];
    const int c = threadIdx.x;
    double s = 0.0;
    for (int b0 = 0; b0 < nblocks; b0 += kSumRows) {
        const int n = min(kSumRows, nblocks - b0);
        for (int e = threadIdx.x; e < n * width; e += blockDim.x) sh[e] = partials[(long long)b0 * width + e];
        __syncthreads();
        if (c < width) {
#pragma unroll 8
            for (int b = 0; b < n; b++) s += sh[b * width + c];
        }
        __syncthreads();
    }
    if (c < width) out[c] = s;
}

// ---- merge, FDM, gather, push, excite ------------------------------------
template <typename T>
__global__ void k_merge(long long G, T *U, const T *__restrict__ phi) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < G) U[i] += phi[i];
}

// compute_volumetric_forces_fdm (include/physics.hpp:159-200)
template <typename T>
__global__ void k_fdm(Geom g, T dx, T dy, T dz, const T *__restrict__ Uall, T *Fx, T *Fy, T *Fz) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * g.G) return;
    const long long off = i >= g.G ? g.G : 0;
    const long long id = i - off;
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const long long sx = (long long)ny * nz, sy = nz;
    const int k = (int)(id % nz), j = (int)((id / nz) % ny), ii = (int)(id / sx);
    const T *U = Uall + off;
    T gx, gy, gz;
    if (ii == 0) gx = (U[id + sx] - U[id]) / dx;
    else if (ii == nx - 1) gx = (U[id] - U[id - sx]) / dx;
    else gx = (U[id + sx] - U[id - sx]) / (T(2.0) * dx);
    if (j == 0) gy = (U[id + sy] - U[id]) / dy;
    else if (j == ny - 1) gy = (U[id] - U[id - sy]) / dy;
    else gy = (U[id + sy] - U[id - sy]) / (T(2.0) * dy);
    if (k == 0) gz = (U[id + 1] - U[id]) / dz;
    else if (k == nz - 1) gz = (U[id] - U[id - 1]) / dz;
    else gz = (U[id + 1] - U[id - 1]) / (T(2.0) * dz);
    Fx[i] = -gx;
    Fy[i] = -gy;
    Fz[i] = -gz;
}

// distribute_forces_to_particles_cic (include/tools.hpp:98-168)
template <typename T>
__global__ void k_gather(Geom g, int protons, int total, const T *__restrict__ x,
                         const T *__restrict__ y, const T *__restrict__ z, const T *__restrict__ Fx,
                         const T *__restrict__ Fy, const T *__restrict__ Fz, T *fx, T *fy, T *fz) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    T cx = cell_coord<T>(x[i], T(g.dmx), nx);
    T cy = cell_coord<T>(y[i], T(g.dmy), ny);
    T cz = cell_coord<T>(z[i], T(g.dmz), nz);
    if (!in_grid<T>(cx, cy, cz, nx, ny, nz)) {
        fx[i] = T(0.0);
        fy[i] = T(0.0);
        fz[i] = T(0.0);
        return;
    }
    int x0 = (int)cx, y0 = (int)cy, z0 = (int)cz;
    int x1 = x0 + 1, y1 = y0 + 1, z1 = z0 + 1;
    T d_x = cx - x0, d_y = cy - y0, d_z = cz - z0;
    T t_x = T(1.0) - d_x, t_y = T(1.0) - d_y, t_z = T(1.0) - d_z;
    const long long off = (i < protons) ? 0 : g.G;
    const long long sx = (long long)ny * nz, sy = nz;
    T ax = T(0.0), ay = T(0.0), az = T(0.0);
    auto acc = [&](int a, int b, int c, T w) {
        long long id = a * sx + b * sy + c + off;
        ax += w * Fx[id];
        ay += w * Fy[id];
        az += w * Fz[id];
    };
    acc(x0, y0, z0, t_x * t_y * t_z);
    if (x1 < nx) acc(x1, y0, z0, d_x * t_y * t_z);
    if (y1 < ny) acc(x0, y1, z0, t_x * d_y * t_z);
    if (x1 < nx && y1 < ny) acc(x1, y1, z0, d_x * d_y * t_z);
    if (z1 < nz) acc(x0, y0, z1, t_x * t_y * d_z);
    if (x1 < nx && z1 < nz) acc(x1, y0, z1, d_x * t_y * d_z);
    if (y1 < ny && z1 < nz) acc(x0, y1, z1, t_x * d_y * d_z);
    if (x1 < nx && y1 < ny && z1 < nz) acc(x1, y1, z1, d_x * d_y * d_z);
    fx[i] = ax;
    fy[i] = ay;
    fz[i] = az;
}

// update_momenta_half / update_positions_full (include/physics.hpp:248-270):
// a += fact * b on three arrays.
template <typename T>
__global__ void k_axpy3(int total, T fact, T *a0, T *a1, T *a2, const T *__restrict__ b0,
                        const T *__restrict__ b1, const T *__restrict__ b2) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    a0[i] += fact * b0[i];
    a1[i] += fact * b1[i];
    a2[i] += fact * b2[i];
}

// nuclear_excitation (include/physics.hpp:236-246)
template <typename T>
__global__ void k_excite(int protons, int total, T dp, T dn, T *kz) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    if (i < protons) kz[i] += dp;
    else kz[i] -= dn;
}

// center_of_mass / mean_squared_radius partials (include/tools.hpp:302-338):
// per block {sum z_p, sum z_n, sum r2_p, sum r2_n, n_in_p, n_in_n}.
template <typename T>
__global__ void k_observe_partials(Geom g, int protons, int total, const T *__restrict__ x,
                                   const T *__restrict__ y, const T *__restrict__ z, double *partials) {
    double v[6] = {0, 0, 0, 0, 0, 0};
    const T dmx = T(g.dmx), dmy = T(g.dmy), dmz = T(g.dmz);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        int s = i < protons ? 0 : 1;
        T xi = x[i], yi = y[i], zi = z[i];
        v[s] += (double)zi;
        if (xi < -dmx || xi > +dmx || yi < -dmy || yi > +dmy || zi < -dmz || zi > +dmz) continue;
        T r2 = xi * xi + yi * yi + zi * zi;
        v[2 + s] += (double)r2;
        v[4 + s] += 1.0;
    }
    __shared__ double sh[6][kBlock];
    for (int c = 0; c < 6; c++) sh[c][threadIdx.x] = v[c];
    __syncthreads();
    for (int o = kBlock / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o)
            for (int c = 0; c < 6; c++) sh[c][threadIdx.x] += sh[c][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x < 6) partials[6 * blockIdx.x + threadIdx.x] = sh[threadIdx.x][0];
}

inline int blocks_for(long long n) { return div_up(n > 0 ? n : 1, kBlock); }

}  // namespace

// ======================= launchers ========================================

template <typename T>
hv_status launch_deposit_atomic(hv_ctx *c, const T *x, const T *y, const T *z, T *rho) {
    HV_CUDA(cudaMemsetAsync(rho, 0, sizeof(T) * 2 * c->geom.G, c->stream));
    if (c->total > 0)
        k_deposit_atomic<T><<<blocks_for(c->total), kBlock, 0, c->stream>>>(c->geom, c->protons, c->total, x, y, z, rho);
    HV_CUDA(cudaGetLastError());
    return HV_OK;
}

template <typename T>
hv_status launch_deposit_sorted(hv_ctx *c, const T *x, const T *y, const T *z, T *rho) {
    const long long ncell = 2 * c->geom.G;
    Scratch &s = c->scratch;
    if (c->total == 0) {
        HV_CUDA(cudaMemsetAsync(rho, 0, sizeof(T) * ncell, c->stream));
        return HV_OK;
    }
    k_cell_keys<T><<<blocks_for(c->total), kBlock, 0, c->stream>>>(c->geom, c->protons, c->total, x, y, z, s.keys, s.vals);
    HV_CUDA(cudaGetLastError());
    int end_bit = 1;
    while ((1ull << end_bit) <= (unsigned long long)ncell) end_bit++;
    size_t bytes = s.cub_tmp_bytes;
    HV_CUDA(cub::DeviceRadixSort::SortPairs(s.cub_tmp, bytes, s.keys, s.keys_alt, s.vals, s.vals_alt,
                                            c->total, 0, end_bit, c->stream));
    HV_CUDA(cudaMemsetAsync(s.cell_start, 0xff, sizeof(int) * (size_t)ncell, c->stream));
    Entry<T> *ent = static_cast<Entry<T> *>(s.entries);
    const SortedParticles<T> part{x, y, z, s.keys_alt, s.vals_alt, c->total};
    k_deposit_entries<T><<<blocks_for(c->total), kBlock, 0, c->stream>>>(c->geom, part, s.cell_start, ent);
    HV_CUDA(cudaGetLastError());
    const Geom &g = c->geom;
    const int zt = std::min(128, (g.nz + 31) / 32 * 32);
    const dim3 grid((g.nz + zt - 1) / zt, g.ny, 2 * g.nx);
    auto *merge = c->total > kMaxIndex32 ? (ent ? k_deposit_merge<T, unsigned long long, true>
                                                : k_deposit_merge<T, unsigned long long, false>)
                  : ent                  ? k_deposit_merge<T, unsigned, true>
                                         : k_deposit_merge<T, unsigned, false>;
    merge<<<grid, zt, 0, c->stream>>>(g, ent, s.cell_start, s.vals_alt, part, rho);
    HV_CUDA(cudaGetLastError());
    return HV_OK;
}

// Bytes of the sorted deposit's entries.
size_t sorted_deposit_entry_bytes(int total, hv_precision prec) {
    return (size_t)total * (prec == HV_F64 ? sizeof(Entry<double>) : sizeof(Entry<float>));
}

// Bytes of CUB temporary storage for a sort of `total` keys.
size_t sorted_deposit_tmp_bytes(int total) {
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairs((void *)nullptr, bytes, (unsigned int *)nullptr, (unsigned int *)nullptr,
                                    (int *)nullptr, (int *)nullptr, total > 0 ? total : 1, 0, 32);
    return bytes;
}

template <typename T>
hv_status launch_smooth(hv_ctx *c, const T *rho_raw, T *rho) {
    const hv_run_params &p = c->params;
    // normalisation term in T, evaluated as the reference does (physics.hpp:229)
    const T sig = T(p.sigma_r);
    const T term = (T(1.0) / p.part_per_nucleon) *
                   (T(1.0) / std::pow(T(2.0) * T(kPi) * sig * sig, T(1.5)));
    const T *w = reinterpret_cast<const T *>(sizeof(T) == 8 ? (void *)c->d64.taps_w : (void *)c->d32.taps_w);
    // staged rows where a block's slab fits in the default shared memory (z
    // rows of at most 512 nodes and stencils of up to ~12 nodes at 128^3 in
    // double), else tap by tap
    const Geom &g = c->geom;
    const int *lim = c->taps.lim;
    RowTile rt;
    rt.qz = (g.nz + 3) / 4;
    rt.ty = std::max(1, std::min(kRowThreads / rt.qz, g.ny));
    rt.pitch = (4 * rt.qz + 2 * lim[2] + 3) / 4 + 1;
    rt.words = (rt.ty + 2 * lim[1]) * 4 * rt.pitch;
    rt.wmax = (2 * lim[1] + 1) * (2 * lim[2] + 1);
    const size_t smem = sizeof(T) * (size_t)(rt.words + rt.wmax);
    if (rt.qz <= kRowThreads && smem <= 48 * 1024 && c->taps.runs > 0 && c->taps_runs) {
        k_smooth_rows<T><<<dim3((g.ny + rt.ty - 1) / rt.ty, g.nx, 2), kRowThreads, smem, c->stream>>>(
            g, rt, lim[0], lim[1], lim[2], c->taps.runs, c->taps_runs, w, term, rho_raw, rho);
        HV_CUDA(cudaGetLastError());
        return HV_OK;
    }
    k_smooth_direct<T><<<blocks_for(2 * c->geom.G), kBlock, 0, c->stream>>>(
        c->geom, c->taps_count, c->taps.lim[0], c->taps.lim[1], c->taps.lim[2], c->taps_dev, w, term, rho_raw, rho);
    HV_CUDA(cudaGetLastError());
    return HV_OK;
}

template <typename T>
hv_status launch_skyrme(hv_ctx *c, const T *rho, T *U) {
    const hv_skyrme &s = c->params.skyrme;
    k_skyrme<T><<<blocks_for(c->geom.G), kBlock, 0, c->stream>>>(c->geom.G, T(s.A), T(s.B), T(s.C), T(s.gamma), rho, U);
    HV_CUDA(cudaGetLastError());
    return HV_OK;
}

template <typename T>
hv_status launch_boundary(hv_ctx *c, T *phi) {
    k_boundary<T, T><<<blocks_for(c->geom.G), kBlock, 0, c->stream>>>(c->geom, c->params.z, phi);
    HV_CUDA(cudaGetLastError());
    return HV_OK;
}

// How the solver's quotients by h^2 are formed (stencil_sum's kDiv): a power of
// two divides exactly by its reciprocal; Markstein's form in double, where h^2
// and its reciprocal are far inside the range.
template <typename T>
static int division_form(const PlainSor<T> &a) {
    int ex;
    auto pow2 = [&](T v) { return std::frexp(v, &ex) == T(0.5); };
    auto mid = [](T v) { return v >= T(1e-20) && v <= T(1e20); };
    if (pow2(a.hx2) && pow2(a.hy2) && pow2(a.hz2)) return 1;
    return sizeof(T) == 8 && mid(a.hx2) && mid(a.hy2) && mid(a.hz2) ? 2 : 0;
}

// Launches the cluster form where it is the faster one: up to three points of a
// colour a thread (about 48^3).  Per half sweep it takes 1.7 us and 0.66 a
// point, the grid form 3.1 and 0.2 (32^3: 2.3 against 3.3, 64^3: 6.6 against 4.5).
template <typename T>
static hv_status sor_cluster_launch(hv_ctx *c, const PlainSor<T> &a, int div, bool *launched) {
    *launched = false;
    const int ranks = kSorRanks, P = (a.nx - 2 + ranks - 1) / ranks;
    const size_t smem = sizeof(T) * (size_t)P * a.ny * 2 * ((a.nz + 1) / 2);
    if (smem > kSorClusterSmem || (long long)P * (a.ny - 2) * a.half > 3 * kClusterThreads) return HV_OK;
    const void *k = div == 1   ? (const void *)k_sor_cluster<T, 1>
                    : div == 2 ? (const void *)k_sor_cluster<T, 2>
                               : (const void *)k_sor_cluster<T, 0>;
    HV_TRY(allow_max_dynamic_smem(k, c->device));
    HV_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ranks);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ranks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) != cudaSuccess || clusters < 1) {
        cudaGetLastError();
        return HV_OK;
    }
    PlainSor<T> arg = a;
    int arg_ranks = ranks, arg_P = P;
    void *args[] = {&arg, &arg_ranks, &arg_P};
    HV_CUDA(cudaLaunchKernelExC(&cfg, k, args));
    *launched = true;
    return HV_OK;
}

template <typename T>
hv_status launch_sor_plain(hv_ctx *c, T *phi, const T *rho, int *iters, double *metric) {
    const Geom &g = c->geom;
    const hv_sor_params &sp = c->params.sor;
    const T dx = T(2.0) * T(g.dmx) / g.nx, dy = T(2.0) * T(g.dmy) / g.ny, dz = T(2.0) * T(g.dmz) / g.nz;
    const T hx2 = dx * dx, hy2 = dy * dy, hz2 = dz * dz;
    const T inv_dx2 = T(1.0) / (T(2.0) / hx2 + T(2.0) / hy2 + T(2.0) / hz2);
    // the solver's work space is the context's: the saved values lie where the
    // sorted deposit keeps its cells' first particles (2 G + 1 ints, written
    // anew by every deposit), the partial results and the barrier among the
    // reductions' words
    Scratch &sc = c->scratch;
    PlainSor<T> a;
    a.nx = g.nx;
    a.ny = g.ny;
    a.nz = g.nz;
    a.half = (g.nz - 1) / 2;  // upper bound of colour points per (i, j) line
    a.count = (int)((long long)(g.nx - 2) * (g.ny - 2) * a.half);
    a.omega = T(sp.omega);
    a.inv_dx2 = inv_dx2;
    a.hx2 = hx2;
    a.hy2 = hy2;
    a.hz2 = hz2;
    a.src_c = T(4.0) * T(kPi) * T(1.44);
    a.tol_t = T(sp.tol);
    a.tol = sp.tol;
    // residual in double from double spacings
    const double ddx = 2.0 * g.dmx / g.nx, ddy = 2.0 * g.dmy / g.ny, ddz = 2.0 * g.dmz / g.nz;
    a.ix2 = 1.0 / (ddx * ddx);
    a.iy2 = 1.0 / (ddy * ddy);
    a.iz2 = 1.0 / (ddz * ddz);
    a.diag = 2.0 * a.ix2 + 2.0 * a.iy2 + 2.0 * a.iz2;
    a.bsrc = 4.0 * kPi * 1.44;
    a.criterion = sp.criterion;
    a.max_iter = sp.max_iter;
    a.rx = T(1.0) / hx2;
    a.ry = T(1.0) / hy2;
    a.rz = T(1.0) / hz2;
    // a thread per colour point up to one block per SM
    a.nblocks = std::min(c->sm_count, std::max(1, div_up(a.count, kSorBlock)));
    a.max_spin = kDefaultSpin;
    a.phi = phi;
    a.saved = reinterpret_cast<T *>(sc.cell_start);
    a.rho = rho;
    a.partials = sc.partials;  // 32 doubles per SM and more
    a.bar = reinterpret_cast<unsigned *>(sc.result + 56);
    a.status = reinterpret_cast<int *>(a.bar + 2);
    a.metric = reinterpret_cast<double *>(a.bar + 8);
    HV_CUDA(cudaMemsetAsync(a.bar, 0, 64, c->stream));
    bool launched = false;
    const int div = division_form(a);
    HV_TRY(sor_cluster_launch<T>(c, a, div, &launched));
    if (!launched) {
        void *args[] = {&a};
        const void *k = div == 1   ? (const void *)k_sor_plain<T, 1>
                        : div == 2 ? (const void *)k_sor_plain<T, 2>
                                   : (const void *)k_sor_plain<T, 0>;
        HV_CUDA(cudaLaunchCooperativeKernel(k, dim3(a.nblocks), dim3(kSorBlock), args, 0, c->stream));
    }
    HV_CUDA(cudaMemcpyAsync(sc.h_result, a.bar, 64, cudaMemcpyDeviceToHost, c->stream));
    HV_CUDA(cudaStreamSynchronize(c->stream));
    const int *st = reinterpret_cast<const int *>(sc.h_result) + 2;
    if (st[0]) {
        set_last_error("SOR: a bounded device-side wait timed out");
        return HV_ERR_TIMEOUT;
    }
    if (iters) *iters = st[1];
    if (metric) *metric = sc.h_result[4];
    return st[2] == 1 ? HV_OK : st[2] == 2 ? HV_ERR_NONFINITE : HV_ERR_NOT_CONVERGED;
}

template <typename T>
hv_status launch_merge(hv_ctx *c, T *U, const T *phi) {
    k_merge<T><<<blocks_for(c->geom.G), kBlock, 0, c->stream>>>(c->geom.G, U, phi);
    HV_CUDA(cudaGetLastError());
    return HV_OK;
}

template <typename T>
hv_status launch_fdm(hv_ctx *c, const T *U, T *Fx, T *Fy, T *Fz) {
    const Geom &g = c->geom;
    const T dx = T(2.0) * T(g.dmx) / g.nx, dy = T(2.0) * T(g.dmy) / g.ny, dz = T(2.0) * T(g.dmz) / g.nz;
    k_fdm<T><<<blocks_for(2 * g.G), kBlock, 0, c->stream>>>(g, dx, dy, dz, U, Fx, Fy, Fz);
    HV_CUDA(cudaGetLastError());
    return HV_OK;
}

template <typename T>
hv_status launch_gather(hv_ctx *c, const T *x, const T *y, const T *z, const T *Fx, const T *Fy, const T *Fz,
                        T *fx, T *fy, T *fz) {
    if (c->total == 0) return HV_OK;
    k_gather<T><<<blocks_for(c->total), kBlock, 0, c->stream>>>(c->geom, c->protons, c->total, x, y, z, Fx, Fy, Fz,
                                                               fx, fy, fz);
    HV_CUDA(cudaGetLastError());
    return HV_OK;
}

template <typename T>
hv_status launch_kick(hv_ctx *c, T *kx, T *ky, T *kz, const T *fx, const T *fy, const T *fz, double dt) {
    if (c->total == 0) return HV_OK;
    const T fact = T(dt) / (T(2.0) * T(kHbarC));  // physics.hpp:251
    k_axpy3<T><<<blocks_for(c->total), kBlock, 0, c->stream>>>(c->total, fact, kx, ky, kz, fx, fy, fz);
    HV_CUDA(cudaGetLastError());
    return HV_OK;
}

template <typename T>
hv_status launch_drift(hv_ctx *c, T *x, T *y, T *z, const T *kx, const T *ky, const T *kz, double dt) {
    if (c->total == 0) return HV_OK;
    const T fact = (T(dt) * T(kHbarC)) / T(kMc2);  // physics.hpp:263
    k_axpy3<T><<<blocks_for(c->total), kBlock, 0, c->stream>>>(c->total, fact, x, y, z, kx, ky, kz);
    HV_CUDA(cudaGetLastError());
    return HV_OK;
}

template <typename T>
hv_status launch_excite(hv_ctx *c, T *kz, double eta) {
    if (c->total == 0) return HV_OK;
    const T zz = T(c->params.z), nn = T(c->params.n), e = T(eta);
    const T dp = e * nn / (zz + nn), dn = e * zz / (zz + nn);  // physics.hpp:241,244
    k_excite<T><<<blocks_for(c->total), kBlock, 0, c->stream>>>(c->protons, c->total, dp, dn, kz);
    HV_CUDA(cudaGetLastError());
    return HV_OK;
}

template <typename T>
hv_status launch_observe(hv_ctx *c, const T *x, const T *y, const T *z, hv_observables *out) {
    const int nb = 2 * c->sm_count;
    k_observe_partials<T><<<nb, kBlock, 0, c->stream>>>(c->geom, c->protons, c->total, x, y, z, c->scratch.partials);
    k_sum_partials<<<1, 512, 0, c->stream>>>(c->scratch.partials, nb, 6, c->scratch.result);
    HV_CUDA(cudaGetLastError());
    HV_CUDA(cudaMemcpyAsync(c->scratch.h_result, c->scratch.result, 6 * sizeof(double), cudaMemcpyDeviceToHost,
                            c->stream));
    HV_CUDA(cudaStreamSynchronize(c->stream));
    const double *v = c->scratch.h_result;
    out->zcm_p = v[0] / (double)c->protons;
    out->zcm_n = v[1] / (double)c->neutrons;
    out->rms_p = std::sqrt(v[2] / v[4]);
    out->rms_n = std::sqrt(v[3] / v[5]);
    const double zz = c->params.z, nn = c->params.n;
    out->dipole = (nn * zz) / (nn + zz) * (out->zcm_p - out->zcm_n);
    return HV_OK;
}

#define HV_INST(T)                                                                                         \
    template hv_status launch_deposit_atomic<T>(hv_ctx *, const T *, const T *, const T *, T *);           \
    template hv_status launch_deposit_sorted<T>(hv_ctx *, const T *, const T *, const T *, T *);           \
    template hv_status launch_smooth<T>(hv_ctx *, const T *, T *);                                         \
    template hv_status launch_skyrme<T>(hv_ctx *, const T *, T *);                                         \
    template hv_status launch_boundary<T>(hv_ctx *, T *);                                                  \
    template hv_status launch_sor_plain<T>(hv_ctx *, T *, const T *, int *, double *);                     \
    template hv_status launch_merge<T>(hv_ctx *, T *, const T *);                                          \
    template hv_status launch_fdm<T>(hv_ctx *, const T *, T *, T *, T *);                                  \
    template hv_status launch_gather<T>(hv_ctx *, const T *, const T *, const T *, const T *, const T *,   \
                                        const T *, T *, T *, T *);                                         \
    template hv_status launch_kick<T>(hv_ctx *, T *, T *, T *, const T *, const T *, const T *, double);   \
    template hv_status launch_drift<T>(hv_ctx *, T *, T *, T *, const T *, const T *, const T *, double);  \
    template hv_status launch_excite<T>(hv_ctx *, T *, double);                                            \
    template hv_status launch_observe<T>(hv_ctx *, const T *, const T *, const T *, hv_observables *);

HV_INST(double)
HV_INST(float)

}  // namespace hv
