// Direct Coulomb solve of the fused path: every correction of the carried FP64
// residual is solved exactly on the run's own grid.
//
// The cycle is the persistent SOR's (k_sor_fast.cu): phi in double, the double
// residual r = b + lap_h phi, the stopping rule tested on it, and a correction
// delta in the context's precision with -lap_h delta = r, folded in as phi +=
// delta.  Only the way delta is found differs.  The red-black sweeps need dozens of exchanges
// between blocks per solve, each a round trip through L2; here delta comes
// from sine transforms along y and z (dense matrices, exact for every
// extent) and a tridiagonal elimination along x, so that a solve is a fixed
// four phases with a grid barrier after each:
//   A  per x plane: r (double, from the extrapolated phi), the two forward
//      transforms of the plane in shared memory
//   B  per group of (ky, kz) columns: the tridiagonal systems along x
//   C  per x plane: the two inverse transforms, delta
//   D  per x plane: phi += delta, the history rotated, |r + lap delta|^2
// and the rule is tested after A and after D.  A float correction leaves the
// residual's rounding noise, ~1e-6 of it for the rough residual of an
// extrapolated start and ~3e-4 for the smooth one of a first guess, so a step
// takes one correction and a first solve two or three.  A double one leaves
// less than any rule that lets a double context take this form.
//
// A symmetric half-length form of the transforms halves their work: row j and
// its mirror are replaced by their sum and difference, of which the odd and
// the even wavenumbers see only one.  A plane is stored as its first half, a
// gap that aligns the second half to 8 columns, and the second half; sums and
// differences take the places of the two rows they come from.
//
// Why dense transforms: the sine transform of n - 2 interior nodes has length
// 2 (n - 1), and n - 1 is odd or prime for the usual even n, so no short FFT
// applies.  The four half-length passes are n^3 / 2 multiply-adds a plane each.
//
// Measured (208Pb, one step's solve, CUDA events; the sweeps it replaces in
// brackets): 128^3 114 us (354), 64^3 41 us (227), 32^3 33 us (203), 75 x 61 x
// 50 40 us (734: such extents had no coarse-grid correction and no tagged
// exchange).  At 128^3, in thousands of cycles of one block: A walk 28 (latency
// of its loads), transforms 35 (the shared loads of their operands, not the
// multiply-adds), B 19 (its loads and the chain of eliminations), C 54, D 50
// (latency), the four barriers with the wait for the slowest block about 25.
// In double, a step's solve at a rule of 1e-10: 32^3 35 us, 64^3 59, 96^3 132,
// 128^3 229 (float corrections, two of them for such a rule: 51, 69, 139, 208).
//
// All forms spill at 128 registers a thread: 136 to 180 bytes those of planes
// up to about 150 x 150 in float, 330 and 950 with two and three tiles a warp,
// 470 to 550 in double (the two walks' operands, not the transforms').
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "grid_sync.cuh"
#include "hv_internal.h"

namespace hv {
namespace {

// Double solves take the direct form when their rule is at least this tight: it
// then pins phi far below what the way to it could show.  At looser rules the
// point where the sweeps stop is part of a double run's result, and stays.
constexpr double kDoubleTol = 1e-9;
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;

template <typename T>
struct DirectArgs {
    int nx, ny, nz, mx, my, mz;   // nodes, interior nodes
    int hy, hz;                   // first halves: (m + 1) / 2 rows or columns
    int off, wz, ps;              // second half's column, columns of a stored plane, its pitch in shared memory
    int py;                       // pitch of the y matrices
    int nblocks, cw, cpitch;      // columns of a phase-B group, their pitch
    int zlen, ylen;               // words of one z (y) matrix pair (a word: one T)
    int shared_tab, tabs;         // y matrices are the z ones; matrices in shared memory: 2 both directions,
                                  // 1 one direction at a time, 0 one axis of one direction
    int front;                    // words of shared memory before the matrices
    double dhx2i, dhy2i, dhz2i, ddiag, src_c, tol;
    T scale;                      // hx^2: the elimination's equations are scaled by it
    int max_iter, extrapolate;
    long long max_spin;
    const T *rho;
    double *phi, *prev, *guess, *resid;  // guess: the next solve's start (interior nodes)
    T *work, *delta;              // [mx][my][wz] spectrum, [nx][ny][nz] correction (zero on the faces)
    const T *wz_f, *wz_i, *wy_f, *wy_i;  // matrix pairs: forward and inverse
    const T *lamy, *lamz;         // eigenvalues times hx^2 in stored order (zero in the gaps)
    double *partials;
    unsigned *bar;
    int *status;
    double *metric;
    int *ctl, *its_ring;
    int ring;
    const DirectArgs *batch;      // several solves in one launch: block -> instance, its first block
    const int *binst, *bfirst;
};

// Four words of a row: what a thread loads, stores and holds of a plane.
template <typename T>
struct Quad;
template <>
struct Quad<float> {
    using type = float4;
};
struct __align__(16) Double4 {
    double x, y, z, w;
};
template <>
struct Quad<double> {
    using type = Double4;
};
template <typename T>
using quad = typename Quad<T>::type;

template <typename T>
__device__ __forceinline__ quad<T> ld4(const T *p) { return *reinterpret_cast<const quad<T> *>(p); }
template <typename T>
__device__ __forceinline__ void st4(T *p, const quad<T> &v) { *reinterpret_cast<quad<T> *>(p) = v; }
__device__ __forceinline__ float4 ldcg4(const float *p) { return __ldcg(reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ Double4 ldcg4(const double *p) {
    const double2 a = __ldcg(reinterpret_cast<const double2 *>(p)), b = __ldcg(reinterpret_cast<const double2 *>(p) + 1);
    return Double4{a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ void stcg4(float *p, const float4 &v) { __stcg(reinterpret_cast<float4 *>(p), v); }
__device__ __forceinline__ void stcg4(double *p, const Double4 &v) {
    __stcg(reinterpret_cast<double2 *>(p), make_double2(v.x, v.y));
    __stcg(reinterpret_cast<double2 *>(p) + 1, make_double2(v.z, v.w));
}

__device__ __forceinline__ float rcp_of(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ double rcp_of(double v) { return 1.0 / v; }

template <typename T>
__device__ __forceinline__ T lds(unsigned p) {
    if constexpr (sizeof(T) == 4) {
        float v;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(p) : "memory");
        return v;
    } else {
        double v;
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(p) : "memory");
        return v;
    }
}
__device__ __forceinline__ void sts(unsigned p, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(p), "f"(v) : "memory"); }
__device__ __forceinline__ void sts(unsigned p, double v) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(p), "d"(v) : "memory"); }

// The matrices' copy to shared memory runs under the work before their first
// use (tab_wait and a block barrier).
template <typename T>
__device__ __forceinline__ void load_tab(T *dst, const T *src, int n) {
    constexpr int kPer = 16 / sizeof(T);
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    for (int e = kPer * threadIdx.x; e < n; e += kPer * kThreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + (unsigned)sizeof(T) * e), "l"(src + e) : "memory");
}
__device__ __forceinline__ void tab_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Tile of a warp in a transform: parity (half), column groups of four and row
// groups; lanes are 8 column groups x 4 row groups, so that a warp's loads of
// the plane and of the matrix are each one 128-byte wavefront.
struct Tile {
    int par, cg, rg;
    bool on;
};
template <int RT>
__device__ __forceinline__ Tile tile_of(int wt, int CG, int RG) {
    const int CB = (CG + 7) >> 3, RB = (RG + 3) >> 2, per = CB * RB, lane = threadIdx.x & 31;
    Tile t;
    t.par = wt / per;
    const int rem = wt - t.par * per;
    t.cg = (rem % CB) * 8 + (lane & 7);
    t.rg = (rem / CB) * 4 + (lane >> 3);
    t.on = t.par < 2 && t.cg < CG && t.rg < RG;
    if (!t.on) t.par = t.cg = t.rg = 0;
    return t;
}

// plane := plane x W along z, in place (the results wait in registers for the
// whole block to have read its operands).  Thread tile: rows rg + RG i, four
// columns; 12 shared loads of 16 bytes per 4 x 32 multiply-adds (RT = 8).
template <typename T, int RT, int NT>
__device__ __forceinline__ void transform_z(const DirectArgs<T> &a, T *P, const T *W) {
    const int RG = (a.my + RT - 1) / RT, CG = a.off / 4, warp = threadIdx.x >> 5, ps = a.ps;
    const int k1 = a.wz - a.off;
    T acc[NT][RT][4];
    Tile t[NT];
#pragma unroll
    for (int n = 0; n < NT; n++) {
        t[n] = tile_of<RT>(warp + n * kWarps, CG, RG);
        if (t[n].par && 4 * t[n].cg >= k1) t[n].on = false, t[n].cg = 0;
#pragma unroll
        for (int i = 0; i < RT; i++) acc[n][i][0] = acc[n][i][1] = acc[n][i][2] = acc[n][i][3] = T(0);
        if (!__any_sync(0xffffffffu, t[n].on)) continue;
        const T *w = W + t[n].par * a.off * a.off + 4 * t[n].cg;
        const T *p = P + t[n].rg * ps + t[n].par * a.off;
        const int K = t[n].par ? k1 : a.off;
        for (int k = 0; k < K; k += 4) {
            quad<T> v[RT];
#pragma unroll
            for (int i = 0; i < RT; i++) v[i] = ld4(p + RG * i * ps + k);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const quad<T> m = ld4(w + (k + q) * a.off);
#pragma unroll
                for (int i = 0; i < RT; i++) {
                    const T s = q == 0 ? v[i].x : q == 1 ? v[i].y : q == 2 ? v[i].z : v[i].w;
                    acc[n][i][0] = fma(s, m.x, acc[n][i][0]);
                    acc[n][i][1] = fma(s, m.y, acc[n][i][1]);
                    acc[n][i][2] = fma(s, m.z, acc[n][i][2]);
                    acc[n][i][3] = fma(s, m.w, acc[n][i][3]);
                }
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < NT; n++) {
        if (!t[n].on) continue;
#pragma unroll
        for (int i = 0; i < RT; i++) {
            const int r = t[n].rg + RG * i;
            if (r < a.my)
                st4(P + r * ps + t[n].par * a.off + 4 * t[n].cg,
                    quad<T>{acc[n][i][0], acc[n][i][1], acc[n][i][2], acc[n][i][3]});
        }
    }
    __syncthreads();
}

// plane := W^T x plane along y: rows kk0 + i of a half from its nk rows.
// `out` (pitch op) receives the plane; in place after a barrier when it is P.
template <typename T, int RT, int NT>
__device__ __forceinline__ void transform_y(const DirectArgs<T> &a, const T *P, const T *W, T *out, int op,
                                            bool in_place) {
    const int RG = (a.hy + RT - 1) / RT, CG = a.wz / 4, warp = threadIdx.x >> 5, ps = a.ps;
    T acc[NT][RT][4];
    Tile t[NT];
#pragma unroll
    for (int n = 0; n < NT; n++) {
        t[n] = tile_of<RT>(warp + n * kWarps, CG, RG);
#pragma unroll
        for (int i = 0; i < RT; i++) acc[n][i][0] = acc[n][i][1] = acc[n][i][2] = acc[n][i][3] = T(0);
        if (!__any_sync(0xffffffffu, t[n].on)) continue;
        const int nk = t[n].par ? a.my - a.hy : a.hy;
        const T *w = W + t[n].par * a.py * a.py + t[n].rg * RT;
        const T *p = P + t[n].par * a.hy * ps + 4 * t[n].cg;
#pragma unroll 4
        for (int k = 0; k < nk; k++) {
            const quad<T> v = ld4(p + k * ps);
            T m[RT];
#pragma unroll
            for (int i = 0; i < RT; i += 4)
                *reinterpret_cast<quad<T> *>(m + i) = ld4(w + k * a.py + i);
#pragma unroll
            for (int i = 0; i < RT; i++) {
                acc[n][i][0] = fma(m[i], v.x, acc[n][i][0]);
                acc[n][i][1] = fma(m[i], v.y, acc[n][i][1]);
                acc[n][i][2] = fma(m[i], v.z, acc[n][i][2]);
                acc[n][i][3] = fma(m[i], v.w, acc[n][i][3]);
            }
        }
    }
    if (in_place) __syncthreads();
#pragma unroll
    for (int n = 0; n < NT; n++) {
        if (!t[n].on) continue;
        const int nk = t[n].par ? a.my - a.hy : a.hy;
#pragma unroll
        for (int i = 0; i < RT; i++) {
            const int kk = t[n].rg * RT + i;
            if (kk < nk)
                st4(out + (size_t)(t[n].par * a.hy + kk) * op + 4 * t[n].cg,
                    quad<T>{acc[n][i][0], acc[n][i][1], acc[n][i][2], acc[n][i][3]});
        }
    }
    __syncthreads();
}

// Sums and differences of mirrored columns (rows), in the places of the pair.
template <typename T>
__device__ __forceinline__ void butterfly_z(const DirectArgs<T> &a, T *P) {
    const int ha = a.mz - a.hz;
    for (int r = threadIdx.x >> 5; r < a.my; r += kWarps)
        for (int j = threadIdx.x & 31; j < ha; j += 32) {
            T *u = P + r * a.ps + j, *v = P + r * a.ps + a.off + ha - 1 - j;
            const T s = *u, d = *v;
            *u = s + d;
            *v = s - d;
        }
    __syncthreads();
}
template <typename T>
__device__ __forceinline__ void butterfly_y(const DirectArgs<T> &a, T *P) {
    const int ha = a.my - a.hy;
    for (int j = threadIdx.x >> 5; j < ha; j += kWarps)
        for (int c = 4 * (threadIdx.x & 31); c < a.wz; c += 128) {
            T *u = P + j * a.ps + c, *v = P + (a.my - 1 - j) * a.ps + c;
            const quad<T> s = ld4(u), d = ld4(v);
            st4(u, quad<T>{s.x + d.x, s.y + d.y, s.z + d.z, s.w + d.w});
            st4(v, quad<T>{s.x - d.x, s.y - d.y, s.z - d.z, s.w - d.w});
        }
    __syncthreads();
}

// Walks the interior rows of x plane i, or of its part `part` of `parts`: each
// warp takes 32 consecutive z of a run of y rows, kU rows at a time.  load(id, interior) is the field whose
// 7-point stencil is formed: its y neighbours roll through registers, its z
// neighbours come from the lanes (the edge lanes load theirs), its x
// neighbours are loaded.  pre(id) reads what use() needs besides at a node.
// All loads of the kU rows are issued before anything is used or stored: the
// walk is bound by the latency of its loads.
template <int kU, typename T, typename Load, typename Pre, typename Use>
__device__ __forceinline__ void walk_plane(const DirectArgs<T> &a, int i, int part, int parts, Load load, Pre pre,
                                           Use use) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nchunk = (a.mz + 31) >> 5, nseg = max(1, kWarps / nchunk);
    const int first = part * a.my / parts, last = (part + 1) * a.my / parts, rows = (last - first + nseg - 1) / nseg;
    const long long sx = (long long)a.ny * a.nz;
    const bool xm_in = i > 1, xp_in = i < a.nx - 2;
    for (int item = warp; item < nchunk * nseg; item += kWarps) {
        const int ch = item % nchunk, sg = item / nchunk;
        const int y0 = 1 + first + sg * rows, y1 = min(y0 + rows, 1 + last);
        if (y0 >= y1) continue;
        const int z0 = 1 + 32 * ch, zr = z0 + lane, z = min(zr, a.nz - 1);
        const bool zin = zr <= a.nz - 2;
        // the node past the lane's end of the run (z0 - 1 or z0 + 32)
        const bool edge = lane == 0 || (lane == 31 && zr + 1 <= a.nz - 1);
        const int ze = lane == 0 ? z0 - 1 : min(zr + 1, a.nz - 1);
        const bool ze_in = ze >= 1 && ze <= a.nz - 2;
        long long id = i * sx + (long long)y0 * a.nz + z, ide = i * sx + (long long)y0 * a.nz + ze;
        auto ym = load(id - a.nz, zin && y0 > 1), c = load(id, zin);
        using V = decltype(c);
        for (int y = y0; y < y1; y += kU) {
            V yn[kU], xm[kU], xp[kU], e[kU];
            decltype(pre(id)) n[kU];
#pragma unroll
            for (int u = 0; u < kU; u++) {
                // rows past the run's end repeat its last one
                const int q = min(u, y1 - 1 - y), d = q * a.nz;
                yn[u] = load(id + d + a.nz, zin && y + q + 1 <= a.ny - 2);
                xm[u] = load(id + d - sx, xm_in && zin);
                xp[u] = load(id + d + sx, xp_in && zin);
                n[u] = pre(id + d);
                e[u] = V(0);
                if (edge) e[u] = load(ide + d, ze_in);
            }
#pragma unroll
            for (int u = 0; u < kU; u++) {
                const V up = __shfl_up_sync(0xffffffffu, c, 1), dn = __shfl_down_sync(0xffffffffu, c, 1);
                if (zin && y + u < y1)
                    use(id + u * a.nz, y + u, zr, c, (double)xm[u] + (double)xp[u], (double)ym + (double)yn[u],
                        (double)(lane == 0 ? e[u] : up) + (double)(lane == 31 ? e[u] : dn), n[u]);
                ym = c;
                c = yn[u];
            }
            id += kU * a.nz;
            ide += kU * a.nz;
        }
    }
}

// Phase B: the systems (2 + l) x_i - x_(i-1) - x_(i+1) = f_i of a group of
// columns, l the column's hx^2 (lam_y + lam_z).  Elimination from both ends
// towards the middle by two half-warps (the coefficients c_i = 1 / (2 + l -
// c_(i-1)) are the same from either end), then substitution outwards.  e = 1 -
// c is carried instead of c, e' = (l + e) / (1 + l + e): all terms positive,
// so the smooth columns (l ~ 1e-3) keep full relative accuracy.  Bound by the
// serial chain, mx / 2 steps of an add, a reciprocal and two products.
template <typename T>
__device__ __forceinline__ void solve_columns(const DirectArgs<T> &a, T *sm, int group) {
    const int ncol = a.my * a.wz, c0 = group * a.cw, n = min(a.cw, ncol - c0), mx = a.mx, pitch = a.cpitch;
    T *f = sm, *cc = sm + (size_t)mx * pitch;
    const int quads = n >> 2, xs = kThreads / quads, xq = threadIdx.x / quads, q4 = 4 * (threadIdx.x - xq * quads);
    T *const g = a.work + c0 + q4;
    constexpr int kU = 8;  // rows in flight per thread
    for (int x = xq < xs ? xq : mx; x < mx; x += kU * xs) {
        quad<T> v[kU];
#pragma unroll
        for (int u = 0; u < kU; u++)
            if (x + u * xs < mx) v[u] = ldcg4(g + (size_t)(x + u * xs) * ncol);
#pragma unroll
        for (int u = 0; u < kU; u++)
            if (x + u * xs < mx) st4(f + (x + u * xs) * pitch + q4, v[u]);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, col = (threadIdx.x >> 5) * 16 + (lane & 15), side = lane >> 4;
    const int h = mx >> 1;
    if ((threadIdx.x >> 5) * 16 < n) {
        // columns past the group's end (n is a multiple of four) run on what
        // their place holds; nothing reads their results
        const int gcol = c0 + min(col, n - 1), ky = gcol / a.wz;
        const T l = __ldg(a.lamy + ky) + __ldg(a.lamz + gcol - ky * a.wz);
        // byte addresses in shared memory: the column's rows from this side's
        // end, and its coefficients
        const int pb = (int)sizeof(T) * pitch, step = side ? -pb : pb;
        unsigned fp = (unsigned)__cvta_generic_to_shared(f + col + (side ? (mx - 1) * pitch : 0));
        unsigned cp = (unsigned)__cvta_generic_to_shared(cc + col);
        T e = T(1), y = T(0), rc = T(0);
        auto forward = [&](T fv) {
            const T t = l + e;
            rc = rcp_of(T(1) + t);
            e = t * rc;
            y = (fv + y) * rc;
            sts(fp, y);
            sts(cp, rc);  // both sides write the column's one coefficient
            fp += step;
            cp += pb;
        };
        int i = 0;
        for (; i + 4 <= h; i += 4) {
            const T f0 = lds<T>(fp), f1 = lds<T>(fp + step), f2 = lds<T>(fp + 2 * step), f3 = lds<T>(fp + 3 * step);
            forward(f0);
            forward(f1);
            forward(f2);
            forward(f3);
        }
        for (; i < h; i++) forward(lds<T>(fp));
        const T other = __shfl_xor_sync(0xffffffffu, y, 16);
        T x;
        if (mx & 1) {
            // the middle node, between the two sides' last ones: their sum
            // first, so that both sides form the same bits, and one of them
            // stores it (y and other change places between the sides)
            x = (lds<T>(fp) + (y + other)) / (l + T(2) * e);
            __syncwarp();
            if (!side) sts(fp, x);
        } else {
            // the other side's last node: x_other = (y_other + c y) / (1 - c^2)
            x = (other + rc * y) / (e * (T(1) + rc));
        }
        __syncwarp();
        auto back = [&](T cv, T yv) {
            x = fma(cv, x, yv);
            fp -= step;
            sts(fp, x);
        };
        for (; i >= 4; i -= 4) {
            const T c3 = lds<T>(cp - pb), c2 = lds<T>(cp - 2 * pb), c1 = lds<T>(cp - 3 * pb), c0v = lds<T>(cp - 4 * pb);
            const T y3 = lds<T>(fp - step), y2 = lds<T>(fp - 2 * step), y1 = lds<T>(fp - 3 * step), y0 = lds<T>(fp - 4 * step);
            back(c3, y3);
            back(c2, y2);
            back(c1, y1);
            back(c0v, y0);
            cp -= 4 * pb;
        }
        for (; i > 0; i--) {
            back(lds<T>(cp - pb), lds<T>(fp - step));
            cp -= pb;
        }
    }
    __syncthreads();
    for (int x = xq < xs ? xq : mx; x < mx; x += xs)
        stcg4(g + (size_t)x * ncol, ld4(f + x * pitch + q4));
    __syncthreads();
}

// What the last phase reads at a node: the residual, the solve's start, phi
// and the solution before it.
struct Node {
    double r, start, phi, prev;
};

template <typename T, int RT, int NT>
__device__ __forceinline__ void direct_body(const DirectArgs<T> &a, const int b) {
    extern __shared__ __align__(16) unsigned char direct_smem[];
    T *sm = reinterpret_cast<T *>(direct_smem);
    __shared__ double s_tot[2];
    const int tid = threadIdx.x;
    int *err = a.status;
    // shared memory: plane | z matrices | y matrices (| the inverse ones).
    // Phase B's columns lie where the plane lies; matrices that do not fit
    // beside them are loaded anew by each phase
    T *P = sm, *tz = sm + a.front;
    // (one axis at a time: the y matrices replace the z ones between the two
    // transforms of every plane)
    constexpr bool kOneAxis = sizeof(T) == 8;
    const bool one_axis = kOneAxis && a.tabs == 0;
    T *ty = a.shared_tab || one_axis ? tz : tz + a.zlen;
    const int one = a.zlen + (a.shared_tab ? 0 : a.ylen);
    T *tzi = a.tabs == 2 ? tz + one : tz, *tyi = a.tabs == 2 ? ty + one : ty;
    const int step = a.ctl[0];
    const int hist = a.extrapolate ? a.ctl[2] : 0;
    const long long sx = (long long)a.ny * a.nz;
    auto lap = [&](double xs, double ys, double zs, T c) {
        return xs * a.dhx2i + ys * a.dhy2i + zs * a.dhz2i - a.ddiag * (double)c;
    };

    auto load_dir = [&](bool inverse) {
        if (a.tabs != 1) return;
        load_tab(tz, inverse ? a.wz_i : a.wz_f, a.zlen);
        if (!a.shared_tab) load_tab(ty, inverse ? a.wy_i : a.wy_f, a.ylen);
    };
    auto load_y = [&](bool inverse) {
        if (one_axis) load_tab(tz, inverse ? a.wy_i : a.wy_f, a.ylen);
    };
    auto wait_y = [&]() {
        if (!one_axis) return;
        tab_wait();
        __syncthreads();
    };
    if (a.tabs == 2) {
        load_tab(tz, a.wz_f, a.zlen);
        load_tab(tzi, a.wz_i, a.zlen);
        if (!a.shared_tab) {
            load_tab(ty, a.wy_f, a.ylen);
            load_tab(tyi, a.wy_i, a.ylen);
        }
    }
    // the start: the extrapolation that the last solve left (none without
    // earlier solutions), the boundary values of phi on the faces
    const double *start = hist > 0 ? a.guess : a.phi;
    auto load_start = [&](long long id, bool interior) { return (interior ? start : a.phi)[id]; };
    auto load_delta = [&](long long id, bool) { return __ldcg(a.delta + id); };
    auto to_plane = [&](int y, int z, double r) {
        const int q = z - 1;
        P[(y - 1) * a.ps + (q < a.hz ? q : a.off + q - a.hz)] = (T)r * a.scale;
    };
    auto totals = [&](double &u, double &v) {
        if (tid < 32) {
            double su = 0.0, sv = 0.0;
            for (int q = tid; q < a.nblocks; q += 32) {
                su += __ldcg(a.partials + 2 * q);
                sv += __ldcg(a.partials + 2 * q + 1);
            }
            for (int o = 16; o > 0; o >>= 1) {
                su += __shfl_xor_sync(0xffffffffu, su, o);
                sv += __shfl_xor_sync(0xffffffffu, sv, o);
            }
            if (tid == 0) {
                s_tot[0] = su;
                s_tot[1] = sv;
            }
        }
        __syncthreads();
        u = s_tot[0];
        v = s_tot[1];
    };
    // The first correction of a solve: phi := v, the solution before it moves
    // to prev, and the next solve's start is extrapolated in time while all its
    // terms are at hand -- 3 v - 3 phi + prev, or 2 v - phi while only one
    // earlier solution is held (a cubic guess measured worse: it amplifies the
    // step-to-step particle noise).  Reading that one field in the next solve's
    // stencil instead of three moves 36 bytes a node fewer.
    auto store_first = [&](long long id, double v, double phi, double prev) {
        if (a.extrapolate) {
            a.guess[id] = a.extrapolate == 2 && hist > 0 ? 3.0 * (v - phi) + prev : 2.0 * v - phi;
            a.prev[id] = phi;
        }
        a.phi[id] = v;
    };
    // a later one adds its share of the extrapolation too
    const double again = a.extrapolate == 2 && hist > 0 ? 3.0 : 2.0;

    unsigned target = epoch_base(a.bar);
    int its = 0;
    double rel = 0.0, bsum = 0.0;
    bool converged = false;
    while (true) {
        // ---- A: residual of the plane and its forward transforms -----------
        double rr = 0.0, bb = 0.0;
        load_dir(false);
        // the stored plane's gaps are zero and stay so until phase B
        const int gap0 = a.off - a.hz, gaps = a.wz - a.mz;
        for (int e = tid; e < a.my * gaps; e += kThreads) {
            const int r = e / gaps, q = e - r * gaps;
            P[r * a.ps + (q < gap0 ? a.hz + q : a.wz - gaps + q)] = 0.0f;
        }
        for (int i = 1 + b; i <= a.mx; i += a.nblocks) {
            if (one_axis) load_tab(tz, a.wz_f, a.zlen);
            if (its == 0) {
                walk_plane<4>(
                    a, i, 0, 1, load_start, [&](long long id) { return __ldg(a.rho + id); },
                    [&](long long id, int y, int z, double c, double xs, double ys, double zs, T rho) {
                        const double bv = a.src_c * (double)rho;
                        const double r = bv + xs * a.dhx2i + ys * a.dhy2i + zs * a.dhz2i - a.ddiag * c;
                        a.resid[id] = r;
                        rr += r * r;
                        bb += bv * bv;
                        to_plane(y, z, r);
                    });
            } else {
                walk_plane<4>(
                    a, i, 0, 1, load_delta, [&](long long id) { return a.resid[id]; },
                    [&](long long id, int y, int z, T c, double xs, double ys, double zs, double r0) {
                        const double r = r0 + lap(xs, ys, zs, c);
                        a.resid[id] = r;
                        to_plane(y, z, r);
                    });
            }
            tab_wait();
            __syncthreads();
            butterfly_z(a, P);
            transform_z<T, RT, NT>(a, P, tz);
            load_y(false);
            butterfly_y(a, P);
            wait_y();
            transform_y<T, RT, NT>(a, P, ty, a.work + (size_t)(i - 1) * a.my * a.wz, a.wz, false);
        }
        if (its == 0) {
            block_sum2(rr, bb);
            if (tid == 0) {
                a.partials[2 * b] = rr;
                a.partials[2 * b + 1] = bb;
            }
        }
        if (!epoch_barrier(a.bar, target, a.nblocks, err, a.max_spin)) return;
        if (its == 0) {
            double u;
            totals(u, bsum);
            rel = bsum > 0.0 ? sqrt(u / bsum) : sqrt(u);
            converged = rel <= a.tol;
            if (converged || !(rel == rel)) {
                for (int i = 1 + b; i <= a.mx; i += a.nblocks)
                    for (int e = tid; e < a.my * a.mz; e += kThreads) {
                        const long long id = i * sx + (long long)(1 + e / a.mz) * a.nz + 1 + e % a.mz;
                        store_first(id, start[id], a.phi[id], a.prev[id]);
                    }
                break;
            }
        }
        // ---- B: along x -------------------------------------------------------
        const int groups = (a.my * a.wz + a.cw - 1) / a.cw;
        for (int g = b; g < groups; g += a.nblocks) solve_columns(a, sm, g);
        if (!epoch_barrier(a.bar, target, a.nblocks, err, a.max_spin)) return;
        // ---- C: inverse transforms -------------------------------------------
        load_dir(true);
        for (int i = 1 + b; i <= a.mx; i += a.nblocks) {
            if (one_axis) load_tab(tz, a.wz_i, a.zlen);
            const T *src = a.work + (size_t)(i - 1) * a.my * a.wz;
            // a row per group of lanes, eight rows in flight per thread
            const int quads = a.wz >> 2, rs = kThreads / quads, rq = tid / quads, q4 = 4 * (tid - rq * quads);
            for (int r = rq < rs ? rq : a.my; r < a.my; r += 8 * rs) {
                quad<T> v[8];
#pragma unroll
                for (int u = 0; u < 8; u++)
                    if (r + u * rs < a.my) v[u] = ldcg4(src + (r + u * rs) * a.wz + q4);
#pragma unroll
                for (int u = 0; u < 8; u++)
                    if (r + u * rs < a.my) st4(P + (r + u * rs) * a.ps + q4, v[u]);
            }
            tab_wait();
            __syncthreads();
            transform_z<T, RT, NT>(a, P, tzi);
            load_y(true);
            butterfly_z(a, P);
            wait_y();
            transform_y<T, RT, NT>(a, P, tyi, P, a.ps, true);
            const int hay = a.my - a.hy;
            for (int j = tid >> 5; j < a.hy; j += kWarps)
                for (int q = tid & 31; q < a.mz; q += 32) {
                    const int c = q < a.hz ? q : a.off + q - a.hz;
                    const T o = P[j * a.ps + c];
                    T *d = a.delta + i * sx + q + 1;
                    if (j < hay) {
                        const T e = P[(a.my - 1 - j) * a.ps + c];
                        __stcg(d + (long long)(j + 1) * a.nz, o + e);
                        __stcg(d + (long long)(a.my - j) * a.nz, o - e);
                    } else {
                        __stcg(d + (long long)(j + 1) * a.nz, o);
                    }
                }
            __syncthreads();
        }
        if (!epoch_barrier(a.bar, target, a.nblocks, err, a.max_spin)) return;
        // ---- D: phi += delta, the FP64 residual of the new phi ---------------
        rr = bb = 0.0;
        // a grid with half as many planes as blocks shares each plane out (64^3:
        // 62 planes, 124 blocks; 16 steps 1181 -> 1162 us)
        const int parts = max(1, a.nblocks / a.mx);
        for (int q = b; q < parts * a.mx; q += a.nblocks) {
            const int i = 1 + q / parts, part = q % parts;
            if (its == 0)
                walk_plane<4>(
                    a, i, part, parts, load_delta,
                    [&](long long id) { return Node{a.resid[id], start[id], a.phi[id], a.prev[id]}; },
                    [&](long long id, int, int, T c, double xs, double ys, double zs, const Node &n) {
                        const double r = n.r + lap(xs, ys, zs, c);
                        rr += r * r;
                        store_first(id, n.start + (double)c, n.phi, n.prev);
                    });
            else
                walk_plane<4>(
                    a, i, part, parts, load_delta,
                    [&](long long id) { return Node{a.resid[id], a.extrapolate ? a.guess[id] : 0.0, a.phi[id], 0.0}; },
                    [&](long long id, int, int, T c, double xs, double ys, double zs, const Node &n) {
                        const double r = n.r + lap(xs, ys, zs, c);
                        rr += r * r;
                        a.phi[id] = n.phi + (double)c;
                        if (a.extrapolate) a.guess[id] = n.start + again * (double)c;
                    });
        }
        block_sum2(rr, bb);
        if (tid == 0) a.partials[2 * b] = rr;
        if (!epoch_barrier(a.bar, target, a.nblocks, err, a.max_spin)) return;
        double u, none;
        totals(u, none);
        rel = bsum > 0.0 ? sqrt(u / bsum) : sqrt(u);
        converged = rel <= a.tol;
        its++;
        if (converged || its >= a.max_iter || !(rel == rel)) break;
    }
    if (b == 0 && tid == 0) {
        epoch_end(a.bar, target);
        a.status[1] = its;
        a.status[2] = converged ? 1 : 0;
        a.status[3] = its + 1;
        a.metric[0] = rel;
        a.ctl[1] = max(its, 1);
        // solutions held before phi; a start from phi leaves none
        a.ctl[2] = a.extrapolate ? min(a.ctl[2] + 1, 2) : 0;
        // negative where the rule was not met, also by a solve that was not
        // finite before its first correction
        if (a.its_ring) a.its_ring[step % a.ring] = converged ? its : -max(its, 1);
    }
}

// One solve, or several in one launch (kBatch): block blockIdx.x works on
// instance binst[blockIdx.x], as its block blockIdx.x - bfirst[instance].
template <typename T, int RT, int NT, bool kBatch>
__global__ void __launch_bounds__(kThreads, 1) k_poisson_direct(DirectArgs<T> p) {
    if constexpr (kBatch) {
        __shared__ DirectArgs<T> inst;
        const int q = p.binst[blockIdx.x];
        if (threadIdx.x == 0) inst = p.batch[q];
        __syncthreads();
        direct_body<T, RT, NT>(inst, (int)blockIdx.x - p.bfirst[q]);
    } else {
        direct_body<T, RT, NT>(p, (int)blockIdx.x);
    }
}

int up(int v, int q) { return (v + q - 1) / q * q; }

// The tile counts of both transforms for row tiles of RT.
int warp_tiles(const Geom &g, int off, int wz, int RT) {
    auto tiles = [](int CG, int RG) { return 2 * ((CG + 7) / 8) * ((RG + 3) / 4); };
    const int my = g.ny - 2, hy = (my + 1) / 2;
    return std::max(tiles(off / 4, (my + RT - 1) / RT), tiles(wz / 4, (hy + RT - 1) / RT));
}

// One axis' matrix pair (odd and even wavenumbers), forward [position][k] and
// inverse [k][position], in zeroed `pitch` squares.
template <typename T>
void sine_tables(int m, int pitch, T *fwd, T *inv) {
    const int h = (m + 1) / 2, ha = m - h;
    const double s = std::sqrt(2.0 / (m + 1));
    for (int par = 0; par < 2; par++)
        for (int p = 0; p < (par ? ha : h); p++)
            for (int k = 0; k < (par ? ha : h); k++) {
                const int j = par ? ha - 1 - p : p, w = 2 * k + 1 + par;
                // the argument reduced exactly before the sine
                const long long r = ((long long)(j + 1) * w) % (2ll * (m + 1));
                const T v = (T)(s * std::sin(kPi * (double)r / (m + 1)));
                fwd[((size_t)par * pitch + p) * pitch + k] = v;
                inv[((size_t)par * pitch + k) * pitch + p] = v;
            }
}

// Shared memory of a solve with nblocks blocks.  Phase B's columns, an equal
// share per block in sixteens (a half-warp each from either end; at most 256,
// all 16 warps), and their coefficients lie where the plane lies; the matrices
// follow, both directions where they fit, else over the columns.  No more is
// asked for than that: what is left of the SM's 256 KB caches the walks' loads
// (128^3: 114 us with 149 KB, 123 with 220).
struct Layout {
    bool ok;
    int cw, front, tabs;
    size_t smem;
};
Layout layout(const PoissonDirect &d, const Geom &g, int nblocks) {
    const int mx = g.nx - 2, ncol = (g.ny - 2) * d.wz;
    const size_t col = (size_t)(mx + mx / 2 + 1), plane = d.plane, one = d.one, word = d.word;
    int cw = std::min(up((ncol + nblocks - 1) / nblocks, 16), 256);
    while (cw > 16 && col * cw * word > d.limit) cw -= 16;
    auto total = [&](int w) { return (std::max(plane, col * w) + 2 * one) * word; };
    while (cw > 64 && total(cw) > d.limit) cw -= 16;
    Layout l;
    l.cw = cw;
    // the transforms wait for matrices brought in axis by axis; only a double
    // plane whose matrices of one direction do not fit takes that form
    l.tabs = total(cw) <= d.limit ? 2 : word == 4 || (plane + one) * word <= d.limit ? 1 : 0;
    l.front = (int)(l.tabs == 2 ? std::max(plane, col * cw) : plane);
    l.smem = l.tabs == 2 ? total(cw) : std::max(plane + (l.tabs ? one : (size_t)d.axis), col * cw) * word;
    l.ok = l.smem <= d.limit;
    return l;
}

template <typename T, bool kBatch>
const void *direct_kernel(int rt, int nt) {
    if constexpr (sizeof(T) == 8) {
        return nt == 1 ? (const void *)k_poisson_direct<T, 4, 1, kBatch> : (const void *)k_poisson_direct<T, 4, 2, kBatch>;
    } else {
        if (rt == 4) return (const void *)k_poisson_direct<T, 4, 1, kBatch>;
        return nt == 1   ? (const void *)k_poisson_direct<T, 8, 1, kBatch>
               : nt == 2 ? (const void *)k_poisson_direct<T, 8, 2, kBatch>
                         : (const void *)k_poisson_direct<T, 8, 3, kBatch>;
    }
}

template <typename T>
DirectArgs<T> direct_args(hv_ctx *c, const T *rho, int *ctl, int *its_ring, int ring, int nblocks) {
    const PoissonDirect &d = c->fused.direct;
    const Geom &g = c->geom;
    DirectArgs<T> a;
    std::memset(&a, 0, sizeof(a));
    a.nx = g.nx;
    a.ny = g.ny;
    a.nz = g.nz;
    a.mx = g.nx - 2;
    a.my = g.ny - 2;
    a.mz = g.nz - 2;
    a.hy = (a.my + 1) / 2;
    a.hz = (a.mz + 1) / 2;
    a.off = d.off;
    a.wz = d.wz;
    a.ps = d.ps;
    a.py = d.py;
    a.zlen = 2 * d.off * d.off;
    a.ylen = 2 * d.py * d.py;
    a.shared_tab = d.shared_tab;
    const Layout lay = layout(d, g, nblocks);
    a.tabs = lay.tabs;
    a.front = lay.front;
    a.nblocks = nblocks;
    a.cw = lay.cw;
    a.cpitch = a.cw;
    const double dx = 2.0 * g.dmx / g.nx, dy = 2.0 * g.dmy / g.ny, dz = 2.0 * g.dmz / g.nz;
    a.dhx2i = 1.0 / (dx * dx);
    a.dhy2i = 1.0 / (dy * dy);
    a.dhz2i = 1.0 / (dz * dz);
    a.ddiag = 2.0 * (a.dhx2i + a.dhy2i + a.dhz2i);
    a.src_c = 4.0 * kPi * kE2;
    a.scale = (T)(dx * dx);
    a.tol = c->params.sor.tol;
    a.max_iter = c->params.sor.max_iter;
    a.extrapolate = c->fast.sor_warm_start == HV_WARM_EXTRAPOLATE ? 1 : c->fast.sor_warm_start == HV_WARM_QUADRATIC ? 2 : 0;
    a.max_spin = c->fast.sor_wait_limit > 0 ? c->fast.sor_wait_limit : kDefaultSpin;
    a.rho = rho;
    a.phi = c->fused.phi64;
    a.prev = c->fused.phi64_prev;
    a.guess = c->fused.phi64_prev2;
    a.resid = c->fused.sor.resid;
    a.work = static_cast<T *>(d.work);
    a.delta = static_cast<T *>(d.delta);
    a.wz_f = static_cast<const T *>(d.tables);
    a.wz_i = a.wz_f + a.zlen;
    a.wy_f = a.wz_i + a.zlen;
    a.wy_i = a.wy_f + a.ylen;
    a.lamy = a.wy_i + a.ylen;
    a.lamz = a.lamy + up(a.my, 4);
    a.partials = d.partials;
    a.bar = d.bar;
    a.status = c->fused.sor.status;
    a.metric = c->fused.sor.metric;
    a.ctl = ctl;
    a.its_ring = its_ring;
    a.ring = ring;
    return a;
}

}  // namespace

namespace {

// Fills the sine matrices of z and y (both directions) and the eigenvalues
// times hx^2 in stored order, zero in the gaps.
template <typename T>
std::vector<T> direct_tables(const PoissonDirect &d, const Geom &g) {
    const int my = g.ny - 2, mz = g.nz - 2, hy = (my + 1) / 2, hz = (mz + 1) / 2;
    const size_t zlen = (size_t)2 * d.off * d.off, ylen = (size_t)2 * d.py * d.py;
    std::vector<T> all(2 * zlen + 2 * ylen + up(my, 4) + d.wz, T(0));
    T *y = all.data() + 2 * zlen, *lam = y + 2 * ylen;
    sine_tables(mz, d.off, all.data(), all.data() + zlen);
    sine_tables(my, d.py, y, y + ylen);
    const double dx = 2.0 * g.dmx / g.nx, dy = 2.0 * g.dmy / g.ny, dz = 2.0 * g.dmz / g.nz;
    auto eigen = [](int m, int w) { const double s = std::sin(kPi * w / (2.0 * (m + 1))); return 4.0 * s * s; };
    for (int r = 0; r < my; r++)
        lam[r] = (T)(eigen(my, r < hy ? 2 * r + 1 : 2 * (r - hy) + 2) * (dx * dx) / (dy * dy));
    for (int q = 0; q < mz; q++)
        lam[up(my, 4) + (q < hz ? q : d.off + q - hz)] =
            (T)(eigen(mz, q < hz ? 2 * q + 1 : 2 * (q - hz) + 2) * (dx * dx) / (dz * dz));
    return all;
}

template <typename T>
hv_status plan_direct(hv_ctx *c) {
    PoissonDirect &d = c->fused.direct;
    const Geom &g = c->geom;
    const int mx = g.nx - 2, my = g.ny - 2, mz = g.nz - 2;
    const int hy = (my + 1) / 2, hz = (mz + 1) / 2;
    constexpr bool f64 = sizeof(T) == 8;
    d.word = sizeof(T);
    d.off = up(hz, 8);
    d.wz = d.off + up(mz - hz, 4);
    d.py = up(hy, 8);
    d.ps = d.wz;
    while (d.ps % 32 != 4 && d.ps % 32 != 12 && d.ps % 32 != 20 && d.ps % 32 != 28) d.ps += 4;
    // tiles of four rows while one a warp covers the plane, else of eight; in
    // double eight rows would not fit in registers, but planes that take more
    // than two tiles of four do not fit in shared memory either
    const int nt4 = (warp_tiles(g, d.off, d.wz, 4) + kWarps - 1) / kWarps;
    d.nt8 = (warp_tiles(g, d.off, d.wz, 8) + kWarps - 1) / kWarps;
    if (f64 ? nt4 > 2 : d.nt8 > 3) return HV_OK;
    d.rt = f64 || nt4 == 1 ? 4 : 8;
    d.nt = d.rt == 4 ? nt4 : d.nt8;
    int optin = 0;
    HV_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
    const size_t plane = (size_t)up(my, 8) * d.ps, zl = (size_t)2 * d.off * d.off, yl = (size_t)2 * d.py * d.py;
    d.shared_tab = my == mz ? 1 : 0;
    const int ncol = my * d.wz;
    // one block per x plane, more where they shorten phase B
    d.nblocks = std::min(c->sm_count, std::max(mx, (ncol + 31) / 32));
    d.plane = (int)plane;
    d.one = (int)(zl + (d.shared_tab ? 0 : yl));
    d.axis = (int)std::max(zl, yl);
    d.limit = optin - 4096;  // the kernels' static shared memory
    const Layout lay = layout(d, g, d.nblocks);
    if (!lay.ok) return HV_OK;
    d.smem = lay.smem;
    const void *kernels[2] = {direct_kernel<T, false>(d.rt, d.nt), nullptr};
    if constexpr (!f64) kernels[1] = direct_kernel<T, true>(d.rt, d.nt);
    for (const void *k : kernels) {
        if (!k) continue;
        HV_TRY(allow_max_dynamic_smem(k, c->device));
        int per_sm = 0;
        HV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kThreads, d.smem));
        if (per_sm < 1) return HV_OK;
    }
    const std::vector<T> all = direct_tables<T>(d, g);
    // one allocation: the tables, the spectrum, the correction (zero on the
    // faces), the partial sums and the barrier words
    const size_t nw = (size_t)mx * ncol, np = 2 * (size_t)c->sm_count;
    const size_t at_work = (all.size() + 63) / 64 * 64, at_delta = at_work + (nw + 63) / 64 * 64;
    const size_t at_part = at_delta + ((size_t)g.G + 63) / 64 * 64;
    const size_t bytes = at_part * sizeof(T) + np * sizeof(double) + 256;
    // where that does not fit in memory, the sweeps run as they would without it
    if (cudaMalloc(&d.tables, bytes) != cudaSuccess) {
        cudaGetLastError();
        d.tables = nullptr;
        return HV_OK;
    }
    T *base = static_cast<T *>(d.tables);
    d.work = base + at_work;
    d.delta = base + at_delta;
    d.partials = reinterpret_cast<double *>(base + at_part);
    d.bar = reinterpret_cast<unsigned *>(d.partials + np);
    HV_CUDA(cudaMemsetAsync(d.delta, 0, bytes - at_delta * sizeof(T), c->stream));
    HV_CUDA(cudaMemcpyAsync(d.tables, all.data(), all.size() * sizeof(T), cudaMemcpyHostToDevice, c->stream));
    HV_CUDA(cudaStreamSynchronize(c->stream));
    d.ok = true;
    return HV_OK;
}

}  // namespace

// Plans the direct solve: it runs on every grid whose y-z plane, with the
// transforms' matrices of one direction (in double: of one axis of it), fits in
// one block's shared memory and in the registers of the forms above -- square
// planes of up to 194 x 194 nodes in float, 130 x 130 in double -- of float contexts, and of double ones with a
// rule of kDoubleTol or tighter.  The others keep the sweeps.
hv_status poisson_plan(hv_ctx *c) {
    c->fused.direct.ok = false;
    if (c->prec == HV_F32) return plan_direct<float>(c);
    return c->params.sor.tol <= kDoubleTol ? plan_direct<double>(c) : HV_OK;
}

void poisson_release(hv_ctx *c) {
    PoissonDirect &d = c->fused.direct;
    if (d.tables) cudaFree(d.tables);
    d = PoissonDirect();
}

// Whether this context's solves take the direct form: the relative-residual
// rule and the default solver options (the corrected cycles on, the tagged
// exchange not replaced by phase counters).
bool poisson_direct_runs(const hv_ctx *c) {
    return c->fused.direct.ok && c->fast.sor_coarse && c->fast.sor_exchange == HV_SOR_EXCHANGE_AUTO &&
           c->params.sor.criterion == HV_SOR_REL_RESIDUAL;
}

void poisson_tile(const hv_ctx *c, int blocks, int *planes, int *rows) {
    *planes = div_up(c->geom.nx - 2, blocks);
    *rows = c->geom.ny;
}

namespace {
template <typename T>
hv_status launch_one(hv_ctx *c, DirectArgs<T> &a) {
    const PoissonDirect &d = c->fused.direct;
    void *args[] = {&a};
    HV_CUDA(cudaLaunchCooperativeKernel(direct_kernel<T, false>(d.rt, d.nt), dim3(d.nblocks), dim3(kThreads), args,
                                        d.smem, c->stream));
    return HV_OK;
}
}  // namespace

template <typename T>
hv_status poisson_launch(hv_ctx *c, const T *rho, int *ctl, int *its_ring, int ring, bool step_solve) {
    DirectArgs<T> a = direct_args<T>(c, rho, ctl, its_ring, ring, c->fused.direct.nblocks);
    if (!step_solve) a.extrapolate = 0;
    return launch_one(c, a);
}
template hv_status poisson_launch<float>(hv_ctx *, const float *, int *, int *, int, bool);
template hv_status poisson_launch<double>(hv_ctx *, const double *, int *, int *, int, bool);

// The adjoint's transposed solve, lap mu = -4 pi e^2 src, with its own history
// and control words.
hv_status poisson_launch_adjoint(hv_ctx *c, const double *src, double *mu, double *mu_prev, double *mu_guess,
                                 int *ctl) {
    DirectArgs<double> a = direct_args<double>(c, src, ctl, nullptr, 0, c->fused.direct.nblocks);
    a.phi = mu;
    a.prev = mu_prev;
    a.guess = mu_guess;
    return launch_one(c, a);
}

// Several direct solves in one cooperative launch: the blocks of the SMs are
// shared out by the instances' work, so that they end together.
hv_status poisson_wave_build(SorWave &w, const std::vector<hv_ctx *> &cs, const std::vector<const float *> &rho,
                             const std::vector<int *> &ctl, const std::vector<int *> &its_ring, int ring,
                             std::vector<int> &blocks) {
    sor_wave_release(w);
    const int n = (int)cs.size(), sms = cs[0]->sm_count;
    if (n > sms) return HV_ERR_UNSUPPORTED;
    // time of an instance ~ planes per block x work of a plane (the walks, and
    // the transforms, as much again for 64 rows and columns)
    auto most = [&](int i) { return cs[i]->fused.direct.nblocks; };
    auto cost = [&](int i) {
        const Geom &g = cs[i]->geom;
        const double plane = (double)g.ny * g.nz * (1.0 + (g.ny + g.nz) / 128.0);
        return plane * ((g.nx - 2 + blocks[i] - 1) / blocks[i]);
    };
    blocks.assign(n, 1);
    for (int left = sms - n; left > 0;) {
        int worst = -1;
        for (int i = 0; i < n; i++)
            if (blocks[i] < most(i) && (worst < 0 || cost(i) > cost(worst))) worst = i;
        if (worst < 0) break;
        // enough blocks for one plane per block fewer, or what is left
        const int mx = cs[worst]->geom.nx - 2, per = (mx + blocks[worst] - 1) / blocks[worst];
        const int next = per > 1 ? (mx + per - 2) / (per - 1) : most(worst);
        const int add = std::min(left, std::max(1, std::min(next, most(worst)) - blocks[worst]));
        blocks[worst] += add;
        left -= add;
    }
    std::vector<DirectArgs<float>> args;
    std::vector<int> binst, bfirst(n);
    int rt = 4, nt = 1;
    size_t smem = 0;
    for (int i = 0; i < n; i++) {
        const PoissonDirect &d = cs[i]->fused.direct;
        args.push_back(direct_args<float>(cs[i], rho[i], ctl[i], its_ring[i], ring, blocks[i]));
        bfirst[i] = (int)binst.size();
        binst.insert(binst.end(), blocks[i], i);
        if (d.rt == 8) rt = 8;
        smem = std::max(smem, layout(d, cs[i]->geom, blocks[i]).smem);
    }
    if (rt == 8)
        for (hv_ctx *c : cs) nt = std::max(nt, c->fused.direct.nt8);
    w.kern = direct_kernel<float, true>(rt, nt);
    HV_TRY(allow_max_dynamic_smem(w.kern, cs[0]->device));
    int per_sm = 0;
    HV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, w.kern, kThreads, smem));
    if ((long long)per_sm * sms < (long long)binst.size()) return HV_ERR_UNSUPPORTED;
    HV_CUDA(cudaMalloc(&w.args, sizeof(DirectArgs<float>) * n));
    HV_CUDA(cudaMalloc((void **)&w.binst, sizeof(int) * binst.size()));
    HV_CUDA(cudaMalloc((void **)&w.bfirst, sizeof(int) * n));
    HV_CUDA(cudaMemcpy(w.args, args.data(), sizeof(DirectArgs<float>) * n, cudaMemcpyHostToDevice));
    HV_CUDA(cudaMemcpy(w.binst, binst.data(), sizeof(int) * binst.size(), cudaMemcpyHostToDevice));
    HV_CUDA(cudaMemcpy(w.bfirst, bfirst.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
    // a cudaMemcpy from pageable memory may return before its DMA ends; the
    // wave's kernels run later on other streams
    HV_CUDA(cudaDeviceSynchronize());
    w.ctx = cs;
    w.nblocks = (int)binst.size();
    w.smem = smem;
    w.direct = true;
    return HV_OK;
}

hv_status poisson_wave_launch(const SorWave &w, cudaStream_t st) {
    DirectArgs<float> p;
    std::memset(&p, 0, sizeof(p));
    p.batch = reinterpret_cast<const DirectArgs<float> *>(w.args);
    p.binst = w.binst;
    p.bfirst = w.bfirst;
    void *args[] = {&p};
    HV_CUDA(cudaLaunchCooperativeKernel(w.kern, dim3(w.nblocks), dim3(kThreads), args, w.smem, st));
    return HV_OK;
}

// The barrier words of a solve that gave up are not back at zero.
hv_status poisson_clear(hv_ctx *c) {
    if (c->fused.direct.bar) HV_CUDA(cudaMemsetAsync(c->fused.direct.bar, 0, sizeof(unsigned) * 2, c->stream));
    return HV_OK;
}

}  // namespace hv
