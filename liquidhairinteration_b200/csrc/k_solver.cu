// k_solver.cu -- CGSolver<3> on the device: per-level ghost-fluid matrix
// assembly, SpMV, damped red-black Gauss-Seidel, restriction/prolongation,
// the V-cycle preconditioner and the PCG loop, which runs on the device.
//
// Matrix storage: per level, diag plus one coefficient per +x/+y/+z face and
// a cell type byte (0: phi > 0, 1: phi == 0, 2: phi < 0).  The reference's
// per-row coefficient (PressureSolver.cpp:556-662) is -term when the
// neighbour has phi < 0 and 0 otherwise, and rows with phi > 0 are empty; the
// face term is the same expression seen from both rows, so
//   A(i, j) = [type_i >= 1] [type_j == 2] * face_coef(i, j).
//
// Sparsity: rows with phi > 0 are empty, so every sweep visits only the
// level's active 8 x 8 x 32 tiles (cells with phi <= 0, plus tiles covering
// an active finer tile so that restricted residuals are carried down).  Cells
// outside active tiles are air cells whose values no row ever reads.
//
// The coarse levels whose rows fit the registers of one 16-CTA cluster are
// solved in one launch, staged in its shared memory: their pre-smoothing,
// restriction, coarsest sweeps, prolongation, post-smoothing.
//
// The PCG loop keeps every scalar on the device.  By default one solve is
// one CUDA graph: the initial V-cycle, then a conditional while node whose
// body is one PCG iteration; the kernel that applies the stopping rule sets
// the loop condition.  With eager = 1 the host drives the same kernels and
// reads the stop flag after every iteration.
#include <algorithm>
#include <random>
#include <string>
#include <type_traits>

#include "impl.cuh"
#include "layouts.cuh"

namespace lhi {

namespace {

constexpr int kGraphIterationCap = 100000;  // hard stop of the device-side loop

// Limit of the solver kernels' waits on their TMA staging copies (200 ms;
// lhi_debug_set_stage_wait_limit lowers it to test the timeout path).  On
// a timeout a CTA records it, waits (200 ms at most) for every copy of its
// own still in flight, and leaves.
__device__ unsigned long long g_stage_wait_ns = kWaitLimitNs;

template <class T> struct LevelK {
    int nx, ny, nz;
    const T* diag;
    const T* cx;
    const T* cy;
    const T* cz;
    const uint8_t* type;
};

template <class T> LevelK<T> lk(const LevelDev<T>& L) {
    return LevelK<T>{L.nx, L.ny, L.nz, L.diag, L.cf[0], L.cf[1], L.cf[2], L.type};
}

// the mixed mode's FP64 finest-level matrix with the level's cell types
template <class T, class TX> LevelK<double> lk_hi(const LiquidImpl<T, TX>& s) {
    const LevelDev<T>& L = s.lv_[0];
    return LevelK<double>{L.nx, L.ny, L.nz, s.diag_hi_, s.cf_hi_[0], s.cf_hi_[1], s.cf_hi_[2], L.type};
}

__device__ __forceinline__ void decode(long long i, int ny, int nz, int& x, int& y, int& z) { idx3(i, ny, nz, x, y, z); }

// CGSolver<3>::GetAx (PressureSolver.cpp:700-717), computed in C
template <class C, class T, class V>
__device__ __forceinline__ C ax_at(const LevelK<T>& L, const V* __restrict__ x, long long i, int xi, int yi, int zi) {
    if (L.type[i] == 0) return C(0);
    const long long sy = L.nz, sx = (long long)L.ny * L.nz;
    C r = C(x[i]) * C(L.diag[i]);
    if (xi + 1 < L.nx && L.type[i + sx] == 2) r += C(x[i + sx]) * C(L.cx[i]);
    if (xi - 1 >= 0 && L.type[i - sx] == 2) r += C(x[i - sx]) * C(L.cx[i - sx]);
    if (yi + 1 < L.ny && L.type[i + sy] == 2) r += C(x[i + sy]) * C(L.cy[i]);
    if (yi - 1 >= 0 && L.type[i - sy] == 2) r += C(x[i - sy]) * C(L.cy[i - sy]);
    if (zi + 1 < L.nz && L.type[i + 1] == 2) r += C(x[i + 1]) * C(L.cz[i]);
    if (zi - 1 >= 0 && L.type[i - 1] == 2) r += C(x[i - 1]) * C(L.cz[i - 1]);
    return r;
}

// The 7-point row of one cell, loaded without data-dependent branches so a
// thread can put the loads of several cells in flight before any arithmetic.
// Out-of-range neighbours read the cell itself and are masked by `in`.
template <class T, class V> struct Cell7 {
    V zc, zn[6];
    T d, cf[6];
    unsigned m;  // bit k: neighbour k exists and has phi < 0
    uint8_t tc;
};

template <class T, class V>
__device__ __forceinline__ void load7(const LevelK<T>& L, const V* __restrict__ x, long long i, int xi, int yi, int zi,
                                      Cell7<T, V>& s) {
    const long long sy = L.nz, sx = (long long)L.ny * L.nz;
    const bool in[6] = {xi + 1 < L.nx, xi > 0, yi + 1 < L.ny, yi > 0, zi + 1 < L.nz, zi > 0};
    const long long j[6] = {in[0] ? i + sx : i, in[1] ? i - sx : i, in[2] ? i + sy : i,
                            in[3] ? i - sy : i, in[4] ? i + 1 : i,  in[5] ? i - 1 : i};
    s.tc = L.type[i];
    s.d = L.diag[i];
    s.zc = x[i];
    uint8_t tn[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        tn[k] = L.type[j[k]];
        s.zn[k] = x[j[k]];
    }
    s.cf[0] = L.cx[i];
    s.cf[1] = L.cx[j[1]];
    s.cf[2] = L.cy[i];
    s.cf[3] = L.cy[j[3]];
    s.cf[4] = L.cz[i];
    s.cf[5] = L.cz[j[5]];
    unsigned m = 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) m |= (in[k] && tn[k] == 2) ? (1u << k) : 0u;
    s.m = m;
}

// ax_at on a loaded row: same terms in the same order (+x, -x, +y, -y, +z, -z)
template <class C, class T, class V> __device__ __forceinline__ C ax7(const Cell7<T, V>& s) {
    if (s.tc == 0) return C(0);
    C r = C(s.zc) * C(s.d);
#pragma unroll
    for (int k = 0; k < 6; ++k)
        if (s.m & (1u << k)) r += C(s.zn[k]) * C(s.cf[k]);
    return r;
}

// A cell's new z from its old one and the quotient (PressureSolver.cpp:830-834),
// the roundings written out so that every kernel has the same
template <class T> __device__ __forceinline__ T smooth_update(T zc, T term, T w, int variant) {
    if (variant == LHI_SMOOTHER_DAMPED_GS) return fma(w, term, zc);
    if constexpr (sizeof(T) == 8) return fma(w, term, X<T>::mul(T(1) - w, zc));
    else return T(fma(1.0 - double(w), double(zc), double(X<T>::mul(w, term))));
}

// CGSolver<3>::Smooth update of one cell from its loaded row (PressureSolver.cpp:830-834)
template <class T>
__device__ __forceinline__ bool smooth7(const Cell7<T, T>& s, T rv, T w, int variant, T& out) {
    if (is_small(s.d)) return false;
    out = smooth_update(s.zc, (rv - ax7<T>(s)) / s.d, w, variant);
    return true;
}

// PCG update region: fluid cells of [1, N-2]^3 (PressureSolver.cpp:874-899)
// or, with LHI_REGION_FLUID, every fluid cell.
__device__ __forceinline__ bool in_region(int x, int y, int z, int nx, int ny, int nz, int region) {
    return region == LHI_REGION_FLUID || (x >= 1 && x <= nx - 2 && y >= 1 && y <= ny - 2 && z >= 1 && z <= nz - 2);
}

// ------------------------------------------------------------- assembly
struct LevelGeom {
    int nx, ny, nz;     // this level
    int fnx, fny, fnz;  // level 0
    int level;
};

// GetApproxLiquidPhi (PressureSolver.cpp:476-493): trilerp of the 2x2x2
// central fine cells with factors 0.5.
template <class T> __device__ __forceinline__ T approx_phi(const T* __restrict__ f, LevelGeom g, int xi, int yi, int zi) {
    if (g.level == 0) return f[((long long)xi * g.fny + yi) * g.fnz + zi];
    const int fac = 1 << g.level, h = (1 << (g.level - 1)) - 1;
    const int bx = fac * xi + h, by = fac * yi + h, bz = fac * zi + h;
    const long long sy = g.fnz, sx = (long long)g.fny * g.fnz;
    const T* b = f + bx * sx + by * sy + bz;
    return trilerp(b[0], b[sx], b[sy], b[sx + sy], b[1], b[sx + 1], b[sy + 1], b[sx + sy + 1], T(0.5), T(0.5), T(0.5));
}
// GetApproxWx / Wy / Wz (PressureSolver.cpp:495-542)
template <class T> __device__ __forceinline__ T approx_w(const T* __restrict__ w, LevelGeom g, int a, int xi, int yi, int zi) {
    const int fy = g.fny + (a == 1), fz = g.fnz + (a == 2);
    if (g.level == 0) return w[((long long)xi * fy + yi) * fz + zi];
    const int fac = 1 << g.level, h = (1 << (g.level - 1)) - 1;
    const long long sy = fz, sx = (long long)fy * fz;
    if (a == 0) {
        const T* b = w + (long long)(fac * xi) * sx + (long long)(fac * yi + h) * sy + (fac * zi + h);
        return bilerp(b[0], b[sy], b[1], b[sy + 1], T(0.5), T(0.5));
    } else if (a == 1) {
        const T* b = w + (long long)(fac * xi + h) * sx + (long long)(fac * yi) * sy + (fac * zi + h);
        return bilerp(b[0], b[sx], b[1], b[sx + 1], T(0.5), T(0.5));
    }
    const T* b = w + (long long)(fac * xi + h) * sx + (long long)(fac * yi + h) * sy + (fac * zi);
    return bilerp(b[0], b[sx], b[sy], b[sx + sy], T(0.5), T(0.5));
}

// Also marks the level's tile of every cell with phi <= 0 as active.
template <class T>
__global__ void k_level_phi(LevelGeom g, const T* __restrict__ fine_phi, T* __restrict__ phi, uint8_t* __restrict__ type,
                            uint8_t* __restrict__ tile_flag, int tdy, int tdz) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long n = (long long)g.nx * g.ny * g.nz;
    if (i >= n) return;
    int x, y, z;
    decode(i, g.ny, g.nz, x, y, z);
    T ph = approx_phi(fine_phi, g, x, y, z);
    if (g.level > 0) phi[i] = ph;
    const uint8_t t = (ph > T(0)) ? 0 : ((ph < T(0)) ? 2 : 1);
    type[i] = t;
    if (t != 0) tile_flag[((long long)(x / kTileX) * tdy + y / kTileY) * tdz + z / kTileZ] = 1;
}

// CGSolver<3>::BuildLHS for one level (PressureSolver.cpp:544-664), in T
// from fields of type TI (TI = float, T = double: the FP64 finest-level
// matrix the mixed mode's outer residual uses).
template <class T, class TI = T>
__device__ __forceinline__ void level_matrix_cell(long long i, LevelGeom g, const TI* __restrict__ phi,
                                                  const TI* __restrict__ lwx, const TI* __restrict__ lwy,
                                                  const TI* __restrict__ lwz, T h0, T h1, T h2, T dt, T rho,
                                                  T* __restrict__ diag, T* __restrict__ cx, T* __restrict__ cy,
                                                  T* __restrict__ cz, uint8_t* __restrict__ type,
                                                  uint8_t* __restrict__ tile_flag, int tdy, int tdz,
                                                  uint8_t* __restrict__ mask, int mpitch) {
    // the FP64 copy is read only on rows with phi <= 0 (and their fluid
    // neighbours): air cells need no entries
    if constexpr (!std::is_same<T, TI>::value)
        if (T(phi[i]) > T(0)) return;
    int x, y, z;
    decode(i, g.ny, g.nz, x, y, z);
    const long long sy = g.nz, sx = (long long)g.ny * g.nz;
    const TI* lw[3] = {lwx, lwy, lwz};
    const T hh[3] = {h0, h1, h2};
    auto term_of = [&](int a, T w) -> T {
        return X<T>::div(X<T>::mul(w, dt), X<T>::mul(X<T>::mul(rho, hh[a]), hh[a]));
    };
    // The six faces (right, left, top, bottom, front, back) and the
    // neighbours' phi, loaded up front so the loads overlap; each face's term
    // w dt / (rho h^2) is formed once (the +x/+y/+z terms serve both this
    // cell's couplings and its diagonal), in the reference's arithmetic.
    const int xs[6] = {x + 1, x, x, x, x, x};
    const int ys[6] = {y, y, y + 1, y, y, y};
    const int zs[6] = {z, z, z, z, z + 1, z};
    const int ax[6] = {0, 0, 1, 1, 2, 2};
    const long long off[6] = {sx, -sx, sy, -sy, 1, -1};
    const bool exists[6] = {x + 1 < g.nx, x - 1 >= 0, y + 1 < g.ny, y - 1 >= 0, z + 1 < g.nz, z - 1 >= 0};
    const T center = T(phi[i]);
    const bool row = !(center > T(0));
    T w6[6], nphi6[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        w6[k] = exists[k] ? T(approx_w(lw[ax[k]], g, ax[k], xs[k], ys[k], zs[k])) : T(0);
        nphi6[k] = exists[k] ? T(phi[i + off[k]]) : T(0);
    }
    T term6[6];
#pragma unroll
    for (int k = 0; k < 6; ++k)  // the -x/-y/-z terms only for a row of the matrix
        term6[k] = (w6[k] > T(0) && ((k & 1) == 0 || row)) ? term_of(ax[k], w6[k]) : T(0);
    // own +x/+y/+z face coefficients
    cx[i] = (w6[0] > T(0)) ? -term6[0] : T(0);
    cy[i] = (w6[2] > T(0)) ? -term6[2] : T(0);
    cz[i] = (w6[4] > T(0)) ? -term6[4] : T(0);
    // the finest level (type != nullptr) also classifies the cell, marks its
    // tile active (k_level_phi's work) and, where the fused sweep runs, writes
    // its neighbour mask (k_level_mask's), from the phi values at hand
    if (type) {
        const uint8_t t = (center > T(0)) ? 0 : ((center < T(0)) ? 2 : 1);
        type[i] = t;
        if (t != 0) tile_flag[((long long)(x / kTileX) * tdy + y / kTileY) * tdz + z / kTileZ] = 1;
        if (mask) {
            unsigned m = t != 0 ? 64u : 0u;
#pragma unroll
            for (int k = 0; k < 6; ++k)
                if (exists[k] && nphi6[k] < T(0)) m |= 1u << k;  // right, left, top, bottom, front, back
            mask[((long long)x * g.ny + y) * mpitch + z] = uint8_t(m);
        }
    }
    T d = T(0);
    if (row) {
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            if (!exists[k] || !(w6[k] > T(0))) continue;
            const T term = term6[k];
            const T nphi = nphi6[k];
            if (nphi < T(0)) d = X<T>::add(d, term);
            else d = X<T>::add(d, X<T>::div(term, frac_floor(fraction_in_region(center, nphi))));
        }
    }
    diag[i] = d;
}

template <class T, class TI = T>
__global__ void k_level_matrix(LevelGeom g, const TI* __restrict__ phi, const TI* __restrict__ lwx,
                               const TI* __restrict__ lwy, const TI* __restrict__ lwz, T h0, T h1, T h2, T dt, T rho,
                               T* __restrict__ diag, T* __restrict__ cx, T* __restrict__ cy, T* __restrict__ cz,
                               uint8_t* __restrict__ type, uint8_t* __restrict__ tile_flag, int tdy, int tdz,
                               uint8_t* __restrict__ mask, int mpitch) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)g.nx * g.ny * g.nz) return;
    level_matrix_cell<T, TI>(i, g, phi, lwx, lwy, lwz, h0, h1, h2, dt, rho, diag, cx, cy, cz, type, tile_flag, tdy,
                             tdz, mask, mpitch);
}

// The mixed mode's finest level: the FP32 matrix (with the cell classes,
// tile flags and neighbour mask) and the FP64 matrix of the outer residual
// from one read of the fields, each in its own arithmetic (the same bits as
// two k_level_matrix launches).
template <class T>
__global__ void k_level_matrix_mixed(LevelGeom g, const T* __restrict__ phi, const T* __restrict__ lwx,
                                     const T* __restrict__ lwy, const T* __restrict__ lwz, T h0, T h1, T h2, T dt,
                                     T rho, T* __restrict__ diag, T* __restrict__ cx, T* __restrict__ cy,
                                     T* __restrict__ cz, uint8_t* __restrict__ type, uint8_t* __restrict__ tile_flag,
                                     int tdy, int tdz, uint8_t* __restrict__ mask, int mpitch, double hd0, double hd1,
                                     double hd2, double dtd, double rhod, double* __restrict__ diag_hi,
                                     double* __restrict__ cx_hi, double* __restrict__ cy_hi,
                                     double* __restrict__ cz_hi) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)g.nx * g.ny * g.nz) return;
    level_matrix_cell<T, T>(i, g, phi, lwx, lwy, lwz, h0, h1, h2, dt, rho, diag, cx, cy, cz, type, tile_flag, tdy,
                            tdz, mask, mpitch);
    level_matrix_cell<double, T>(i, g, phi, lwx, lwy, lwz, hd0, hd1, hd2, dtd, rhod, diag_hi, cx_hi, cy_hi, cz_hi,
                                 nullptr, nullptr, 0, 0, nullptr, 0);
}

// Galerkin coarse level (LHI_COARSE_GALERKIN): A_c = P^T A P / 8 of the
// finer level f under the V-cycle's transfers (constant injection P, the
// 1/8 averaging restriction), with A_ij = [type_i >= 1][type_j == 2] c_ij as
// every kernel of the solver applies it.  Coarse cell I takes its 8
// children's diagonals and the couplings between them; the coupling of I
// with its +x / +y / +z neighbour is the sum over the 4 child pairs across
// that face.  type_I = 2 if a child is fluid, else 1 if a child has phi = 0.
template <class T>
__global__ void k_level_galerkin(LevelK<T> F, int cnx, int cny, int cnz, T* __restrict__ diag, T* __restrict__ cx,
                                 T* __restrict__ cy, T* __restrict__ cz, uint8_t* __restrict__ type,
                                 uint8_t* __restrict__ tile_flag, int tdy, int tdz) {
    long long I = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long n = (long long)cnx * cny * cnz;
    if (I >= n) return;
    int X, Y, Z;
    decode(I, cny, cnz, X, Y, Z);
    const long long fsy = F.nz, fsx = (long long)F.ny * F.nz;
    auto fi = [&](int x, int y, int z) -> long long { return ((long long)x * F.ny + y) * F.nz + z; };
    // A_ij of fine cells i and its +axis neighbour j = i + step: rows couple to fluid columns only
    auto a_ij = [&](long long i, long long j, T c) -> T {
        return (F.type[i] >= 1 && F.type[j] == 2) ? c : T(0);
    };
    T d = T(0);
    uint8_t t = 0;
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2; ++b)
            for (int c = 0; c < 2; ++c) {
                const long long i = fi(2 * X + a, 2 * Y + b, 2 * Z + c);
                const uint8_t ti = F.type[i];
                t = (ti == 2 || t == 2) ? 2 : (ti == 1 ? uint8_t(1) : t);
                if (ti >= 1) d += F.diag[i];
                // couplings inside the coarse cell, both directions
                if (a == 0) d += a_ij(i, i + fsx, F.cx[i]) + a_ij(i + fsx, i, F.cx[i]);
                if (b == 0) d += a_ij(i, i + fsy, F.cy[i]) + a_ij(i + fsy, i, F.cy[i]);
                if (c == 0) d += a_ij(i, i + 1, F.cz[i]) + a_ij(i + 1, i, F.cz[i]);
            }
    T ccx = T(0), ccy = T(0), ccz = T(0);
    for (int u = 0; u < 2; ++u)
        for (int v = 0; v < 2; ++v) {
            if (X + 1 < cnx) {
                const long long i = fi(2 * X + 1, 2 * Y + u, 2 * Z + v);
                ccx += a_ij(i, i + fsx, F.cx[i]);
            }
            if (Y + 1 < cny) {
                const long long i = fi(2 * X + u, 2 * Y + 1, 2 * Z + v);
                ccy += a_ij(i, i + fsy, F.cy[i]);
            }
            if (Z + 1 < cnz) {
                const long long i = fi(2 * X + u, 2 * Y + v, 2 * Z + 1);
                ccz += a_ij(i, i + 1, F.cz[i]);
            }
        }
    const T s = T(0.125);
    diag[I] = d * s;
    cx[I] = ccx * s;
    cy[I] = ccy * s;
    cz[I] = ccz * s;
    type[I] = t;
    if (t != 0) tile_flag[((long long)(X / kTileX) * tdy + Y / kTileY) * tdz + Z / kTileZ] = 1;
}

// CGSolver<3>::BuildRHS (PressureSolver.cpp:682-698)
// (TI = float, T = double: the FP64 right-hand side of the mixed mode's
// outer residual, from the same float fields)
template <class T, class TI = T>
__device__ __forceinline__ void build_rhs_cell(long long i, int nx, int ny, int nz, T h0, T h1, T h2,
                                               const TI* __restrict__ phi, const TI* __restrict__ lwx,
                                               const TI* __restrict__ lwy, const TI* __restrict__ lwz,
                                               const TI* __restrict__ vx, const TI* __restrict__ vy,
                                               const TI* __restrict__ vz, T* __restrict__ rhs) {
    (void)nx;
    if constexpr (!std::is_same<T, TI>::value)  // the FP64 copy is read only where phi <= 0
        if (T(phi[i]) > T(0)) return;
    T b = T(0);
    if (!(T(phi[i]) > T(0))) {
        int x, y, z;
        decode(i, ny, nz, x, y, z);
        long long fxi = ((long long)x * ny + y) * nz + z, fxs = (long long)ny * nz;
        long long fyi = ((long long)x * (ny + 1) + y) * nz + z, fys = nz;
        long long fzi = ((long long)x * ny + y) * (nz + 1) + z;
        b = X<T>::sub(b, X<T>::div(X<T>::mul(T(lwx[fxi + fxs]), T(vx[fxi + fxs])), h0));
        b = X<T>::add(b, X<T>::div(X<T>::mul(T(lwx[fxi]), T(vx[fxi])), h0));
        b = X<T>::sub(b, X<T>::div(X<T>::mul(T(lwy[fyi + fys]), T(vy[fyi + fys])), h1));
        b = X<T>::add(b, X<T>::div(X<T>::mul(T(lwy[fyi]), T(vy[fyi])), h1));
        b = X<T>::sub(b, X<T>::div(X<T>::mul(T(lwz[fzi + 1]), T(vz[fzi + 1])), h2));
        b = X<T>::add(b, X<T>::div(X<T>::mul(T(lwz[fzi]), T(vz[fzi])), h2));
    }
    rhs[i] = b;
}

template <class T, class TI = T>
__global__ void k_build_rhs(int nx, int ny, int nz, T h0, T h1, T h2, const TI* __restrict__ phi,
                            const TI* __restrict__ lwx, const TI* __restrict__ lwy, const TI* __restrict__ lwz,
                            const TI* __restrict__ vx, const TI* __restrict__ vy, const TI* __restrict__ vz,
                            T* __restrict__ rhs) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nx * ny * nz) return;
    build_rhs_cell<T, TI>(i, nx, ny, nz, h0, h1, h2, phi, lwx, lwy, lwz, vx, vy, vz, rhs);
}

// The mixed mode's two right-hand sides (FP32 for the loop, FP64 for the
// outer residual) from one read of the fields, each in its own arithmetic.
template <class T>
__global__ void k_build_rhs_mixed(int nx, int ny, int nz, T h0, T h1, T h2, double hd0, double hd1, double hd2,
                                  const T* __restrict__ phi, const T* __restrict__ lwx, const T* __restrict__ lwy,
                                  const T* __restrict__ lwz, const T* __restrict__ vx, const T* __restrict__ vy,
                                  const T* __restrict__ vz, T* __restrict__ rhs, double* __restrict__ rhs_hi) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nx * ny * nz) return;
    build_rhs_cell<T, T>(i, nx, ny, nz, h0, h1, h2, phi, lwx, lwy, lwz, vx, vy, vz, rhs);
    build_rhs_cell<double, T>(i, nx, ny, nz, hd0, hd1, hd2, phi, lwx, lwy, lwz, vx, vy, vz, rhs_hi);
}

// ------------------------------------------------------------ active tiles
struct TileK {
    const int32_t* ids;
    const int* count;
    int tdy, tdz;
    int ysplit;  // work units per tile: each takes every ysplit-th row
};

// Visits every in-grid cell of the active tiles.  A work unit is (tile, row
// subset); persistent CTAs take units blockIdx.x, blockIdx.x + gridDim.x, ...;
// warp w takes x = x0 + w and lane l takes z = z0 + l.  Small levels use
// ysplit = 8 (one row per thread) so their few tiles still fill the GPU.
template <class F> __device__ __forceinline__ void for_tiles(const TileK& tk, int nx, int ny, int nz, F&& f) {
    const int units = *tk.count * tk.ysplit;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
        const int t = u / tk.ysplit, sub = u - t * tk.ysplit;
        const int id = tk.ids[t];
        const int tz = id % tk.tdz, rest = id / tk.tdz;
        const int ty = rest % tk.tdy, tx = rest / tk.tdy;
        const int x = tx * kTileX + w, z = tz * kTileZ + lane;
        if (x >= nx || z >= nz) continue;
        const int y0 = ty * kTileY, y1 = min(y0 + kTileY, ny);
        for (int y = y0 + sub; y < y1; y += tk.ysplit) f(x, y, z, ((long long)x * ny + y) * nz + z);
    }
}

// for_tiles with a thread's rows of a work unit handed over together:
// f(x, z, i0, rows, ys) where row k < rows is cell i0 + k * ys * nz (y
// ascending).  Kernels load every row before using any, so a thread keeps
// up to 8 rows of loads in flight; per-thread sums keep for_tiles' order.  The
// kernels' R is the most rows a unit has (kTileY, or 2 on small levels: fewer
// registers, so more of the launch runs at once).
template <class F> __device__ __forceinline__ void for_tile_cols(const TileK& tk, int nx, int ny, int nz, F&& f) {
    const int units = *tk.count * tk.ysplit;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
        const int t = u / tk.ysplit, sub = u - t * tk.ysplit;
        const int id = tk.ids[t];
        const int tz = id % tk.tdz, rest = id / tk.tdz;
        const int ty = rest % tk.tdy, tx = rest / tk.tdy;
        const int x = tx * kTileX + w, z = tz * kTileZ + lane;
        if (x >= nx || z >= nz) continue;
        const int yb = ty * kTileY + sub, ye = min(ty * kTileY + kTileY, ny);
        const int rows = yb < ye ? (ye - yb + tk.ysplit - 1) / tk.ysplit : 0;
        f(x, z, ((long long)x * ny + yb) * nz + z, yb, rows, tk.ysplit);
    }
}

struct TileLevels {
    int nlev;
    int tdim[kMaxLevels][3];
    uint8_t* flag[kMaxLevels];
    int32_t* ids[kMaxLevels];
};

// One CTA: level l's flags |= its 2x2x2 child tiles' flags at level l - 1
// (finest first), then each level's active tiles are listed in increasing
// order (deterministic) with their count in counts[l].
__global__ void __launch_bounds__(1024) k_tiles_finalize(TileLevels tl, int* __restrict__ counts) {
    __shared__ int warp_tot[32];
    __shared__ int base;
    for (int l = 0; l < tl.nlev; ++l) {
        const int ax = tl.tdim[l][0], ay = tl.tdim[l][1], az = tl.tdim[l][2];
        const int n = ax * ay * az;
        if (l > 0) {
            const int fx = tl.tdim[l - 1][0], fy = tl.tdim[l - 1][1], fz = tl.tdim[l - 1][2];
            for (int t = threadIdx.x; t < n; t += blockDim.x) {
                const int tz = t % az, ty = (t / az) % ay, tx = t / (az * ay);
                uint8_t f = tl.flag[l][t];
                for (int c = 0; c < 8 && !f; ++c) {
                    const int cx = 2 * tx + (c >> 2), cy = 2 * ty + ((c >> 1) & 1), cz = 2 * tz + (c & 1);
                    if (cx < fx && cy < fy && cz < fz) f |= tl.flag[l - 1][(cx * fy + cy) * fz + cz];
                }
                tl.flag[l][t] = f;
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) base = 0;
        __syncthreads();
        for (int c0 = 0; c0 < n; c0 += blockDim.x) {
            const int t = c0 + threadIdx.x;
            const int f = (t < n && tl.flag[l][t]) ? 1 : 0;
            const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
            const unsigned m = __ballot_sync(0xffffffffu, f);
            if (lane == 0) warp_tot[w] = __popc(m);
            __syncthreads();
            int off = 0;
            for (int k = 0; k < w; ++k) off += warp_tot[k];
            const int rank = base + off + __popc(m & ((1u << lane) - 1u));
            if (f) tl.ids[l][rank] = t;
            __syncthreads();
            if (threadIdx.x == 0) {
                int tot = 0;
                for (int k = 0; k < int(blockDim.x >> 5); ++k) tot += warp_tot[k];
                base += tot;
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) counts[l] = base;
        __syncthreads();
    }
}

// ----------------------------------------------------------- V-cycle
// CGSolver<3>::Smooth (PressureSolver.cpp:821-837): one colour of damped
// red-black Gauss-Seidel on one level's active tiles.  A work unit is one of the
// four rows y of that colour in a tile, a thread its cell at (x, z).  Latency
// bounds it: one row a thread takes 40 registers, so that six CTAs an SM are
// at work (FP64: three); four rows, loaded ahead, took 128 and two CTAs
// (93 x 70 x 61: 7.4 -> 5.3 us; a PCG iteration of 125 x 141 x 99 187 -> 167,
// of 128^3 in FP64 236 -> 213).
constexpr int kSweepSplit = kTileY / 2;
template <class T>
__global__ void __launch_bounds__(kTileThreads, sizeof(T) == 4 ? 6 : 3)
    k_sweep(LevelK<T> L, TileK tk, const T* __restrict__ r, T* __restrict__ z, T w, int variant, int phase,
            const int* __restrict__ stop) {
    if (*stop) return;
    const int units = *tk.count * kSweepSplit;
    const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
        const int t = u / kSweepSplit, row = u - t * kSweepSplit;
        const int id = tk.ids[t];
        const int tz = id % tk.tdz, rest = id / tk.tdz;
        const int ty = rest % tk.tdy, tx = rest / tk.tdy;
        const int x = tx * kTileX + wp, zz = tz * kTileZ + lane;
        const int y0 = ty * kTileY, y = y0 + ((phase + x + zz + y0) & 1) + 2 * row;
        if (x >= L.nx || zz >= L.nz || y >= L.ny) continue;
        const long long i = ((long long)x * L.ny + y) * L.nz + zz;
        Cell7<T, T> c;
        load7(L, z, i, x, y, zz, c);
        T out;
        if (smooth7(c, r[i], w, variant, out)) z[i] = out;
    }
}

// ------------------------------------------------- fused red-black sweep
// One damped red-black Gauss-Seidel sweep (both colours) of an FP32 level in
// one pass.  A CTA takes an active 8 x 8 x 32 tile T and stages by TMA:
//   Z  (z_in)    T grown by 2 cells in x and y, z from z0-4: 12 x 12 x 40
//   R, D, CZ     T grown by 1 in x and y:                    10 x 10 x 40
//   CX           as R with x from x0-2:                      11 x 10 x 40
//   CY           as R with y from y0-2:                      10 x 11 x 40
//   M (bytes)    T grown by 1, z from z0-16:                 10 x 10 x 64
// It updates colour 0 on T grown by one cell (the ring recomputes exactly
// what the neighbouring tiles compute), then colour 1 on T, in place in
// shared memory, and writes T to z_out.  Reading z_in and writing z_out
// keeps the neighbours' halo reads on the old values.  Each cell's update is
// the arithmetic of smooth7 in the same order, so the values equal those of
// two k_sweep launches.  Cells outside the grid read diag 0 and are skipped.
namespace rb {
constexpr int kZW = layout::kZW;
constexpr int kZ = layout::kZBox;
constexpr int kR = layout::kRBox;
constexpr int kC = layout::kCBox;
constexpr int kMW = layout::kMW;
constexpr int kM = layout::kMBox;
constexpr uint32_t kTx = uint32_t((kZ + 3 * kR + 2 * kC) * 4 + kM);  // bytes the 7 boxes deliver
constexpr int al(int b) { return (b + 127) & ~127; }
// offsets inside one stage
constexpr int oZ = 0;
constexpr int oR = oZ + al(kZ * 4);
constexpr int oD = oR + al(kR * 4);
constexpr int oCZ = oD + al(kR * 4);
constexpr int oCX = oCZ + al(kR * 4);
constexpr int oCY = oCX + al(kC * 4);
constexpr int oM = oCY + al(kC * 4);
constexpr int kStage = oM + al(kM);
constexpr int kBase = 128;  // two mbarriers, then two stages
constexpr int kSmem = kBase + 2 * kStage;
constexpr int kThreads = 512;
}  // namespace rb

// Mask bits of a cell: 0..5 neighbour +x, -x, +y, -y, +z, -z exists with phi < 0;
// 6: the cell's own type is not 0.
__device__ __forceinline__ bool rb_eval(const float* __restrict__ Zs, const float* __restrict__ Rs,
                                        const float* __restrict__ Ds, const float* __restrict__ CZs,
                                        const float* __restrict__ CXs, const float* __restrict__ CYs,
                                        const uint8_t* __restrict__ Ms, int lx, int ly, int lz, float w, int variant,
                                        int& zi, float& out) {
    const int ri = layout::rb_r(lx, ly, lz);
    zi = layout::rb_z(lx, ly, lz);
    const float d = Ds[ri];
    if (is_small(d)) return false;
    const unsigned m = Ms[layout::rb_m(lx, ly, lz)];
    const float zc = Zs[zi];
    float ax = 0.f;
    if (m & 64u) {
        const int xi = layout::rb_cx(lx, ly, lz);
        const int yi = layout::rb_cy(lx, ly, lz);
        ax = zc * d;
        if (m & 1u) ax += Zs[zi + layout::kZStepX] * CXs[xi];
        if (m & 2u) ax += Zs[zi - layout::kZStepX] * CXs[xi - layout::kCXStepX];
        if (m & 4u) ax += Zs[zi + layout::kZStepY] * CYs[yi];
        if (m & 8u) ax += Zs[zi - layout::kZStepY] * CYs[yi - layout::kCYStepY];
        if (m & 16u) ax += Zs[zi + 1] * CZs[ri];
        if (m & 32u) ax += Zs[zi - 1] * CZs[ri - 1];
    }
    const float term = (Rs[ri] - ax) / d;
    if (variant == LHI_SMOOTHER_DAMPED_GS) out = zc + w * term;
    else out = float((1.0 - double(w)) * double(zc) + double(float(w * term)));
    return true;
}

// Tile id u of the active list -> origin of its 8 x 8 x 32 cells.
__device__ __forceinline__ void tile_origin_of(int id, int tdy, int tdz, int& x0, int& y0, int& z0) {
    const int tz = id % tdz, rest = id / tdz;
    z0 = tz * kTileZ;
    y0 = (rest % tdy) * kTileY;
    x0 = (rest / tdy) * kTileX;
}
__device__ __forceinline__ void tile_origin(const int32_t* __restrict__ ids, int u, int tdy, int tdz, int& x0, int& y0,
                                            int& z0) {
    tile_origin_of(ids[u], tdy, tdz, x0, y0, z0);
}

__device__ __forceinline__ void rb_issue(unsigned char* st, uint64_t* bar, const CUtensorMap* mz, const CUtensorMap* mr,
                                         const CUtensorMap* md, const CUtensorMap* mcx, const CUtensorMap* mcy,
                                         const CUtensorMap* mcz, const CUtensorMap* mm, int x0, int y0, int z0) {
    fence_proxy_async();
    bar_expect_tx(bar, rb::kTx);
    tma_load_box(st + rb::oZ, mz, z0 - 4, y0 - 2, x0 - 2, bar);
    tma_load_box(st + rb::oR, mr, z0 - 4, y0 - 1, x0 - 1, bar);
    tma_load_box(st + rb::oD, md, z0 - 4, y0 - 1, x0 - 1, bar);
    tma_load_box(st + rb::oCZ, mcz, z0 - 4, y0 - 1, x0 - 1, bar);
    tma_load_box(st + rb::oCX, mcx, z0 - 4, y0 - 1, x0 - 2, bar);
    tma_load_box(st + rb::oCY, mcy, z0 - 4, y0 - 2, x0 - 1, bar);
    tma_load_box(st + rb::oM, mm, z0 - 16, y0 - 1, x0 - 1, bar);
}

// One CTA per SM walks its tiles through two shared-memory stages: the
// boxes of the next tile are in flight while the current one is smoothed.
__global__ void __launch_bounds__(rb::kThreads, 1)
    k_rb_fused(const __grid_constant__ CUtensorMap mz, const __grid_constant__ CUtensorMap mr,
               const __grid_constant__ CUtensorMap md, const __grid_constant__ CUtensorMap mcx,
               const __grid_constant__ CUtensorMap mcy, const __grid_constant__ CUtensorMap mcz,
               const __grid_constant__ CUtensorMap mm, int nx, int ny, int nz, const int32_t* __restrict__ ids,
               const int* __restrict__ count, int tdy, int tdz, float* __restrict__ zout, float w, int variant,
               SolveScalars* __restrict__ sc, const float* __restrict__ ap, double* __restrict__ partials,
               unsigned* __restrict__ counter, int final_dot, int region, int flexible) {
    extern __shared__ __align__(128) unsigned char sm[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm);
    double v[2] = {0.0, 0.0};  // r.z and Ap.z of the swept tiles (final_dot)
    // the loads that lead to the first copy, all at once (the list has at
    // least gridDim.x entries whatever the count), and the maps' descriptors,
    // before the CTA's barrier: a PCG iteration of 64^3 takes 150 us, 152 with
    // one after another; 128^3 174 and 176, 192^3 310 and 318, 256^3 the same
    const int stop = sc->stop, units = *count, id0 = ids[blockIdx.x];
    if (threadIdx.x == 0) {
        prefetch_map(&mz);
        prefetch_map(&mr);
        prefetch_map(&md);
        prefetch_map(&mcx);
        prefetch_map(&mcy);
        prefetch_map(&mcz);
        prefetch_map(&mm);
        bar_init(&bar[0], 1);
        bar_init(&bar[1], 1);
    }
    if (stop) return;
    if (threadIdx.x == 0 && int(blockIdx.x) < units) {
        int a, b, c;
        tile_origin_of(id0, tdy, tdz, a, b, c);
        rb_issue(sm + rb::kBase, &bar[0], &mz, &mr, &md, &mcx, &mcy, &mcz, &mm, a, b, c);
    }
    __syncthreads();
    int it = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x, ++it) {
        const int s = it & 1;
        unsigned char* st = sm + rb::kBase + s * rb::kStage;
        int x0, y0, z0;
        tile_origin(ids, u, tdy, tdz, x0, y0, z0);
        const int un = u + int(gridDim.x);
        if (threadIdx.x == 0 && un < units) {  // the other stage was released by the last barrier
            int a, b, c;
            tile_origin(ids, un, tdy, tdz, a, b, c);
            rb_issue(sm + rb::kBase + (s ^ 1) * rb::kStage, &bar[s ^ 1], &mz, &mr, &md, &mcx, &mcy, &mcz, &mm, a, b,
                     c);
        }
        if (__syncthreads_or(!bar_wait(&bar[s], (it >> 1) & 1, g_stage_wait_ns))) {  // every thread leaves together
            if (threadIdx.x == 0) {
                sc->timeout = 1;
                sc->status = LHI_E_TIMEOUT;
                sc->stop = 1;
                // no copy of this CTA may still be landing when it exits: the one given up on and the prefetch
                bar_wait(&bar[s], (it >> 1) & 1);
                if (un < units) bar_wait(&bar[s ^ 1], ((it + 1) >> 1) & 1);
            }
            break;  // a CTA that gave up still takes part in the grid-wide sum below
        }
        // final_dot: this thread's float4 of Ap (the tile's 512 float4s, one
        // per thread), loaded now so the load overlaps the two colour phases
        static_assert(64 * 8 == rb::kThreads, "one float4 of the tile per thread");
        float4 apv = make_float4(0.f, 0.f, 0.f, 0.f);
        if (final_dot) {
            const int row = threadIdx.x >> 3, c = threadIdx.x & 7;
            const int x = x0 + (row >> 3), y = y0 + (row & 7), z = z0 + 4 * c;
            if (x < nx && y < ny && z < nz) apv = *reinterpret_cast<const float4*>(ap + ((long long)x * ny + y) * nz + z);
        }
        float* Zs = reinterpret_cast<float*>(st + rb::oZ);
        const float* Rs = reinterpret_cast<const float*>(st + rb::oR);
        const float* Ds = reinterpret_cast<const float*>(st + rb::oD);
        const float* CZs = reinterpret_cast<const float*>(st + rb::oCZ);
        const float* CXs = reinterpret_cast<const float*>(st + rb::oCX);
        const float* CYs = reinterpret_cast<const float*>(st + rb::oCY);
        const uint8_t* Ms = st + rb::oM;
        // colour 0 ((x + y + z) even) on T grown by one cell: 10 x 10 rows of 17
        // a colour's updates read only the other colour: a thread evaluates
        // all of its cells before storing any, so their loads overlap
        {
            constexpr int kN = (layout::kRbColour0Items + rb::kThreads - 1) / rb::kThreads;
            int zi[kN];
            float out[kN];
            bool upd[kN];
#pragma unroll
            for (int n = 0; n < kN; ++n) {
                const int q = threadIdx.x + n * rb::kThreads;
                upd[n] = false;
                if (q < layout::kRbColour0Items) {
                    int lx, ly, lz;
                    layout::rb_colour0(q, x0, y0, z0, lx, ly, lz);
                    upd[n] = rb_eval(Zs, Rs, Ds, CZs, CXs, CYs, Ms, lx, ly, lz, w, variant, zi[n], out[n]);
                }
            }
#pragma unroll
            for (int n = 0; n < kN; ++n)
                if (upd[n]) Zs[zi[n]] = out[n];
        }
        __syncthreads();
        // colour 1 on T: 8 x 8 rows of 16
        {
            constexpr int kN = layout::kRbColour1Items / rb::kThreads;
            int zi[kN];
            float out[kN];
            bool upd[kN];
#pragma unroll
            for (int n = 0; n < kN; ++n) {
                const int q = threadIdx.x + n * rb::kThreads;
                int lx, ly, lz;
                layout::rb_colour1(q, x0, y0, z0, lx, ly, lz);
                upd[n] = rb_eval(Zs, Rs, Ds, CZs, CXs, CYs, Ms, lx, ly, lz, w, variant, zi[n], out[n]);
            }
#pragma unroll
            for (int n = 0; n < kN; ++n)
                if (upd[n]) Zs[zi[n]] = out[n];
        }
        __syncthreads();
        for (int q = threadIdx.x; q < layout::kRbOutItems; q += rb::kThreads) {
            int lx, ly, c;
            const int zo = layout::rb_out(q, lx, ly, c);
            const int x = x0 + lx, y = y0 + ly, z = z0 + 4 * c;
            if (x < nx && y < ny && z < nz) {
                const float4 zv = *reinterpret_cast<const float4*>(Zs + zo);
                *reinterpret_cast<float4*>(zout + ((long long)x * ny + y) * nz + z) = zv;
                if (final_dot) {  // k_cg_dot_rz's sums over the swept cells
                    const float zz[4] = {zv.x, zv.y, zv.z, zv.w}, aa[4] = {apv.x, apv.y, apv.z, apv.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int lz = 4 * c + j;
                        const float rv = Rs[layout::rb_r(lx, ly, lz)];
                        v[0] += double(rv) * double(zz[j]);
                        const unsigned m = Ms[layout::rb_m(lx, ly, lz)];
                        if ((m & 64u) && in_region(x, y, z + j, nx, ny, nz, region))
                            v[1] += double(aa[j]) * double(zz[j]);
                    }
                }
            }
        }
        __syncthreads();
    }
    if (!final_dot) return;
    double tot[2];
    if (!grid_sum_last<2>(v, partials, counter, tot)) return;
    const double rz_new = tot[0], apz = tot[1];
    sc->rz_new = rz_new;
    sc->apz = apz;
    sc->beta = flexible ? (-sc->alpha * apz / sc->rz_old) : (rz_new / sc->rz_old);
    sc->rz_old = rz_new;
}

// Neighbour masks of one level for the fused sweep (bits as rb_eval reads them).
template <class T>
__global__ void k_level_mask(LevelK<T> L, uint8_t* __restrict__ mask, int pitch) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long n = (long long)L.nx * L.ny * L.nz;
    if (i >= n) return;
    int x, y, z;
    decode(i, L.ny, L.nz, x, y, z);
    const long long sy = L.nz, sx = (long long)L.ny * L.nz;
    unsigned m = L.type[i] != 0 ? 64u : 0u;
    if (x + 1 < L.nx && L.type[i + sx] == 2) m |= 1u;
    if (x > 0 && L.type[i - sx] == 2) m |= 2u;
    if (y + 1 < L.ny && L.type[i + sy] == 2) m |= 4u;
    if (y > 0 && L.type[i - sy] == 2) m |= 8u;
    if (z + 1 < L.nz && L.type[i + 1] == 2) m |= 16u;
    if (z > 0 && L.type[i - 1] == 2) m |= 32u;
    mask[((long long)x * L.ny + y) * pitch + z] = uint8_t(m);
}

// CGSolver<3>::Restrict (PressureSolver.cpp:796-819) at one coarse cell: the
// coarse residual is accumulated in Scalar with 0.125 * (...) evaluated in
// double; z_c = 0.  The 8 children's rows are loaded 4 at a time before use;
// the children are summed in the reference's order.
template <class T>
__device__ __forceinline__ void restrict_cell_batched(const LevelK<T>& F, const T* __restrict__ rf,
                                                      const T* __restrict__ zf, int x, int y, int z, long long i,
                                                      T* __restrict__ rc, T* __restrict__ zc) {
    const long long sy = F.nz, sx = (long long)F.ny * F.nz;
    const int bx = x << 1, by = y << 1, bz = z << 1;
    T acc = T(0);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        Cell7<T, T> c[4];
        T rv[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int a = h, b = (k >> 1) & 1, cc = k & 1;
            const long long f = (long long)(bx + a) * sx + (by + b) * sy + (bz + cc);
            load7(F, zf, f, bx + a, by + b, bz + cc, c[k]);
            rv[k] = rf[f];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const T res = rv[k] - ax7<T>(c[k]);
            acc = T(double(acc) + 0.125 * double(res));
        }
    }
    rc[i] = acc;
    zc[i] = T(0);
}

template <class T>
__global__ void __launch_bounds__(kTileThreads, 2) k_restrict_t(LevelK<T> F, const T* __restrict__ rf, const T* __restrict__ zf,
                                                             int cnx, int cny, int cnz, TileK tk, T* __restrict__ rc,
                                                             T* __restrict__ zc, const int* __restrict__ stop) {
    if (*stop) return;
    for_tiles(tk, cnx, cny, cnz,
              [&](int x, int y, int z, long long i) { restrict_cell_batched(F, rf, zf, x, y, z, i, rc, zc); });
}

// Every cell of a coarse level, eight lanes a cell: each lane forms one child's
// residual, all of its loads at once, and the children are summed in the
// reference's order over shuffles.  Latency bounds it: one thread a cell put
// too few warps on the chip and walked eight rows of dependent loads
// (93 x 70 x 61: 19 us before, 7.3 now).
template <class T>
__global__ void __launch_bounds__(256) k_restrict_dense(LevelK<T> F, const T* __restrict__ rf, const T* __restrict__ zf,
                                                        int cnx, int cny, int cnz, T* __restrict__ rc,
                                                        T* __restrict__ zc, const int* __restrict__ stop) {
    if (*stop) return;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, i = t >> 3;
    if (i >= (long long)cnx * cny * cnz) return;  // all eight lanes of a cell, or none
    const int k = int(t & 7);  // child (0,0,0) (0,0,1) (0,1,0) ...
    int x, y, z;
    decode(i, cny, cnz, x, y, z);
    x = 2 * x + (k >> 2);
    y = 2 * y + ((k >> 1) & 1);
    z = 2 * z + (k & 1);
    const long long f = ((long long)x * F.ny + y) * F.nz + z;
    Cell7<T, T> c;
    load7(F, zf, f, x, y, z, c);
    const T res = rf[f] - ax7<T>(c);
    const unsigned lanes = 0xffu << (threadIdx.x & 24);
    T acc = T(0);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc = T(double(acc) + 0.125 * double(__shfl_sync(lanes, res, j, 8)));
    if (k == 0) rc[i] = acc;
    if (k == 1) zc[i] = T(0);
}

// CGSolver<3>::Prolong (PressureSolver.cpp:774-794): piecewise-constant,
// written per fine cell (fine cells beyond 2 * coarse extent get nothing).
template <class T, int R>
__global__ void __launch_bounds__(kTileThreads) k_prolong_t(int fnx, int fny, int fnz, TileK tk, const T* __restrict__ zc,
                                                            int cnx, int cny, int cnz, T* __restrict__ zf,
                                                            const int* __restrict__ stop) {
    if (*stop) return;
    for_tile_cols(tk, fnx, fny, fnz, [&](int x, int z, long long i0, int yb, int rows, int ys) {
        const long long st = (long long)ys * fnz;
        const int cx = x >> 1, cz = z >> 1;
        bool on[R];
        T fv[R], cv[R];
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int cy = (yb + k * ys) >> 1;
            on[k] = k < rows && cx < cnx && cy < cny && cz < cnz;
            if (on[k]) {
                fv[k] = zf[i0 + k * st];
                cv[k] = zc[((long long)cx * cny + cy) * cnz + cz];
            }
        }
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (on[k]) zf[i0 + k * st] = fv[k] + cv[k];
    });
}

// ------------------------------------------------- coarse levels in a cluster
// The V-cycle of the coarse levels [first, last] in one launch, on one
// cluster of up to 16 CTAs.  A level is cut into slabs of planes, one per
// CTA; z, r and the residuals live in the CTAs' shared memory, each slab of z
// with a copy of the neighbouring CTAs' adjacent planes.  Every thread owns
// at most kSlots cells of each colour of its slab and keeps their rows
// (diagonal and its reciprocal, six coefficients, r) in registers for all
// sweeps, so a colour pass loads the neighbours' z from its own shared
// memory, updates, stores, and pushes the cells of a slab's outer planes
// into the neighbours' copies through distributed shared memory; a cluster
// barrier ends the pass.  Levels of one group of slots a thread run on CTA 0
// alone, by as many warps as have cells, between CTA barriers: with one slot
// a pass of 0.3 us against 0.6 us over the cluster (whose barrier with remote
// stores in flight takes 0.45 us); at 16^3 one CTA's shared memory and issue
// slots lose (1.0 us a pass against 0.6).  A warp skips the groups in which it
// has no cell to update (air above the water: 64^3 5+5 147 us an iteration
// against 149, 93 x 70 x 61 113 against 115).
// What bounds it: the instructions and latency of a pass (shared-memory
// loads, the update's dependent arithmetic, the barrier), not bytes.  In
// single precision a thread's slots go in pairs through the packed two-wide
// multiply-add.  Each update is smooth7's arithmetic in the same order, with
// the same bits.  Levels 32^3 to 8^3 of a 64^3 dam break, a V-cycle: 41 us
// with 2+2 sweeps and 20 at the bottom (68 as fused sweeps at 32^3 and one
// CTA below), 57 us with 5+5 (115), each 3 us less since warps skip air.
namespace cl {
constexpr int kThreads = 512;
constexpr int kMaxCtas = 16;
// cells of one colour per thread: 10 registers of row each, two colours
// (float: 80 of the 128 registers a 512-thread CTA allows)
template <class T> constexpr int kSlots = sizeof(T) == 4 ? 4 : 2;
constexpr size_t kSmemBytes = 216 * 1024;
// A slot's row in memory: kVecs 16-byte vectors (-d, -c[6], 1 / d) and a
// word of flags, each kind contiguous over the slots of one colour.
template <class T> constexpr int kVecs = int(8 * sizeof(T) / 16);
template <class T> __host__ __device__ constexpr int row_bytes(int items) { return items * (16 * kVecs<T> + 4); }
// flags: the diagonal is not small (the sweeps update the cell); the slot
// holds a cell; its plane is the slab's first / last with a neighbour CTA on
// that side; the cell has a row (it is not air); neighbours +x, -x, +y, -y,
// +z, -z of the row; its diagonal lies beyond kMaxDiag.  Bits 16 and up: the
// cell's index in the slab's z.
constexpr unsigned kUpdate = 1, kCell = 2, kLeft = 4, kRight = 8, kRow = 16, kNeighbour = 32, kSlow = 32 << 6;
constexpr int kIndexShift = 16;
// ClusterSlots::quotient rounds correctly from numerators of kMinNum to kMaxNum
// under diagonals of at most kMaxDiag (and at least is_small's bound): the
// remainders are then multiples of the least positive number, the quotient a
// normal one.  Smaller numerators are scaled by kScale first.
template <class T> constexpr T kMinNum = sizeof(T) == 4 ? T(0x1p-98) : T(0x1p-900);
template <class T> constexpr T kMaxNum = sizeof(T) == 4 ? T(0x1p98) : T(0x1p900);
template <class T> constexpr T kMaxDiag = sizeof(T) == 4 ? T(0x1p26) : T(0x1p100);
template <class T> constexpr T kScale = sizeof(T) == 4 ? T(0x1p96) : T(0x1p1000);
// half of the least positive number, scaled
template <class T> constexpr T kHalfLeast = sizeof(T) == 4 ? T(0x1p-54) : T(0x1p-75);
}  // namespace cl

// A level in its slabs' axes: planes of x over (y, z), or (SWAP) planes of y
// over (x, z).
template <class T> struct ClusterLevel {
    int nx, ny, nz;  // extent along the planes' axis, along the other one, along z
    int ctas;    // CTAs of the level: 1 (CTA 0 alone) or the whole cluster
    int planes;  // planes per CTA
    int hz;      // cells of one colour per row, rounded up
    int items;   // slots of one colour per CTA: planes * ny * hz, rounded up to 4
    int zoff;    // z in shared memory: planes + 2 planes
    int roff;    // r in shared memory: planes planes
    int rowoff;  // the CTA's rows in shared memory, in bytes (-1: they stay in global memory)
    unsigned char* rows;  // [ctas][2 colours][row_bytes(items)]
    T* r;
    T* z;
    // index in the level's arrays of cell a (plane 0 lies before the slab) of the slab that starts at plane x0
    template <bool SWAP> __device__ __forceinline__ long long global(int a, int x0) const {
        if (!SWAP) return (long long)(x0 - 1) * (ny * nz) + a;
        const int p = a / (ny * nz), rem = a - p * (ny * nz), y = rem / nz;
        return ((long long)y * nx + (x0 - 1 + p)) * nz + (rem - y * nz);
    }
};

template <class T> struct ClusterLevels {
    int first, last;
    int resoff;  // residuals of the level being restricted, in shared memory
    int zend;    // end of the levels' z in shared memory
    ClusterLevel<T> L[kMaxLevels];
};

// Cell of slot q of a colour: its plane within the slab, y and z.
template <class T>
__device__ __forceinline__ bool cluster_slot(const ClusterLevel<T>& L, int cta, int colour, int q, int& p, int& y,
                                             int& z) {
    const int row = q / L.hz;
    p = row / L.ny;
    y = row - p * L.ny;
    const int x = cta * L.planes + p;
    z = 2 * (q - row * L.hz) + ((colour + x + y) & 1);
    return p < L.planes && x < L.nx && z < L.nz;
}

// Rows of every cluster level, once per BuildLHS, in slot order: the visits
// read them coalesced instead of gathering 15 values a cell.
template <class T> struct ClusterMatrix {
    LevelK<T> L[kMaxLevels];
};
template <class T>
__global__ void __launch_bounds__(256) k_cluster_rows(ClusterLevels<T> c, ClusterMatrix<T> A, int swap) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    int l = c.first;
    for (; l <= c.last; ++l) {
        const int n = c.L[l].ctas * 2 * c.L[l].items;
        if (t < n) break;
        t -= n;
    }
    if (l > c.last) return;
    const ClusterLevel<T>& C = c.L[l];
    const LevelK<T>& L = A.L[l];
    const int half = t / C.items, q = t - half * C.items;  // half: (cta, colour)
    const int cta = half >> 1, colour = half & 1;
    const int sy = L.nz, sx = L.ny * L.nz;
    T w[8] = {T(0), T(0), T(0), T(0), T(0), T(0), T(0), T(0)};
    unsigned m = unsigned(C.ny * C.nz) << cl::kIndexShift;  // an empty slot still points into the slab
    int p, y, z;
    if (cluster_slot(C, cta, colour, q, p, y, z)) {
        const int plane = cta * C.planes + p;
        m = cl::kCell | (unsigned((p + 1) * (C.ny * C.nz) + y * C.nz + z) << cl::kIndexShift);
        if (C.ctas > 1 && p == 0 && plane > 0) m |= cl::kLeft;
        if (C.ctas > 1 && p == C.planes - 1 && plane + 1 < C.nx) m |= cl::kRight;
        const int x = swap ? y : plane;
        if (swap) y = plane;
        const int i = x * sx + y * sy + z;
        if (L.type[i] != 0) {  // an air cell's row is empty
            const T d = L.diag[i];
            m |= cl::kRow;
            w[0] = -d;
            const bool on[6] = {x + 1 < L.nx && L.type[i + sx] == 2, x > 0 && L.type[i - sx] == 2,
                                y + 1 < L.ny && L.type[i + sy] == 2, y > 0 && L.type[i - sy] == 2,
                                z + 1 < L.nz && L.type[i + 1] == 2,  z > 0 && L.type[i - 1] == 2};
            if (on[0]) w[1] = -L.cx[i];
            if (on[1]) w[2] = -L.cx[i - sx];
            if (on[2]) w[3] = -L.cy[i];
            if (on[3]) w[4] = -L.cy[i - sy];
            if (on[4]) w[5] = -L.cz[i];
            if (on[5]) w[6] = -L.cz[i - 1];
#pragma unroll
            for (int e = 0; e < 6; ++e) m |= on[e] ? cl::kNeighbour << e : 0u;
            if (!is_small(d)) {
                m |= cl::kUpdate;
                w[7] = X<T>::div(T(1), d);
                if (!(fabs(d) <= cl::kMaxDiag<T>)) m |= cl::kSlow;
            }
        }
    }
    unsigned char* row = C.rows + size_t(half) * cl::row_bytes<T>(C.items);
    constexpr int per = 16 / int(sizeof(T));
#pragma unroll
    for (int v = 0; v < cl::kVecs<T>; ++v)
#pragma unroll
        for (int j = 0; j < per; ++j) reinterpret_cast<T*>(row + (size_t(v) * C.items + q) * 16)[j] = w[v * per + j];
    reinterpret_cast<uint32_t*>(row + size_t(cl::kVecs<T>) * C.items * 16)[q] = m;
}

// Copies of a slot's z in the neighbouring CTAs' halo planes: the first
// plane goes after the left CTA's last (which holds `planes` planes), the
// last one before the right CTA's first.
struct ClusterSides {
    uint32_t left, right;  // z index 0's address in the neighbours, moved by the slab
};
template <class T>
__device__ __forceinline__ ClusterSides cluster_sides(const ClusterLevel<T>& L, unsigned rank, const T* z) {
    ClusterSides o{0, 0};
    if (L.ctas > 1) {
        const int slab = L.planes * L.ny * L.nz * int(sizeof(T));
        if (rank > 0) o.left = map_rank(smem_addr(z), rank - 1) + slab;
        if (int(rank) + 1 < L.ctas) o.right = map_rank(smem_addr(z), rank + 1) - slab;
    }
    return o;
}
template <class T> __device__ __forceinline__ void cluster_push(const ClusterSides& o, unsigned m, int a, T v) {
    if (m & (cl::kLeft | cl::kRight)) {
        if (m & cl::kLeft) st_cluster(o.left + a * int(sizeof(T)), v);
        if (m & cl::kRight) st_cluster(o.right + a * int(sizeof(T)), v);
    }
}

template <class T>
__device__ __forceinline__ const unsigned char* cluster_rows(const ClusterLevel<T>& L, int cta, const T* sm, int c) {
    const unsigned char* rows = L.rowoff >= 0 ? reinterpret_cast<const unsigned char*>(sm) + L.rowoff
                                              : L.rows + size_t(cta) * 2 * cl::row_bytes<T>(L.items);
    return rows + c * cl::row_bytes<T>(L.items);
}

// The residual of slot q of a colour as the tile kernels form it for every
// operand: an absent neighbour is not read (0 times an infinity there is not
// 0).  d: the cell's diagonal.
template <class T, bool SWAP>
__device__ __forceinline__ T cluster_exact(const ClusterLevel<T>& L, int cta, int c, int q, T rv, T& d) {
    extern __shared__ __align__(16) unsigned char smem[];
    const T* sm = reinterpret_cast<const T*>(smem);
    const unsigned char* row = cluster_rows(L, cta, sm, c);
    const unsigned m = reinterpret_cast<const uint32_t*>(row + size_t(cl::kVecs<T>) * L.items * 16)[q];
    T w[8];
#pragma unroll
    for (int v = 0; v < cl::kVecs<T>; ++v) {
        const uint4 u = reinterpret_cast<const uint4*>(row)[v * L.items + q];
        memcpy(&w[v * (16 / int(sizeof(T)))], &u, 16);
    }
    const int sx = SWAP ? L.nz : L.ny * L.nz, sy = SWAP ? L.ny * L.nz : L.nz, step[6] = {sx, -sx, sy, -sy, 1, -1};
    const T* z = sm + L.zoff + (m >> cl::kIndexShift);
    d = -w[0];
    T ax = T(0);
    if (m & cl::kRow) {
        ax = X<T>::mul(z[0], d);
#pragma unroll
        for (int e = 0; e < 6; ++e)
            if (m & (cl::kNeighbour << e)) ax = fma(z[step[e]], -w[1 + e], ax);
    }
    return X<T>::sub(rv, ax);
}
// For the operands that ClusterSlots leaves to them: the residual, and a
// sweep's update of the cell (m: its flags) and of its copies.
template <class T, bool SWAP>
__device__ __noinline__ T cluster_exact_residual(const ClusterLevel<T>& L, int cta, int c, int q, T rv) {
    T d;
    return cluster_exact<T, SWAP>(L, cta, c, q, rv, d);
}
template <class T, bool SWAP>
__device__ __forceinline__ void cluster_exact_update(const ClusterLevel<T>& L, int cta, int c, int q, T rv, unsigned m,
                                                     T w, int variant) {
    extern __shared__ __align__(16) unsigned char smem[];
    T* z = reinterpret_cast<T*>(smem) + L.zoff;
    const int a = int(m >> cl::kIndexShift);
    T d;
    const T res = cluster_exact<T, SWAP>(L, cta, c, q, rv, d);
    z[a] = smooth_update(z[a], X<T>::div(res, d), w, variant);
    cluster_push(cluster_sides(L, unsigned(cta), z), m, a, z[a]);
}

// Rows of a thread's slots: NK of each colour, in groups of W.
template <class T, int NK, bool SWAP> struct ClusterSlots {
    static constexpr int W = (sizeof(T) == 4 && NK >= 2) ? 2 : 1, G = NK / W;
    using V = Lanes<T, W>;
    using P = typename V::P;
    P nd[2][G], y[2][G], r[2][G], nc[2][G][6];  // -d, 1 / d, r, -c
    unsigned m[2][NK];
    bool slow;  // a diagonal of this thread's is beyond kMaxDiag
    __device__ __forceinline__ int a(int c, int k) const { return int(m[c][k] >> cl::kIndexShift); }

    __device__ __forceinline__ void load(const ClusterLevel<T>& L, int cta, const T* __restrict__ sm, bool r_global) {
        slow = false;
        const int sx = L.ny * L.nz;
        const T* rs = sm + L.roff - sx;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const unsigned char* row = cluster_rows(L, cta, sm, c);
#pragma unroll
            for (int g = 0; g < G; ++g) {
                T w[W][8], rv[W];
#pragma unroll
                for (int j = 0; j < W; ++j) {
                    const int k = g * W + j, q = int(threadIdx.x) + k * cl::kThreads;
                    m[c][k] = unsigned(sx) << cl::kIndexShift;  // empty: points into the slab, no flags
                    rv[j] = T(0);
#pragma unroll
                    for (int e = 0; e < 8; ++e) w[j][e] = T(0);
                    if (q >= L.items) continue;
                    m[c][k] = reinterpret_cast<const uint32_t*>(row + size_t(cl::kVecs<T>) * L.items * 16)[q];
#pragma unroll
                    for (int v = 0; v < cl::kVecs<T>; ++v) {
                        const uint4 u = reinterpret_cast<const uint4*>(row)[v * L.items + q];
                        memcpy(&w[j][v * (16 / int(sizeof(T)))], &u, 16);
                    }
                    slow |= (m[c][k] & cl::kSlow) != 0;
                    if (m[c][k] & cl::kCell) rv[j] = r_global ? L.r[L.template global<SWAP>(a(c, k), cta * L.planes)] : rs[a(c, k)];
                }
                T t[W];
                auto gather = [&](int e) {
#pragma unroll
                    for (int j = 0; j < W; ++j) t[j] = w[j][e];
                    return V::pack(t);
                };
                nd[c][g] = gather(0);
#pragma unroll
                for (int e = 0; e < 6; ++e) nc[c][g][e] = gather(1 + e);
                y[c][g] = gather(7);
                r[c][g] = V::pack(rv);
            }
        }
    }

    // r - A z of group g of a colour, in ax7's order on negated coefficients (the same roundings); an absent
    // neighbour adds 0 (its coefficient), or makes the result NaN where its z is not finite.  zc: the cells' own z.
    __device__ __forceinline__ P residual(int c, int g, const T* z, int plane, int row, P& zc) const {
        const int sx = SWAP ? row : plane, sy = SWAP ? plane : row;  // steps of the grid's x and y
        T v[7][W];
#pragma unroll
        for (int j = 0; j < W; ++j) {
            const T* p = z + a(c, g * W + j);
            v[0][j] = p[sx];
            v[1][j] = p[-sx];
            v[2][j] = p[sy];
            v[3][j] = p[-sy];
            v[4][j] = p[1];
            v[5][j] = p[-1];
            v[6][j] = p[0];
        }
        zc = V::pack(v[6]);
        P ax = V::mul(zc, nd[c][g]);
#pragma unroll
        for (int e = 0; e < 6; ++e) ax = V::fmadd(V::pack(v[e]), nc[c][g][e], ax);
        return V::add(r[c][g], ax);
    }

    // n / d, correctly rounded, from y = 1 / d correctly rounded: two
    // corrected quotients with exact remainders (P. Markstein, "Computation
    // of elementary functions on the IBM RISC System/6000 processor", IBM J.
    // Res. Dev. 34(1), 1990: a quotient within one unit in the last place,
    // corrected by its exact remainder times the correctly rounded
    // reciprocal, is the rounded quotient).  Five dependent multiply-adds,
    // two cells at a time, instead of a division each.  Holds for operands
    // that rare() does not name.
    __device__ __forceinline__ P quotient(int c, int g, P n) const {
        const P q0 = V::mul(n, y[c][g]);
        const P q1 = V::fmadd(V::fmadd(nd[c][g], q0, n), y[c][g], q0);
        return V::fmadd(V::fmadd(nd[c][g], q1, n), y[c][g], q1);
    }

    // rare: one of the group's numerators lies outside kMinNum .. kMaxNum and
    // is not 0 (less one, the pattern of 0 is the largest), or a diagonal of
    // the thread is too large.  Tested on bit patterns, off the quotients'
    // chain and behind the stores, so that no pass waits for it (comparisons
    // of every numerator within the chain: 0.06 us of a 0.26 us pass).  Solves
    // do meet such numerators, where z decays through air gaps, so they have a
    // path of their own (93 x 70 x 61: all of them through
    // cluster_exact_update cost 8% of an iteration).
    static __device__ __forceinline__ unsigned key(float n) { return 2u * __float_as_uint(n); }
    static __device__ __forceinline__ unsigned key(double n) {
        return 2u * unsigned(__double2hiint(n)) | unsigned(__double2loint(n) != 0);
    }
    static __device__ __forceinline__ bool small(T n) { return key(n) - 1u < key(cl::kMinNum<T>) - 1u; }
    __device__ __forceinline__ bool rare(P n) const {
        T nv[W];
        V::unpack(n, nv);
        unsigned least = ~0u, most = 0u;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            least = min(least, key(nv[j]) - 1u);
            most = max(most, key(nv[j]));
        }
        return least < key(cl::kMinNum<T>) - 1u || most > key(cl::kMaxNum<T>) || slow;
    }
    // The group's quotients q again where numerators are small: scaled by a
    // power of two they round as the others; scaled back they are exact where
    // they are normal numbers, and below rounded once more, which differs from
    // one rounding only where the scaled quotient lies half-way between two
    // numbers.  exact: the lanes left to cluster_exact_update.
    __device__ __forceinline__ P scaled_quotient(int c, int g, P n, P q, unsigned& exact) const {
        const T up[2] = {cl::kScale<T>, cl::kScale<T>}, down[2] = {T(1) / cl::kScale<T>, T(1) / cl::kScale<T>};
        const P large = quotient(c, g, V::mul(n, V::pack(up))), back = V::mul(large, V::pack(down));
        T nv[W], qv[W], lv[W], bv[W];
        V::unpack(n, nv);
        V::unpack(q, qv);
        V::unpack(large, lv);
        V::unpack(back, bv);
        exact = 0u;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            const bool once = fabs(lv[j] - bv[j] * cl::kScale<T>) != cl::kHalfLeast<T>;
            const bool ok = !(m[c][g * W + j] & cl::kSlow) && (small(nv[j]) ? once : key(nv[j]) <= key(cl::kMaxNum<T>));
            if (small(nv[j])) qv[j] = bv[j];
            if (!ok && (m[c][g * W + j] & cl::kUpdate)) exact |= 1u << j;
        }
        return V::pack(qv);
    }
};

// Ends a step of level l: the cluster's barrier, or that of CTA 0's warps
// that have cells of the level.  Every level has a CTA barrier of its own:
// warps without cells of a level wait at the next finer level's barrier
// meanwhile, and one barrier takes one thread count.
static_assert(kMaxLevels + 1 <= 16, "a hardware barrier per level beside __syncthreads's");
__device__ __forceinline__ void cluster_step(bool wide, int l, int threads) {
    if (wide) cluster_barrier();
    else asm volatile("bar.sync %0, %1;" ::"r"(l + 1), "r"(threads) : "memory");
}

constexpr int kVisitDown = 0, kVisitLast = 1, kVisitUp = 2;

// One visit of level l on the way down (smooth, restrict: PressureSolver.cpp:796-819),
// at the bottom (smooth), or on the way up (prolong: :774-794, smooth).
// threads: the threads of this CTA that take part (all of them where the level is the cluster's).
template <class T, int NK, bool SWAP>
__device__ __noinline__ void cluster_visit(const ClusterLevels<T>& c, int l, int mode, unsigned rank, T w, int variant,
                                           int sweeps, int threads) {
    extern __shared__ __align__(16) unsigned char smem[];  // named here too, so that every access is a shared one
    T* sm = reinterpret_cast<T*>(smem);
    using S = ClusterSlots<T, NK, SWAP>;
    using V = typename S::V;
    using P = typename S::P;
    constexpr int W = S::W, G = S::G;
    const ClusterLevel<T>& F = c.L[l];
    const bool wide = F.ctas > 1;
    const int sy = F.nz, sx = F.ny * F.nz, x0 = int(rank) * F.planes;
    T* z = sm + F.zoff;
    const ClusterSides side = cluster_sides(F, rank, z);
    S s;
    s.load(F, int(rank), sm, l == c.first);
    if (mode == kVisitUp) {
        const ClusterLevel<T>& C = c.L[l + 1];
        const int csx = C.ny * C.nz;
        if (C.ctas == 1) cluster_step(wide, l, threads);  // the coarser level is CTA 0's, by fewer warps perhaps
        // the coarse planes above this slab's planes: C's own z, or copies in place of the residuals
        const int X0 = x0 >> 1;
        const T* zc = sm + C.zoff + csx;
        if (wide) {
            const int X1 = min(((x0 + F.planes - 1) >> 1) + 1, C.nx);
            T* copy = sm + c.resoff;
            for (int i = threadIdx.x; i < (X1 - X0) * csx; i += threads) {
                const int X = X0 + i / csx, own = C.ctas > 1 ? X / C.planes : 0;
                copy[i] = ld_cluster<T>(map_rank(smem_addr(zc + (X - own * C.planes) * csx + i % csx), own));
            }
            zc = copy;
            __syncthreads();
        }
#pragma unroll
        for (int cc = 0; cc < 2; ++cc)
#pragma unroll
            for (int k = 0; k < NK; ++k) {
                if (!(s.m[cc][k] & cl::kCell)) continue;
                const int a = s.a(cc, k), p = a / sx - 1, rem = a - (p + 1) * sx, y = rem / sy;
                const int X = (x0 + p) >> 1, Y = y >> 1, Z = (rem - y * sy) >> 1;
                if (X >= C.nx || Y >= C.ny || Z >= C.nz) continue;
                const T v = z[a] + zc[(X - X0) * csx + Y * C.nz + Z];
                z[a] = v;
                cluster_push(side, s.m[cc][k], a, v);
            }
        cluster_step(wide, l, threads);
    }
    T wv[W];
#pragma unroll
    for (int j = 0; j < W; ++j) wv[j] = w;
    const P wp = V::pack(wv);
    unsigned wet = 0;  // groups (colour 0's, colour 1's) in which this warp has a cell to update
#pragma unroll
    for (int k = 0; k < 2 * NK; ++k)
        wet |= __any_sync(0xffffffffu, s.m[k / NK][k % NK] & cl::kUpdate) ? 1u << (k / W) : 0u;
    for (int n = 0; n < sweeps; ++n)
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
#pragma unroll
            for (int g = 0; g < G; ++g) {
                if (!(wet >> (cc * G + g) & 1u)) continue;
                P zc;
                const P res = s.residual(cc, g, z, sx, sy, zc);
                const P t = s.quotient(cc, g, res);
                auto store = [&](P q, unsigned skip) {
                    T out[W];
                    if (variant == LHI_SMOOTHER_DAMPED_GS) {
                        V::unpack(V::fmadd(wp, q, zc), out);
                    } else {
                        T tv[W], zv[W];
                        V::unpack(q, tv);
                        V::unpack(zc, zv);
#pragma unroll
                        for (int j = 0; j < W; ++j) out[j] = smooth_update(zv[j], tv[j], w, variant);
                    }
#pragma unroll
                    for (int j = 0; j < W; ++j) {
                        const unsigned m = s.m[cc][g * W + j];
                        if ((m & cl::kUpdate) && !(skip >> j & 1u)) {
                            z[s.a(cc, g * W + j)] = out[j];
                            cluster_push(side, m, s.a(cc, g * W + j), out[j]);
                        }
                    }
                };
                store(t, 0u);
                if (s.rare(res)) {  // again, behind the stores; the neighbours' z is the other colour's
                    unsigned exact;
                    store(s.scaled_quotient(cc, g, res, t, exact), exact);
                    if (exact) {
                        T zv[W], rv[W];
                        V::unpack(zc, zv);
                        V::unpack(s.r[cc][g], rv);
#pragma unroll
                        for (int j = 0; j < W; ++j)
                            if (exact >> j & 1u) {
                                z[s.a(cc, g * W + j)] = zv[j];
                                cluster_exact_update<T, SWAP>(F, int(rank), cc,
                                                              int(threadIdx.x) + (g * W + j) * cl::kThreads, rv[j],
                                                              s.m[cc][g * W + j], w, variant);
                            }
                    }
                }
            }
            cluster_step(wide, l, threads);
        }
    if (mode != kVisitDown) {
#pragma unroll
        for (int cc = 0; cc < 2; ++cc)
#pragma unroll
            for (int k = 0; k < NK; ++k)
                if (s.m[cc][k] & cl::kCell) F.z[F.template global<SWAP>(s.a(cc, k), x0)] = z[s.a(cc, k)];
        return;
    }
    T* res = sm + c.resoff - sx;
#pragma unroll
    for (int cc = 0; cc < 2; ++cc)
#pragma unroll
        for (int g = 0; g < G; ++g) {
            P zc;
            T rv[W];
            V::unpack(s.residual(cc, g, z, sx, sy, zc), rv);
#pragma unroll
            for (int j = 0; j < W; ++j) {
                if (!(s.m[cc][g * W + j] & cl::kCell)) continue;
                if (rv[j] != rv[j]) {
                    T ro[W];
                    V::unpack(s.r[cc][g], ro);
                    rv[j] = cluster_exact_residual<T, SWAP>(F, int(rank), cc,
                                                            int(threadIdx.x) + (g * W + j) * cl::kThreads, ro[j]);
                }
                res[s.a(cc, g * W + j)] = rv[j];
            }
        }
    // a coarse plane's children can lie in two slabs where the slabs have an odd number of planes
    if (wide && !(F.planes & 1)) __syncthreads();
    else cluster_step(wide, l, threads);
    // the coarse planes whose first child plane lies in this slab; their r goes to its owner
    const ClusterLevel<T>& C = c.L[l + 1];
    const int csx = C.ny * C.nz;
    const int X0 = (x0 + 1) >> 1, X1 = min((x0 + F.planes + 1) >> 1, C.nx);
    for (int i = threadIdx.x; i < (X1 - X0) * csx; i += threads) {
        const int X = X0 + i / csx, rem = i % csx;
        const int Y = rem / C.nz, Z = rem - Y * C.nz;
        T rv[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {  // in the reference's order, x first
            const int kp = SWAP ? (k >> 1) & 1 : k >> 2, ky = SWAP ? k >> 2 : (k >> 1) & 1;
            const int p = 2 * X + kp - x0, fy = 2 * Y + ky, fz = 2 * Z + (k & 1);
            const bool next = p >= F.planes;
            const T* src = sm + c.resoff + ((next ? 0 : p) * F.ny + fy) * F.nz + fz;
            if (next) rv[k] = ld_cluster<T>(map_rank(smem_addr(src), rank + 1));
            else rv[k] = *src;
        }
        T acc = T(0);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc = T(double(acc) + 0.125 * double(rv[k]));
        const int own = C.ctas > 1 ? X / C.planes : 0;
        T* dst = sm + C.roff + (X - own * C.planes) * csx + rem;
        if (own == int(rank)) *dst = acc;
        else st_cluster(map_rank(smem_addr(dst), own), acc);
        C.r[C.template global<SWAP>(csx + rem, X)] = acc;
    }
    cluster_step(wide, l, threads);  // the next level's r is ready, and no CTA still reads these residuals
}

template <class T, bool SWAP>
__global__ void __launch_bounds__(cl::kThreads, 1)
    k_coarse_cycle(const __grid_constant__ ClusterLevels<T> c, T w, int variant, int pre, int post, int fin,
                   const int* __restrict__ stop) {
    if (*stop) return;  // the same for every CTA: no kernel that sets it runs beside this one
    extern __shared__ __align__(16) unsigned char smem[];
    T* sm = reinterpret_cast<T*>(smem);
    const unsigned rank = cluster_rank();
    const bool wide = c.L[c.first].ctas > 1;  // more CTAs than one
    // the rows that are read from shared memory start on their way (every
    // thread waits for its own copies before the first barrier)
    for (int l = c.first; l <= c.last; ++l) {
        const ClusterLevel<T>& L = c.L[l];
        if (L.rowoff < 0 || (L.ctas == 1 && rank != 0)) continue;
        const int n16 = 2 * cl::row_bytes<T>(L.items) / 16;
        const unsigned char* src = L.rows + size_t(rank) * 2 * cl::row_bytes<T>(L.items);
        for (int i = threadIdx.x; i < n16; i += cl::kThreads) copy16_async(smem + L.rowoff + 16 * i, src + 16 * i);
    }
    for (int i = threadIdx.x; i < c.zend; i += cl::kThreads) sm[i] = T(0);
    copy_async_wait();
    if (wide) cluster_barrier();
    else __syncthreads();
    const int n = c.last - c.first;
    for (int step = 0; step <= 2 * n; ++step) {
        const int l = step <= n ? c.first + step : c.last - (step - n);
        const int mode = step < n ? kVisitDown : step == n ? kVisitLast : kVisitUp;
        const int sweeps = mode == kVisitDown ? pre : mode == kVisitLast ? fin : post;
        const ClusterLevel<T>& L = c.L[l];
        const int threads = L.ctas > 1 ? cl::kThreads : max(32, min(cl::kThreads, (L.items + 31) & ~31));
        if ((L.ctas == 1 && rank != 0) || int(threadIdx.x) >= threads) continue;
        if (L.items <= cl::kThreads) cluster_visit<T, 1, SWAP>(c, l, mode, rank, w, variant, sweeps, threads);
        else if (L.items <= 2 * cl::kThreads) cluster_visit<T, 2, SWAP>(c, l, mode, rank, w, variant, sweeps, threads);
        else cluster_visit<T, cl::kSlots<T>, SWAP>(c, l, mode, rank, w, variant, sweeps, threads);
    }
    if (wide) cluster_barrier();  // no CTA leaves while another may still reach its shared memory
}

template <class T>
__global__ void __launch_bounds__(kTileThreads) k_precond_none_t(LevelK<T> L, TileK tk, const T* __restrict__ r,
                                                                 T* __restrict__ z, const int* __restrict__ stop) {
    if (*stop) return;
    for_tiles(tk, L.nx, L.ny, L.nz, [&](int x, int y, int zz, long long i) {
        if (L.type[i] != 0) z[i] = r[i];
    });
}
template <class T>
__global__ void __launch_bounds__(kTileThreads) k_precond_jacobi_t(LevelK<T> L, TileK tk, const T* __restrict__ r,
                                                                   T* __restrict__ z, const int* __restrict__ stop) {
    if (*stop) return;
    for_tiles(tk, L.nx, L.ny, L.nz, [&](int x, int y, int zz, long long i) {
        T d = L.diag[i];
        if (!is_small(d)) z[i] = r[i] / d;
    });
}

// ---------------------------------------------------------------- PCG
struct CgConf {
    int region;
    int maxit;
    int every;       // true residual every k iterations (0 = never)
    int flexible;
    int rel;         // LHI_TOL_RELATIVE
    double tol;
    cudaGraphConditionalHandle cond;
    int use_cond;
    int warm;        // LHI_GUESS_PREVIOUS: the relative threshold comes from ||b||, not ||r0||
};

// Stopping rule after an update of r (PressureSolver.cpp:889-902): with a
// true-residual period, every k-th iteration and every apparent convergence
// is decided on r = b - A x instead (the next kernel computes it).
__device__ void cg_decide(SolveScalars* sc, double res2, const CgConf& cf, bool after_true) {
    const double residual = sqrt(res2);
    sc->residual = residual;
    if (!after_true) {
        sc->iter += 1;
        if (cf.every > 0 && (sc->iter % cf.every == 0 || residual < sc->threshold)) {
            sc->true_now = 1;
            return;
        }
    } else {
        sc->true_now = 0;
    }
    const bool conv = residual < sc->threshold;
    const bool bad = !isfinite(residual);
    const bool stop = conv || bad || sc->iter >= cf.maxit || sc->iter >= kGraphIterationCap;
    sc->status = bad ? LHI_E_NAN : (conv ? LHI_OK : LHI_E_NOT_CONVERGED);
    if (stop) sc->stop = 1;
    if (cf.use_cond) cudaGraphSetConditional(cf.cond, stop ? 0u : 1u);
}

// A loop-body kernel that finds the solve stopped by another kernel (a
// bounded wait that ran out) ends the graph's while loop: the iteration that
// set the conditional to continue did so before the stop.
__device__ __forceinline__ void cg_end_loop(const CgConf& cf) {
    if (cf.use_cond && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(cf.cond, 0u);
}

// r0 = rhs on fluid cells (PressureSolver.cpp:847-856)
template <class T>
__global__ void __launch_bounds__(kTileThreads) k_cg_init_r(LevelK<T> L, TileK tk, const T* __restrict__ rhs, T* __restrict__ r) {
    for_tiles(tk, L.nx, L.ny, L.nz, [&](int x, int y, int z, long long i) {
        if (L.type[i] != 0) r[i] = rhs[i];
    });
}

// LHI_GUESS_PREVIOUS: x keeps the last solve's values on the cells that are
// fluid now and is 0 elsewhere (so the pressure written from it is 0 off
// the liquid, as the reference's cleared grid has it).
template <class TX>
__global__ void k_x_fluid_only(long long n, const uint8_t* __restrict__ type, TX* __restrict__ x) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && type[i] != 2) x[i] = TX(0);
}

// LHI_GUESS_PREVIOUS: r0 = b - A x0 on the cells with a row (where the
// reference's r0 = b is set), and sum b^2 over them into red[0]: the
// relative stopping rule's reference norm.
template <class T, class TX>
__global__ void __launch_bounds__(kTileThreads) k_cg_init_warm(LevelK<T> L, TileK tk, const T* __restrict__ b,
                                                               const TX* __restrict__ x, T* __restrict__ r,
                                                               double* __restrict__ partials,
                                                               unsigned* __restrict__ counter,
                                                               SolveScalars* __restrict__ sc) {
    double v[1] = {0.0};
    for_tiles(tk, L.nx, L.ny, L.nz, [&](int xi, int yi, int zi, long long i) {
        if (L.type[i] == 0) return;
        r[i] = T(double(b[i]) - ax_at<double>(L, x, i, xi, yi, zi));
        v[0] += double(b[i]) * double(b[i]);
    });
    double tot[1];
    if (!grid_sum_last<1>(v, partials, counter, tot)) return;
    sc->red[0] = tot[0];
}

// p = z on fluid cells; rz = r.z and rr = r.r over all cells; the stopping
// threshold from ||r0|| (PressureSolver.cpp:858-871)
template <class T>
__global__ void __launch_bounds__(kTileThreads) k_cg_init_p(LevelK<T> L, TileK tk, const T* __restrict__ r,
                                                            const T* __restrict__ z, T* __restrict__ p,
                                                            double* __restrict__ partials, unsigned* __restrict__ counter,
                                                            SolveScalars* __restrict__ sc, CgConf cf) {
    double v[2] = {0.0, 0.0};
    for_tiles(tk, L.nx, L.ny, L.nz, [&](int x, int y, int zz, long long i) {
        const T zi = z[i], ri = r[i];
        if (L.type[i] != 0) p[i] = zi;
        v[0] += double(ri) * double(zi);
        v[1] += double(ri) * double(ri);
    });
    double tot[2];
    if (!grid_sum_last<2>(v, partials, counter, tot)) return;
    sc->rz_old = tot[0];
    sc->rr_all = tot[1];
    const double r0 = sqrt(tot[1]);
    const T t = T(cf.tol);
    sc->residual0 = r0;
    sc->residual = r0;
    // with a previous solution as the guess, ||r|| is measured against ||b|| (k_cg_init_warm)
    const double ref = cf.warm ? sqrt(sc->red[0]) : r0;
    sc->threshold = cf.rel ? double(T(t * T(ref))) : double(t);
    sc->iter = 0;
    sc->true_now = 0;
    // a zero right-hand side is solved by x = 0 (under the relative rule the
    // threshold is then 0 as well, and r0 < threshold never holds)
    const bool conv = r0 < sc->threshold || r0 == 0.0;
    const bool stop = conv || cf.maxit <= 0;
    sc->status = conv ? LHI_OK : LHI_E_NOT_CONVERGED;
    sc->stop = stop ? 1 : 0;
    if (cf.use_cond) cudaGraphSetConditional(cf.cond, stop ? 0u : 1u);
}

// ------------------------------------------------- TMA-staged SpMV
// Ap = A p with p.Ap for the finest level, one 8 x 8 x 32 tile per step: p
// grown by one cell in x and y (z from z0-4), diag, the coefficients with
// the -x / -y / -z neighbours' faces, and the neighbour mask staged by TMA.
// A thread owns (x0 + warp, z0 + lane) and the tile's 8 rows, as k_cg_spmv
// does; the CTAs take other tiles than k_cg_spmv's, so p.Ap is grouped
// differently in its last bits.
namespace sp {
constexpr int kP = layout::kPBox, kD = layout::kDBox, kCX = layout::kCXBox, kCY = layout::kCYBox,
              kCZ = layout::kCZBox, kM = kD;
constexpr uint32_t kTx = uint32_t((kP + kD + kCX + kCY + kCZ) * 4 + kM);
// offsets inside one stage; two mbarriers, then two stages
constexpr int oP = 0, oD = oP + kP * 4, oCX = oD + kD * 4, oCY = oCX + kCX * 4, oCZ = oCY + kCY * 4,
              oM = oCZ + kCZ * 4, kStage = oM + kM;
constexpr int kBase = 128, kSmem = kBase + 2 * kStage;
static_assert(kP * 4 % 128 == 0 && kCX * 4 % 128 == 0 && kCZ * 4 % 128 == 0 && kStage % 128 == 0,
              "128-byte aligned boxes");
}  // namespace sp

__device__ __forceinline__ void sp_issue(unsigned char* st, uint64_t* bar, const CUtensorMap* mp, const CUtensorMap* md,
                                         const CUtensorMap* mcx, const CUtensorMap* mcy, const CUtensorMap* mcz,
                                         const CUtensorMap* mm, int x0, int y0, int z0) {
    fence_proxy_async();
    bar_expect_tx(bar, sp::kTx);
    tma_load_box(st + sp::oP, mp, z0 - 4, y0 - 1, x0 - 1, bar);
    tma_load_box(st + sp::oD, md, z0, y0, x0, bar);
    tma_load_box(st + sp::oCX, mcx, z0, y0, x0 - 1, bar);
    tma_load_box(st + sp::oCY, mcy, z0, y0 - 1, x0, bar);
    tma_load_box(st + sp::oCZ, mcz, z0 - 4, y0, x0, bar);
    tma_load_box(st + sp::oM, mm, z0, y0, x0, bar);
}

// Two CTAs per SM, each walking its tiles through two stages (the next
// tile's boxes in flight while the current one is multiplied).
__global__ void __launch_bounds__(kTileThreads, 2)
    k_spmv_tma(const __grid_constant__ CUtensorMap mp, const __grid_constant__ CUtensorMap md,
               const __grid_constant__ CUtensorMap mcx, const __grid_constant__ CUtensorMap mcy,
               const __grid_constant__ CUtensorMap mcz, const __grid_constant__ CUtensorMap mm, int nx, int ny, int nz,
               const int32_t* __restrict__ ids, const int* __restrict__ count, int tdy, int tdz, float* __restrict__ ap,
               double* __restrict__ partials, unsigned* __restrict__ counter, SolveScalars* __restrict__ sc,
               CgConf cf) {
    if (sc->stop) return;
    extern __shared__ __align__(128) unsigned char sm[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm);
    if (threadIdx.x == 0) {
        bar_init(&bar[0], 1);
        bar_init(&bar[1], 1);
    }
    __syncthreads();
    double v[1] = {0.0};
    const int units = *count;
    const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0 && int(blockIdx.x) < units) {
        int a, b, c;
        tile_origin(ids, blockIdx.x, tdy, tdz, a, b, c);
        sp_issue(sm + sp::kBase, &bar[0], &mp, &md, &mcx, &mcy, &mcz, &mm, a, b, c);
    }
    bool failed = false;
    int it = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x, ++it) {
        const int s = it & 1;
        const unsigned char* st = sm + sp::kBase + s * sp::kStage;
        int x0, y0, z0;
        tile_origin(ids, u, tdy, tdz, x0, y0, z0);
        const int un = u + int(gridDim.x);
        if (threadIdx.x == 0 && un < units) {  // the other stage was released by the last barrier
            int a, b, c;
            tile_origin(ids, un, tdy, tdz, a, b, c);
            sp_issue(sm + sp::kBase + (s ^ 1) * sp::kStage, &bar[s ^ 1], &mp, &md, &mcx, &mcy, &mcz, &mm, a, b, c);
        }
        if (__syncthreads_or(!bar_wait(&bar[s], (it >> 1) & 1, g_stage_wait_ns))) {  // every thread leaves together
            if (threadIdx.x == 0) {  // drain this CTA's copies in flight (the one given up on, the prefetch)
                bar_wait(&bar[s], (it >> 1) & 1);
                if (un < units) bar_wait(&bar[s ^ 1], ((it + 1) >> 1) & 1);
            }
            failed = true;
            break;
        }
        const float* Ps = reinterpret_cast<const float*>(st + sp::oP);
        const float* Ds = reinterpret_cast<const float*>(st + sp::oD);
        const float* CXs = reinterpret_cast<const float*>(st + sp::oCX);
        const float* CYs = reinterpret_cast<const float*>(st + sp::oCY);
        const float* CZs = reinterpret_cast<const float*>(st + sp::oCZ);
        const uint8_t* Ms = st + sp::oM;
        const int x = x0 + wp, zz = z0 + lane;
        if (x < nx && zz < nz) {
#pragma unroll
            for (int ly = 0; ly < kTileY; ++ly) {
                const int y = y0 + ly;
                if (y >= ny) break;
                const int pi = layout::sp_p(wp, ly, lane);
                const int ci = layout::sp_c(wp, ly, lane);
                const unsigned m = Ms[ci];
                const float pc = Ps[pi];
                float a = 0.f;
                if (m & 64u) {
                    a = pc * Ds[ci];
                    if (m & 1u) a += Ps[pi + layout::kPStepX] * CXs[layout::sp_cx(wp, ly, lane)];
                    if (m & 2u) a += Ps[pi - layout::kPStepX] * CXs[layout::sp_cx_minus(wp, ly, lane)];
                    if (m & 4u) a += Ps[pi + layout::kPStepY] * CYs[layout::sp_cy(wp, ly, lane)];
                    if (m & 8u) a += Ps[pi - layout::kPStepY] * CYs[layout::sp_cy_minus(wp, ly, lane)];
                    if (m & 16u) a += Ps[pi + 1] * CZs[layout::sp_cz(wp, ly, lane)];
                    if (m & 32u) a += Ps[pi - 1] * CZs[layout::sp_cz_minus(wp, ly, lane)];
                }
                ap[((long long)x * ny + y) * nz + zz] = a;
                if ((m & 64u) && in_region(x, y, zz, nx, ny, nz, cf.region)) v[0] += double(pc) * double(a);
            }
        }
        __syncthreads();
    }
    if (failed && threadIdx.x == 0) {
        sc->timeout = 1;
        sc->status = LHI_E_TIMEOUT;
        sc->stop = 1;
    }
    // every CTA takes part in the grid-wide sum, a failed one too
    double tot[1];
    if (!grid_sum_last<1>(v, partials, counter, tot)) return;
    sc->denom = tot[0];
    sc->alpha = sc->rz_old / tot[0];
}

// ------------------------------------------------- TMA restriction
// CGSolver<3>::Restrict from one active fine tile: z grown by one cell, r,
// diag, coefficients and mask staged by TMA; the residual r - A z of the
// tile's 2048 cells goes to shared memory, then each of its 4 x 4 x 16
// coarse cells sums its 8 children in the reference's order (restrict_cell_batched).
// Coarse cells whose children all lie in inactive fine tiles are air cells
// whose restriction is 0, which they already hold.
namespace rs {
constexpr int kR = 8 * 8 * 32;
constexpr int oP = 128, oR = oP + sp::kP * 4, oD = oR + kR * 4, oCX = oD + sp::kD * 4, oCY = oCX + sp::kCX * 4,
              oCZ = oCY + sp::kCY * 4, oM = oCZ + sp::kCZ * 4, oRes = oM + sp::kM, kSmem = oRes + kR * 4;
constexpr uint32_t kTx = sp::kTx + kR * 4;
}  // namespace rs

__global__ void __launch_bounds__(kTileThreads, 3)
    k_restrict_tma(const __grid_constant__ CUtensorMap mz, const __grid_constant__ CUtensorMap mr,
                   const __grid_constant__ CUtensorMap md, const __grid_constant__ CUtensorMap mcx,
                   const __grid_constant__ CUtensorMap mcy, const __grid_constant__ CUtensorMap mcz,
                   const __grid_constant__ CUtensorMap mm, int nx, int ny, int nz, const int32_t* __restrict__ ids,
                   const int* __restrict__ count, int tdy, int tdz, int cnx, int cny, int cnz, float* __restrict__ rc,
                   float* __restrict__ zc, SolveScalars* __restrict__ sc) {
    if (sc->stop) return;
    extern __shared__ __align__(128) unsigned char sm[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm);
    const float* Ps = reinterpret_cast<const float*>(sm + rs::oP);
    const float* Rs = reinterpret_cast<const float*>(sm + rs::oR);
    const float* Ds = reinterpret_cast<const float*>(sm + rs::oD);
    const float* CXs = reinterpret_cast<const float*>(sm + rs::oCX);
    const float* CYs = reinterpret_cast<const float*>(sm + rs::oCY);
    const float* CZs = reinterpret_cast<const float*>(sm + rs::oCZ);
    const uint8_t* Ms = sm + rs::oM;
    float* Res = reinterpret_cast<float*>(sm + rs::oRes);
    if (threadIdx.x == 0) bar_init(bar, 1);
    __syncthreads();
    const int units = *count;
    const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned parity = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
        int x0, y0, z0;
        tile_origin(ids, u, tdy, tdz, x0, y0, z0);
        if (threadIdx.x == 0) {
            fence_proxy_async();
            bar_expect_tx(bar, rs::kTx);
            tma_load_box(sm + rs::oP, &mz, z0 - 4, y0 - 1, x0 - 1, bar);
            tma_load_box(sm + rs::oR, &mr, z0, y0, x0, bar);
            tma_load_box(sm + rs::oD, &md, z0, y0, x0, bar);
            tma_load_box(sm + rs::oCX, &mcx, z0, y0, x0 - 1, bar);
            tma_load_box(sm + rs::oCY, &mcy, z0, y0 - 1, x0, bar);
            tma_load_box(sm + rs::oCZ, &mcz, z0 - 4, y0, x0, bar);
            tma_load_box(sm + rs::oM, &mm, z0, y0, x0, bar);
        }
        if (__syncthreads_or(!bar_wait(bar, parity, g_stage_wait_ns))) {  // every thread leaves together
            if (threadIdx.x == 0) {
                sc->timeout = 1;
                sc->status = LHI_E_TIMEOUT;
                sc->stop = 1;
                bar_wait(bar, parity);  // the copy given up on lands before the CTA exits
            }
            __syncthreads();
            return;
        }
        parity ^= 1u;
        float res[kTileY];  // all rows first, then the stores: their loads overlap
#pragma unroll
        for (int ly = 0; ly < kTileY; ++ly) {
            const int pi = layout::sp_p(wp, ly, lane);
            const int ci = layout::sp_c(wp, ly, lane);
            const unsigned m = Ms[ci];
            const float zc0 = Ps[pi];
            float a = 0.f;
            if (m & 64u) {
                a = zc0 * Ds[ci];
                if (m & 1u) a += Ps[pi + layout::kPStepX] * CXs[layout::sp_cx(wp, ly, lane)];
                if (m & 2u) a += Ps[pi - layout::kPStepX] * CXs[layout::sp_cx_minus(wp, ly, lane)];
                if (m & 4u) a += Ps[pi + layout::kPStepY] * CYs[layout::sp_cy(wp, ly, lane)];
                if (m & 8u) a += Ps[pi - layout::kPStepY] * CYs[layout::sp_cy_minus(wp, ly, lane)];
                if (m & 16u) a += Ps[pi + 1] * CZs[layout::sp_cz(wp, ly, lane)];
                if (m & 32u) a += Ps[pi - 1] * CZs[layout::sp_cz_minus(wp, ly, lane)];
            }
            res[ly] = Rs[ci] - a;
        }
#pragma unroll
        for (int ly = 0; ly < kTileY; ++ly) Res[layout::sp_c(wp, ly, lane)] = res[ly];
        __syncthreads();
        {
            int i, j, k;
            layout::rs_coarse(threadIdx.x, i, j, k);
            const int cx = (x0 >> 1) + i, cy = (y0 >> 1) + j, cz = (z0 >> 1) + k;
            if (cx < cnx && cy < cny && cz < cnz) {
                float acc = 0.f;
#pragma unroll
                for (int c8 = 0; c8 < 8; ++c8) {
                    const float res = Res[layout::rs_child(i, j, k, c8)];
                    acc = float(double(acc) + 0.125 * double(res));
                }
                const long long o = ((long long)cx * cny + cy) * cnz + cz;
                rc[o] = acc;
                zc[o] = 0.f;
            }
        }
        __syncthreads();
    }
}

// Ap = A p; p.Ap over the update region; alpha = rz / p.Ap (PressureSolver.cpp:873-888).
// A work unit is every ysplit-th row (four or eight) of a tile, row by row, for
// the reason of k_sweep (93 x 70 x 61: 13 us with four rows loaded ahead, 10 now).
template <class T>
__global__ void __launch_bounds__(kTileThreads, sizeof(T) == 4 ? 6 : 3)
    k_cg_spmv(LevelK<T> L, TileK tk, const T* __restrict__ p, T* __restrict__ ap, double* __restrict__ partials,
              unsigned* __restrict__ counter, SolveScalars* __restrict__ sc, CgConf cf) {
    if (sc->stop) return;
    double v[1] = {0.0};
    for_tiles(tk, L.nx, L.ny, L.nz, [&](int x, int y, int z, long long i) {
        Cell7<T, T> c;
        load7(L, p, i, x, y, z, c);
        const T a = ax7<T>(c);
        ap[i] = a;
        if (c.tc != 0 && in_region(x, y, z, L.nx, L.ny, L.nz, cf.region)) v[0] += double(c.zc) * double(a);
    });
    double tot[1];
    if (!grid_sum_last<1>(v, partials, counter, tot)) return;
    sc->denom = tot[0];
    sc->alpha = sc->rz_old / tot[0];
}

// x += alpha p; r -= alpha Ap; ||r||^2 over the update region; then the
// stopping rule (PressureSolver.cpp:889-902)
template <class T, class TX, int R>
__global__ void __launch_bounds__(kTileThreads) k_cg_update_xr(LevelK<T> L, TileK tk, const T* __restrict__ p,
                                                               const T* __restrict__ ap, TX* __restrict__ x,
                                                               T* __restrict__ r, double* __restrict__ partials,
                                                               unsigned* __restrict__ counter,
                                                               SolveScalars* __restrict__ sc, CgConf cf) {
    if (sc->stop) {
        cg_end_loop(cf);
        return;
    }
    const double alpha = sc->alpha;
    double v[1] = {0.0};
    for_tile_cols(tk, L.nx, L.ny, L.nz, [&](int xi, int zi, long long i0, int yb, int rows, int ys) {
        const long long st = (long long)ys * L.nz;
        bool on[R];
        TX xv[R];
        T pv[R], rv[R], av[R];
#pragma unroll
        for (int k = 0; k < R; ++k)
            on[k] = k < rows && L.type[i0 + k * st] != 0 && in_region(xi, yb + k * ys, zi, L.nx, L.ny, L.nz, cf.region);
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (on[k]) {
                xv[k] = x[i0 + k * st];
                pv[k] = p[i0 + k * st];
                rv[k] = r[i0 + k * st];
                av[k] = ap[i0 + k * st];
            }
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (on[k]) {
                x[i0 + k * st] = TX(double(xv[k]) + alpha * double(pv[k]));
                const T rn = T(double(rv[k]) - alpha * double(av[k]));
                r[i0 + k * st] = rn;
                v[0] += double(rn) * double(rn);
            }
    });
    double tot[1];
    if (!grid_sum_last<1>(v, partials, counter, tot)) return;
    sc->res2 = tot[0];
    cg_decide(sc, tot[0], cf, false);
}

// r = b - A x on the update region (stored when `store`, as TR), summed
// squares.  The mixed mode passes its FP64 finest-level matrix and
// right-hand side here (T = double) with the FP32 residual (TR = float).
template <class T, class TX, class TR>
__device__ __forceinline__ void true_residual_sweep(const LevelK<T>& L, const TileK& tk, int region, const T* __restrict__ b,
                                                    const TX* __restrict__ x, TR* __restrict__ r, bool store, double& acc) {
    for_tiles(tk, L.nx, L.ny, L.nz, [&](int xi, int yi, int zi, long long i) {
        if (L.type[i] == 0 || !in_region(xi, yi, zi, L.nx, L.ny, L.nz, region)) return;
        const double res = double(b[i]) - ax_at<double>(L, x, i, xi, yi, zi);
        if (store) r[i] = TR(res);
        acc += res * res;
    });
}

template <class T, class TX, class TR = T>
__global__ void __launch_bounds__(kTileThreads) k_cg_true_residual(LevelK<T> L, TileK tk, const T* __restrict__ b,
                                                                   const TX* __restrict__ x, TR* __restrict__ r,
                                                                   double* __restrict__ partials,
                                                                   unsigned* __restrict__ counter,
                                                                   SolveScalars* __restrict__ sc, CgConf cf) {
    if (sc->stop) {
        cg_end_loop(cf);
        return;
    }
    if (!sc->true_now) return;
    double v[1] = {0.0};
    true_residual_sweep(L, tk, cf.region, b, x, r, true, v[0]);
    double tot[1];
    if (!grid_sum_last<1>(v, partials, counter, tot)) return;
    sc->res2 = tot[0];
    sc->true2 = tot[0];
    cg_decide(sc, tot[0], cf, true);
}

// ||b - A x||^2 of the final iterate (not stored)
template <class T, class TX>
__global__ void __launch_bounds__(kTileThreads) k_true_residual_final(LevelK<T> L, TileK tk, int region,
                                                                      const T* __restrict__ b, const TX* __restrict__ x,
                                                                      double* __restrict__ partials,
                                                                      unsigned* __restrict__ counter,
                                                                      double* __restrict__ out) {
    double v[1] = {0.0};
    true_residual_sweep<T, TX, T>(L, tk, region, b, x, nullptr, false, v[0]);
    grid_sum_finish<1>(v, partials, counter, out);
}

// rz_new = r.z over all cells (Array3::Reduce); Ap.z over the update region;
// beta (PressureSolver.cpp:905-912): Fletcher-Reeves, or Polak-Ribiere
// -alpha Ap.z / rz_old when flexible
template <class T, int R>
__global__ void __launch_bounds__(kTileThreads) k_cg_dot_rz(LevelK<T> L, TileK tk, const T* __restrict__ r,
                                                            const T* __restrict__ z, const T* __restrict__ ap,
                                                            double* __restrict__ partials, unsigned* __restrict__ counter,
                                                            SolveScalars* __restrict__ sc, CgConf cf) {
    if (sc->stop) return;
    double v[2] = {0.0, 0.0};
    for_tile_cols(tk, L.nx, L.ny, L.nz, [&](int xi, int zz, long long i0, int yb, int rows, int ys) {
        const long long st = (long long)ys * L.nz;
        bool on[R];
        T zv[R], rv[R], av[R];
#pragma unroll
        for (int k = 0; k < R; ++k) {
            on[k] = k < rows && L.type[i0 + k * st] != 0 && in_region(xi, yb + k * ys, zz, L.nx, L.ny, L.nz, cf.region);
            if (k < rows) {
                zv[k] = z[i0 + k * st];
                rv[k] = r[i0 + k * st];
            }
        }
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (on[k]) av[k] = ap[i0 + k * st];
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if (k >= rows) break;
            v[0] += double(rv[k]) * double(zv[k]);
            if (on[k]) v[1] += double(av[k]) * double(zv[k]);
        }
    });
    double tot[2];
    if (!grid_sum_last<2>(v, partials, counter, tot)) return;
    const double rz_new = tot[0], apz = tot[1];
    sc->rz_new = rz_new;
    sc->apz = apz;
    sc->beta = cf.flexible ? (-sc->alpha * apz / sc->rz_old) : (rz_new / sc->rz_old);
    sc->rz_old = rz_new;
}

// p = z + beta p on fluid cells (PressureSolver.cpp:913-921)
template <class T, int R>
__global__ void __launch_bounds__(kTileThreads) k_cg_update_p(LevelK<T> L, TileK tk, const T* __restrict__ z,
                                                              T* __restrict__ p, const SolveScalars* __restrict__ sc) {
    if (sc->stop) return;
    const double beta = sc->beta;
    for_tile_cols(tk, L.nx, L.ny, L.nz, [&](int x, int zz, long long i0, int yb, int rows, int ys) {
        const long long st = (long long)ys * L.nz;
        bool on[R];
        T zv[R], pv[R];
#pragma unroll
        for (int k = 0; k < R; ++k) on[k] = k < rows && L.type[i0 + k * st] != 0;
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (on[k]) {
                zv[k] = z[i0 + k * st];
                pv[k] = p[i0 + k * st];
            }
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (on[k]) p[i0 + k * st] = T(double(zv[k]) + beta * double(pv[k]));
    });
}

template <class T, class TX> __global__ void k_x_to_pressure(long long n, const TX* __restrict__ x, T* __restrict__ pr) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) pr[i] = T(x[i]);
}

template <class T>
__global__ void k_get_ax(LevelK<T> L, const T* __restrict__ x, T* __restrict__ out) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long n = (long long)L.nx * L.ny * L.nz;
    if (i >= n) return;
    int xi, yi, zi;
    decode(i, L.ny, L.nz, xi, yi, zi);
    out[i] = ax_at<T>(L, x, i, xi, yi, zi);
}

// m_Acoef[level] expanded to 6 per cell: right, left, top, bottom, front, back
template <class T> __global__ void k_expand_acoef(LevelK<T> L, T* __restrict__ out) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long n = (long long)L.nx * L.ny * L.nz;
    if (i >= n) return;
    int x, y, z;
    decode(i, L.ny, L.nz, x, y, z);
    const long long sy = L.nz, sx = (long long)L.ny * L.nz;
    T c[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
    if (L.type[i] != 0) {
        if (x + 1 < L.nx && L.type[i + sx] == 2) c[0] = L.cx[i];
        if (x - 1 >= 0 && L.type[i - sx] == 2) c[1] = L.cx[i - sx];
        if (y + 1 < L.ny && L.type[i + sy] == 2) c[2] = L.cy[i];
        if (y - 1 >= 0 && L.type[i - sy] == 2) c[3] = L.cy[i - sy];
        if (z + 1 < L.nz && L.type[i + 1] == 2) c[4] = L.cz[i];
        if (z - 1 >= 0 && L.type[i - 1] == 2) c[5] = L.cz[i - 1];
    }
    for (int k = 0; k < 6; ++k) out[6 * i + k] = c[k];
}

// --------------------------------------------------- learned preconditioner
// Cell-centre solid flag: mean of the cell's 8 node SDF values < 0.
template <class T>
__global__ void k_solid_cells(const T* __restrict__ sp, int nx, int ny, int nz, uint8_t* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long n = (long long)nx * ny * nz;
    if (i >= n) return;
    int x, y, z;
    decode(i, ny, nz, x, y, z);
    const long long sy = nz + 1, sx = (long long)(ny + 1) * (nz + 1);
    const T* b = sp + x * sx + y * sy + z;
    const double m = double(b[0]) + b[1] + b[sy] + b[sy + 1] + b[sx] + b[sx + 1] + b[sx + sy] + b[sx + sy + 1];
    out[i] = m < 0.0 ? 1 : 0;
}

// The network's cell classes: the level-0 type, with rows that the solver
// skips (diagonal below EPSILON: cells cut off by solid walls) marked 0.
template <class T>
__global__ void k_net_type(const uint8_t* __restrict__ type, const T* __restrict__ diag, long long n,
                           uint8_t* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = is_small(diag[i]) ? 0 : type[i];
}

// e = A z - r; sums of e^2 and r^2 over all cells
template <class T>
__global__ void k_loss_residual(LevelK<T> L, const float* __restrict__ z, const T* __restrict__ r, float* __restrict__ e,
                                double* __restrict__ partials, unsigned* __restrict__ counter, double* __restrict__ out) {
    double v[2] = {0.0, 0.0};
    const long long n = (long long)L.nx * L.ny * L.nz;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        int x, y, zz;
        decode(i, L.ny, L.nz, x, y, zz);
        const double ei = ax_at<double>(L, z, i, x, y, zz) - double(r[i]);
        e[i] = float(ei);
        v[0] += ei * ei;
        v[1] += double(r[i]) * double(r[i]);
    }
    grid_sum_finish<2>(v, partials, counter, out);
}

// dz = 2 A^T e / (sum r^2 * batch); the loss sum e^2 / sum r^2 / batch is added to out[2]
template <class T>
__global__ void k_loss_grad(LevelK<T> L, const float* __restrict__ e, int batch, float* __restrict__ dz,
                            double* __restrict__ red) {
    const long long n = (long long)L.nx * L.ny * L.nz;
    const double rr = red[1] > 0 ? red[1] : 1.0;
    const double scale = 2.0 / (rr * batch);
    const long long sy = L.nz, sx = (long long)L.ny * L.nz;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        int x, y, z;
        decode(i, L.ny, L.nz, x, y, z);
        const uint8_t ti = L.type[i];
        double acc = 0.0;
        if (ti != 0) acc = double(L.diag[i]) * e[i];
        if (ti == 2) {  // A(j, i) = [t_j >= 1][t_i == 2] c_ij
            if (x + 1 < L.nx && L.type[i + sx] != 0) acc += double(L.cx[i]) * e[i + sx];
            if (x > 0 && L.type[i - sx] != 0) acc += double(L.cx[i - sx]) * e[i - sx];
            if (y + 1 < L.ny && L.type[i + sy] != 0) acc += double(L.cy[i]) * e[i + sy];
            if (y > 0 && L.type[i - sy] != 0) acc += double(L.cy[i - sy]) * e[i - sy];
            if (z + 1 < L.nz && L.type[i + 1] != 0) acc += double(L.cz[i]) * e[i + 1];
            if (z > 0 && L.type[i - 1] != 0) acc += double(L.cz[i - 1]) * e[i - 1];
        }
        dz[i] = float(scale * acc);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) red[2] += red[0] / rr / batch;
}

}  // namespace

// ------------------------------------------------------------- host side
// Work units per tile: enough units to fill `grid` CTAs, at least min_split.
static int ysplit_for(int ntiles, int grid, int min_split) {
    int s = min_split;
    while (s < kTileY && ntiles * s * 2 <= grid) s *= 2;
    return s;
}
template <class T> static TileK tile_k(const LevelDev<T>& L, const int* count, int grid, int min_split = 1) {
    return TileK{L.tiles, count, L.tdim[1], L.tdim[2], ysplit_for(L.ntiles, grid, min_split)};
}
// persistent CTAs for a tile kernel on level L (0 when the level is empty)
template <class T> static unsigned tile_blocks(const LevelDev<T>& L, int grid, int min_split = 1) {
    const long long units = (long long)L.ntiles * ysplit_for(L.ntiles, grid, min_split);
    return unsigned(std::min<long long>(units, grid));
}
constexpr int kFewRows = 2;              // rows of a unit at a split of kSplit
constexpr int kSplit = kTileY / kFewRows;  // of k_cg_spmv and, on levels of few tiles, of the column kernels
// The column kernels (prolongation, CG vectors) hold all rows of a unit: two on
// levels of up to kColsTiles tiles, where more CTAs at work count for more than
// the loads a thread has in flight, eight above.  A PCG iteration with two and
// with eight: 432 tiles (96^3, FP64) 163 and 169 us, 1024 (128^3, FP64) 213 and
// 218, 1152 (125 x 141 x 99) 161.0 and 159.3, 2000 (160^3, mixed) 231 and 229.5.
constexpr int kColsTiles = 1024;
template <class T> static int cols_split(const LevelDev<T>& L) { return L.ntiles <= kColsTiles ? kSplit : 1; }

template <class T, class TX> double LiquidImpl<T, TX>::read_scalar(const double* dptr) {
    double v;
    LHI_CUDA(cudaMemcpyAsync(&v, dptr, sizeof(double), cudaMemcpyDeviceToHost, stream_));
    LHI_CUDA(cudaStreamSynchronize(stream_));
    return v;
}

template <class T, class TX> void LiquidImpl<T, TX>::read_scalars() {
    LHI_CUDA(cudaMemcpyAsync(sc_host_, sc_, sizeof(SolveScalars), cudaMemcpyDeviceToHost, stream_));
    LHI_CUDA(cudaStreamSynchronize(stream_));
}

// CGSolver<3>::Init (PressureSolver.cpp:666-680)
template <class T, class TX> void LiquidImpl<T, TX>::solver_init() {
    LHI_CUDA(cudaMemsetAsync(p_, 0, sizeof(T) * ncell_, cur_));
    if (sp_.initial_guess != LHI_GUESS_PREVIOUS)  // else the last solution is the guess (k_x_fluid_only)
        LHI_CUDA(cudaMemsetAsync(x_, 0, sizeof(TX) * ncell_, cur_));
    LHI_CUDA(cudaMemsetAsync(rhs_, 0, sizeof(T) * ncell_, cur_));
    for (int l = 0; l < nlev_; ++l) {
        LevelDev<T>& L = lv_[l];
        if (L.n == 0) continue;
        LHI_CUDA(cudaMemsetAsync(L.r, 0, sizeof(T) * L.n, cur_));
        LHI_CUDA(cudaMemsetAsync(L.z, 0, sizeof(T) * L.n, cur_));
        LHI_CUDA(cudaMemsetAsync(L.diag, 0, sizeof(T) * L.n, cur_));
        for (int a = 0; a < 3; ++a) LHI_CUDA(cudaMemsetAsync(L.cf[a], 0, sizeof(T) * L.n, cur_));
    }
    LHI_CUDA(cudaMemsetAsync(sc_, 0, sizeof(SolveScalars), cur_));
}

template <class T, class TX> void LiquidImpl<T, TX>::build_rhs() {
    auto ps_ = scope(LHI_KERNEL_GRID);
    if constexpr (kHiResidual) {
        k_build_rhs_mixed<T><<<blocks_for(ncell_, 256), 256, 0, cur_>>>(
            nx_, ny_, nz_, dx_[0], dx_[1], dx_[2], dxd_[0], dxd_[1], dxd_[2], liquid_phi_, lw_[0], lw_[1], lw_[2],
            v_[0], v_[1], v_[2], rhs_, rhs_hi_);
    } else {
        k_build_rhs<T><<<blocks_for(ncell_, 256), 256, 0, cur_>>>(nx_, ny_, nz_, dx_[0], dx_[1], dx_[2], liquid_phi_,
                                                                  lw_[0], lw_[1], lw_[2], v_[0], v_[1], v_[2], rhs_);
    }
    LHI_LAUNCH_CHECK();
}

// CGSolver<3>::BuildLHS (PressureSolver.cpp:544-664) for every level, then
// the levels' active-tile lists.
template <class T, class TX> void LiquidImpl<T, TX>::build_lhs(double rho, double dt) {
    auto ps_ = scope(LHI_KERNEL_LHS);
    for (int l = 0; l < nlev_; ++l) {
        LevelDev<T>& L = lv_[l];
        if (L.n == 0) continue;
        LevelGeom g{L.nx, L.ny, L.nz, nx_, ny_, nz_, l};
        LHI_CUDA(cudaMemsetAsync(L.tile_flag, 0, size_t(L.ntiles), cur_));
        if (l > 0 && sp_.coarse_operator == LHI_COARSE_GALERKIN) {
            k_level_galerkin<T><<<blocks_for(L.n, 256), 256, 0, cur_>>>(lk(lv_[l - 1]), L.nx, L.ny, L.nz, L.diag,
                                                                        L.cf[0], L.cf[1], L.cf[2], L.type,
                                                                        L.tile_flag, L.tdim[1], L.tdim[2]);
            LHI_LAUNCH_CHECK();
            continue;
        }
        if (l > 0) {  // the finest level's classes, tile flags and mask come with its matrix
            k_level_phi<T><<<blocks_for(L.n, 256), 256, 0, cur_>>>(g, liquid_phi_, L.phi, L.type, L.tile_flag,
                                                                  L.tdim[1], L.tdim[2]);
            LHI_LAUNCH_CHECK();
        }
        const T* phi = (l == 0) ? liquid_phi_ : L.phi;
        bool done = false;
        if constexpr (kHiResidual) {
            if (l == 0) {  // with the FP64 matrix of the outer residual
                k_level_matrix_mixed<T><<<blocks_for(L.n, 256), 256, 0, cur_>>>(
                    g, phi, lw_[0], lw_[1], lw_[2], L.h[0], L.h[1], L.h[2], T(dt), T(rho), L.diag, L.cf[0], L.cf[1],
                    L.cf[2], L.type, L.tile_flag, L.tdim[1], L.tdim[2], L.fused ? L.mask : nullptr, L.mpitch, dxd_[0],
                    dxd_[1], dxd_[2], dt, rho, diag_hi_, cf_hi_[0], cf_hi_[1], cf_hi_[2]);
                LHI_LAUNCH_CHECK();
                done = true;
            }
        }
        if (!done) {
            k_level_matrix<T><<<blocks_for(L.n, 256), 256, 0, cur_>>>(
                g, phi, lw_[0], lw_[1], lw_[2], L.h[0], L.h[1], L.h[2], T(dt), T(rho), L.diag, L.cf[0], L.cf[1],
                L.cf[2], l == 0 ? L.type : nullptr, L.tile_flag, L.tdim[1], L.tdim[2],
                (l == 0 && L.fused) ? L.mask : nullptr, L.mpitch);
            LHI_LAUNCH_CHECK();
        }
    }
    build_tiles();
    build_masks();
    net_type_fresh_ = false;
}

// The coarse kernel's view of levels [first, nlev): slabs, shared-memory
// layout, rows.  In shared memory: every level's z, every level's r, the
// residuals, then the rows of the levels below the first, and the first
// level's where they still fit (they are read twice a cycle).
template <class T, class TX> static ClusterLevels<T> coarse_view(const LiquidImpl<T, TX>& s, int first) {
    const bool swap = s.coarse_swap_;  // slabs of y
    ClusterLevels<T> c{};
    c.first = first;
    c.last = s.nlev_ - 1;
    long long off = 4, slab = 0;  // the neighbours of an empty slot may lie just outside its level's z
    unsigned char* rows = static_cast<unsigned char*>(s.coarse_rows_);
    for (int l = c.first; l <= c.last; ++l) {
        const LevelDev<T>& D = s.lv_[l];
        ClusterLevel<T>& L = c.L[l];
        L.nx = swap ? D.ny : D.nx;
        L.ny = swap ? D.nx : D.ny;
        L.nz = D.nz;
        L.hz = (D.nz + 1) / 2;
        // CTA 0 alone where its threads hold the whole level in one group of slots each (FP32: a pair).  8 x 12 x 16
        // cells at the bottom of a two-level cycle: 68 us an iteration against 72 over the cluster, 12^3 below 24^3:
        // 91 and 95; in more slots the cluster is better (11 x 14 x 16: 73 and 84, 14^3: 77 and 90, 12^3 in FP64: 106
        // and 113)
        const bool solo = (long long)D.nx * D.ny * L.hz <= (sizeof(T) == 4 ? 2 : 1) * cl::kThreads;
        L.ctas = solo ? 1 : s.coarse_ctas_;
        L.planes = (L.nx + L.ctas - 1) / L.ctas;
        L.items = int(std::min(((long long)L.planes * L.ny * L.hz + 3) / 4 * 4, 1LL << 24));
        L.zoff = int(off);
        off += (long long)(L.planes + 2) * L.ny * L.nz;
        L.rows = rows;
        if (rows) rows += size_t(L.ctas) * 2 * cl::row_bytes<T>(L.items);
        L.r = D.r;
        L.z = D.z;
        slab = std::max(slab, (long long)L.planes * L.ny * L.nz);
    }
    off += 4;
    c.zend = int(off);
    for (int l = c.first; l <= c.last; ++l) {
        c.L[l].roff = int(off);
        off += (long long)c.L[l].planes * c.L[l].ny * c.L[l].nz;
    }
    c.resoff = int(off);
    off = ((off + slab) * (long long)sizeof(T) + 15) / 16 * 16;  // bytes from here on
    for (int l = c.last; l >= c.first; --l) {
        const long long bytes = 2LL * cl::row_bytes<T>(c.L[l].items);
        const bool fits = off + bytes <= (long long)cl::kSmemBytes;
        c.L[l].rowoff = fits ? int(off) : -1;
        if (fits) off += bytes;
    }
    return c;
}
template <class T> static size_t coarse_smem(const ClusterLevels<T>& c) {
    long long slab = 0, end = 0;
    for (int l = c.first; l <= c.last; ++l) {
        const ClusterLevel<T>& L = c.L[l];
        slab = std::max(slab, (long long)L.planes * L.ny * L.nz);
        if (L.rowoff >= 0) end = std::max(end, L.rowoff + 2LL * cl::row_bytes<T>(L.items));
    }
    return size_t(std::max(end, ((c.resoff + slab) * (long long)sizeof(T) + 15) / 16 * 16));
}

template <class T, class TX> void LiquidImpl<T, TX>::build_masks() {
    for (int l = 1; l < coarse_level_; ++l) {  // level 0's mask comes with its matrix (k_level_matrix)
        LevelDev<T>& L = lv_[l];
        if (!L.fused) continue;
        k_level_mask<T><<<blocks_for(L.n, 256), 256, 0, cur_>>>(lk(L), L.mask, L.mpitch);
        LHI_LAUNCH_CHECK();
    }
    if (coarse_level_ < nlev_) {
        ClusterMatrix<T> m{};
        for (int l = coarse_level_; l < nlev_; ++l) m.L[l] = lk(lv_[l]);
        k_cluster_rows<T><<<blocks_for(coarse_rows_n_, 256), 256, 0, cur_>>>(coarse_view(*this, coarse_level_), m,
                                                                              int(coarse_swap_));
        LHI_LAUNCH_CHECK();
    }
}

// Levels that the fused sweep can take: FP32, z extent a multiple of 4 (TMA
// strides are multiples of 16 bytes), at least 12 cells in x and y and one
// tile (32 cells) in z.  Boxes may reach past the level in z; TMA fills that
// part with zeros, which reads as diag 0 and an empty mask.
template <class T, class TX> void LiquidImpl<T, TX>::setup_fused() {
    if constexpr (std::is_same<T, float>::value) {
        LHI_CUDA(cudaFuncSetAttribute(k_rb_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, rb::kSmem));
        LHI_CUDA(cudaFuncSetAttribute(k_restrict_tma, cudaFuncAttributeMaxDynamicSharedMemorySize, rs::kSmem));
        for (int l = 0; l < coarse_level_; ++l) {  // setup_coarse has run
            LevelDev<T>& L = lv_[l];
            if (L.n == 0 || L.nz % 4 != 0 || L.nx < 12 || L.ny < 12 || L.nz < kTileZ) continue;
            L.mpitch = (L.nz + 15) / 16 * 16;
            const size_t mb = size_t(L.nx) * L.ny * L.mpitch;
            LHI_CUDA(cudaMalloc(&L.zb, sizeof(T) * L.n));
            LHI_CUDA(cudaMalloc(&L.mask, mb));
            LHI_CUDA(cudaMemsetAsync(L.zb, 0, sizeof(T) * L.n, stream_));
            LHI_CUDA(cudaMemsetAsync(L.mask, 0, mb, stream_));
            const auto F32 = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
            L.tm_z = make_box_map(L.z, F32, 4, L.nx, L.ny, L.nz, L.nz, 12, 12, rb::kZW);
            L.tm_zb = make_box_map(L.zb, F32, 4, L.nx, L.ny, L.nz, L.nz, 12, 12, rb::kZW);
            L.tm_r = make_box_map(L.r, F32, 4, L.nx, L.ny, L.nz, L.nz, 10, 10, rb::kZW);
            L.tm_d = make_box_map(L.diag, F32, 4, L.nx, L.ny, L.nz, L.nz, 10, 10, rb::kZW);
            L.tm_cz = make_box_map(L.cf[2], F32, 4, L.nx, L.ny, L.nz, L.nz, 10, 10, rb::kZW);
            L.tm_cx = make_box_map(L.cf[0], F32, 4, L.nx, L.ny, L.nz, L.nz, 11, 10, rb::kZW);
            L.tm_cy = make_box_map(L.cf[1], F32, 4, L.nx, L.ny, L.nz, L.nz, 10, 11, rb::kZW);
            L.tm_m = make_box_map(L.mask, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, L.nx, L.ny, L.nz, L.mpitch, 10, 10,
                                  rb::kMW);
            L.ts_z = make_box_map(L.z, F32, 4, L.nx, L.ny, L.nz, L.nz, 10, 10, 40);
            L.ts_zb = make_box_map(L.zb, F32, 4, L.nx, L.ny, L.nz, L.nz, 10, 10, 40);
            L.ts_r = make_box_map(L.r, F32, 4, L.nx, L.ny, L.nz, L.nz, 8, 8, 32);
            L.ts_d = make_box_map(L.diag, F32, 4, L.nx, L.ny, L.nz, L.nz, 8, 8, 32);
            L.ts_cx = make_box_map(L.cf[0], F32, 4, L.nx, L.ny, L.nz, L.nz, 9, 8, 32);
            L.ts_cy = make_box_map(L.cf[1], F32, 4, L.nx, L.ny, L.nz, L.nz, 8, 9, 32);
            L.ts_cz = make_box_map(L.cf[2], F32, 4, L.nx, L.ny, L.nz, L.nz, 8, 8, 36);
            L.ts_m = make_box_map(L.mask, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, L.nx, L.ny, L.nz, L.mpitch, 8, 8, 32);
            L.fused = true;
        }
    }
}

// Tensor maps of the finest level's TMA SpMV (on the CG direction p).
template <class T, class TX> void LiquidImpl<T, TX>::setup_spmv() {
    if constexpr (std::is_same<T, float>::value) {
        LevelDev<T>& L = lv_[0];
        if (!L.fused) return;
        LHI_CUDA(cudaFuncSetAttribute(k_spmv_tma, cudaFuncAttributeMaxDynamicSharedMemorySize, sp::kSmem));
        const auto F32 = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
        tm_sp_[0] = make_box_map(p_, F32, 4, L.nx, L.ny, L.nz, L.nz, 10, 10, 40);
        tm_sp_[1] = make_box_map(L.diag, F32, 4, L.nx, L.ny, L.nz, L.nz, 8, 8, 32);
        tm_sp_[2] = make_box_map(L.cf[0], F32, 4, L.nx, L.ny, L.nz, L.nz, 9, 8, 32);
        tm_sp_[3] = make_box_map(L.cf[1], F32, 4, L.nx, L.ny, L.nz, L.nz, 8, 9, 32);
        tm_sp_[4] = make_box_map(L.cf[2], F32, 4, L.nx, L.ny, L.nz, L.nz, 8, 8, 36);
        tm_sp_[5] = make_box_map(L.mask, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, L.nx, L.ny, L.nz, L.mpitch, 8, 8, 32);
        spmv_tma_ = true;
    }
}

template <class T, class TX> void LiquidImpl<T, TX>::build_tiles() {
    TileLevels tl{};
    tl.nlev = 0;
    for (int l = 0; l < nlev_ && lv_[l].n > 0; ++l) {
        for (int a = 0; a < 3; ++a) tl.tdim[l][a] = lv_[l].tdim[a];
        tl.flag[l] = lv_[l].tile_flag;
        tl.ids[l] = lv_[l].tiles;
        tl.nlev = l + 1;
    }
    if (tl.nlev == 0) return;
    k_tiles_finalize<<<1, 1024, 0, cur_>>>(tl, sc_->tile_count);
    LHI_LAUNCH_CHECK();
}

template <class T, class TX> bool LiquidImpl<T, TX>::smooth(int level, int sweeps, bool final_dot) {
    LevelDev<T>& L = lv_[level];
    const unsigned G = unsigned(std::min((long long)L.ntiles * kSweepSplit, (long long)tile_grid_));
    if (L.n == 0 || sweeps <= 0 || G == 0) return false;
    const T w = T(sp_.smoothing_factor);
    const int cat = (level == 0) ? LHI_KERNEL_SMOOTH_FINE : LHI_KERNEL_SMOOTH_COARSE;
    if (L.fused && sp_.sweep_kernel == LHI_SWEEP_FUSED) {
        const unsigned GF = unsigned(std::min(L.ntiles, kSMs));
        for (int s = 0; s < sweeps; ++s) {
            auto ps_ = scope(cat);
            const int fd = (final_dot && s + 1 == sweeps) ? 1 : 0;
            k_rb_fused<<<GF, rb::kThreads, rb::kSmem, cur_>>>(
                L.tm_z, L.tm_r, L.tm_d, L.tm_cx, L.tm_cy, L.tm_cz, L.tm_m, L.nx, L.ny, L.nz, L.tiles,
                &sc_->tile_count[level], L.tdim[1], L.tdim[2], reinterpret_cast<float*>(L.zb), float(w),
                sp_.smoother, sc_, reinterpret_cast<const float*>(ap_), partials_, counter_, fd, sp_.update_region,
                sp_.cg_variant == LHI_CG_FLEXIBLE ? 1 : 0);
            LHI_LAUNCH_CHECK();
            std::swap(L.z, L.zb);
            std::swap(L.tm_z, L.tm_zb);
            std::swap(L.ts_z, L.ts_zb);
        }
        return final_dot;
    }
    const TileK tk{L.tiles, &sc_->tile_count[level], L.tdim[1], L.tdim[2], 1};  // k_sweep splits tiles by itself
    for (int s = 0; s < sweeps; ++s)
        for (int phase = 0; phase < 2; ++phase) {
            auto ps_ = scope(cat);
            k_sweep<T><<<G, kTileThreads, 0, cur_>>>(lk(L), tk, L.r, L.z, w, sp_.smoother, phase, &sc_->stop);
            LHI_LAUNCH_CHECK();
        }
    return false;
}

template <class T, class TX> void LiquidImpl<T, TX>::restrict_to(int level) {
    LevelDev<T>& C = lv_[level];
    LevelDev<T>& F = lv_[level - 1];
    if (C.n == 0) return;
    auto ps_ = scope(LHI_KERNEL_RESTRICT);
    if (F.fused && sp_.sweep_kernel == LHI_SWEEP_FUSED) {
        const unsigned GR = unsigned(std::min(F.ntiles, 3 * kSMs));
        k_restrict_tma<<<GR, kTileThreads, rs::kSmem, cur_>>>(
            F.ts_z, F.ts_r, F.ts_d, F.ts_cx, F.ts_cy, F.ts_cz, F.ts_m, F.nx, F.ny, F.nz, F.tiles,
            &sc_->tile_count[level - 1], F.tdim[1], F.tdim[2], C.nx, C.ny, C.nz, reinterpret_cast<float*>(C.r),
            reinterpret_cast<float*>(C.z), sc_);
    } else if (level >= coarse_level_) {
        k_restrict_dense<T><<<blocks_for(8 * C.n, 256), 256, 0, cur_>>>(lk(F), F.r, F.z, C.nx, C.ny, C.nz, C.r, C.z,
                                                                     &sc_->stop);
    } else {
        const unsigned G = tile_blocks(C, tile_grid_);
        k_restrict_t<T><<<G, kTileThreads, 0, cur_>>>(lk(F), F.r, F.z, C.nx, C.ny, C.nz,
                                                      tile_k(C, &sc_->tile_count[level], tile_grid_), C.r, C.z,
                                                      &sc_->stop);
    }
    LHI_LAUNCH_CHECK();
}

template <class T, class TX> void LiquidImpl<T, TX>::prolong_to(int level) {
    LevelDev<T>& C = lv_[level + 1];
    LevelDev<T>& F = lv_[level];
    const unsigned G = tile_blocks(F, tile_grid_, cols_split(F));
    if (C.n == 0 || F.n == 0 || G == 0) return;
    auto ps_ = scope(LHI_KERNEL_PROLONG);
    const TileK tk = tile_k(F, &sc_->tile_count[level], tile_grid_, cols_split(F));
    const auto kern = tk.ysplit >= kSplit ? k_prolong_t<T, kFewRows> : k_prolong_t<T, kTileY>;
    kern<<<G, kTileThreads, 0, cur_>>>(F.nx, F.ny, F.nz, tk, C.z, C.nx, C.ny, C.nz, F.z, &sc_->stop);
    LHI_LAUNCH_CHECK();
}

// CTAs of the coarse kernel's cluster (its non-portable maximum where the
// device has room for one).
template <class T> static int coarse_cluster_ctas() {
    for (const auto k : {k_coarse_cycle<T, false>, k_coarse_cycle<T, true>}) {
        LHI_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(cl::kSmemBytes)));
        LHI_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    }
    for (int n = cl::kMaxCtas; n > 8; n /= 2) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(unsigned(n));
        cfg.blockDim = dim3(cl::kThreads);
        cfg.dynamicSmemBytes = cl::kSmemBytes;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = unsigned(n);
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, k_coarse_cycle<T, false>, &cfg) == cudaSuccess && fit > 0) return n;
        cudaGetLastError();
    }
    return 8;
}

// Picks the first level (below the finest) from which on every level's slabs
// fit the cluster: at most coarse_cells cells where the caller set that, and
// slabs of at most two colours of kSlots cells a thread.  Slabs are planes of
// x, or planes of y where those let a finer level in: a level flat in x is a
// slab of its own otherwise (1 x 50 x 50 in FP64, 20 sweeps at the bottom of a
// two-level cycle: 139 us
// an iteration on the tile kernels, 76 with slabs of y).  The kernel is
// compiled for either, so that the common one's steps stay in few registers.
template <class T, class TX> void LiquidImpl<T, TX>::setup_coarse() {
    coarse_level_ = nlev_;
    coarse_smem_ = 0;
    if (nlev_ < 2) return;
    const int ctas = coarse_cluster_ctas<T>();
    const long long slots = (long long)cl::kSlots<T> * cl::kThreads;
    auto finest = [&](bool swap) {  // the finest first level that still fits
        coarse_swap_ = swap;
        int fit = nlev_;
        for (int first = nlev_ - 1; first >= 1; --first) {
            if (sp_.coarse_cells > 0 && lv_[first].n > sp_.coarse_cells) break;
            coarse_ctas_ = ctas;
            const ClusterLevels<T> c = coarse_view(*this, first);
            if (c.L[first].items > slots || coarse_smem(c) > cl::kSmemBytes) break;
            fit = first;
        }
        return fit;
    };
    const int by_y = finest(true), by_x = finest(false);
    coarse_swap_ = by_y < by_x;
    coarse_level_ = std::min(by_x, by_y);
    if (coarse_level_ == nlev_) return;
    ClusterLevels<T> c = coarse_view(*this, coarse_level_);
    coarse_ctas_ = c.L[coarse_level_].ctas;
    c = coarse_view(*this, coarse_level_);
    coarse_smem_ = coarse_smem(c);
    coarse_rows_n_ = 0;
    size_t bytes = 0;
    for (int l = c.first; l <= c.last; ++l) {
        coarse_rows_n_ += 2LL * c.L[l].ctas * c.L[l].items;
        bytes += size_t(2) * c.L[l].ctas * cl::row_bytes<T>(c.L[l].items);
    }
    LHI_CUDA(cudaMalloc(&coarse_rows_, std::max(bytes, size_t(16))));
}

// CGSolver<3>::ApplyPreconditioner multigrid branch (PressureSolver.cpp:730-771)
template <class T, class TX> void LiquidImpl<T, TX>::enqueue_vcycle() {
    T* z_at_start[kMaxLevels];
    for (int l = 0; l < nlev_; ++l) z_at_start[l] = lv_[l].z;
    enqueue_vcycle_levels();
    // an odd number of fused sweeps on a level leaves its result in the other
    // buffer: copy it back so every V-cycle starts and ends on the same one
    for (int l = 0; l < nlev_; ++l) {
        LevelDev<T>& L = lv_[l];
        if (L.z == z_at_start[l]) continue;
        LHI_CUDA(cudaMemcpyAsync(L.zb, L.z, sizeof(T) * L.n, cudaMemcpyDeviceToDevice, cur_));
        std::swap(L.z, L.zb);
        std::swap(L.tm_z, L.tm_zb);
        std::swap(L.ts_z, L.ts_zb);
    }
}

template <class T, class TX> void LiquidImpl<T, TX>::enqueue_vcycle_levels() {
    const int last = nlev_ - 1;
    const int Lc = coarse_level_;
    if (Lc <= last) {
        for (int l = 0; l < Lc; ++l) {
            smooth(l, sp_.num_pre_smooth);
            restrict_to(l + 1);
        }
        {
            auto ps_ = scope(LHI_KERNEL_SMOOTH_COARSE);
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(unsigned(coarse_ctas_));
            cfg.blockDim = dim3(cl::kThreads);
            cfg.dynamicSmemBytes = coarse_smem_;
            cfg.stream = cur_;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = unsigned(coarse_ctas_);
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            LHI_CUDA(cudaLaunchKernelEx(&cfg, coarse_swap_ ? k_coarse_cycle<T, true> : k_coarse_cycle<T, false>,
                                        coarse_view(*this, coarse_level_), T(sp_.smoothing_factor), int(sp_.smoother),
                                        int(sp_.num_pre_smooth), int(sp_.num_post_smooth), int(sp_.num_final_smooth),
                                        static_cast<const int*>(&sc_->stop)));
            LHI_LAUNCH_CHECK();
        }
        for (int l = Lc - 1; l >= 0; --l) {
            prolong_to(l);
            dot_fused_ |= smooth(l, sp_.num_post_smooth, l == 0 && fuse_dot_);
        }
    } else {
        for (int l = 0; l < last; ++l) {
            smooth(l, sp_.num_pre_smooth);
            restrict_to(l + 1);
        }
        smooth(last, sp_.num_final_smooth);
        for (int l = last - 1; l >= 0; --l) {
            prolong_to(l);
            dot_fused_ |= smooth(l, sp_.num_post_smooth, l == 0 && fuse_dot_);
        }
    }
}

template <class T, class TX> void LiquidImpl<T, TX>::vcycle() { enqueue_vcycle(); }

template <class T, class TX> void LiquidImpl<T, TX>::enqueue_precond() {
    LevelDev<T>& L0 = lv_[0];
    const unsigned G = tile_blocks(L0, tile_grid_);
    switch (sp_.preconditioner) {
        case LHI_PRECOND_NONE:
            if (G == 0) break;
            k_precond_none_t<T><<<G, kTileThreads, 0, cur_>>>(lk(L0), tile_k(L0, &sc_->tile_count[0], tile_grid_),
                                                              L0.r, L0.z, &sc_->stop);
            LHI_LAUNCH_CHECK();
            break;
        case LHI_PRECOND_JACOBI:
            if (G == 0) break;
            k_precond_jacobi_t<T><<<G, kTileThreads, 0, cur_>>>(lk(L0), tile_k(L0, &sc_->tile_count[0], tile_grid_),
                                                                L0.r, L0.z, &sc_->stop);
            LHI_LAUNCH_CHECK();
            break;
        case LHI_PRECOND_LEARNED:
            if (net_ && !use_fallback_) {
                ensure_solid_cells();
                ensure_net_type();
                const int dims[3] = {nx_, ny_, nz_};
                if (net_->sparse_enabled_ && (net_plan_stale_ || net_->plan_type_ != net_type_)) {
                    net_->plan_sparse(dims, net_type_, cur_);
                    net_plan_stale_ = false;
                }
                net_->forward(dims, reinterpret_cast<const float*>(L0.r), net_type_, solid_cell_,
                              reinterpret_cast<float*>(L0.z), 0.0, cur_, true);
                break;
            }
            enqueue_vcycle();
            break;
        default: enqueue_vcycle();
    }
}

// CGSolver<3>::ApplyPreconditioner (PressureSolver.cpp:719-772) as a stage
template <class T, class TX> void LiquidImpl<T, TX>::apply_preconditioner() {
    LHI_CUDA(cudaMemsetAsync(&sc_->stop, 0, sizeof(int), cur_));
    enqueue_precond();
}

static CgConf make_conf(const lhi_solver_params& sp, unsigned long long cond, int use_cond) {
    CgConf c;
    c.region = sp.update_region;
    c.maxit = sp.max_iterations;
    c.every = sp.true_residual_every;
    c.flexible = sp.cg_variant == LHI_CG_FLEXIBLE ? 1 : 0;
    c.rel = sp.tolerance_mode == LHI_TOL_RELATIVE ? 1 : 0;
    c.tol = sp.tolerance;
    c.cond = cond;
    c.use_cond = use_cond;
    c.warm = sp.initial_guess == LHI_GUESS_PREVIOUS ? 1 : 0;
    return c;
}

// r = b; z = M r; p = z; rz; ||r0||; threshold (PressureSolver.cpp:845-871)
template <class T, class TX> void LiquidImpl<T, TX>::enqueue_init(unsigned long long cond, int use_cond) {
    LevelDev<T>& L0 = lv_[0];
    const TileK tk = tile_k(L0, &sc_->tile_count[0], tile_grid_);
    const unsigned G = std::max(1u, tile_blocks(L0, tile_grid_));
    const CgConf cf = make_conf(sp_, cond, use_cond);
    {
        auto ps_ = scope(LHI_KERNEL_CG_VECTOR);
        if (sp_.initial_guess == LHI_GUESS_PREVIOUS) {
            k_x_fluid_only<TX><<<blocks_for(ncell_, 256), 256, 0, cur_>>>(ncell_, L0.type, x_);
            LHI_LAUNCH_CHECK();
            k_cg_init_warm<T, TX><<<G, kTileThreads, 0, cur_>>>(lk(L0), tk, rhs_, x_, L0.r, partials_, counter_, sc_);
        } else {
            k_cg_init_r<T><<<G, kTileThreads, 0, cur_>>>(lk(L0), tk, rhs_, L0.r);
        }
        LHI_LAUNCH_CHECK();
    }
    record_snapshot();
    enqueue_precond();
    {
        auto ps_ = scope(LHI_KERNEL_CG_VECTOR);
        k_cg_init_p<T><<<G, kTileThreads, 0, cur_>>>(lk(L0), tk, L0.r, L0.z, p_, partials_, counter_, sc_, cf);
        LHI_LAUNCH_CHECK();
    }
}

// One PCG iteration (PressureSolver.cpp:870-922).
template <class T, class TX> void LiquidImpl<T, TX>::enqueue_body(unsigned long long cond, int use_cond) {
    LevelDev<T>& L0 = lv_[0];
    const TileK tk = tile_k(L0, &sc_->tile_count[0], tile_grid_, cols_split(L0));
    const unsigned G = std::max(1u, tile_blocks(L0, tile_grid_, cols_split(L0)));
    const CgConf cf = make_conf(sp_, cond, use_cond);
    {
        auto ps_ = scope(LHI_KERNEL_SPMV);
        if (spmv_tma_ && sp_.sweep_kernel == LHI_SWEEP_FUSED)
            k_spmv_tma<<<std::min(G, unsigned(2 * kSMs)), kTileThreads, sp::kSmem, cur_>>>(
                tm_sp_[0], tm_sp_[1], tm_sp_[2], tm_sp_[3], tm_sp_[4], tm_sp_[5], L0.nx, L0.ny, L0.nz, L0.tiles,
                &sc_->tile_count[0], L0.tdim[1], L0.tdim[2], reinterpret_cast<float*>(ap_), partials_, counter_, sc_,
                cf);
        else
            k_cg_spmv<T><<<std::max(1u, tile_blocks(L0, tile_grid_, kSplit)), kTileThreads, 0, cur_>>>(
                lk(L0), tile_k(L0, &sc_->tile_count[0], tile_grid_, kSplit), p_, ap_, partials_, counter_, sc_, cf);
        LHI_LAUNCH_CHECK();
    }
    {
        auto ps_ = scope(LHI_KERNEL_CG_VECTOR);
        const auto kern = tk.ysplit >= kSplit ? k_cg_update_xr<T, TX, kFewRows> : k_cg_update_xr<T, TX, kTileY>;
        kern<<<G, kTileThreads, 0, cur_>>>(lk(L0), tk, p_, ap_, x_, L0.r, partials_, counter_, sc_, cf);
        LHI_LAUNCH_CHECK();
        if (sp_.true_residual_every > 0) {
            if constexpr (kHiResidual)
                k_cg_true_residual<double, TX, T><<<G, kTileThreads, 0, cur_>>>(lk_hi(*this), tk, rhs_hi_, x_, L0.r,
                                                                                partials_, counter_, sc_, cf);
            else
                k_cg_true_residual<T, TX><<<G, kTileThreads, 0, cur_>>>(lk(L0), tk, rhs_, x_, L0.r, partials_,
                                                                        counter_, sc_, cf);
            LHI_LAUNCH_CHECK();
        }
    }
    record_snapshot();
    // with the multigrid preconditioner the last level-0 sweep of the V-cycle
    // also forms r.z and Ap.z (and beta), which saves k_cg_dot_rz's pass
    fuse_dot_ = sp_.preconditioner == LHI_PRECOND_MULTIGRID;
    dot_fused_ = false;
    enqueue_precond();
    fuse_dot_ = false;
    {
        auto ps_ = scope(LHI_KERNEL_CG_VECTOR);
        if (!dot_fused_) {
            const auto kern = tk.ysplit >= kSplit ? k_cg_dot_rz<T, kFewRows> : k_cg_dot_rz<T, kTileY>;
            kern<<<G, kTileThreads, 0, cur_>>>(lk(L0), tk, L0.r, L0.z, ap_, partials_, counter_, sc_, cf);
            LHI_LAUNCH_CHECK();
        }
        const auto kern = tk.ysplit >= kSplit ? k_cg_update_p<T, kFewRows> : k_cg_update_p<T, kTileY>;
        kern<<<G, kTileThreads, 0, cur_>>>(lk(L0), tk, L0.z, p_, sc_);
        LHI_LAUNCH_CHECK();
    }
}

// grid.pressure = x (PressureSolver.cpp:933) and the final true residual
template <class T, class TX> void LiquidImpl<T, TX>::enqueue_final() {
    LevelDev<T>& L0 = lv_[0];
    const unsigned G = std::max(1u, tile_blocks(L0, tile_grid_));
    auto ps_ = scope(LHI_KERNEL_CG_VECTOR);
    k_x_to_pressure<T, TX><<<blocks_for(ncell_, 256), 256, 0, cur_>>>(ncell_, x_, pressure_);
    LHI_LAUNCH_CHECK();
    if constexpr (kHiResidual)
        k_true_residual_final<double, TX><<<G, kTileThreads, 0, cur_>>>(
            lk_hi(*this), tile_k(L0, &sc_->tile_count[0], tile_grid_), sp_.update_region, rhs_hi_, x_, partials_, counter_,
            &sc_->true2);
    else
        k_true_residual_final<T, TX><<<G, kTileThreads, 0, cur_>>>(lk(L0), tile_k(L0, &sc_->tile_count[0], tile_grid_),
                                                                   sp_.update_region, rhs_, x_, partials_, counter_,
                                                                   &sc_->true2);
    LHI_LAUNCH_CHECK();
}

// The solve after BuildLHS as one graph: init; while (!stop) { iteration };
// final.  Pointers and parameters are fixed for the handle's lifetime, so
// the graph is built on the first solve and replayed after.
// with_init: the whole solve (init, the loop, the final pass).  Without it:
// the loop from the current iterate on and the final pass (the tail of a
// solve whose first iterations ran host-driven); its loop condition starts
// at 1 at every launch, and a solve that has already stopped leaves the
// loop in its first body's first kernel.
template <class T, class TX> void LiquidImpl<T, TX>::build_solve_graph(bool with_init) {
    cudaGraph_t g = nullptr;
    LHI_CUDA(cudaStreamSynchronize(stream_));  // surfaces any earlier asynchronous error before capturing
    LHI_CUDA(cudaGetLastError());
    LHI_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
    try {
        cudaStreamCaptureStatus st;
        const cudaGraphNode_t* deps = nullptr;
        size_t nd = 0;
        cudaGraph_t cg = nullptr;
        LHI_CUDA(cudaStreamGetCaptureInfo(stream_, &st, nullptr, &cg, nullptr, nullptr));
        cudaGraphConditionalHandle h;
        if (with_init)
            LHI_CUDA(cudaGraphConditionalHandleCreate(&h, cg, 0, 0));
        else
            LHI_CUDA(cudaGraphConditionalHandleCreate(&h, cg, 1, cudaGraphCondAssignDefault));
        const long long c0 = g_kernel_launches.load();
        if (with_init) enqueue_init(h, 1);
        const long long c1 = g_kernel_launches.load();
        LHI_CUDA(cudaStreamGetCaptureInfo(stream_, &st, nullptr, &cg, &deps, &nd));
        cudaGraphNodeParams cp = {};
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = h;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        cudaGraphNode_t node;
        LHI_CUDA(cudaGraphAddNode(&node, cg, deps, nd, &cp));
        cudaGraph_t body = cp.conditional.phGraph_out[0];
        LHI_CUDA(cudaStreamUpdateCaptureDependencies(stream_, &node, 1, cudaStreamSetCaptureDependencies));
        LHI_CUDA(cudaStreamBeginCaptureToGraph(side_, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
        cur_ = side_;
        long long c2 = 0;
        try {
            enqueue_body(h, 1);
            c2 = g_kernel_launches.load();
        } catch (...) {
            cur_ = stream_;
            cudaGraph_t b2 = nullptr;
            cudaStreamEndCapture(side_, &b2);
            throw;
        }
        cur_ = stream_;
        cudaGraph_t body_out = nullptr;
        LHI_CUDA(cudaStreamEndCapture(side_, &body_out));
        enqueue_final();
        const long long c3 = g_kernel_launches.load();
        LHI_CUDA(cudaStreamEndCapture(stream_, &g));
        if (with_init) graph_init_kernels_ = c1 - c0;
        graph_body_kernels_ = c2 - c1;
        graph_final_kernels_ = c3 - c2;
        // captured launches did not run: the replays below count what runs
        g_kernel_launches.fetch_sub(c3 - c0);
    } catch (...) {
        cur_ = stream_;
        cudaGraph_t g2 = nullptr;
        cudaStreamEndCapture(stream_, &g2);
        if (g2) cudaGraphDestroy(g2);
        throw;
    }
    cudaGraphExec_t exec = nullptr;
    cudaGraphInstantiateParams ip = {};
    cudaError_t e = cudaGraphInstantiateWithParams(&exec, g, &ip);
    std::string why;
    if (e != cudaSuccess) {
        cudaGraphNodeType nt = cudaGraphNodeTypeEmpty;
        if (ip.errNode_out) cudaGraphNodeGetType(ip.errNode_out, &nt);
        why = std::string("solve graph instantiation failed: ") + cudaGetErrorString(e) + " (result " +
              std::to_string(int(ip.result_out)) + ", node type " + std::to_string(int(nt)) + ")";
        cudaGetLastError();
    }
    cudaGraphDestroy(g);
    if (e != cudaSuccess) throw CudaError(e, why);
    (with_init ? solve_exec_ : tail_exec_) = exec;
}

// CGSolver<3>::Solve (PressureSolver.cpp:839-934)
template <class T, class TX> int LiquidImpl<T, TX>::solve(double rho, double dt) {
    if (stats_pending_) finish_stats();
    LHI_CUDA(cudaEventRecord(ev0_, stream_));
    solver_init();
    build_rhs();
    build_lhs(rho, dt);
    bool graph_replayed = false;
    const bool learned = sp_.preconditioner == LHI_PRECOND_LEARNED;
    if (learned && !net_) throw std::invalid_argument("LHI_PRECOND_LEARNED without a network (lhi_solver_set_network)");
    use_fallback_ = false;
    learned_iters_ = 0;
    fallback_at_ = -1;
    // The first solve of a handle runs host-driven: it launches (and so
    // loads) every kernel of the loop once, which must not happen for the
    // first time inside a stream capture; later solves replay the graph.
    const bool graph_ok = solved_once_;
    solved_once_ = true;
    if (!sp_.eager && !prof_.on && !learned && snap_cap_ == 0 && graph_ok && graph_error_.empty() && !solve_exec_) {
        try {
            build_solve_graph(true);
        } catch (const CudaError& err) {
            graph_error_ = err.what();  // keep solving, host-driven (lhi_solver_graph_error)
            cudaGetLastError();         // the failed capture's error is not this solve's
        }
    }
    if (!sp_.eager && !prof_.on && !learned && snap_cap_ == 0 && graph_ok && solve_exec_) {
        LHI_CUDA(cudaGraphLaunch(solve_exec_, stream_));
        graph_replayed = true;
    } else {
        // host-driven loop; with the learned preconditioner the host also
        // applies the fallback rule between iterations
        const bool no_fallback = fallback_iters_ < 0;
        const int cap = fallback_iters_ > 0 ? fallback_iters_ : sp_.max_iterations;
        enqueue_init(0, 0);
        if (learned) {
            learned_iters_ = 1;
            read_scalars();
            if (!no_fallback && !(sc_host_->rz_old > 0.0) && !sc_host_->stop) {
                // r.M(r) <= 0: the network gives no descent direction; start over with the V-cycle
                use_fallback_ = true;
                fallback_at_ = 0;
                learned_iters_ = 0;
                enqueue_init(0, 0);
            }
        }
        double prev = -1.0;
        // after the fallback (and once one V-cycle body has run here, so no
        // kernel loads for the first time inside a capture) the rest of the
        // solve is one replay of the tail graph
        const bool tail_ok = learned && !sp_.eager && !prof_.on && snap_cap_ == 0;
        bool tail = false;
        for (;;) {
            read_scalars();
            if (sc_host_->stop) break;
            if (learned && !use_fallback_ && !no_fallback) {
                const double res = sc_host_->residual;
                const bool slow = prev > 0 && res > 0.95 * prev;
                if (slow || sc_host_->iter >= cap) {
                    use_fallback_ = true;
                    fallback_at_ = sc_host_->iter;
                }
                prev = res;
            }
            if (learned && !use_fallback_) ++learned_iters_;
            if (tail_ok && use_fallback_ && fallback_body_ran_ && tail_error_.empty()) {
                if (!tail_exec_) {
                    try {
                        build_solve_graph(false);
                    } catch (const CudaError& err) {
                        tail_error_ = err.what();  // keep the loop host-driven
                        cudaGetLastError();
                    }
                }
                if (tail_exec_) {
                    tail_from_iter_ = sc_host_->iter;
                    LHI_CUDA(cudaGraphLaunch(tail_exec_, stream_));
                    tail = true;
                    break;
                }
            }
            enqueue_body(0, 0);
            if (use_fallback_) fallback_body_ran_ = true;
        }
        if (!tail) enqueue_final();
    }
    LHI_CUDA(cudaEventRecord(ev1_, stream_));
    last_solve_graph_ = graph_replayed;
    stats_pending_ = true;
    if (async_ && graph_replayed) return LHI_OK;  // read by stats() later
    finish_stats();
    // a network application whose pipeline wait ran out left no usable direction
    if (learned && net_ && net_->check_status(stream_) != LHI_OK) stats_.status = LHI_E_TIMEOUT;
    return stats_.status;
}

// Statistics of the last solve from the device scalars (synchronises).
template <class T, class TX> void LiquidImpl<T, TX>::finish_stats() {
    read_scalars();
    float ms = 0.f;
    LHI_CUDA(cudaEventElapsedTime(&ms, ev0_, ev1_));
    if (last_solve_graph_)  // kernels the replay ran: init, one body per loop trip, final
        g_kernel_launches.fetch_add(graph_init_kernels_ + graph_final_kernels_ +
                                    graph_body_kernels_ * (long long)std::max(sc_host_->iter, 0));
    if (tail_from_iter_ >= 0)  // the tail graph: one body per loop trip from where it started (at least one), final
        g_kernel_launches.fetch_add(graph_final_kernels_ +
                                    graph_body_kernels_ * (long long)std::max(sc_host_->iter - tail_from_iter_, 1));
    tail_from_iter_ = -1;
    stats_.iterations = sc_host_->iter;
    stats_.initial_residual = sc_host_->residual0;
    stats_.final_residual = sc_host_->residual;
    stats_.true_residual = std::sqrt(sc_host_->true2);
    stats_.solve_ms = ms;
    stats_.status = sc_host_->timeout ? LHI_E_TIMEOUT : sc_host_->status;
    stats_pending_ = false;
}

template <class T, class TX> void LiquidImpl<T, TX>::spmv(int level, const T* x, T* y) {
    LevelDev<T>& L = lv_[level];
    if (L.n == 0) return;
    k_get_ax<T><<<blocks_for(L.n, 256), 256, 0, cur_>>>(lk(L), x, y);
    LHI_LAUNCH_CHECK();
}

// One SpMV of the PCG body on the handle's p, through the same launch as
// enqueue_body's (so the same kernel and tile order); p.Ap comes back from
// the device scalars.
template <class T, class TX> double LiquidImpl<T, TX>::spmv_p(int* tma) {
    LevelDev<T>& L0 = lv_[0];
    if (L0.n == 0) return 0.0;
    cur_ = stream_;
    LHI_CUDA(cudaMemsetAsync(&sc_->stop, 0, sizeof(int), stream_));  // a finished solve leaves stop set
    const TileK tk = tile_k(L0, &sc_->tile_count[0], tile_grid_);
    const unsigned G = std::max(1u, tile_blocks(L0, tile_grid_));
    const CgConf cf = make_conf(sp_, 0, 0);
    const bool use_tma = spmv_tma_ && sp_.sweep_kernel == LHI_SWEEP_FUSED;
    {
        auto ps_ = scope(LHI_KERNEL_SPMV);
        if (use_tma)
            k_spmv_tma<<<std::min(G, unsigned(2 * kSMs)), kTileThreads, sp::kSmem, cur_>>>(
                tm_sp_[0], tm_sp_[1], tm_sp_[2], tm_sp_[3], tm_sp_[4], tm_sp_[5], L0.nx, L0.ny, L0.nz, L0.tiles,
                &sc_->tile_count[0], L0.tdim[1], L0.tdim[2], reinterpret_cast<float*>(ap_), partials_, counter_, sc_,
                cf);
        else
            k_cg_spmv<T><<<std::max(1u, tile_blocks(L0, tile_grid_, kSplit)), kTileThreads, 0, cur_>>>(
                lk(L0), tile_k(L0, &sc_->tile_count[0], tile_grid_, kSplit), p_, ap_, partials_, counter_, sc_, cf);
        LHI_LAUNCH_CHECK();
    }
    read_scalars();
    if (sc_host_->timeout) throw std::runtime_error("SpMV: a bounded wait on a staging copy timed out");
    if (tma) *tma = use_tma ? 1 : 0;
    return sc_host_->denom;
}

template <class T, class TX> void LiquidImpl<T, TX>::get_ax(int level, const void* x, void* out) {
    if (level < 0 || level >= nlev_) throw std::invalid_argument("bad level");
    LevelDev<T>& L = lv_[level];
    if (L.n == 0) return;
    T *dx = nullptr, *dy = nullptr;
    LHI_CUDA(cudaMalloc(&dx, sizeof(T) * L.n));
    LHI_CUDA(cudaMalloc(&dy, sizeof(T) * L.n));
    LHI_CUDA(cudaMemcpyAsync(dx, x, sizeof(T) * L.n, cudaMemcpyHostToDevice, stream_));
    spmv(level, dx, dy);
    LHI_CUDA(cudaMemcpyAsync(out, dy, sizeof(T) * L.n, cudaMemcpyDeviceToHost, stream_));
    LHI_CUDA(cudaStreamSynchronize(stream_));
    cudaFree(dx);
    cudaFree(dy);
}

template <class T, class TX>
void LiquidImpl<T, TX>::active_tiles(int level, int32_t* active, int32_t* total, int32_t* coarse) {
    if (level < 0 || level >= nlev_) throw std::invalid_argument("bad level");
    read_scalars();
    *active = sc_host_->tile_count[level];
    *total = lv_[level].ntiles;
    *coarse = (level >= coarse_level_) ? 1 : 0;
}

template <class T, class TX> void LiquidImpl<T, TX>::set_network(LearnedNet* net, int fallback_iterations) {
    if (sp_.preconditioner != LHI_PRECOND_LEARNED)
        throw std::invalid_argument("lhi_solver_set_network needs a handle created with LHI_PRECOND_LEARNED");
    if (fallback_iterations < -1) throw std::invalid_argument("fallback_iterations must be >= -1");
    net_ = net;
    fallback_iters_ = fallback_iterations;
}

template <class T, class TX> void LiquidImpl<T, TX>::ensure_solid_cells() {
    if (!solid_cell_) LHI_CUDA(cudaMalloc(&solid_cell_, size_t(ncell_)));
    if (solid_cell_fresh_) return;
    k_solid_cells<T><<<blocks_for(ncell_, 256), 256, 0, cur_>>>(solid_phi_, nx_, ny_, nz_, solid_cell_);
    LHI_LAUNCH_CHECK();
    solid_cell_fresh_ = true;
}

template <class T, class TX> void LiquidImpl<T, TX>::ensure_net_type() {
    if (!net_type_) LHI_CUDA(cudaMalloc(&net_type_, size_t(ncell_)));
    if (net_type_fresh_) return;
    k_net_type<T><<<blocks_for(ncell_, 256), 256, 0, cur_>>>(lv_[0].type, lv_[0].diag, ncell_, net_type_);
    LHI_LAUNCH_CHECK();
    net_type_fresh_ = true;
    net_plan_stale_ = true;
}

template <class T, class TX> void LiquidImpl<T, TX>::record_residuals(int max_snapshots) {
    if (max_snapshots < 0 || max_snapshots > 100000) throw std::invalid_argument("max_snapshots out of range");
    if (snaps_) cudaFree(snaps_);
    snaps_ = nullptr;
    snap_cap_ = max_snapshots;
    snap_count_ = snap_next_ = 0;
    if (max_snapshots > 0) LHI_CUDA(cudaMalloc(&snaps_, sizeof(float) * size_t(ncell_) * size_t(max_snapshots)));
}

// Copy of level-0 r (as FP32) into the next snapshot slot (ring buffer).
template <class T, class TX> void LiquidImpl<T, TX>::record_snapshot() {
    if (snap_cap_ == 0) return;
    float* dst = snaps_ + size_t(snap_next_) * size_t(ncell_);
    if (sizeof(T) == sizeof(float)) {
        LHI_CUDA(cudaMemcpyAsync(dst, lv_[0].r, sizeof(float) * ncell_, cudaMemcpyDeviceToDevice, cur_));
    } else {
        throw std::invalid_argument("residual recording needs an FP32 or MIXED handle");
    }
    snap_next_ = (snap_next_ + 1) % snap_cap_;
    snap_count_ = std::min(snap_count_ + 1, snap_cap_);
}

template <class T, class TX>
void LiquidImpl<T, TX>::train(LearnedNet* net, int steps, int batch, double lr, uint64_t seed, double* first,
                              double* last) {
    if (sizeof(T) != sizeof(float)) throw std::invalid_argument("training needs an FP32 or MIXED handle");
    if (snap_count_ == 0) throw std::invalid_argument("no recorded residuals (lhi_solver_record_residuals + solve)");
    if (steps < 1 || batch < 1) throw std::invalid_argument("steps and batch must be >= 1");
    if (!train_z_) {
        LHI_CUDA(cudaMalloc(&train_z_, sizeof(float) * ncell_));
        LHI_CUDA(cudaMalloc(&train_dz_, sizeof(float) * ncell_));
        LHI_CUDA(cudaMalloc(&train_e_, sizeof(float) * ncell_));
        LHI_CUDA(cudaMalloc(&train_red_, sizeof(double) * 4));
    }
    ensure_solid_cells();
    ensure_net_type();
    LevelDev<T>& L0 = lv_[0];
    const int dims[3] = {nx_, ny_, nz_};
    const unsigned nbk = std::min<unsigned>(blocks_for(ncell_, 256), unsigned(sum_blocks_));
    std::mt19937_64 rng(seed);
    double first_loss = 0.0, last_loss = 0.0;
    for (int st = 0; st < steps; ++st) {
        net->zero_grad(cur_);
        LHI_CUDA(cudaMemsetAsync(train_red_ + 2, 0, sizeof(double), cur_));
        for (int b = 0; b < batch; ++b) {
            const int k = int(rng() % uint64_t(snap_count_));
            const float* r = snaps_ + size_t(k) * size_t(ncell_);
            net->forward(dims, r, net_type_, solid_cell_, train_z_, 0.0, cur_);
            k_loss_residual<T><<<nbk, 256, 0, cur_>>>(lk(L0), train_z_, reinterpret_cast<const T*>(r), train_e_,
                                                      partials_, counter_, train_red_);
            LHI_LAUNCH_CHECK();
            k_loss_grad<T><<<nbk, 256, 0, cur_>>>(lk(L0), train_e_, batch, train_dz_, train_red_);
            LHI_LAUNCH_CHECK();
            net->backward(train_dz_, cur_);
        }
        net->adam_step(lr, 0.9, 0.999, 1e-8, cur_);
        if (st == 0 || st == steps - 1) {
            double loss = 0.0;
            LHI_CUDA(cudaMemcpyAsync(&loss, train_red_ + 2, sizeof(double), cudaMemcpyDeviceToHost, cur_));
            LHI_CUDA(cudaStreamSynchronize(cur_));
            if (st == 0) first_loss = loss;
            last_loss = loss;
        }
    }
    if (net->check_status(cur_) != LHI_OK) throw CudaError(cudaErrorLaunchTimeout, "tensor-core pipeline wait timed out");
    *first = first_loss;
    *last = last_loss;
}

template <class T, class TX> void LiquidImpl<T, TX>::get_acoef(int level, T* host_out) {
    LevelDev<T>& L = lv_[level];
    if (L.n == 0) return;
    T* d = nullptr;
    LHI_CUDA(cudaMalloc(&d, sizeof(T) * 6 * L.n));
    k_expand_acoef<T><<<blocks_for(L.n, 256), 256, 0, stream_>>>(lk(L), d);
    LHI_LAUNCH_CHECK();
    LHI_CUDA(cudaMemcpyAsync(host_out, d, sizeof(T) * 6 * L.n, cudaMemcpyDeviceToHost, stream_));
    LHI_CUDA(cudaStreamSynchronize(stream_));
    cudaFree(d);
}

void set_stage_wait_limit_ns(unsigned long long ns) {
    LHI_CUDA(cudaMemcpyToSymbol(g_stage_wait_ns, &ns, sizeof(ns)));
}

template class LiquidImpl<float, float>;
template class LiquidImpl<float, double>;
template class LiquidImpl<double, double>;

}  // namespace lhi
