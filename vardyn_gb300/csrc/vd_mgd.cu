// Node-centred Dirichlet multigrid for the masked Helmholtz problems of the
// multilayer QG PV inversion (mapping/models/model_qgsw/qg.py:222-298): per
// vertical mode m, on the interior nodes of the psi grid,
//     (u_E + u_W - 2u)/d0^2 + (u_N + u_S - 2u)/d1^2 - lambda_m u = b
// at ocean nodes, u = 0 at land nodes and beyond the outer boundary. The
// reference solves the same discrete problem with a DST solve and a
// capacitance-matrix correction at the irregular boundary points
// (helmholtz.py:146-184), which needs one DST solve per irregular point and an
// M x M inverse; at 20 % land that is tens of thousands of solves. Here a
// geometric V-cycle solves it directly:
//   - node-centred coarsening (coarse node I at fine node 2I+1; n -> (n+1)/2-1),
//     a coarse node an unknown where its 3 x 3 fine neighbourhood is, the
//     operator rediscretised on every level;
//   - red-black Gauss-Seidel smoothing (2 + 2 sweeps), full-weighting
//     restriction and bilinear prolongation of the correction, both masked;
//   - the coarsest level solved exactly with a float64 inverse built on the host;
//   - the symmetric V-cycle (red-black pre-smoothing, black-red post-smoothing)
//     preconditions conjugate gradients: the conservative coarse masks keep
//     the coarse levels from bridging land, and the Krylov iteration removes
//     the few coastal modes they resolve poorly;
//   - the scalars of every system live in device memory, the float64 dot
//     products are reduced in a fixed order (per-block partial sums, added up by
//     the system's last block); when ||r|| <= tol ||b|| a system's flag makes every
//     later kernel of that system return at once, so a solve is a fixed
//     launch sequence (it can be captured in a CUDA graph) that stops
//     computing at the tolerance.
// A V-cycle is two launches a level (descent and ascent, tiles with halos in
// shared memory) and one block per system for the small levels, an iteration two
// more: 14 launches where separate sweeps, residuals, restrictions and vector
// updates took 95. Measured on three systems of 1023 x 767 in float64, 1e-8:
// 17.4 -> 5.3 ms a solve; one system of 511 x 767 8.4 -> 2.8 ms.
// Systems are [nsys = nmode * batch] slices of the caller's arrays with a row
// pitch `ld` and a system stride `fs` (the interior of a (nx+1) x (ny+1) psi
// field in place).
#include "vd_internal.cuh"
#include <algorithm>
#include <cmath>
#include <new>
#include <vector>

namespace vd {

struct MgdLevel {
    int n0, n1;
    double d0, d1;
    int8_t* mask;       // [n0][n1] device
};

// One level of one solve. coef[m] = {1/D, c0/D, c1/D, D} of mode m with
// c0 = 1/d0^2, c1 = 1/d1^2 and the diagonal D = 2 c0 + 2 c1 + lambda_m: a
// Gauss-Seidel update is c0/D (u_N + u_S) + c1/D (u_E + u_W) - b/D, four FP64
// instructions and no division (this part issues 2 FP64 FMAs a clock and SM, and
// a division costs more than ten of them).
template <typename T>
struct MgdLev {
    int n0, n1;
    const int8_t* mask;
    const T* coef;       // [nmode][4]
    int batch;           // systems per mode
    const int* done;     // [nsys] converged flags
};

constexpr int MGD_SCAL = 4;            // per system: ||b||^2, rho, alpha, relative residual
constexpr int MGD_NT = 256;            // threads of the tile kernels

// Scalars of the conjugate gradients, reduced in a fixed order: every block
// leaves its partial sum, the last block of a system adds them up and forms the
// scalar that the next kernel reads.
struct MgdDot {
    int what;            // 0 = ||b||^2, 1 = rho = r.z, 2 = alpha = rho / (p.Ap), 3 = test on r.r, 4 = beta, rho
    double tol;
    double* part;        // [nsys][blocks of a system]
    int* count;          // [nsys] arrivals, back to 0 after each reduction
    int* done;
    double* sc;          // [nsys][MGD_SCAL]
    double* beta;        // [nsys]
    double* rel;         // [nsys] or nullptr
};

__device__ __forceinline__ double mgd_block_sum(double a)
{
    __shared__ double sh[MGD_NT / 32];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = a;
    __syncthreads();
    double v = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < MGD_NT / 32; ++k) v += sh[k];
    return v;                           // thread 0 holds the sum
}

// Called by every thread of every block of system s (grid x * y blocks).
__device__ __forceinline__ void mgd_dot(const MgdDot& D, int s, double a)
{
    __shared__ bool last;
    const int nblk = gridDim.x * gridDim.y, blk = blockIdx.y * gridDim.x + blockIdx.x;
    double v = mgd_block_sum(a);
    if (threadIdx.x == 0) {
        D.part[(long long)s * nblk + blk] = v;
        __threadfence();
        last = atomicAdd(D.count + s, 1) == nblk - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    a = 0.0;
    for (int k = threadIdx.x; k < nblk; k += MGD_NT) a += __ldcg(D.part + (long long)s * nblk + k);
    v = mgd_block_sum(a);
    if (threadIdx.x != 0) return;
    D.count[s] = 0;
    double* c = D.sc + (long long)s * MGD_SCAL;
    if (D.what == 0) {
        c[0] = v;
        if (v == 0.0) { D.done[s] = 1; c[3] = 0.0; if (D.rel) D.rel[s] = 0.0; }
    } else if (D.what == 1) {
        c[1] = v;
    } else if (D.what == 2) {
        c[2] = v != 0.0 ? c[1] / v : 0.0;
    } else if (D.what == 3) {
        const double q = c[0] > 0.0 ? sqrt(v / c[0]) : 0.0;
        c[3] = q;
        if (D.rel) D.rel[s] = q;
        if (q <= D.tol) D.done[s] = 1;
    } else {
        D.beta[s] = c[1] != 0.0 ? v / c[1] : 0.0;
        c[1] = v;
    }
}

// One Gauss-Seidel half sweep over the points of parity `color` of the local
// rows [A0, A1] x columns [B0, B1] of a shared-memory tile with pitch P.
template <typename T, int P, int A0, int A1, int B0, int B1>
__device__ __forceinline__ void mgd_half(int color, T* u, const T* bs, const int8_t* ms, T k0, T k1)
{
    constexpr int NR = A1 - A0 + 1, NC = (B1 - B0 + 2) / 2;
    for (int idx = threadIdx.x; idx < NR * NC; idx += MGD_NT) {
        const int r = idx / NC, a = A0 + r;
        const int b = B0 + 2 * (idx - r * NC) + ((a + B0 + color) & 1);
        const int o = a * P + b;
        if (b <= B1 && ms[o])
            u[o] = fma(k1, u[o - 1] + u[o + 1], fma(k0, u[o - P] + u[o + P], -bs[o]));
    }
    __syncthreads();
}

// Tiles of TI x TJ fine points with 4 points of halo before and 5 after (the
// four half sweeps and the residual each consume one ring). TI and TJ are even:
// a point's colour is the parity of its local indices.
template <typename T, int TI, int TJ>
struct MgdTile {
    static constexpr int NR = TI + 9, P = TJ + 10;
    static constexpr size_t bytes = size_t(NR) * P * (2 * sizeof(T) + 1);
};

// Descent of the V-cycle on one level, all in one pass over memory: u from 0 by
// red, black, red, black half sweeps; the residual (exactly 0 at the black
// points just solved); its full weighting, the right-hand side of the level
// below. The level used to take four sweep launches, a residual, a restriction
// and a fill, each a pass over the level.
template <typename T, int TI, int TJ>
__global__ void __launch_bounds__(MGD_NT)
k_mgd_pre(MgdLev<T> A, const T* __restrict__ b, T* __restrict__ u, int n0c, int n1c,
          const int8_t* __restrict__ maskc, T* __restrict__ bc)
{
    using Tl = MgdTile<T, TI, TJ>;
    constexpr int P = Tl::P;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* us = reinterpret_cast<T*>(smem_raw);
    T* bs = us + Tl::NR * P;
    int8_t* ms = reinterpret_cast<int8_t*>(bs + Tl::NR * P);
    const int s = blockIdx.z;
    if (A.done[s]) return;
    const int i0 = blockIdx.y * TI, j0 = blockIdx.x * TJ;
    const T* co = A.coef + 4 * (s / A.batch);
    const T inv = co[0], k0 = co[1], k1 = co[2];
    const T* bg = b + (long long)s * A.n0 * A.n1;
    constexpr int W = TJ + 9;
    for (int idx = threadIdx.x; idx < Tl::NR * W; idx += MGD_NT) {
        const int a = idx / W, c = idx - a * W;
        const int i = i0 + a - 4, j = j0 + c - 4;
        T v = T(0);
        int8_t m = 0;
        if (i >= 0 && i < A.n0 && j >= 0 && j < A.n1) {
            m = A.mask[i * A.n1 + j];
            if (m) v = bg[(long long)i * A.n1 + j] * inv;
        }
        bs[a * P + c] = v;
        us[a * P + c] = ((a + c) & 1) ? T(0) : -v;      // the first red half sweep
        ms[a * P + c] = m;
    }
    __syncthreads();
    mgd_half<T, P, 1, TI + 7, 1, TJ + 7>(1, us, bs, ms, k0, k1);
    mgd_half<T, P, 2, TI + 6, 2, TJ + 6>(0, us, bs, ms, k0, k1);
    mgd_half<T, P, 3, TI + 5, 3, TJ + 5>(1, us, bs, ms, k0, k1);
    T* ug = u + (long long)s * A.n0 * A.n1;
    for (int idx = threadIdx.x; idx < TI * TJ; idx += MGD_NT) {
        const int a = idx / TJ, c = idx - a * TJ;
        const int i = i0 + a, j = j0 + c;
        if (i < A.n0 && j < A.n1) ug[(long long)i * A.n1 + j] = us[(a + 4) * P + c + 4];
    }
    // residual over D at the red points, in place of b/D
    {
        constexpr int NR = TI + 1, NC = (TJ + 2) / 2;
        for (int idx = threadIdx.x; idx < NR * NC; idx += MGD_NT) {
            const int r = idx / NC, a = 4 + r;
            const int c = 4 + 2 * (idx - r * NC) + (a & 1);
            const int o = a * P + c;
            if (c <= TJ + 4)
                bs[o] = ms[o] ? us[o] - fma(k1, us[o - 1] + us[o + 1], fma(k0, us[o - P] + us[o + P], -bs[o])) : T(0);
        }
    }
    __syncthreads();
    const T D16 = co[3] * T(0.0625);
    T* bcs = bc + (long long)s * n0c * n1c;
    for (int idx = threadIdx.x; idx < (TI / 2) * (TJ / 2); idx += MGD_NT) {
        const int a = idx / (TJ / 2), c = idx - a * (TJ / 2);
        const int I = i0 / 2 + a, J = j0 / 2 + c;
        if (I >= n0c || J >= n1c) continue;
        const int o = (2 * a + 5) * P + 2 * c + 5;
        bcs[(long long)I * n1c + J] = maskc[I * n1c + J]
            ? D16 * (T(4) * bs[o] + ((bs[o - P - 1] + bs[o - P + 1]) + (bs[o + P - 1] + bs[o + P + 1]))) : T(0);
    }
}

template <typename T>
__device__ __forceinline__ T mgd_get(const T* u, int n0, int n1, int i, int j)
{
    return (i >= 0 && i < n0 && j >= 0 && j < n1) ? u[(long long)i * n1 + j] : T(0);
}

// bilinear interpolation of the coarse correction at fine point (i, j): fine
// index 2I+1 is coarse I, an even fine index lies between I-1 and I
template <typename T>
__device__ __forceinline__ T mgd_interp(const T* e, int n0c, int n1c, int i, int j)
{
    const int I = (i - 1) >> 1, J = (j - 1) >> 1;
    auto E = [&](int a, int c) { return mgd_get(e, n0c, n1c, a, c); };
    if (i & 1) return (j & 1) ? E(I, J) : T(0.5) * (E(I, J) + E(I, J + 1));
    if (j & 1) return T(0.5) * (E(I, J) + E(I + 1, J));
    return T(0.25) * ((E(I, J) + E(I + 1, J)) + (E(I, J + 1) + E(I + 1, J + 1)));
}

// Ascent on one level: u + interpolated correction, then black, red, black, red
// half sweeps (the descent's order reversed, so that the cycle is a symmetric
// preconditioner), written to z. DOT (level 0): the sum of b z as well.
template <typename T, int TI, int TJ, bool DOT>
__global__ void __launch_bounds__(MGD_NT)
k_mgd_post(MgdLev<T> A, const T* __restrict__ b, const T* __restrict__ u, int n0c, int n1c,
           const T* __restrict__ ec, T* __restrict__ z, MgdDot D)
{
    using Tl = MgdTile<T, TI, TJ>;
    constexpr int P = Tl::P;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* us = reinterpret_cast<T*>(smem_raw);
    T* bs = us + Tl::NR * P;
    int8_t* ms = reinterpret_cast<int8_t*>(bs + Tl::NR * P);
    const int s = blockIdx.z;
    if (A.done[s]) return;
    const int i0 = blockIdx.y * TI, j0 = blockIdx.x * TJ;
    const T* co = A.coef + 4 * (s / A.batch);
    const T inv = co[0], k0 = co[1], k1 = co[2];
    const long long fs = (long long)A.n0 * A.n1;
    const T* bg = b + s * fs;
    const T* ug = u + s * fs;
    const T* e = ec + (long long)s * n0c * n1c;
    constexpr int W = TJ + 8;
    for (int idx = threadIdx.x; idx < (TI + 8) * W; idx += MGD_NT) {
        const int a = idx / W, c = idx - a * W;
        const int i = i0 + a - 4, j = j0 + c - 4;
        T v = T(0), x = T(0);
        int8_t m = 0;
        if (i >= 0 && i < A.n0 && j >= 0 && j < A.n1) {
            m = A.mask[i * A.n1 + j];
            if (m) {
                v = bg[(long long)i * A.n1 + j] * inv;
                // the first half sweep overwrites the black points inside the halo
                if (!((a + c) & 1)) x = ug[(long long)i * A.n1 + j] + mgd_interp(e, n0c, n1c, i, j);
            }
        }
        bs[a * P + c] = v;
        us[a * P + c] = x;
        ms[a * P + c] = m;
    }
    __syncthreads();
    mgd_half<T, P, 1, TI + 6, 1, TJ + 6>(1, us, bs, ms, k0, k1);
    mgd_half<T, P, 2, TI + 5, 2, TJ + 5>(0, us, bs, ms, k0, k1);
    mgd_half<T, P, 3, TI + 4, 3, TJ + 4>(1, us, bs, ms, k0, k1);
    mgd_half<T, P, 4, TI + 3, 4, TJ + 3>(0, us, bs, ms, k0, k1);
    T* zg = z + s * fs;
    double acc = 0.0;
    for (int idx = threadIdx.x; idx < TI * TJ; idx += MGD_NT) {
        const int a = idx / TJ, c = idx - a * TJ;
        const int i = i0 + a, j = j0 + c;
        if (i < A.n0 && j < A.n1) {
            const int o = (a + 4) * P + c + 4;
            zg[(long long)i * A.n1 + j] = us[o];
            if (DOT) acc += (double)bg[(long long)i * A.n1 + j] * (double)us[o];
        }
    }
    if (DOT) mgd_dot(D, s, acc);
}

// coarsest level: u[idx[m]] = sum_k inv[mode][m][k] b[idx[k]] in float64, one
// warp a row
template <typename T>
__global__ void k_mgd_coarse(int nb, int ncell, int batch, const int* __restrict__ done, const int32_t* __restrict__ idx,
                             const double* __restrict__ inv, const T* __restrict__ b, T* __restrict__ u)
{
    const int s = blockIdx.y;
    if (done[s]) return;
    const int m = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (m >= nb) return;
    const double* row = inv + ((long long)(s / batch) * nb + m) * nb;
    const T* bs = b + (long long)s * ncell;
    double acc = 0.0;
    for (int k = lane; k < nb; k += 32) acc += row[k] * (double)bs[idx[k]];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) u[(long long)s * ncell + idx[m]] = (T)acc;
}

// The levels of at most MGD_CHAIN_CELLS cells, down to the exact coarsest solve
// and back, in one block per system: u and b of every level in shared memory,
// the same half sweeps between block barriers. A level this small is shorter
// than a launch.
constexpr int MGD_CHAIN_CELLS = 1024;
constexpr int MGD_CHAIN_UNKNOWNS = 128;    // largest coarsest system of the one-block form
constexpr int MGD_CHAIN_LEVELS = 12;

template <typename T>
struct MgdChain {
    int nlev;
    MgdLev<T> lv[MGD_CHAIN_LEVELS];
    int nb;
    const int32_t* cidx;
    const double* cinv;
};

template <typename T>
__global__ void __launch_bounds__(MGD_NT)
k_mgd_chain(MgdChain<T> C, const T* __restrict__ b, T* __restrict__ u)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* sm = reinterpret_cast<T*>(smem_raw);
    const int s = blockIdx.x;
    if (C.lv[0].done[s]) return;
    const int mode = s / C.lv[0].batch;
    const int cells0 = C.lv[0].n0 * C.lv[0].n1;
    // level l: u at 2 * off, b behind it; levels one after the other
    for (int k = threadIdx.x; k < cells0; k += MGD_NT) sm[cells0 + k] = b[(long long)s * cells0 + k];
    __syncthreads();
    auto half = [&](const MgdLev<T>& L, const T* co, int color, T* us, const T* bs) {
        const int n0 = L.n0, n1 = L.n1, hc = (n1 + 1) >> 1;
        for (int idx = threadIdx.x; idx < n0 * hc; idx += MGD_NT) {
            const int i = idx / hc, j = 2 * (idx - i * hc) + ((i + color) & 1);
            const int o = i * n1 + j;
            if (j < n1 && L.mask[o])
                us[o] = fma(co[2], mgd_get(us, n0, n1, i, j - 1) + mgd_get(us, n0, n1, i, j + 1),
                            fma(co[1], mgd_get(us, n0, n1, i - 1, j) + mgd_get(us, n0, n1, i + 1, j), -(bs[o] * co[0])));
        }
        __syncthreads();
    };
    int off = 0;
    for (int l = 0; l < C.nlev - 1; ++l) {
        const MgdLev<T>& L = C.lv[l];
        const MgdLev<T>& N = C.lv[l + 1];
        const int n1 = L.n1, cells = L.n0 * L.n1, ncells = N.n0 * N.n1;
        T *us = sm + off, *bs = us + cells, *bn = sm + off + 2 * cells + ncells;
        const T* co = L.coef + 4 * mode;
        for (int k = threadIdx.x; k < cells; k += MGD_NT) us[k] = T(0);
        __syncthreads();
        for (int h = 0; h < 4; ++h) half(L, co, h & 1, us, bs);
        for (int k = threadIdx.x; k < ncells; k += MGD_NT) {
            const int I = k / N.n1, J = k - I * N.n1;
            T v = T(0);
            if (N.mask[k]) {
                // the 3 x 3 neighbourhood of an unknown is ocean; its red points
                auto res = [&](int i, int j) {
                    const int o = i * n1 + j;
                    return us[o] - fma(co[2], mgd_get(us, L.n0, n1, i, j - 1) + mgd_get(us, L.n0, n1, i, j + 1),
                                       fma(co[1], mgd_get(us, L.n0, n1, i - 1, j) + mgd_get(us, L.n0, n1, i + 1, j),
                                           -(bs[o] * co[0])));
                };
                const int i = 2 * I + 1, j = 2 * J + 1;
                v = co[3] * T(0.0625) * (T(4) * res(i, j) + ((res(i - 1, j - 1) + res(i - 1, j + 1)) +
                                                         (res(i + 1, j - 1) + res(i + 1, j + 1))));
            }
            bn[k] = v;
        }
        __syncthreads();
        off += 2 * cells;
    }
    {
        const MgdLev<T>& L = C.lv[C.nlev - 1];
        const int cells = L.n0 * L.n1;
        T *us = sm + off, *bs = us + cells;
        for (int k = threadIdx.x; k < cells; k += MGD_NT) us[k] = T(0);
        __syncthreads();
        const int lane = threadIdx.x & 31;
        for (int m = threadIdx.x >> 5; m < C.nb; m += MGD_NT / 32) {
            const double* row = C.cinv + ((long long)mode * C.nb + m) * C.nb;
            double acc = 0.0;
            for (int k = lane; k < C.nb; k += 32) acc += row[k] * (double)bs[C.cidx[k]];
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
            if (lane == 0) us[C.cidx[m]] = (T)acc;
        }
        __syncthreads();
    }
    for (int l = C.nlev - 2; l >= 0; --l) {
        const MgdLev<T>& L = C.lv[l];
        const MgdLev<T>& N = C.lv[l + 1];
        const int cells = L.n0 * L.n1;
        const T* en = sm + off;
        off -= 2 * cells;
        T *us = sm + off, *bs = us + cells;
        const T* co = L.coef + 4 * mode;
        for (int k = threadIdx.x; k < cells; k += MGD_NT) {
            const int i = k / L.n1, j = k - i * L.n1;
            if (L.mask[k]) us[k] += mgd_interp(en, N.n0, N.n1, i, j);
        }
        __syncthreads();
        for (int h = 1; h < 5; ++h) half(L, co, h & 1, us, bs);
    }
    for (int k = threadIdx.x; k < cells0; k += MGD_NT) u[(long long)s * cells0 + k] = sm[k];
}

// x = 0 on the caller's array (land included), r = b on the ocean nodes (land
// carries no equation), ||b||^2
template <typename T, int TI, int TJ>
__global__ void __launch_bounds__(MGD_NT)
k_mgd_init(MgdLev<T> A, const T* __restrict__ b, long long ldb, long long fsb, T* __restrict__ x, long long ldx,
           long long fsx, T* __restrict__ r, MgdDot D)
{
    const int s = blockIdx.z;
    const int i0 = blockIdx.y * TI, j0 = blockIdx.x * TJ;
    double acc = 0.0;
    for (int idx = threadIdx.x; idx < TI * TJ; idx += MGD_NT) {
        const int i = i0 + idx / TJ, j = j0 + idx % TJ;
        if (i >= A.n0 || j >= A.n1) continue;
        x[s * fsx + (long long)i * ldx + j] = T(0);
        const T v = A.mask[i * A.n1 + j] ? b[s * fsb + (long long)i * ldb + j] : T(0);
        r[((long long)s * A.n0 + i) * A.n1 + j] = v;
        acc += (double)v * (double)v;
    }
    mgd_dot(D, s, acc);
}

// p = z + beta p_old (p = z on the first iteration), q = -A p, p.q. p is read a
// ring beyond the block's tile: p_old and p are different buffers. q carries the
// problem that the iteration solves, so it is formed from differences: with the
// sweeps' rounded 1/D, c0/D, c1/D, D (2 c0/D + 2 c1/D) + lambda would miss D by 1e-7
// D in float32, as much as the lowest modes' eigenvalues (511 x 767, lambda = 0: 9e-4
// of the solution). The V-cycle, which only preconditions, keeps the quotients.
// (7 FP64 instructions a point for 6: 1 % of a float64 solve, 5.25 -> 5.31 ms on three
// systems of 1023 x 767.)
// op[m] = {c0, c1, lambda_m}.
template <typename T, int TI, int TJ>
__global__ void __launch_bounds__(MGD_NT)
k_mgd_pq(MgdLev<T> A, const T* __restrict__ op, int first, const T* __restrict__ z, const T* __restrict__ pold,
         T* __restrict__ pnew, T* __restrict__ q, MgdDot D)
{
    constexpr int P = TJ + 2;
    __shared__ T ps[(TI + 2) * P];
    const int s = blockIdx.z;
    if (A.done[s]) return;
    const int i0 = blockIdx.y * TI, j0 = blockIdx.x * TJ;
    op += 3 * (s / A.batch);
    const T c0 = op[0], c1 = op[1], lam = op[2];
    const long long o0 = (long long)s * A.n0 * A.n1;
    const T be = first ? T(0) : (T)D.beta[s];
    for (int idx = threadIdx.x; idx < (TI + 2) * P; idx += MGD_NT) {
        const int a = idx / P, c = idx - a * P;
        const int i = i0 + a - 1, j = j0 + c - 1;
        T v = T(0);
        if (i >= 0 && i < A.n0 && j >= 0 && j < A.n1) {
            const long long o = o0 + (long long)i * A.n1 + j;
            v = first ? z[o] : z[o] + be * pold[o];
        }
        ps[idx] = v;
    }
    __syncthreads();
    double acc = 0.0;
    for (int idx = threadIdx.x; idx < TI * TJ; idx += MGD_NT) {
        const int a = idx / TJ, c = idx - a * TJ;
        const int i = i0 + a, j = j0 + c;
        if (i >= A.n0 || j >= A.n1) continue;
        const int l = (a + 1) * P + c + 1;
        const long long o = o0 + (long long)i * A.n1 + j;
        const T pc = ps[l];
        T v = T(0);
        if (A.mask[i * A.n1 + j])
            v = fma(-c0, fma(T(-2), pc, ps[l - P] + ps[l + P]), fma(-c1, fma(T(-2), pc, ps[l - 1] + ps[l + 1]), lam * pc));
        pnew[o] = pc;
        q[o] = v;
        acc += (double)pc * (double)v;
    }
    mgd_dot(D, s, acc);
}

// With q = -A p and sc[2] = rho / (p.q) = -alpha: x (strided) += alpha p,
// r -= alpha A p, r.r
template <typename T, int TI, int TJ>
__global__ void __launch_bounds__(MGD_NT)
k_mgd_xr(MgdLev<T> A, const T* __restrict__ pv, const T* __restrict__ qv, T* __restrict__ x, long long ldx,
         long long fsx, T* __restrict__ r, MgdDot D)
{
    const int s = blockIdx.z;
    if (A.done[s]) return;
    const int i0 = blockIdx.y * TI, j0 = blockIdx.x * TJ;
    const T al = (T)D.sc[(long long)s * MGD_SCAL + 2];
    double acc = 0.0;
    for (int idx = threadIdx.x; idx < TI * TJ; idx += MGD_NT) {
        const int i = i0 + idx / TJ, j = j0 + idx % TJ;
        if (i >= A.n0 || j >= A.n1) continue;
        const long long o = ((long long)s * A.n0 + i) * A.n1 + j;
        x[s * fsx + (long long)i * ldx + j] -= al * pv[o];
        const T v = r[o] - al * qv[o];
        r[o] = v;
        acc += (double)v * (double)v;
    }
    mgd_dot(D, s, acc);
}

__global__ void k_mgd_fill_int(int n, int v, int* __restrict__ x)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) x[k] = v;
}

// Gauss-Jordan inverse with partial pivoting of a dense float64 matrix
static bool invert(std::vector<double>& A, int n, std::vector<double>& inv)
{
    inv.assign((size_t)n * n, 0.0);
    for (int i = 0; i < n; ++i) inv[(size_t)i * n + i] = 1.0;
    for (int c = 0; c < n; ++c) {
        int p = c;
        for (int r = c + 1; r < n; ++r)
            if (std::fabs(A[(size_t)r * n + c]) > std::fabs(A[(size_t)p * n + c])) p = r;
        if (A[(size_t)p * n + c] == 0.0) return false;
        if (p != c)
            for (int k = 0; k < n; ++k) {
                std::swap(A[(size_t)p * n + k], A[(size_t)c * n + k]);
                std::swap(inv[(size_t)p * n + k], inv[(size_t)c * n + k]);
            }
        const double d = 1.0 / A[(size_t)c * n + c];
        for (int k = 0; k < n; ++k) { A[(size_t)c * n + k] *= d; inv[(size_t)c * n + k] *= d; }
        for (int r = 0; r < n; ++r) {
            if (r == c) continue;
            const double f = A[(size_t)r * n + c];
            if (f == 0.0) continue;
            for (int k = 0; k < n; ++k) {
                A[(size_t)r * n + k] -= f * A[(size_t)c * n + k];
                inv[(size_t)r * n + k] -= f * inv[(size_t)c * n + k];
            }
        }
    }
    return true;
}

}  // namespace vd

using namespace vd;

struct vd_mgd_plan {
    vd_mgd_desc d;
    std::vector<MgdLevel> lv;
    void* coef = nullptr;           // [level][nmode][4] plan dtype (MgdLev::coef), then op [nmode][3] (k_mgd_pq)
    int nb = 0;                     // coarsest unknowns
    int32_t* cidx = nullptr;        // [nb]
    double* cinv = nullptr;         // [nmode][nb][nb]
};

static int mgd_coarsenable(int n) { return (n + 1) % 2 == 0 && (n + 1) / 2 - 1 >= 3; }

extern "C" vd_status vd_mgd_plan_create(vd_mgd_plan** out, const vd_mgd_desc* d)
{
    if (!out || !d) return VD_ERR_ARG;
    *out = nullptr;
    if (d->n0 < 1 || d->n1 < 1 || d->nmode < 1 || !d->lambda_host || !(d->d0 > 0) || !(d->d1 > 0) ||
        d->max_cycles < 1 || !(d->tol > 0) || (d->dtype != VD_F32 && d->dtype != VD_F64))
        return VD_ERR_ARG;
    vd_mgd_plan* p = new (std::nothrow) vd_mgd_plan();
    if (!p) return VD_ERR_ARG;
    p->d = *d;
    p->d.mask_host = nullptr;
    p->d.lambda_host = nullptr;
    auto fail = [&](int code) { vd_mgd_plan_destroy(p); return code; };
    // level hierarchy on the host
    std::vector<std::vector<int8_t>> masks;
    std::vector<int8_t> m0((size_t)d->n0 * d->n1, 1);
    if (d->mask_host)
        for (size_t k = 0; k < m0.size(); ++k) m0[k] = d->mask_host[k] != 0.0;
    masks.push_back(m0);
    std::vector<int> n0s{d->n0}, n1s{d->n1};
    std::vector<double> d0s{d->d0}, d1s{d->d1};
    while (mgd_coarsenable(n0s.back()) && mgd_coarsenable(n1s.back()) && n0s.back() * n1s.back() > 64) {
        const int n0 = n0s.back(), n1 = n1s.back();
        const int c0 = (n0 + 1) / 2 - 1, c1 = (n1 + 1) / 2 - 1;
        // a coarse node is an unknown only if the 3 x 3 fine nodes around it
        // are: a coarse level never bridges a fine land barrier (which would
        // join basins that the fine problem keeps apart)
        std::vector<int8_t> mc((size_t)c0 * c1);
        const std::vector<int8_t>& mf = masks.back();
        for (int I = 0; I < c0; ++I)
            for (int J = 0; J < c1; ++J) {
                int8_t v = 1;
                for (int a = -1; a <= 1; ++a)
                    for (int c = -1; c <= 1; ++c) v &= mf[(size_t)(2 * I + 1 + a) * n1 + 2 * J + 1 + c];
                mc[(size_t)I * c1 + J] = v;
            }
        masks.push_back(mc);
        n0s.push_back(c0); n1s.push_back(c1);
        d0s.push_back(2 * d0s.back()); d1s.push_back(2 * d1s.back());
    }
    const int nlev = (int)masks.size();
    // coarsest level: float64 inverse per mode over its unknowns
    const int cn0 = n0s.back(), cn1 = n1s.back();
    std::vector<int32_t> idx;
    for (int k = 0; k < cn0 * cn1; ++k)
        if (masks.back()[k]) idx.push_back(k);
    p->nb = (int)idx.size();
    if (p->nb > 4096) return fail(VD_ERR_UNSUPPORTED);
    std::vector<double> invs((size_t)d->nmode * p->nb * p->nb);
    {
        const double a0 = 1.0 / (d0s.back() * d0s.back()), a1 = 1.0 / (d1s.back() * d1s.back());
        std::vector<int> pos((size_t)cn0 * cn1, -1);
        for (int k = 0; k < p->nb; ++k) pos[idx[k]] = k;
        for (int m = 0; m < d->nmode; ++m) {
            std::vector<double> A((size_t)p->nb * p->nb, 0.0), inv;
            for (int k = 0; k < p->nb; ++k) {
                const int i = idx[k] / cn1, j = idx[k] % cn1;
                A[(size_t)k * p->nb + k] = -2 * a0 - 2 * a1 - d->lambda_host[m];
                const int nbs[4][2] = {{i - 1, j}, {i + 1, j}, {i, j - 1}, {i, j + 1}};
                for (int t = 0; t < 4; ++t) {
                    const int ii = nbs[t][0], jj = nbs[t][1];
                    if (ii < 0 || ii >= cn0 || jj < 0 || jj >= cn1) continue;
                    const int q = pos[(size_t)ii * cn1 + jj];
                    if (q >= 0) A[(size_t)k * p->nb + q] += t < 2 ? a0 : a1;
                }
            }
            if (p->nb && !invert(A, p->nb, inv)) return fail(VD_ERR_ARG);
            std::copy(inv.begin(), inv.end(), invs.begin() + (size_t)m * p->nb * p->nb);
        }
    }
    // device tables
    p->lv.resize(nlev);
    for (int l = 0; l < nlev; ++l) {
        MgdLevel& L = p->lv[l];
        L.n0 = n0s[l]; L.n1 = n1s[l]; L.d0 = d0s[l]; L.d1 = d1s[l];
        if (cudaMalloc(&L.mask, masks[l].size()) != cudaSuccess) return fail(VD_ERR_CUDA);
        if (cudaMemcpy(L.mask, masks[l].data(), masks[l].size(), cudaMemcpyHostToDevice) != cudaSuccess)
            return fail(VD_ERR_CUDA);
    }
    const size_t es = d->dtype == VD_F64 ? 8 : 4;
    std::vector<char> co(es * d->nmode * (4 * (size_t)nlev + 3));
    auto put = [&](size_t o, double v) {
        if (es == 8) reinterpret_cast<double*>(co.data())[o] = v;
        else reinterpret_cast<float*>(co.data())[o] = (float)v;
    };
    for (int l = 0; l < nlev; ++l)
        for (int m = 0; m < d->nmode; ++m) {
            const double a0 = 1.0 / (d0s[l] * d0s[l]), a1 = 1.0 / (d1s[l] * d1s[l]);
            const double D = 2 * a0 + 2 * a1 + d->lambda_host[m];
            const double v[4] = {1.0 / D, a0 / D, a1 / D, D};
            for (int k = 0; k < 4; ++k) put(4 * ((size_t)l * d->nmode + m) + k, v[k]);
        }
    for (int m = 0; m < d->nmode; ++m) {
        const size_t o = 4 * (size_t)nlev * d->nmode + 3 * (size_t)m;
        put(o, 1.0 / (d->d0 * d->d0));
        put(o + 1, 1.0 / (d->d1 * d->d1));
        put(o + 2, d->lambda_host[m]);
    }
    if (cudaMalloc(&p->coef, co.size()) != cudaSuccess ||
        cudaMemcpy(p->coef, co.data(), co.size(), cudaMemcpyHostToDevice) != cudaSuccess)
        return fail(VD_ERR_CUDA);
    if (p->nb) {
        if (cudaMalloc(&p->cidx, idx.size() * 4) != cudaSuccess ||
            cudaMemcpy(p->cidx, idx.data(), idx.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
            cudaMalloc(&p->cinv, invs.size() * 8) != cudaSuccess ||
            cudaMemcpy(p->cinv, invs.data(), invs.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess)
            return fail(VD_ERR_CUDA);
    }
    *out = p;
    return VD_OK;
}

extern "C" vd_status vd_mgd_plan_destroy(vd_mgd_plan* p)
{
    if (!p) return VD_OK;
    for (auto& L : p->lv) cudaFree(L.mask);
    cudaFree(p->coef);
    cudaFree(p->cidx);
    cudaFree(p->cinv);
    delete p;
    return VD_OK;
}

extern "C" int vd_mgd_levels(const vd_mgd_plan* p) { return p ? (int)p->lv.size() : 0; }
extern "C" int vd_mgd_coarse_unknowns(const vd_mgd_plan* p) { return p ? p->nb : 0; }

// Tiles of the level kernels: 32 x 64 points, or 8 x 32 where the larger ones
// would leave SMs idle (a level's tile is bound by its SM's FP64 rate: 32 x 64
// points take about 7 us alone, whatever the level's size).
constexpr int MGD_TI = 32, MGD_TJ = 64, MGD_SI = 8, MGD_SJ = 32;

static bool mgd_small_tiles(int n0, int n1, int nsys)
{
    return (long long)((n0 + MGD_TI - 1) / MGD_TI) * ((n1 + MGD_TJ - 1) / MGD_TJ) * nsys < 152;
}

static dim3 mgd_grid(int n0, int n1, int nsys)
{
    if (mgd_small_tiles(n0, n1, nsys)) return dim3((n1 + MGD_SJ - 1) / MGD_SJ, (n0 + MGD_SI - 1) / MGD_SI, nsys);
    return dim3((n1 + MGD_TJ - 1) / MGD_TJ, (n0 + MGD_TI - 1) / MGD_TI, nsys);
}

// per level: the descent's u, the right-hand side and the ascent's u of nsys
// systems; then the conjugate-gradient vectors r, p, q of level 0; flags and
// arrival counts; dot partial sums; scalars; beta. Level 0's right-hand side
// is r itself: its slot is the second buffer of p.
static size_t mgd_layout(const vd_mgd_plan* p, int nsys, std::vector<size_t>* off)
{
    const size_t es = p->d.dtype == VD_F64 ? 8 : 4;
    size_t o = 0;
    auto take = [&](size_t bytes) { const size_t a = o; o = (o + bytes + 255) & ~size_t(255); return a; };
    if (off) off->clear();
    for (size_t l = 0; l < p->lv.size(); ++l)
        for (int w = 0; w < 3; ++w) {
            const size_t a = take(es * (size_t)nsys * p->lv[l].n0 * p->lv[l].n1);
            if (off) off->push_back(a);
        }
    const size_t n0 = es * (size_t)nsys * p->lv[0].n0 * p->lv[0].n1;
    const dim3 g = mgd_grid(p->lv[0].n0, p->lv[0].n1, nsys);
    const size_t cr = take(n0), cp = take(n0), cq = take(n0);
    const size_t fl = take(4 * (size_t)2 * nsys);
    const size_t pa = take(8 * (size_t)nsys * g.x * g.y);
    const size_t sc = take(8 * (size_t)nsys * MGD_SCAL);
    const size_t be = take(8 * (size_t)nsys);
    if (off) for (size_t a : {cr, cp, cq, fl, pa, sc, be}) off->push_back(a);
    return o;
}

extern "C" size_t vd_mgd_workspace_bytes(const vd_mgd_plan* p, int batch)
{
    if (!p || batch < 1) return 0;
    return mgd_layout(p, batch * p->d.nmode, nullptr);
}

template <typename T>
static size_t mgd_chain_smem(const MgdChain<T>& C)
{
    size_t n = 0;
    for (int l = 0; l < C.nlev; ++l) n += 2 * (size_t)C.lv[l].n0 * C.lv[l].n1;
    return n * sizeof(T);
}

static PerDeviceOnce g_mgd_once;

static cudaError_t mgd_configure()
{
    return g_mgd_once.run([]() -> cudaError_t {
        cudaError_t e = cudaSuccess;
        auto set = [&](const void* f, size_t bytes) {
            if (!e) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        };
        constexpr size_t b8 = MgdTile<double, MGD_TI, MGD_TJ>::bytes, b4 = MgdTile<float, MGD_TI, MGD_TJ>::bytes;
        set((const void*)k_mgd_pre<double, MGD_TI, MGD_TJ>, b8);
        set((const void*)k_mgd_post<double, MGD_TI, MGD_TJ, true>, b8);
        set((const void*)k_mgd_post<double, MGD_TI, MGD_TJ, false>, b8);
        set((const void*)k_mgd_pre<float, MGD_TI, MGD_TJ>, b4);
        set((const void*)k_mgd_post<float, MGD_TI, MGD_TJ, true>, b4);
        set((const void*)k_mgd_post<float, MGD_TI, MGD_TJ, false>, b4);
        return e;
    });
}

// The tile kernels of one solve with one tile shape.
template <typename T, int TI, int TJ>
struct MgdLaunch {
    static constexpr size_t smem = MgdTile<T, TI, TJ>::bytes;
    static void pre(dim3 g, cudaStream_t st, const MgdLev<T>& A, const T* b, T* u, const MgdLev<T>& C, T* bc)
    {
        k_mgd_pre<T, TI, TJ><<<g, MGD_NT, smem, st>>>(A, b, u, C.n0, C.n1, C.mask, bc);
    }
    static void post(dim3 g, cudaStream_t st, const MgdLev<T>& A, const T* b, const T* u, const MgdLev<T>& C,
                     const T* ec, T* z, const MgdDot* D)
    {
        if (D) k_mgd_post<T, TI, TJ, true><<<g, MGD_NT, smem, st>>>(A, b, u, C.n0, C.n1, ec, z, *D);
        else k_mgd_post<T, TI, TJ, false><<<g, MGD_NT, smem, st>>>(A, b, u, C.n0, C.n1, ec, z, MgdDot{});
    }
};

template <typename T>
static int mgd_solve_t(const vd_mgd_plan* p, int batch, const T* b, long long ldb, long long fsb, T* u, long long ldu,
                       long long fsu, double* rel, char* ws, cudaStream_t st)
{
    if (mgd_configure() != cudaSuccess) return VD_ERR_CUDA;
    const int nsys = batch * p->d.nmode;
    std::vector<size_t> off;
    mgd_layout(p, nsys, &off);
    const int nlev = (int)p->lv.size();
    auto buf = [&](int l, int w) { return (T*)(ws + off[3 * l + w]); };
    T* cr = (T*)(ws + off[3 * nlev]);
    T* cp[2] = {(T*)(ws + off[3 * nlev + 1]), buf(0, 1)};
    T* cq = (T*)(ws + off[3 * nlev + 2]);
    T* cz = buf(0, 2);
    int* done = (int*)(ws + off[3 * nlev + 3]);
    MgdDot D;
    D.tol = p->d.tol;
    D.count = done + nsys;
    D.part = (double*)(ws + off[3 * nlev + 4]);
    D.sc = (double*)(ws + off[3 * nlev + 5]);
    D.beta = (double*)(ws + off[3 * nlev + 6]);
    D.done = done;
    D.rel = rel;
    auto dot = [&](int what) { D.what = what; return D; };
    auto lev = [&](int l) {
        MgdLev<T> A;
        A.n0 = p->lv[l].n0; A.n1 = p->lv[l].n1;
        A.mask = p->lv[l].mask; A.coef = (const T*)p->coef + 4 * (size_t)l * p->d.nmode;
        A.batch = batch; A.done = done;
        return A;
    };
    auto small = [&](int l) { return mgd_small_tiles(p->lv[l].n0, p->lv[l].n1, nsys); };
    auto grid = [&](int l) { return mgd_grid(p->lv[l].n0, p->lv[l].n1, nsys); };
    // the one-block levels [lc, nlev): none when the coarsest is large
    int lc = nlev;
    MgdChain<T> ch{};
    if (p->nb <= MGD_CHAIN_UNKNOWNS && nlev <= MGD_CHAIN_LEVELS)
        while (lc > 1 && p->lv[lc - 1].n0 * p->lv[lc - 1].n1 <= MGD_CHAIN_CELLS) --lc;
    if (lc < nlev) {
        ch.nlev = nlev - lc;
        for (int l = lc; l < nlev; ++l) ch.lv[l - lc] = lev(l);
        ch.nb = p->nb; ch.cidx = p->cidx; ch.cinv = p->cinv;
    }
    const int lt = std::min(lc, nlev - 1);      // first level without tile kernels
    // z = V(r), with r.z reduced as `what`
    auto precond = [&](int what) -> int {
        auto rhs = [&](int l) { return l ? buf(l, 1) : cr; };
        for (int l = 0; l < lt; ++l) {
            if (small(l)) MgdLaunch<T, MGD_SI, MGD_SJ>::pre(grid(l), st, lev(l), rhs(l), buf(l, 0), lev(l + 1), buf(l + 1, 1));
            else MgdLaunch<T, MGD_TI, MGD_TJ>::pre(grid(l), st, lev(l), rhs(l), buf(l, 0), lev(l + 1), buf(l + 1, 1));
            VD_LAUNCH_CHECK();
        }
        if (lc < nlev) {
            k_mgd_chain<T><<<nsys, MGD_NT, mgd_chain_smem(ch), st>>>(ch, buf(lt, 1), buf(lt, 2));
            VD_LAUNCH_CHECK();
        } else if (p->nb) {
            const int l = nlev - 1;
            k_mgd_coarse<T><<<dim3((p->nb + 7) / 8, nsys), 256, 0, st>>>(p->nb, p->lv[l].n0 * p->lv[l].n1, batch, done,
                                                                          p->cidx, p->cinv, buf(l, 1), buf(l, 2));
            VD_LAUNCH_CHECK();
        }
        const MgdDot d = dot(what);
        for (int l = lt - 1; l >= 0; --l) {
            const MgdDot* dp = l == 0 ? &d : nullptr;
            if (small(l)) MgdLaunch<T, MGD_SI, MGD_SJ>::post(grid(l), st, lev(l), rhs(l), buf(l, 0), lev(l + 1), buf(l + 1, 2), buf(l, 2), dp);
            else MgdLaunch<T, MGD_TI, MGD_TJ>::post(grid(l), st, lev(l), rhs(l), buf(l, 0), lev(l + 1), buf(l + 1, 2), buf(l, 2), dp);
            VD_LAUNCH_CHECK();
        }
        return VD_OK;
    };
    const bool s0 = small(0);
    const dim3 g0 = grid(0);
    const MgdLev<T> A0 = lev(0);
    const T* op = (const T*)p->coef + 4 * (size_t)nlev * p->d.nmode;
    k_mgd_fill_int<<<(2 * nsys + 255) / 256, 256, 0, st>>>(2 * nsys, 0, done);
    VD_LAUNCH_CHECK();
    if (lc == nlev) {
        // k_mgd_coarse writes the unknowns only; land stays 0
        const int l = nlev - 1;
        VD_CUDA_TRY(cudaMemsetAsync(buf(l, 2), 0, sizeof(T) * (size_t)nsys * p->lv[l].n0 * p->lv[l].n1, st));
    }
    if (s0) k_mgd_init<T, MGD_SI, MGD_SJ><<<g0, MGD_NT, 0, st>>>(A0, b, ldb, fsb, u, ldu, fsu, cr, dot(0));
    else k_mgd_init<T, MGD_TI, MGD_TJ><<<g0, MGD_NT, 0, st>>>(A0, b, ldb, fsb, u, ldu, fsu, cr, dot(0));
    VD_LAUNCH_CHECK();
    int rc;
    if ((rc = precond(1))) return rc;
    for (int it = 0; it < p->d.max_cycles; ++it) {
        // sc[2] = rho / (p . q) = -alpha
        T *pn = cp[it & 1], *po = cp[1 - (it & 1)];
        if (s0) k_mgd_pq<T, MGD_SI, MGD_SJ><<<g0, MGD_NT, 0, st>>>(A0, op, it == 0, cz, po, pn, cq, dot(2));
        else k_mgd_pq<T, MGD_TI, MGD_TJ><<<g0, MGD_NT, 0, st>>>(A0, op, it == 0, cz, po, pn, cq, dot(2));
        VD_LAUNCH_CHECK();
        if (s0) k_mgd_xr<T, MGD_SI, MGD_SJ><<<g0, MGD_NT, 0, st>>>(A0, pn, cq, u, ldu, fsu, cr, dot(3));
        else k_mgd_xr<T, MGD_TI, MGD_TJ><<<g0, MGD_NT, 0, st>>>(A0, pn, cq, u, ldu, fsu, cr, dot(3));
        VD_LAUNCH_CHECK();
        if (it + 1 < p->d.max_cycles && (rc = precond(4))) return rc;
    }
    return VD_OK;
}

extern "C" vd_status vd_mgd_solve(const vd_mgd_plan* p, int batch, const void* b, long long ldb, long long fsb,
                                  void* u, long long ldu, long long fsu, double* rel, void* work, size_t work_bytes,
                                  void* stream)
{
    if (!p || batch < 1 || !b || !u || !work || ldb < p->d.n1 || ldu < p->d.n1 || fsb < ldb * p->d.n0 ||
        fsu < ldu * p->d.n0)
        return VD_ERR_ARG;
    if (work_bytes < vd_mgd_workspace_bytes(p, batch)) return VD_ERR_WORKSPACE;
    if (p->lv.size() < 2) return VD_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    return p->d.dtype == VD_F64
               ? mgd_solve_t<double>(p, batch, (const double*)b, ldb, fsb, (double*)u, ldu, fsu, rel, (char*)work, st)
               : mgd_solve_t<float>(p, batch, (const float*)b, ldb, fsb, (float*)u, ldu, fsu, rel, (char*)work, st);
}

