// Masked multigrid Helmholtz solver: div(c grad u) - lambda u = rhs on cell
// centres of a masked domain in an n0 x n1 rectangle, homogeneous Neumann
// walls on cell edges (mapping/models/model_qgsw/helmholtz_multigrid.py,
// MG_Helmholtz 156-419): damped Jacobi (omega = 0.95, 6 sweeps per smooth,
// 73-99), residual (102-114), cell-centred restriction / 9-3-3-1
// prolongation with mask-count divisors (117-151, 265-278), mask and
// coefficient hierarchies (248-293), full-multigrid start then max_ite
// V-cycles (322-419), bottom solve by pseudo-inverse (226-237) or Jacobi.
//
// A batch of nsys systems shares the grid and coefficient; system b uses
// lambda[b]. Arrays are row-major [nsys][n0][n1]. Every level keeps its
// mask, edge coefficients, divisors and Jacobi factor on the device; the
// recursion runs on the host and only launches kernels on the caller's
// stream, so a whole solve can be captured in a CUDA graph.
#include "vd_internal.cuh"
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

namespace {

struct HLevel {
    int n0 = 0, n1 = 0;
    double d0 = 0, d1 = 0;
    std::vector<double> mask, cu, cv, divr, divp, factor;   // factor [nsys][n0][n1]
};

int mg_nlevels(int n)
{
    if (n <= 8) return 1;
    int h = 0;
    while (((n >> h) & 1) == 0) ++h;
    while ((n >> h) < 8) --h;
    return 1 + h;
}

double at(const std::vector<double>& a, int n0, int n1, int i, int j)
{
    return (i < 0 || j < 0 || i >= n0 || j >= n1) ? 0.0 : a[(size_t)i * n1 + j];
}

// pseudo-inverse of a symmetric matrix (cyclic Jacobi eigenvalues; the cut
// |lambda| <= 1e-15 max|lambda| of numpy.linalg.pinv's default rcond)
std::vector<double> pinv_sym(std::vector<double> A, int N)
{
    std::vector<double> V((size_t)N * N, 0.0);
    for (int i = 0; i < N; ++i) V[(size_t)i * N + i] = 1.0;
    for (int sweep = 0; sweep < 100; ++sweep) {
        double off = 0.0, tot = 0.0;
        for (int i = 0; i < N; ++i)
            for (int j = 0; j < N; ++j) {
                const double v = A[(size_t)i * N + j] * A[(size_t)i * N + j];
                tot += v;
                if (i != j) off += v;
            }
        if (off <= 1e-30 * tot) break;
        for (int p = 0; p < N - 1; ++p)
            for (int q = p + 1; q < N; ++q) {
                const double apq = A[(size_t)p * N + q];
                if (apq == 0.0) continue;
                const double app = A[(size_t)p * N + p], aqq = A[(size_t)q * N + q];
                const double theta = (aqq - app) / (2 * apq);
                const double t = (theta >= 0 ? 1.0 : -1.0) / (std::fabs(theta) + std::sqrt(theta * theta + 1));
                const double c = 1 / std::sqrt(t * t + 1), s = t * c;
                for (int k = 0; k < N; ++k) {
                    const double akp = A[(size_t)k * N + p], akq = A[(size_t)k * N + q];
                    A[(size_t)k * N + p] = c * akp - s * akq;
                    A[(size_t)k * N + q] = s * akp + c * akq;
                }
                for (int k = 0; k < N; ++k) {
                    const double apk = A[(size_t)p * N + k], aqk = A[(size_t)q * N + k];
                    A[(size_t)p * N + k] = c * apk - s * aqk;
                    A[(size_t)q * N + k] = s * apk + c * aqk;
                }
                for (int k = 0; k < N; ++k) {
                    const double vkp = V[(size_t)k * N + p], vkq = V[(size_t)k * N + q];
                    V[(size_t)k * N + p] = c * vkp - s * vkq;
                    V[(size_t)k * N + q] = s * vkp + c * vkq;
                }
            }
    }
    double emax = 0.0;
    for (int i = 0; i < N; ++i) emax = std::max(emax, std::fabs(A[(size_t)i * N + i]));
    std::vector<double> P((size_t)N * N, 0.0);
    for (int e = 0; e < N; ++e) {
        const double lam = A[(size_t)e * N + e];
        if (std::fabs(lam) <= 1e-15 * emax) continue;
        for (int i = 0; i < N; ++i)
            for (int j = 0; j < N; ++j) P[(size_t)i * N + j] += V[(size_t)i * N + e] * V[(size_t)j * N + e] / lam;
    }
    return P;
}

}  // namespace

struct vd_mg_plan {
    int n0 = 0, n1 = 0, nsys = 0, dtype = VD_F64, nlev = 0, max_ite = 20, niter_bottom = -1;
    double omega = 0.95;
    std::vector<double> lambda;
    std::vector<HLevel> lv;
    int nb = 0;                          // bottom cells
    int lc = 0;                          // first level run by the one-block coarse kernel (nlev: none)
    void* dev = nullptr;
    struct DLev {
        const void *mask = nullptr, *cu = nullptr, *cv = nullptr, *factor = nullptr, *g = nullptr, *mr = nullptr,
                   *mp = nullptr;
    };
    std::vector<DLev> dl;
    const void* lam = nullptr;           // [nsys]
    const int32_t* bot_idx = nullptr;    // [nb] flat bottom cell index
    const void* bot_inv = nullptr;       // [nsys][nb][nb]
    // the bottom level's 6 niter_bottom damped sweeps as one linear map,
    // f = N rhs (+ M f on a one-level grid): [nsys][N, M][output m][input k]
    const void* bot_sm = nullptr;
    // the whole solve as one CUDA graph on plan-owned rhs / solution buffers
    // (captured at the first solve with a given workspace, replayed after)
    void* gbuf = nullptr;                // [2][nsys][n0][n1]: rhs, solution
    cudaStream_t gstream = nullptr;      // capture stream
    cudaGraphExec_t gexec = nullptr;
    const void* gws = nullptr;           // workspace the graph was captured with
    std::vector<size_t> ws_off;          // per level: f, rhs, tmp, scaled rhs offsets (elements)
    size_t ws_elems = 0;
};

namespace vd {

// One level on the device. The edge coefficients are stored pre-scaled by
// 1/d0^2 and 1/d1^2 and the Jacobi factor pre-multiplied by omega. In float64,
// whose instruction rate bounds the sweeps, they are also stored times the factor
// (g), and the level's right-hand side once times the factor (rr = factor rhs): a
// sweep is then 5 FP64 instructions a cell instead of 7, for as many arrays. In
// float32, bound by memory and launches, the shared coefficients are the fewer bytes.
template <typename T>
struct MgLev {
    int n0, n1;
    const T *mask, *cu, *cv, *factor, *lam;   // cu = c_u/d0^2, cv = c_v/d1^2, factor = omega mask/den
    const T* g;                               // float64: [nsys][4][n0][n1], towards i+1, i-1, j+1, j-1
    const T *mr, *mp;                         // mask / divisor of the restriction here, the prolongation to here
};
template <typename T> constexpr bool mg_scaled = sizeof(T) == 8;

template <typename T>
__device__ __forceinline__ T fat(const T* f, int n0, int n1, int i, int j)
{
    return (i < 0 || j < 0 || i >= n0 || j >= n1) ? T(0) : f[(long long)i * n1 + j];
}

// Per-point arithmetic, shared by the level-wide kernels, the tile kernels and the
// one-block coarse-level kernel so that all give the same bits.

// what a sweep reads of the right-hand side, at cell o of system b
template <typename T>
__device__ __forceinline__ T mg_scaled_rhs(const MgLev<T>& L, T rhs, int b, long long o)
{
    if constexpr (mg_scaled<T>) return __ldg(L.factor + (long long)b * L.n0 * L.n1 + o) * rhs;
    else return rhs;
}

// the first sweep from f = 0
template <typename T>
__device__ __forceinline__ T mg_first(const MgLev<T>& L, T rr, int b, long long o)
{
    if constexpr (mg_scaled<T>) return -rr;
    else return __ldg(L.factor + (long long)b * L.n0 * L.n1 + o) * (T(0) - rr);
}

// one damped Jacobi update of cell (i, j) from its neighbours (helmholtz_multigrid.py:86-98)
template <typename T>
__device__ __forceinline__ T mg_update(const MgLev<T>& L, T fc, T fe, T fw, T fn, T fs, T rr, int b, int i, int j,
                                       T omega)
{
    const long long n = (long long)L.n0 * L.n1, o = (long long)i * L.n1 + j;
    if constexpr (mg_scaled<T>) {
        const T* g = L.g + 4 * b * n + o;
        const T s = (T(1) - omega) * fc - rr;
        return __ldg(g) * fe + (__ldg(g + n) * fw + (__ldg(g + 2 * n) * fn + (__ldg(g + 3 * n) * fs + s)));
    } else {
        const T cup = L.cu[o + L.n1], cui = L.cu[o];
        const T cvp = L.cv[o + i + 1], cvi = L.cv[o + i];
        const T s = cup * fe + cui * fw + cvp * fn + cvi * fs;
        return __ldg(L.factor + b * n + o) * (s - rr) + (T(1) - omega) * fc;
    }
}
template <typename T>
__device__ __forceinline__ T mg_sweep_pt(const MgLev<T>& L, const T* F, T rr, int b, int i, int j, T omega)
{
    return mg_update(L, F[(long long)i * L.n1 + j], fat(F, L.n0, L.n1, i + 1, j), fat(F, L.n0, L.n1, i - 1, j),
                     fat(F, L.n0, L.n1, i, j + 1), fat(F, L.n0, L.n1, i, j - 1), rr, b, i, j, omega);
}

// rhs - mask (div(c grad f) - lambda f) at (i, j)  (helmholtz_multigrid.py:102-114)
template <typename T>
__device__ __forceinline__ T mg_resid(const MgLev<T>& L, T fc, T fe, T fw, T fn, T fs, T rhs, T lam, int i, int j)
{
    const long long o = (long long)i * L.n1 + j;
    const T cup = L.cu[o + L.n1], cui = L.cu[o];
    const T cvp = L.cv[o + i + 1], cvi = L.cv[o + i];
    // (one chain of FMAs: 10 FP64 instructions)
    T h = cup * (fe - fc);
    h = h - cui * (fc - fw);
    h = h + cvp * (fn - fc);
    h = h - cvi * (fc - fs);
    h = h - lam * fc;
    return rhs - h * L.mask[o];
}
template <typename T>
__device__ __forceinline__ T mg_residual_pt(const MgLev<T>& L, const T* F, T rhs, T lam, int i, int j)
{
    return mg_resid(L, F[(long long)i * L.n1 + j], fat(F, L.n0, L.n1, i + 1, j), fat(F, L.n0, L.n1, i - 1, j),
                    fat(F, L.n0, L.n1, i, j + 1), fat(F, L.n0, L.n1, i, j - 1), rhs, lam, i, j);
}

// (sum of the 2x2 fine cells) * (mask / div) at coarse (I, J)  (147-151)
template <typename T>
__device__ __forceinline__ T mg_restrict_pt(const T* fine, int n1c, int I, int J, const T* mr)
{
    const int n1f = 2 * n1c;
    const T* F = fine + (long long)(2 * I) * n1f + 2 * J;
    return (F[0] + F[n1f] + F[1] + F[n1f + 1]) * mr[(long long)I * n1c + J];
}

// f + prolong(coarse) * (mask / div) at a fine cell: 9-3-3-1 weights as two
// interpolations of 3-1, along i then j  (117-144). c: its coarse cell, then the
// coarse neighbours it leans on along i, along j and across
template <typename T>
__device__ __forceinline__ T mg_prolong4(T c, T ci, T cj, T cij, T mp, T f)
{
    return f + (T(3) * (T(3) * c + ci) + (T(3) * cj + cij)) * mp;
}
template <typename T>
__device__ __forceinline__ T mg_prolong_pt(const T* V, int n0c, int n1c, int i_f, int jf, T mp, T f)
{
    const int I = i_f >> 1, J = jf >> 1;
    const int di = (i_f & 1) ? 1 : -1, dj = (jf & 1) ? 1 : -1;
    return mg_prolong4(fat(V, n0c, n1c, I, J), fat(V, n0c, n1c, I + di, J), fat(V, n0c, n1c, I, J + dj),
                       fat(V, n0c, n1c, I + di, J + dj), mp, f);
}

// One sweep of a level. FP64-issue bound in float64 at the large levels (1024 x 768:
// 9.8 us, 7.9 at the pipe's rate; with 7 instructions a cell 13.0 us).
template <typename T>
__global__ void k_mg_sweep(MgLev<T> L, const T* __restrict__ f, const T* __restrict__ rr, T* __restrict__ out,
                           T omega)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y, b = blockIdx.z;
    if (j >= L.n1) return;
    const long long fs = (long long)L.n0 * L.n1, o = (long long)i * L.n1 + j;
    out[b * fs + o] = mg_sweep_pt(L, f + b * fs, rr[b * fs + o], b, i, j, omega);
}

template <typename T>
__global__ void k_mg_residual(MgLev<T> L, const T* __restrict__ f, const T* __restrict__ rhs, T* __restrict__ res)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y, b = blockIdx.z;
    if (j >= L.n1) return;
    const long long fs = (long long)L.n0 * L.n1, o = (long long)i * L.n1 + j;
    res[b * fs + o] = mg_residual_pt(L, f + b * fs, rhs[b * fs + o], L.lam[b], i, j);
}

// The sweep's coefficients (MgLev::g) of a level from its factor and edge coefficients, at
// plan creation. (Formed on the host, with their copy there: 82 ms for a plan of 12
// systems of 512^2, here 31.)
template <typename T>
__global__ void k_mg_coeffs(int n0, int n1, const T* __restrict__ cu, const T* __restrict__ cv,
                            const T* __restrict__ factor, T* __restrict__ g)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y, b = blockIdx.z;
    if (j >= n1) return;
    const long long n = (long long)n0 * n1, o = (long long)i * n1 + j;
    const T w = factor[b * n + o];
    g += 4 * b * n + o;
    g[0] = w * cu[o + n1];
    g[n] = w * cu[o];
    g[2 * n] = w * cv[o + i + 1];
    g[3 * n] = w * cv[o + i];
}

// rr of a level (float64, the finest level's once a solve)
template <typename T>
__global__ void k_mg_scale(MgLev<T> L, const T* __restrict__ rhs, T* __restrict__ rr)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y, b = blockIdx.z;
    if (j >= L.n1) return;
    const long long fs = (long long)L.n0 * L.n1, o = (long long)i * L.n1 + j;
    rr[b * fs + o] = mg_scaled_rhs(L, rhs[b * fs + o], b, o);
}

// What a level keeps of its right-hand side v at cell o: rhs, rr (float64) and,
// where first is given, the result of the first sweep from f = 0.
template <typename T>
struct MgDown {
    T *rhs, *rr, *first;
};
template <typename T>
__device__ __forceinline__ void mg_put_rhs(const MgLev<T>& C, const MgDown<T>& d, T v, int b, long long o)
{
    const long long go = (long long)b * C.n0 * C.n1 + o;
    d.rhs[go] = v;
    const T rr = mg_scaled_rhs(C, v, b, o);
    if constexpr (mg_scaled<T>) d.rr[go] = rr;
    if (d.first) d.first[go] = mg_first(C, rr, b, o);
}

template <typename T>
__global__ void k_mg_restrict(MgLev<T> C, const T* __restrict__ fine, MgDown<T> d)
{
    const int J = blockIdx.x * blockDim.x + threadIdx.x;
    const int I = blockIdx.y, b = blockIdx.z;
    if (J >= C.n1) return;
    const long long fsc = (long long)C.n0 * C.n1;
    mg_put_rhs(C, d, mg_restrict_pt(fine + b * 4 * fsc, C.n1, I, J, C.mr), b, (long long)I * C.n1 + J);
}

// Residual of level L restricted to level C, one thread a coarse cell (its four
// residuals never leave registers). 1024 x 768 float64: 19.7 us (17 + 10 as two kernels
// with a division), 16 at the FP64 rate.
template <typename T>
__global__ void k_mg_resid_restrict(MgLev<T> L, MgLev<T> C, const T* __restrict__ f, const T* __restrict__ rhs,
                                    MgDown<T> d)
{
    const int J = blockIdx.x * blockDim.x + threadIdx.x;
    const int I = blockIdx.y, b = blockIdx.z;
    if (J >= C.n1) return;
    const long long fs = (long long)L.n0 * L.n1;
    f += b * fs;
    rhs += b * fs;
    T r[2][2];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const int i = 2 * I + u, j = 2 * J + v;
            r[u][v] = mg_residual_pt(L, f, rhs[(long long)i * L.n1 + j], L.lam[b], i, j);
        }
    const long long o = (long long)I * C.n1 + J;
    mg_put_rhs(C, d, (r[0][0] + r[1][0] + r[0][1] + r[1][1]) * C.mr[o], b, o);
}

// Prolongation to level L of the coarse field V, one thread a coarse cell: its four
// fine cells share their 3-1 interpolations along i (3.5 FP64 instructions a fine cell,
// a division and 7 more when each fine cell was formed alone: 30 us at 1024 x 768, here
// 8.4).
template <typename T>
__global__ void k_mg_prolong(MgLev<T> L, int n0c, int n1c, const T* __restrict__ V, T* __restrict__ fine, int add)
{
    const int J = blockIdx.x * blockDim.x + threadIdx.x;
    const int I = blockIdx.y, b = blockIdx.z;
    if (J >= n1c) return;
    V += b * (long long)n0c * n1c;
    fine += b * (long long)L.n0 * L.n1;
    T c[3][3];
#pragma unroll
    for (int u = 0; u < 3; ++u)
#pragma unroll
        for (int v = 0; v < 3; ++v) c[u][v] = fat(V, n0c, n1c, I + u - 1, J + v - 1);
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const long long o = (long long)(2 * I + u) * L.n1 + 2 * J + v;
            fine[o] = mg_prolong4(c[1][1], c[2 * u][1], c[1][2 * v], c[2 * u][2 * v], L.mp[o],
                                  add ? fine[o] : T(0));
        }
}

// Six sweeps of a level in one launch, over tiles of RO x CO cells with a halo that
// shrinks by a cell a sweep; for the levels whose sweep is shorter than a launch.
// DOWN: the pre-smoothing, from f or (ZERO) from f = 0, then the residual, restricted
// to the coarser level C; in = f, out = the smoothed field, which goes to another
// buffer since tiles read one another's cells. Up: in + prolonged correction V, then
// the six sweeps.
// A block is bound by its SM's FP64 rate (1.7 lanes a clock), so the tile is as small
// as it takes to cover the SMs: the host picks the size by the sum of the active cells.
template <int RO, int CO, int HALO>
constexpr int mg_tile_work()   // warps' rounds of a block over its sweeps
{
    int n = 0;
    for (int h = HALO - 1; h >= HALO - 6; --h) n += ((RO + 2 * h) * (CO + 2 * h) + 31) / 32;
    return n;
}

template <int RO, int CO> constexpr int mg_tile_nt = RO * CO >= 256 ? 512 : 256;   // threads

template <typename T, int RO, int CO, bool DOWN, bool ZERO>
__global__ void __launch_bounds__(mg_tile_nt<RO, CO>) k_mg_tile(MgLev<T> L, MgLev<T> C, const T* __restrict__ in,
                                                 const T* __restrict__ V, const T* __restrict__ rhs,
                                                 const T* __restrict__ rr, T* __restrict__ out, MgDown<T> d, T omega)
{
    constexpr int H = DOWN ? 7 : 6;                  // halo: the sweeps, and the residual's
    constexpr int NT = mg_tile_nt<RO, CO>;
    constexpr int RR = RO + 2 * H, CC = CO + 2 * H;
    __shared__ T s[2][RR * CC];
    const int b = blockIdx.z, tid = threadIdx.x;
    const int i0 = (int)blockIdx.y * RO - H, j0 = (int)blockIdx.x * CO - H;
    const long long fs = (long long)L.n0 * L.n1;
    rr += b * fs;
    rhs += b * fs;
    auto inside = [&](int i, int j) { return i >= 0 && i < L.n0 && j >= 0 && j < L.n1; };
    for (int e = tid; e < RR * CC; e += NT) {
        const int r = e / CC, c = e % CC, i = i0 + r, j = j0 + c;
        T x = T(0);
        if (inside(i, j)) {
            const long long o = (long long)i * L.n1 + j;
            if constexpr (DOWN && ZERO) {
                x = mg_first(L, rr[o], b, o);
            } else {
                x = in[b * fs + o];
                if constexpr (!DOWN) {
                    const long long fc = (long long)C.n0 * C.n1;
                    x = mg_prolong_pt(V + b * fc, C.n0, C.n1, i, j, L.mp[o], x);
                }
            }
        }
        s[0][e] = x;
        s[1][e] = T(0);   // cells outside the grid stay 0 in both
    }
    __syncthreads();
    constexpr int FIRST = DOWN && ZERO ? 1 : 0;      // sweeps already done
#pragma unroll
    for (int k = FIRST; k < 6; ++k) {
        const T* const src = s[(k - FIRST) & 1];
        T* const dst = s[(k - FIRST + 1) & 1];
        const int m = k + 1, W = CC - 2 * m, N = (RR - 2 * m) * W;
        for (int e = tid; e < N; e += NT) {
            const int r = e / W + m, c = e % W + m, i = i0 + r, j = j0 + c;
            if (inside(i, j)) {
                const T* q = src + r * CC + c;
                dst[r * CC + c] = mg_update(L, q[0], q[CC], q[-CC], q[1], q[-1], rr[(long long)i * L.n1 + j], b, i, j,
                                            omega);
            }
        }
        __syncthreads();
    }
    const T* const res = s[(6 - FIRST) & 1];
    for (int e = tid; e < RO * CO; e += NT) {
        const int r = e / CO + H, c = e % CO + H, i = i0 + r, j = j0 + c;
        if (inside(i, j)) out[b * fs + (long long)i * L.n1 + j] = res[r * CC + c];
    }
    if constexpr (DOWN) {
        const T lam = L.lam[b];
        for (int e = tid; e < RO * CO / 4; e += NT) {
            const int R = e / (CO / 2), Cc = e % (CO / 2);
            if (!inside(i0 + H + 2 * R, j0 + H + 2 * Cc)) continue;
            T x[2][2];
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    const int r = H + 2 * R + u, c = H + 2 * Cc + v, i = i0 + r, j = j0 + c;
                    const T* q = res + r * CC + c;
                    x[u][v] = mg_resid(L, q[0], q[CC], q[-CC], q[1], q[-1], rhs[(long long)i * L.n1 + j], lam, i, j);
                }
            const int I = (int)blockIdx.y * (RO / 2) + R, J = (int)blockIdx.x * (CO / 2) + Cc;
            const long long o = (long long)I * C.n1 + J;
            mg_put_rhs(C, d, (x[0][0] + x[1][0] + x[0][1] + x[1][1]) * C.mr[o], b, o);
        }
    }
}

// bottom: f[b][idx[m]] = sum_l rhs[b][idx[l]] inv[b][l][m]  (341-346)
template <typename T>
__global__ void k_mg_bottom(int nb, long long fs, const int32_t* __restrict__ idx, const T* __restrict__ inv,
                            const T* __restrict__ rhs, T* __restrict__ f)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y;
    if (m >= nb) return;
    const T* R = rhs + b * fs;
    const T* P = inv + (long long)b * nb * nb;
    T s = T(0);
    for (int l = 0; l < nb; ++l) s += R[idx[l]] * P[(long long)l * nb + m];
    f[b * fs + idx[m]] = s;
}

// ---------------------------------------------------------------------------
// Coarse levels in one block (or one cluster of blocks) per system. Below a few thousand cells a level's
// sweep is shorter than a kernel launch, and the bottom smoothing alone is
// 6 x niter_bottom sweeps per V-cycle; this kernel runs everything from level
// l0 down (the V-cycle, or the full-multigrid start) with the block's threads
// striding over the level and a barrier between phases. The solution,
// right-hand side and scratch of every level from l0 down live in shared
// memory (level l0's come in from, and its solution goes back to, global
// memory); the coefficients are read-only global tables; the arithmetic is
// the per-point functions above.
// ---------------------------------------------------------------------------
constexpr int MG_MAXLEV = 16;
constexpr long long MG_TILE_MAX = 65536;

template <typename T>
struct MgCoarseArgs {
    int l0, nlev, niter_bottom, nb, fmg, zero;   // zero: the V-cycle starts from f = 0
    T omega;
    MgLev<T> L[MG_MAXLEV];
    int soff[MG_MAXLEV];        // shared-memory offset of level l: f, rhs, scratch, scaled rhs (n0 n1 each)
    T* f0;                      // level l0 solution (system-0 base): in (V-cycle) and out
    const T* rhs0;              // level l0 right-hand side (system-0 base)
    const int32_t* bot_idx;
    const T* bot_inv;
    const T* bot_sm;            // bottom smoothing as matrices, or nullptr
};

template <typename T>
struct MgcLevel {
    T *f, *rhs, *tmp, *rr;   // rr: what the sweeps read (mg_scaled_rhs)
    int n;
};

template <typename T>
__device__ __forceinline__ MgcLevel<T> mgc_level(const MgCoarseArgs<T>& A, T* sm, int l)
{
    MgcLevel<T> v;
    v.n = A.L[l].n0 * A.L[l].n1;
    v.f = sm + A.soff[l];
    v.rhs = v.f + v.n;
    v.tmp = v.rhs + v.n;
    v.rr = mg_scaled<T> ? v.tmp + v.n : v.rhs;
    return v;
}

// The threads of one system's coarse kernel: one block, or a cluster of blocks (CL)
// that each hold every level in their own shared memory, take a share of the cells of
// a phase, and store a result into all of the copies. A phase then reads locally and
// ends at a cluster barrier instead of a block barrier.
template <typename T, bool CL>
struct McTeam {
    int rank, nb;   // block of the cluster, blocks
    __device__ __forceinline__ int first() const { return rank * (int)blockDim.x + (int)threadIdx.x; }
    __device__ __forceinline__ int step() const { return nb * (int)blockDim.x; }
    __device__ __forceinline__ void put(T* p, T v) const
    {
        if constexpr (CL) {
            const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
            for (int r = 0; r < nb; ++r) {
                uint32_t q;
                asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(q) : "r"(a), "r"(r));
                if constexpr (sizeof(T) == 8)
                    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(q), "d"(v) : "memory");
                else
                    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(q), "f"(v) : "memory");
            }
        } else {
            *p = v;
        }
    }
    __device__ __forceinline__ void sync() const
    {
        if constexpr (CL) {
            asm volatile("barrier.cluster.arrive.release;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        } else {
            __syncthreads();
        }
    }
};

template <typename T, bool CL>
__device__ void mgc_smooth(const MgCoarseArgs<T>& A, const McTeam<T, CL>& tm, T* sm, int l, int b, int times)
{
    const MgLev<T>& L = A.L[l];
    const MgcLevel<T> v = mgc_level(A, sm, l);
    for (int t = 0; t < times; ++t)
        for (int s = 0; s < 6; ++s) {
            const T* src = (s % 2 == 0) ? v.f : v.tmp;
            T* dst = (s % 2 == 0) ? v.tmp : v.f;
            for (int o = tm.first(); o < v.n; o += tm.step()) {
                const int i = o / L.n1, j = o - i * L.n1;
                tm.put(dst + o, mg_sweep_pt(L, src, v.rr[o], b, i, j, A.omega));
            }
            tm.sync();
        }
}

template <typename T> __device__ __forceinline__ T mg_warp_sum(T x)
{
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) x += __shfl_xor_sync(0xffffffffu, x, k);
    return x;
}

template <typename T, bool CL>
__device__ void mgc_bottom(const MgCoarseArgs<T>& A, const McTeam<T, CL>& tm, T* sm, int b)
{
    const int l = A.nlev - 1;
    const MgcLevel<T> v = mgc_level(A, sm, l);
    if (A.niter_bottom > 0 && A.bot_sm != nullptr) {
        // f = N rhs (+ M f when the grid has one level; below it f is zero here), a warp
        // a cell: the rows of N and M are contiguous
        const long long n2 = (long long)v.n * v.n;
        const T* Nm = A.bot_sm + (long long)b * 2 * n2;
        const T* Mm = Nm + n2;
        const int lane = threadIdx.x & 31;
        for (int m = tm.first() >> 5; m < v.n; m += tm.step() >> 5) {
            T s = T(0);
            for (int k = lane; k < v.n; k += 32) s += __ldg(Nm + (long long)m * v.n + k) * v.rhs[k];
            if (A.nlev == 1)
                for (int k = lane; k < v.n; k += 32) s += __ldg(Mm + (long long)m * v.n + k) * v.f[k];
            s = mg_warp_sum(s);
            if (lane == 0) tm.put(v.tmp + m, s);
        }
        tm.sync();
        for (int m = threadIdx.x; m < v.n; m += blockDim.x) v.f[m] = v.tmp[m];   // every block its own copy
        tm.sync();
        return;
    }
    if (A.niter_bottom > 0) {
        mgc_smooth(A, tm, sm, l, b, A.niter_bottom);
        return;
    }
    for (int o = threadIdx.x; o < v.n; o += blockDim.x) v.f[o] = T(0);
    tm.sync();
    const T* P = A.bot_inv + (long long)b * A.nb * A.nb;
    for (int m = tm.first(); m < A.nb; m += tm.step()) {
        T s = T(0);
        for (int k = 0; k < A.nb; ++k) s += v.rhs[__ldg(A.bot_idx + k)] * __ldg(P + (long long)k * A.nb + m);
        tm.put(v.f + __ldg(A.bot_idx + m), s);
    }
    tm.sync();
}

// rhs of level lc from a fine-level field (shared memory)
template <typename T, bool CL>
__device__ void mgc_restrict(const MgCoarseArgs<T>& A, const McTeam<T, CL>& tm, T* sm, const T* fine, int lc, int b)
{
    const MgLev<T>& C = A.L[lc];
    const MgcLevel<T> v = mgc_level(A, sm, lc);
    for (int o = tm.first(); o < v.n; o += tm.step()) {
        const int I = o / C.n1, J = o - I * C.n1;
        const T x = mg_restrict_pt(fine, C.n1, I, J, C.mr);
        tm.put(v.rhs + o, x);
        if constexpr (mg_scaled<T>) tm.put(v.rr + o, mg_scaled_rhs(C, x, b, o));
    }
}

template <typename T, bool CL>
__device__ void mgc_prolong(const MgCoarseArgs<T>& A, const McTeam<T, CL>& tm, T* sm, int l, bool add)
{
    const MgLev<T>& Fl = A.L[l];
    const MgLev<T>& C = A.L[l + 1];
    const MgcLevel<T> vf = mgc_level(A, sm, l), vc = mgc_level(A, sm, l + 1);
    for (int o = tm.first(); o < vf.n; o += tm.step()) {
        const int i = o / Fl.n1, j = o - i * Fl.n1;
        tm.put(vf.f + o, mg_prolong_pt(vc.f, C.n0, C.n1, i, j, Fl.mp[o], add ? vf.f[o] : T(0)));
    }
    tm.sync();
}

template <typename T, bool CL>
__device__ void mgc_vcycle(const MgCoarseArgs<T>& A, const McTeam<T, CL>& tm, T* sm, int l0, int b)
{
    const int last = A.nlev - 1;
    for (int l = l0; l < last; ++l) {
        mgc_smooth(A, tm, sm, l, b, 1);
        const MgLev<T>& L = A.L[l];
        const MgcLevel<T> v = mgc_level(A, sm, l);
        for (int o = tm.first(); o < v.n; o += tm.step()) {
            const int i = o / L.n1, j = o - i * L.n1;
            tm.put(v.tmp + o, mg_residual_pt(L, v.f, v.rhs[o], L.lam[b], i, j));
        }
        tm.sync();
        mgc_restrict(A, tm, sm, v.tmp, l + 1, b);
        const MgcLevel<T> c = mgc_level(A, sm, l + 1);
        for (int o = threadIdx.x; o < c.n; o += blockDim.x) c.f[o] = T(0);
        tm.sync();
    }
    mgc_bottom(A, tm, sm, b);
    for (int l = last - 1; l >= l0; --l) {
        mgc_prolong(A, tm, sm, l, true);
        mgc_smooth(A, tm, sm, l, b, 1);
    }
}

template <typename T, bool CL>
__global__ void __launch_bounds__(1024) k_mg_coarse(MgCoarseArgs<T> A)
{
    extern __shared__ __align__(16) unsigned char mg_smem[];
    T* sm = reinterpret_cast<T*>(mg_smem);
    McTeam<T, CL> tm;
    tm.rank = 0;
    tm.nb = 1;
    if constexpr (CL) {
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(tm.rank));
        asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(tm.nb));
    }
    const int b = blockIdx.x / tm.nb;
    const MgcLevel<T> v0 = mgc_level(A, sm, A.l0);
    const long long g0 = (long long)b * v0.n;
    // (every block reads the whole level into its copy; the barrier also says that
    // every block of the cluster has started, before the first store into it)
    for (int o = threadIdx.x; o < v0.n; o += blockDim.x) {
        v0.rhs[o] = A.rhs0[g0 + o];
        if constexpr (mg_scaled<T>) v0.rr[o] = mg_scaled_rhs(A.L[A.l0], v0.rhs[o], b, o);
        if (!A.fmg) v0.f[o] = A.zero ? T(0) : A.f0[g0 + o];
    }
    tm.sync();
    if (!A.fmg) {
        mgc_vcycle(A, tm, sm, A.l0, b);
    } else {
        const int last = A.nlev - 1;
        for (int l = A.l0 + 1; l <= last; ++l) {
            mgc_restrict(A, tm, sm, mgc_level(A, sm, l - 1).rhs, l, b);
            tm.sync();
        }
        const MgcLevel<T> vb = mgc_level(A, sm, last);
        for (int o = threadIdx.x; o < vb.n; o += blockDim.x) vb.f[o] = T(0);
        tm.sync();
        mgc_bottom(A, tm, sm, b);
        for (int l = last - 1; l >= A.l0; --l) {
            mgc_prolong(A, tm, sm, l, false);
            mgc_vcycle(A, tm, sm, l, b);
        }
    }
    // (the last phase's barrier: no block stores into another any more)
    for (int o = tm.first(); o < v0.n; o += tm.step()) A.f0[g0 + o] = v0.f[o];
}

template <typename T>
__global__ void k_mg_zero(long long n, T* __restrict__ x)
{
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) x[k] = T(0);
}

}  // namespace vd

namespace {

constexpr int MG_COARSE_CL = 256;   // threads of a clustered block (512: 6.26 ms a solve for 6.16)

template <typename T>
struct MgRun {
    const vd_mg_plan* p;
    T* ws;
    cudaStream_t st;

    vd::MgLev<T> lev(int l) const
    {
        const vd_mg_plan::DLev& D = p->dl[l];
        vd::MgLev<T> L;
        L.n0 = p->lv[l].n0;
        L.n1 = p->lv[l].n1;
        L.mask = (const T*)D.mask;
        L.cu = (const T*)D.cu;
        L.cv = (const T*)D.cv;
        L.factor = (const T*)D.factor;
        L.g = (const T*)D.g;
        L.mr = (const T*)D.mr;
        L.mp = (const T*)D.mp;
        L.lam = (const T*)p->lam;
        return L;
    }
    T* buf(int l, int which) const { return ws + p->ws_off[4 * l + which]; }
    // what the sweeps of level l read for the right-hand side rhs
    const T* scaled(int l, const T* rhs) const { return vd::mg_scaled<T> ? buf(l, 3) : rhs; }
    vd::MgDown<T> down(int l) const
    {
        vd::MgDown<T> d;
        d.rhs = buf(l, 1);
        d.rr = vd::mg_scaled<T> ? buf(l, 3) : nullptr;
        d.first = (l < p->lc && !tiled(l)) ? buf(l, 2) : nullptr;
        return d;
    }
    long long nel(int l) const { return (long long)p->nsys * p->lv[l].n0 * p->lv[l].n1; }
    dim3 grid(int n0, int n1) const { return dim3((unsigned)((n1 + 127) / 128), (unsigned)n0, (unsigned)p->nsys); }

    // Levels whose six sweeps run as one tile kernel: those of at most MG_TILE_MAX cells
    // (all systems), where a sweep is shorter than its launch; above, the halo's extra
    // FP64 work costs more than the launches. A 1024 x 768 float64 solve with the line at
    // 0, 4096, 16384, 65536 and 262144 cells: 6.61, 6.40, 6.25, 6.16 and 6.45 ms.
    bool tiled(int l) const { return l < p->nlev - 1 && l < p->lc && nel(l) <= vd::MG_TILE_MAX; }

    int zero(T* x, long long n) const
    {
        vd::k_mg_zero<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, x);
        VD_LAUNCH_CHECK();
        return VD_OK;
    }
    // `times` smooths of 6 damped sweeps, ping-pong through the level's tmp buffer;
    // started: the first sweep is in tmp already (from f = 0)
    int smooth(int l, T* f, const T* rhs, int times, bool started = false) const
    {
        const vd::MgLev<T> L = lev(l);
        T* tmp = buf(l, 2);
        const T* rr = scaled(l, rhs);
        const dim3 g = grid(L.n0, L.n1);
        for (int s = started ? 1 : 0; s < 6 * times; ++s) {
            const T* src = (s % 2 == 0) ? f : tmp;
            T* dst = (s % 2 == 0) ? tmp : f;
            vd::k_mg_sweep<T><<<g, 128, 0, st>>>(L, src, rr, dst, T(p->omega));
            VD_LAUNCH_CHECK();
        }
        return VD_OK;
    }
    template <int RO, int CO>
    int tile(int l, bool dn, bool started, const T* in, const T* V, const T* rhs, T* out) const
    {
        const vd::MgLev<T> L = lev(l), C = lev(l + 1);
        const dim3 g((unsigned)((L.n1 + CO - 1) / CO), (unsigned)((L.n0 + RO - 1) / RO), (unsigned)p->nsys);
        const int nt = vd::mg_tile_nt<RO, CO>;
        const T w = T(p->omega);
        const T* rr = scaled(l, rhs);
        const vd::MgDown<T> d = down(l + 1);
        if (!dn) vd::k_mg_tile<T, RO, CO, false, false><<<g, nt, 0, st>>>(L, C, in, V, rhs, rr, out, d, w);
        else if (started) vd::k_mg_tile<T, RO, CO, true, true><<<g, nt, 0, st>>>(L, C, in, V, rhs, rr, out, d, w);
        else vd::k_mg_tile<T, RO, CO, true, false><<<g, nt, 0, st>>>(L, C, in, V, rhs, rr, out, d, w);
        VD_LAUNCH_CHECK();
        return VD_OK;
    }
    // the tile that keeps the busiest SM shortest: work of a block x blocks an SM
    int tile_any(int l, bool dn, bool started, const T* in, const T* V, const T* rhs, T* out) const
    {
        auto cost = [&](int ro, int co, int work) {
            const long long nb = (long long)((p->lv[l].n0 + ro - 1) / ro) * ((p->lv[l].n1 + co - 1) / co) * p->nsys;
            return ((nb + 151) / 152) * work;
        };
        const long long c0 = cost(8, 8, vd::mg_tile_work<8, 8, 6>()), c1 = cost(8, 16, vd::mg_tile_work<8, 16, 6>()),
                        c2 = cost(16, 16, vd::mg_tile_work<16, 16, 6>()),
                        c3 = cost(16, 32, vd::mg_tile_work<16, 32, 6>());
        const long long m = std::min(std::min(c0, c1), std::min(c2, c3));
        if (c3 == m) return tile<16, 32>(l, dn, started, in, V, rhs, out);
        if (c2 == m) return tile<16, 16>(l, dn, started, in, V, rhs, out);
        if (c1 == m) return tile<8, 16>(l, dn, started, in, V, rhs, out);
        return tile<8, 8>(l, dn, started, in, V, rhs, out);
    }
    // started: f starts from zero (and its first sweep is in tmp)
    int bottom(T* f, const T* rhs, bool started) const
    {
        const int l = p->nlev - 1;
        if (p->niter_bottom <= 0) {
            const long long fs = (long long)p->lv[l].n0 * p->lv[l].n1;
            int rc = zero(f, nel(l));
            if (rc) return rc;
            if (p->nb > 0) {
                vd::k_mg_bottom<T><<<dim3((unsigned)((p->nb + 127) / 128), (unsigned)p->nsys), 128, 0, st>>>(
                    p->nb, fs, p->bot_idx, (const T*)p->bot_inv, rhs, f);
                VD_LAUNCH_CHECK();
            }
            return VD_OK;
        }
        return smooth(l, f, rhs, p->niter_bottom, started);
    }
    // levels >= l0 in one block per system (p->lc <= l0): a V-cycle on (f, rhs)
    // at l0 (from f = 0 where zero_f), or (fmg) the full-multigrid start from the
    // restricted rhs at l0
    int coarse(T* f, const T* rhs, int l0, bool fmg, bool zero_f) const
    {
        vd::MgCoarseArgs<T> A;
        A.l0 = l0; A.nlev = p->nlev; A.niter_bottom = p->niter_bottom; A.nb = p->nb; A.fmg = fmg ? 1 : 0;
        A.zero = zero_f ? 1 : 0;
        A.omega = T(p->omega);
        int off = 0;
        for (int l = 0; l < p->nlev; ++l) {
            A.L[l] = lev(l);
            A.soff[l] = off;
            if (l >= l0) off += (vd::mg_scaled<T> ? 4 : 3) * p->lv[l].n0 * p->lv[l].n1;
        }
        A.f0 = f;
        A.rhs0 = rhs;
        A.bot_idx = p->bot_idx;
        A.bot_inv = (const T*)p->bot_inv;
        A.bot_sm = (const T*)p->bot_sm;
        const size_t smem = (size_t)off * sizeof(T);
        // blocks a system: one in float32 (a phase is shorter than a cluster barrier);
        // in float64, where one SM's FP64 rate is the bound, a cluster of up to 8 while
        // the systems' clusters fit the GPU at once (15 of 8). Levels of 768 and 192 cells:
        // 43.5 us a V-cycle with one block, 31.8 with 8, now bound by the barriers. What
        // gains is the bottom solve, by its cells squared as a matrix or an exact inverse;
        // each level above loses 10 to 14 us of sweeps to the barriers. Solves with one
        // block / 8, by the cells of these levels:
        //   bottom sweeps as a matrix (up to 512 cells): 60 332 / 256 us, 384 3031 / 1901,
        //   480 + 120 1562 / 1515, 384 + 96 1381 / 1502, 1024 + 256 + 64 1550 / 1697
        //   bottom sweeps one by one: 672 5433 / 6248, 896 6606 / 6443
        //   exact bottom: 288 3620 / 3626, 384 2574 / 2367, 768 + 192 1928 / 1996
        const int above = p->nlev - 1 - l0, cells = p->lv.back().n0 * p->lv.back().n1;
        const bool wide = p->niter_bottom <= 0 ? above == 0 && cells >= 320
                          : p->bot_sm          ? cells >= 32 + 80 * above
                                               : cells >= 864;
        int nc = 1;
        if (vd::mg_scaled<T> && wide)
            while (nc < 8 && (long long)p->nsys * 2 * nc <= 120) nc *= 2;
        if (nc == 1) {
            vd::k_mg_coarse<T, false><<<(unsigned)p->nsys, 1024, smem, st>>>(A);
        } else if constexpr (vd::mg_scaled<T>) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3((unsigned)(p->nsys * nc));
            cfg.blockDim = dim3(MG_COARSE_CL);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = st;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = (unsigned)nc;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            VD_CUDA_TRY(cudaLaunchKernelEx(&cfg, vd::k_mg_coarse<T, true>, A));
        }
        VD_LAUNCH_CHECK();
        return VD_OK;
    }
    // one V-cycle on (f, rhs) at level l. started: from f = 0, with the first sweep
    // in tmp where the level's sweeps are single launches
    int vcycle(T* f, const T* rhs, int l, bool started) const
    {
        if (l >= p->lc) return coarse(f, rhs, l, false, started);
        if (l == p->nlev - 1) return bottom(f, rhs, started);
        int rc;
        const vd::MgLev<T> L = lev(l), C = lev(l + 1);
        T* rcz = buf(l + 1, 1);
        T* ec = buf(l + 1, 0);
        if (tiled(l)) {
            if ((rc = tile_any(l, true, started, f, nullptr, rhs, buf(l, 2)))) return rc;
            if ((rc = vcycle(ec, rcz, l + 1, true))) return rc;
            return tile_any(l, false, false, buf(l, 2), ec, rhs, f);
        }
        if ((rc = smooth(l, f, rhs, 1, started))) return rc;
        vd::k_mg_resid_restrict<T><<<grid(C.n0, C.n1), 128, 0, st>>>(L, C, f, rhs, down(l + 1));
        VD_LAUNCH_CHECK();
        if ((rc = vcycle(ec, rcz, l + 1, true))) return rc;
        vd::k_mg_prolong<T><<<grid(C.n0, C.n1), 128, 0, st>>>(L, C.n0, C.n1, ec, f, 1);
        VD_LAUNCH_CHECK();
        return smooth(l, f, rhs, 1);
    }
    // FMG_Helmholtz (helmholtz_multigrid.py:380-419)
    int solve(const T* rhs, T* out) const
    {
        const int n = p->nlev;
        int rc;
        if (vd::mg_scaled<T>) {
            vd::k_mg_scale<T><<<grid(p->n0, p->n1), 128, 0, st>>>(lev(0), rhs, buf(0, 3));
            VD_LAUNCH_CHECK();
        }
        if (n == 1) {
            if ((rc = zero(out, nel(0)))) return rc;
            if ((rc = bottom(out, rhs, false))) return rc;
        } else {
            // right-hand sides down to the coarse kernel's first level or the bottom,
            // the start there, and a V-cycle on every level up
            const int lb = p->lc < n ? p->lc : n - 1;
            for (int i = 1; i <= lb; ++i) {
                vd::k_mg_restrict<T><<<grid(p->lv[i].n0, p->lv[i].n1), 128, 0, st>>>(
                    lev(i), (i == 1) ? rhs : buf(i - 1, 1), down(i));
                VD_LAUNCH_CHECK();
            }
            T* fb = lb == 0 ? out : buf(lb, 0);
            const T* rb = lb == 0 ? rhs : buf(lb, 1);
            if (p->lc < n) {
                if ((rc = coarse(fb, rb, lb, true, false))) return rc;
            } else {
                if ((rc = zero(fb, nel(lb)))) return rc;
                if ((rc = bottom(fb, rb, false))) return rc;
            }
            for (int L = lb - 1; L >= 0; --L) {
                T* fL = (L == 0) ? out : buf(L, 0);
                const T* rL = (L == 0) ? rhs : buf(L, 1);
                vd::k_mg_prolong<T><<<grid(p->lv[L + 1].n0, p->lv[L + 1].n1), 128, 0, st>>>(
                    lev(L), p->lv[L + 1].n0, p->lv[L + 1].n1, buf(L + 1, 0), fL, 0);
                VD_LAUNCH_CHECK();
                if ((rc = vcycle(fL, rL, L, false))) return rc;
            }
        }
        for (int it = 0; it < p->max_ite; ++it)
            if ((rc = vcycle(out, rhs, 0, false))) return rc;
        return VD_OK;
    }
};

// ---- hierarchy construction (host, float64; helmholtz_multigrid.py:248-293) ----
std::vector<double> restrict_h(const std::vector<double>& v, int n0, int n1, const std::vector<double>* div, double d)
{
    const int n0c = n0 / 2, n1c = n1 / 2;
    std::vector<double> o((size_t)n0c * n1c);
    for (int I = 0; I < n0c; ++I)
        for (int J = 0; J < n1c; ++J) {
            const double s = v[(size_t)(2 * I) * n1 + 2 * J] + v[(size_t)(2 * I + 1) * n1 + 2 * J] +
                             v[(size_t)(2 * I) * n1 + 2 * J + 1] + v[(size_t)(2 * I + 1) * n1 + 2 * J + 1];
            o[(size_t)I * n1c + J] = s / (div ? (*div)[(size_t)I * n1c + J] : d);
        }
    return o;
}

std::vector<double> prolong_h(const std::vector<double>& v, int n0c, int n1c)
{
    const int n0 = 2 * n0c, n1 = 2 * n1c;
    std::vector<double> o((size_t)n0 * n1);
    for (int i = 0; i < n0; ++i)
        for (int j = 0; j < n1; ++j) {
            const int I = i >> 1, J = j >> 1, di = (i & 1) ? 1 : -1, dj = (j & 1) ? 1 : -1;
            o[(size_t)i * n1 + j] = 9 * at(v, n0c, n1c, I, J) + 3 * (at(v, n0c, n1c, I, J + dj) +
                                    at(v, n0c, n1c, I + di, J)) + at(v, n0c, n1c, I + di, J + dj);
        }
    return o;
}

void uv_masks(const std::vector<double>& m, int n0, int n1, std::vector<double>& mu, std::vector<double>& mv)
{
    mu.assign((size_t)(n0 + 1) * n1, 0.0);
    mv.assign((size_t)n0 * (n1 + 1), 0.0);
    for (int i = 0; i <= n0; ++i)
        for (int j = 0; j < n1; ++j) mu[(size_t)i * n1 + j] = (at(m, n0, n1, i - 1, j) + at(m, n0, n1, i, j)) > 1.5;
    for (int i = 0; i < n0; ++i)
        for (int j = 0; j <= n1; ++j)
            mv[(size_t)i * (n1 + 1) + j] = (at(m, n0, n1, i, j - 1) + at(m, n0, n1, i, j)) > 1.5;
}

// H f on one level (helmholtz_multigrid.py:53-62), for the bottom matrix
void helm_apply(const HLevel& L, double lam, const std::vector<double>& f, std::vector<double>& out)
{
    const int n0 = L.n0, n1 = L.n1;
    out.assign((size_t)n0 * n1, 0.0);
    for (int i = 0; i < n0; ++i)
        for (int j = 0; j < n1; ++j) {
            const double fc = f[(size_t)i * n1 + j];
            const double hx = L.cu[(size_t)(i + 1) * n1 + j] * (at(f, n0, n1, i + 1, j) - fc) -
                              L.cu[(size_t)i * n1 + j] * (fc - at(f, n0, n1, i - 1, j));
            const double hy = L.cv[(size_t)i * (n1 + 1) + j + 1] * (at(f, n0, n1, i, j + 1) - fc) -
                              L.cv[(size_t)i * (n1 + 1) + j] * (fc - at(f, n0, n1, i, j - 1));
            out[(size_t)i * n1 + j] = (hx / (L.d0 * L.d0) + hy / (L.d1 * L.d1) - lam * fc) * L.mask[(size_t)i * n1 + j];
        }
}

// The bottom level's K damped Jacobi sweeps (the device formula, in float64)
// as f_K = M f_0 + N rhs, by sweeping unit vectors; appended to `out` as
// N then M (zeros when !with_m), each [output m][input k].
void bottom_sweep_matrices(const HLevel& L, const double* factor, double omega, int K, bool with_m,
                           std::vector<double>& out)
{
    const int n0 = L.n0, n1 = L.n1, n = n0 * n1;
    const double dxm2 = 1.0 / (L.d0 * L.d0), dym2 = 1.0 / (L.d1 * L.d1);
    std::vector<double> f(n), g(n), r(n);
    auto sweep = [&](const std::vector<double>& src, std::vector<double>& dst) {
        for (int i = 0; i < n0; ++i)
            for (int j = 0; j < n1; ++j) {
                const size_t o = (size_t)i * n1 + j;
                const double sx = L.cu[(size_t)(i + 1) * n1 + j] * at(src, n0, n1, i + 1, j) +
                                  L.cu[o] * at(src, n0, n1, i - 1, j);
                const double sy = L.cv[(size_t)i * (n1 + 1) + j + 1] * at(src, n0, n1, i, j + 1) +
                                  L.cv[(size_t)i * (n1 + 1) + j] * at(src, n0, n1, i, j - 1);
                const double s = dxm2 * sx + dym2 * sy;
                dst[o] = omega * factor[o] * (s - r[o]) + (1.0 - omega) * src[o];
            }
    };
    const size_t base = out.size();
    out.resize(base + 2 * (size_t)n * n, 0.0);
    for (int pass = 0; pass < (with_m ? 2 : 1); ++pass)
        for (int k = 0; k < n; ++k) {
            std::fill(f.begin(), f.end(), 0.0);
            std::fill(r.begin(), r.end(), 0.0);
            (pass == 0 ? r : f)[k] = 1.0;
            for (int t = 0; t < K; ++t) {
                sweep(f, g);
                f.swap(g);
            }
            double* dst = out.data() + base + (size_t)pass * n * n + k;
            for (int m = 0; m < n; ++m) dst[(size_t)m * n] = f[m];
        }
}

struct Blob {
    std::vector<unsigned char> b;
    size_t add(const void* p, size_t n)
    {
        const size_t off = (b.size() + 255) & ~size_t(255);
        b.resize(off + n + 1);
        if (n) std::memcpy(b.data() + off, p, n);
        return off;
    }
    template <typename T>
    size_t addv(const std::vector<double>& v)
    {
        std::vector<T> t(v.begin(), v.end());
        return add(t.data(), t.size() * sizeof(T));
    }
};

template <typename T>
int mg_upload(vd_mg_plan* p, const std::vector<int32_t>& idx, const std::vector<double>& inv,
              const std::vector<double>& bsm)
{
    Blob bl;
    struct Off { size_t mask, cu, cv, factor, g, mr, mp; };
    std::vector<Off> off(p->nlev);
    for (int l = 0; l < p->nlev; ++l) {
        const HLevel& L = p->lv[l];
        off[l].mask = bl.addv<T>(L.mask);
        const double dxm2 = 1.0 / (L.d0 * L.d0), dym2 = 1.0 / (L.d1 * L.d1);
        std::vector<double> cus(L.cu), cvs(L.cv), fw(L.factor);
        for (double& v : cus) v *= dxm2;
        for (double& v : cvs) v *= dym2;
        for (double& v : fw) v *= p->omega;
        off[l].cu = bl.addv<T>(cus);
        off[l].cv = bl.addv<T>(cvs);
        off[l].factor = bl.addv<T>(fw);
        // restriction and prolongation: mask / divisor
        std::vector<double> mr(L.divr), mp(L.divp);
        for (size_t k = 0; k < mr.size(); ++k) mr[k] = L.mask[k] / mr[k];
        for (size_t k = 0; k < mp.size(); ++k) mp[k] = L.mask[k] / mp[k];
        off[l].mr = mr.empty() ? 0 : bl.addv<T>(mr);
        off[l].mp = mp.empty() ? 0 : bl.addv<T>(mp);
    }
    const size_t o_lam = bl.addv<T>(p->lambda);
    const size_t o_idx = bl.add(idx.data(), idx.size() * sizeof(int32_t));
    const size_t o_inv = bl.addv<T>(inv);
    const size_t o_bsm = bl.addv<T>(bsm);
    size_t total = bl.b.size();
    for (int l = 0; l < p->nlev; ++l) {
        off[l].g = total = (total + 255) & ~size_t(255);
        if (vd::mg_scaled<T>) total += sizeof(T) * 4 * (size_t)p->nsys * p->lv[l].n0 * p->lv[l].n1;
    }
    VD_CUDA_TRY(cudaMalloc(&p->dev, total));
    VD_CUDA_TRY(cudaMemcpy(p->dev, bl.b.data(), bl.b.size(), cudaMemcpyHostToDevice));
    unsigned char* b = (unsigned char*)p->dev;
    p->dl.resize(p->nlev);
    for (int l = 0; l < p->nlev; ++l) {
        p->dl[l].mask = b + off[l].mask;
        p->dl[l].cu = b + off[l].cu;
        p->dl[l].cv = b + off[l].cv;
        p->dl[l].factor = b + off[l].factor;
        p->dl[l].g = vd::mg_scaled<T> ? b + off[l].g : nullptr;
        p->dl[l].mr = p->lv[l].divr.empty() ? nullptr : b + off[l].mr;
        p->dl[l].mp = p->lv[l].divp.empty() ? nullptr : b + off[l].mp;
    }
    p->lam = b + o_lam;
    p->bot_idx = (const int32_t*)(b + o_idx);
    p->bot_inv = b + o_inv;
    p->bot_sm = bsm.empty() ? nullptr : b + o_bsm;
    if (vd::mg_scaled<T>) {
        for (int l = 0; l < p->nlev; ++l) {
            const HLevel& L = p->lv[l];
            vd::k_mg_coeffs<T><<<dim3((unsigned)((L.n1 + 127) / 128), (unsigned)L.n0, (unsigned)p->nsys), 128>>>(
                L.n0, L.n1, (const T*)p->dl[l].cu, (const T*)p->dl[l].cv, (const T*)p->dl[l].factor, (T*)(b + off[l].g));
            VD_LAUNCH_CHECK();
        }
        VD_CUDA_TRY(cudaStreamSynchronize(0));
    }
    return VD_OK;
}

}  // namespace

extern "C" vd_status vd_mg_plan_create(vd_mg_plan** out, const vd_mg_desc* d)
{
    if (!out || !d) return VD_ERR_ARG;
    *out = nullptr;
    if (d->n0 < 1 || d->n1 < 1 || d->nsys < 1 || !d->lambda_host || !d->coef_u_host || !d->coef_v_host ||
        !(d->d0 > 0) || !(d->d1 > 0) || d->max_ite < 0 || (d->dtype != VD_F32 && d->dtype != VD_F64))
        return VD_ERR_ARG;
    const int nlev = d->n_levels > 0 ? d->n_levels : std::min(mg_nlevels(d->n0), mg_nlevels(d->n1));
    const int N = 1 << (nlev - 1);
    if (d->n0 % N || d->n1 % N) return VD_ERR_ARG;
    vd_mg_plan* p = new (std::nothrow) vd_mg_plan();
    if (!p) return VD_ERR_ARG;
    p->n0 = d->n0; p->n1 = d->n1; p->nsys = d->nsys; p->dtype = d->dtype; p->nlev = nlev;
    p->max_ite = d->max_ite; p->niter_bottom = d->niter_bottom;
    p->lambda.assign(d->lambda_host, d->lambda_host + d->nsys);
    // level 0
    p->lv.resize(nlev);
    HLevel& L0 = p->lv[0];
    L0.n0 = d->n0; L0.n1 = d->n1; L0.d0 = d->d0; L0.d1 = d->d1;
    L0.mask.assign((size_t)d->n0 * d->n1, 1.0);
    if (d->mask_host) std::copy(d->mask_host, d->mask_host + (size_t)d->n0 * d->n1, L0.mask.begin());
    std::vector<double> mu, mv;
    uv_masks(L0.mask, L0.n0, L0.n1, mu, mv);
    std::vector<double> cu0(d->coef_u_host, d->coef_u_host + (size_t)(d->n0 + 1) * d->n1);
    std::vector<double> cv0(d->coef_v_host, d->coef_v_host + (size_t)d->n0 * (d->n1 + 1));
    std::vector<double> coef((size_t)d->n0 * d->n1);
    for (int i = 0; i < d->n0; ++i)
        for (int j = 0; j < d->n1; ++j)
            coef[(size_t)i * d->n1 + j] = 0.25 * (cu0[(size_t)(i + 1) * d->n1 + j] + cu0[(size_t)i * d->n1 + j] +
                                                  cv0[(size_t)i * (d->n1 + 1) + j + 1] +
                                                  cv0[(size_t)i * (d->n1 + 1) + j]);
    L0.cu.resize(cu0.size());
    L0.cv.resize(cv0.size());
    for (size_t k = 0; k < cu0.size(); ++k) L0.cu[k] = cu0[k] * mu[k];
    for (size_t k = 0; k < cv0.size(); ++k) L0.cv[k] = cv0[k] * mv[k];
    for (int l = 1; l < nlev; ++l) {
        const HLevel& F = p->lv[l - 1];
        HLevel& C = p->lv[l];
        C.n0 = F.n0 / 2; C.n1 = F.n1 / 2; C.d0 = F.d0 * 2; C.d1 = F.d1 * 2;
        std::vector<double> m4 = restrict_h(F.mask, F.n0, F.n1, nullptr, 4.0);
        C.mask.resize(m4.size());
        for (size_t k = 0; k < m4.size(); ++k) C.mask[k] = m4[k] > 0.5;
        C.divr = restrict_h(F.mask, F.n0, F.n1, nullptr, 1.0);
        for (double& v : C.divr) v = std::max(v, 1.0);
        coef = restrict_h(coef, F.n0, F.n1, &C.divr, 0.0);
        for (size_t k = 0; k < coef.size(); ++k) coef[k] *= C.mask[k];
        uv_masks(C.mask, C.n0, C.n1, mu, mv);
        C.cu.assign((size_t)(C.n0 + 1) * C.n1, 0.0);
        C.cv.assign((size_t)C.n0 * (C.n1 + 1), 0.0);
        for (int i = 0; i <= C.n0; ++i)
            for (int j = 0; j < C.n1; ++j)
                C.cu[(size_t)i * C.n1 + j] = (at(coef, C.n0, C.n1, i - 1, j) + at(coef, C.n0, C.n1, i, j)) / 2 *
                                             mu[(size_t)i * C.n1 + j];
        for (int i = 0; i < C.n0; ++i)
            for (int j = 0; j <= C.n1; ++j)
                C.cv[(size_t)i * (C.n1 + 1) + j] = (at(coef, C.n0, C.n1, i, j - 1) + at(coef, C.n0, C.n1, i, j)) /
                                                   2 * mv[(size_t)i * (C.n1 + 1) + j];
    }
    for (int l = 0; l + 1 < nlev; ++l) {
        p->lv[l].divp = prolong_h(p->lv[l + 1].mask, p->lv[l + 1].n0, p->lv[l + 1].n1);
        for (double& v : p->lv[l].divp) v = std::max(v, 1.0);
    }
    for (int l = 0; l < nlev; ++l) {
        HLevel& L = p->lv[l];
        const double dxm2 = 1.0 / (L.d0 * L.d0), dym2 = 1.0 / (L.d1 * L.d1);
        L.factor.assign((size_t)p->nsys * L.n0 * L.n1, 0.0);
        for (int b = 0; b < p->nsys; ++b)
            for (int i = 0; i < L.n0; ++i)
                for (int j = 0; j < L.n1; ++j) {
                    const double den = p->lambda[b] +
                                       dxm2 * (L.cu[(size_t)(i + 1) * L.n1 + j] + L.cu[(size_t)i * L.n1 + j]) +
                                       dym2 * (L.cv[(size_t)i * (L.n1 + 1) + j + 1] + L.cv[(size_t)i * (L.n1 + 1) + j]);
                    L.factor[((size_t)b * L.n0 + i) * L.n1 + j] = L.mask[(size_t)i * L.n1 + j] / den;
                }
    }
    // bottom pseudo-inverse
    std::vector<int32_t> idx;
    std::vector<double> inv;
    const HLevel& Bt = p->lv[nlev - 1];
    if (p->niter_bottom <= 0) {
        for (int i = 0; i < Bt.n0; ++i)
            for (int j = 0; j < Bt.n1; ++j)
                if (Bt.mask[(size_t)i * Bt.n1 + j] != 0) idx.push_back(i * Bt.n1 + j);
        p->nb = (int)idx.size();
        if (p->nb > 4096) {
            delete p;
            return VD_ERR_UNSUPPORTED;
        }
        inv.assign((size_t)p->nsys * p->nb * p->nb, 0.0);
        std::vector<double> e((size_t)Bt.n0 * Bt.n1), He;
        for (int b = 0; b < p->nsys; ++b) {
            std::vector<double> H((size_t)p->nb * p->nb);
            for (int k = 0; k < p->nb; ++k) {
                std::fill(e.begin(), e.end(), 0.0);
                e[idx[k]] = 1.0;
                helm_apply(Bt, p->lambda[b], e, He);
                for (int jrow = 0; jrow < p->nb; ++jrow) H[(size_t)jrow * p->nb + k] = He[idx[jrow]];
            }
            const std::vector<double> P = pinv_sym(H, p->nb);
            std::copy(P.begin(), P.end(), inv.begin() + (size_t)b * p->nb * p->nb);
        }
    }
    // workspace: per level f, rhs, tmp and, in float64, the scaled rhs
    size_t offw = 0;
    p->ws_off.resize(4 * nlev);
    const int nbuf = p->dtype == VD_F64 ? 4 : 3;
    for (int l = 0; l < nlev; ++l)
        for (int w = 0; w < nbuf; ++w) {
            p->ws_off[4 * l + w] = offw;
            offw += (size_t)p->nsys * p->lv[l].n0 * p->lv[l].n1;
            offw = (offw + 63) & ~size_t(63);
        }
    p->ws_elems = offw;
    // the one-block coarse kernel takes the levels of at most 4096 cells (1024
    // in float64: one SM's FP64 rate is ~1/64 of its FP32 rate, so a float64
    // level of 3072 cells runs faster spread over the GPU) whose solution, rhs
    // and scratch fit 200 KB of shared memory
    p->lc = nlev;
    const size_t esz = p->dtype == VD_F64 ? 8 : 4;
    const long long max_cells = p->dtype == VD_F64 ? 1024 : 4096;
    for (int l = 0; l < nlev; ++l) {
        size_t sm = 0;
        for (int k = l; k < nlev; ++k) sm += nbuf * (size_t)p->lv[k].n0 * p->lv[k].n1 * esz;
        if ((long long)p->lv[l].n0 * p->lv[l].n1 <= max_cells && sm <= 200 * 1024) {
            p->lc = l;
            break;
        }
    }
    if (nlev > vd::MG_MAXLEV) p->lc = nlev;
    if (p->lc < nlev) {
        const cudaError_t e = p->dtype == VD_F64
            ? cudaFuncSetAttribute(vd::k_mg_coarse<double, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024)
            : cudaFuncSetAttribute(vd::k_mg_coarse<float, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        const cudaError_t e2 = cudaFuncSetAttribute(vd::k_mg_coarse<double, true>,
                                                    cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess || e2 != cudaSuccess) {
            if (p->dev) cudaFree(p->dev);
            delete p;
            return VD_ERR_CUDA;
        }
    }
    // bottom smoothing of the coarse kernel as matrices (bottom levels of at
    // most 512 cells: 2 x 512^2 entries a system, built in well under a second)
    std::vector<double> bsm;
    if (p->niter_bottom > 0 && p->lc < nlev && (long long)Bt.n0 * Bt.n1 <= 512) {
        const size_t nbc = (size_t)Bt.n0 * Bt.n1;
        for (int b = 0; b < p->nsys; ++b)
            bottom_sweep_matrices(Bt, Bt.factor.data() + b * nbc, p->omega, 6 * p->niter_bottom, nlev == 1, bsm);
    }
    const int st = p->dtype == VD_F64 ? mg_upload<double>(p, idx, inv, bsm) : mg_upload<float>(p, idx, inv, bsm);
    if (st != VD_OK) {
        if (p->dev) cudaFree(p->dev);
        delete p;
        return st;
    }
    *out = p;
    return VD_OK;
}

extern "C" vd_status vd_mg_plan_destroy(vd_mg_plan* p)
{
    if (!p) return VD_ERR_ARG;
    if (p->gexec) cudaGraphExecDestroy(p->gexec);
    if (p->gstream) cudaStreamDestroy(p->gstream);
    if (p->gbuf) cudaFree(p->gbuf);
    if (p->dev) cudaFree(p->dev);
    delete p;
    return VD_OK;
}

extern "C" int vd_mg_levels(const vd_mg_plan* p) { return p ? p->nlev : 0; }

extern "C" size_t vd_mg_workspace_bytes(const vd_mg_plan* p)
{
    return p ? p->ws_elems * (p->dtype == VD_F64 ? 8 : 4) : 0;
}

static int mg_run(const vd_mg_plan* p, const void* rhs, void* f, void* ws, cudaStream_t st)
{
    if (p->dtype == VD_F64) {
        MgRun<double> r{p, (double*)ws, st};
        return r.solve((const double*)rhs, (double*)f);
    }
    MgRun<float> r{p, (float*)ws, st};
    return r.solve((const float*)rhs, (float*)f);
}

// (Re)capture the solve on the plan's buffers with workspace ws.
static int mg_capture(vd_mg_plan* p, void* ws)
{
    const size_t bytes = (size_t)p->nsys * p->n0 * p->n1 * (p->dtype == VD_F64 ? 8 : 4);
    if (!p->gbuf) VD_CUDA_TRY(cudaMalloc(&p->gbuf, 2 * bytes));
    if (!p->gstream) VD_CUDA_TRY(cudaStreamCreateWithFlags(&p->gstream, cudaStreamNonBlocking));
    if (p->gexec) {
        cudaGraphExecDestroy(p->gexec);
        p->gexec = nullptr;
    }
    char* g = (char*)p->gbuf;
    VD_CUDA_TRY(cudaStreamBeginCapture(p->gstream, cudaStreamCaptureModeRelaxed));
    const int rc = mg_run(p, g, g + bytes, ws, p->gstream);
    cudaGraph_t graph = nullptr;
    const cudaError_t ec = cudaStreamEndCapture(p->gstream, &graph);
    if (rc != VD_OK) {
        if (graph) cudaGraphDestroy(graph);
        return rc;
    }
    VD_CUDA_TRY(ec);
    const cudaError_t ei = cudaGraphInstantiate(&p->gexec, graph, 0);
    cudaGraphDestroy(graph);
    VD_CUDA_TRY(ei);
    p->gws = ws;
    return VD_OK;
}

extern "C" vd_status vd_mg_solve(const vd_mg_plan* p, const void* rhs, void* f, void* ws, size_t wsb, void* stream)
{
    if (!p || !rhs || !f || !ws) return VD_ERR_ARG;
    if (wsb < vd_mg_workspace_bytes(p)) return VD_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    // a caller that is itself capturing records the launches directly
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    VD_CUDA_TRY(cudaStreamIsCapturing(st, &cs));
    if (cs != cudaStreamCaptureStatusNone) return mg_run(p, rhs, f, ws, st);
    // a solve is ~25 kernel launches per level per V-cycle; replaying them as
    // one graph removes their host launch cost
    vd_mg_plan* q = const_cast<vd_mg_plan*>(p);
    if (!q->gexec || q->gws != ws) {
        const int rc = mg_capture(q, ws);
        if (rc != VD_OK) return rc;
    }
    const size_t bytes = (size_t)p->nsys * p->n0 * p->n1 * (p->dtype == VD_F64 ? 8 : 4);
    char* g = (char*)q->gbuf;
    VD_CUDA_TRY(cudaMemcpyAsync(g, rhs, bytes, cudaMemcpyDeviceToDevice, st));
    VD_CUDA_TRY(cudaGraphLaunch(q->gexec, st));
    VD_CUDA_TRY(cudaMemcpyAsync(f, g + bytes, bytes, cudaMemcpyDeviceToDevice, st));
    return VD_OK;
}

extern "C" vd_status vd_mg_residual(const vd_mg_plan* p, const void* f, const void* rhs, void* res, void* stream)
{
    if (!p || !f || !rhs || !res) return VD_ERR_ARG;
    const dim3 g((unsigned)((p->n1 + 127) / 128), (unsigned)p->n0, (unsigned)p->nsys);
    if (p->dtype == VD_F64) {
        MgRun<double> r{p, nullptr, (cudaStream_t)stream};
        vd::k_mg_residual<double><<<g, 128, 0, (cudaStream_t)stream>>>(r.lev(0), (const double*)f,
                                                                       (const double*)rhs, (double*)res);
    } else {
        MgRun<float> r{p, nullptr, (cudaStream_t)stream};
        vd::k_mg_residual<float><<<g, 128, 0, (cudaStream_t)stream>>>(r.lev(0), (const float*)f, (const float*)rhs,
                                                                      (float*)res);
    }
    VD_LAUNCH_CHECK();
    return VD_OK;
}
