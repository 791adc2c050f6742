// Helmholtz PV->SSH inversion on a rectangle with Dirichlet walls.
//
// The reference inverts g/f*lap5 - g*f/c^2 by a 2-D orthonormal DST-I,
// division by the operator's eigenvalues and a second 2-D DST-I
// (mapping/models/model_qg1l/jqgm.py:75-91, eigenvalues 166-172). DST-I
// vectors are the exact eigenvectors of the 1-D Dirichlet second difference,
// so the same solution is obtained with ONE transform direction:
//
//   1. DST-I along x of every interior row          (dense half-size GEMMs)
//   2. for every x-wavenumber k, the tridiagonal system along y
//        a*X[j-1] + b_k*X[j] + a*X[j+1] = F[j],  a = g/f/dy^2,
//        b_k = g/f*(-2/dy^2 + mu_k) - g*f/c^2,  mu_k = 2(cos(pi(k+1)/(nx-1))-1)/dx^2
//      (Thomas algorithm with precomputed multipliers)
//   3. DST-I along x again (the orthonormal DST-I is its own inverse).
//
// DST-I even/odd split: with n = nx-2, S[p][k] = sqrt(2/(n+1)) sin(pi(p+1)(k+1)/(n+1))
// satisfies S[n-1-p][k] = (-1)^k S[p][k], so
//   forward:  F_even-k = (x[p] + x[n-1-p]) . Wodd,   F_odd-k = (x[p] - x[n-1-p]) . Weven
//   inverse:  A = Xe . Wodd^T, B = Xo . Weven;  y[p] = A+B, y[n-1-p] = A-B
// which halves the multiply-adds of a dense transform. Spectral rows are kept
// in parity-split order: columns [0, ne) hold k = 0,2,4..., [ne, n) hold k = 1,3,...
#include "vd_internal.cuh"
#include <vector>
#include <mutex>
#include <algorithm>
#include <cmath>

namespace vd {

template <typename T> struct Vec8;
template <> struct Vec8<float> {
    static __device__ __forceinline__ void load(const float* p, float (&r)[8]) {
        float4 a = *reinterpret_cast<const float4*>(p);
        float4 b = *reinterpret_cast<const float4*>(p + 4);
        r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w;
        r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
    }
};
struct GemmGeom {
    int n, ne, no, my, nx;
    long long fs;
    int R;          // rows = nfields * my
    int kpad, ldw, lds;
};

enum { MODE_FWD = 0, MODE_INV = 1 };

template <int TR> struct GemmShape {
    static constexpr int NT = 2 * (TR / 8) * 16;   // threads per CTA
};

template <typename T, int TR>
__host__ __device__ constexpr size_t gemm_smem_elems(int kpad) {
    return size_t(2) * kpad * TR +
           (size_t(2) * DST_KC * DST_NC > size_t(TR) * DST_NC ? size_t(2) * DST_KC * DST_NC
                                                              : size_t(TR) * DST_NC);
}

// One CTA: TR interior rows x DST_NC output columns of BOTH halves.
// Threads [0, NT/2) multiply by W1 (the even-k half), [NT/2, NT) by W2.
template <typename T, int TR, int MODE, int EPI>
__global__ void __launch_bounds__(GemmShape<TR>::NT)
dst_gemm_kernel(GemmGeom g, const T* __restrict__ W1, const T* __restrict__ W2,
                const T* __restrict__ src, const T* __restrict__ sub, int sub_batches,
                T* __restrict__ spec, T* __restrict__ out, const T* __restrict__ add,
                int add_batches, const int8_t* __restrict__ mask)
{
    constexpr int NT = GemmShape<TR>::NT;
    constexpr int NC = DST_NC;
    constexpr int KC = DST_KC;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* As = reinterpret_cast<T*>(smem_raw);
    T* Bs = As + size_t(g.kpad) * TR;
    T* Ws = Bs + size_t(g.kpad) * TR;     // W1 chunk | W2 chunk, later the exchange tile
    T* W1s = Ws;
    T* W2s = Ws + KC * NC;

    const int tid = threadIdx.x;
    const int row0 = blockIdx.y * TR;
    const int c0 = blockIdx.x * NC;
    const int n = g.n, ne = g.ne, no = g.no, my = g.my;

    // ---- prologue: operands, transposed to [k][row] -------------------------
    for (int idx = tid; idx < g.kpad * TR; idx += NT) {
        const int r = idx % TR;
        const int p = idx / TR;
        const int row = row0 + r;
        T a = T(0), b = T(0);
        if (row < g.R) {
            if (MODE == MODE_FWD) {
                if (p < ne) {
                    const int f = row / my;
                    const int j = row - f * my + 1;
                    const T* s = src + f * g.fs + (long long)j * g.nx + 1;
                    const T* sb = (sub != nullptr && f < sub_batches)
                                      ? sub + f * g.fs + (long long)j * g.nx + 1 : nullptr;
                    T x1 = s[p];
                    if (sb) x1 -= sb[p];
                    if (p < no) {
                        T x2 = s[n - 1 - p];
                        if (sb) x2 -= sb[n - 1 - p];
                        a = x1 + x2;
                        b = x1 - x2;
                    } else {
                        a = x1;   // middle point of an odd-length transform
                    }
                }
            } else {
                const T* s = spec + (long long)row * g.lds;
                if (p < ne) a = s[p];
                if (p < no) b = s[ne + p];
            }
        }
        As[p * TR + r] = a;
        Bs[p * TR + r] = b;
    }

    const int grp = tid / (NT / 2);
    const int lt = tid % (NT / 2);
    const int ty = lt / 16;
    const int tx = lt % 16;
    const T* Aop = grp == 0 ? As : Bs;
    const T* Wop = grp == 0 ? W1s : W2s;

    T acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = T(0);

    for (int k0 = 0; k0 < g.kpad; k0 += KC) {
        __syncthreads();
        for (int e = tid; e < KC * NC; e += NT) {
            const int kk = e / NC;
            const int cc = e - kk * NC;
            const size_t goff = size_t(k0 + kk) * g.ldw + c0 + cc;
            W1s[e] = W1[goff];
            W2s[e] = W2[goff];
        }
        __syncthreads();
#pragma unroll 4
        for (int kk = 0; kk < KC; ++kk) {
            T a[8], w[8];
            Vec8<T>::load(Aop + (k0 + kk) * TR + ty * 8, a);
            Vec8<T>::load(Wop + kk * NC + tx * 8, w);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fma(a[i], w[j], acc[i][j]);
        }
    }

    const int rb = row0 + ty * 8;
    const int cb = c0 + tx * 8;
    if (MODE == MODE_FWD) {
        const int lim = grp == 0 ? ne : no;
        const int coff = grp == 0 ? 0 : ne;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int row = rb + i;
            if (row >= g.R) continue;
            T* d = spec + (long long)row * g.lds + coff;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int t = cb + j;
                if (t < lim) d[t] = acc[i][j];
            }
        }
    } else {
        __syncthreads();
        T* X = Ws;   // [TR][NC] exchange tile
        if (grp == 1) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) X[(ty * 8 + i) * NC + tx * 8 + j] = acc[i][j];
        }
        __syncthreads();
        if (grp == 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int row = rb + i;
                if (row >= g.R) continue;
                const int f = row / my;
                const int j = row - f * my + 1;
                const long long base = f * g.fs + (long long)j * g.nx + 1;
#pragma unroll
                for (int jj = 0; jj < 8; ++jj) {
                    const int p = cb + jj;
                    if (p >= ne) continue;
                    const T A = acc[i][jj];
                    const T B = (p < no) ? X[(ty * 8 + i) * NC + tx * 8 + jj] : T(0);
                    const int ps[2] = {p, n - 1 - p};
                    const T ys[2] = {A + B, A - B};
                    const int cnt = (p < no) ? 2 : 1;
                    for (int u = 0; u < cnt; ++u) {
                        const long long o = base + ps[u];
                        if (EPI == EPI_H) {
                            T y = ys[u];
                            if (add != nullptr && f < add_batches) y += add[o];
                            out[o] = y;
                        } else {
                            const int mi = j * g.nx + 1 + ps[u];
                            out[o] = (mask[mi] == 3) ? ys[u] + add[o] : T(0);
                        }
                    }
                }
            }
        }
    }
}

// Dense form of the float64 pass. The part runs 2 FP64 FMAs a clock and SM, one
// warp instruction per 64 clocks on each of an SM's four schedulers, so the
// kernel is bound by the FP64 pipe as soon as every scheduler holds a warp:
// operands are read straight from L1 / L2 (one W load per R FMAs), and the work
// is cut finely enough to fill all 608 schedulers even for one 128^2 field.
// A warp owns 32 output columns of one half (even-k or odd-k sums) of R rows;
// a CTA's warps are both halves x CWC column groups x RG row groups over the
// butterflied rows in shared memory. PF (one row a warp): the next 8 entries of W are
// loaded while the last 8 are used; with a warp or two on a scheduler nothing else
// covers an L2 load.
// Measured on one 128^2 field: a pass 6.3 us forward and 6.6 us inverse (8.0 and 13.2
// without the prefetch and with CTAs of two rows on 63 SMs); the whole solve 340 us with
// the 8 x 8 register tile of the float32 kernel (8 CTAs of two warps a pass); 119 us on
// one 384^2 field.
template <int R, int CWC, int RG, bool PF, int MODE, int EPI>
__global__ void __launch_bounds__(64 * CWC * RG)
dst_dense64_kernel(GemmGeom g, const double* __restrict__ W1, const double* __restrict__ W2,
                   const double* __restrict__ src, const double* __restrict__ sub, int sub_batches,
                   double* __restrict__ spec, double* __restrict__ out, const double* __restrict__ add,
                   int add_batches, const int8_t* __restrict__ mask)
{
    constexpr int TR = R * RG, NC = 32 * CWC, NW = CWC * RG, NT = 64 * NW;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* As = reinterpret_cast<double*>(smem_raw);    // [ne][TR]
    double* Bs = As + (size_t)g.ne * TR;                 // [no][TR]
    const int n = g.n, ne = g.ne, no = g.no, my = g.my;
    const int cg = (ne + NC - 1) / NC;                   // column groups: the CTAs of the same rows follow one another
    const int row0 = (int)(blockIdx.x / (unsigned)cg) * TR, c0 = (int)(blockIdx.x % (unsigned)cg) * NC;

    for (int idx = threadIdx.x; idx < ne * TR; idx += NT) {
        const int r = idx / ne, p = idx - r * ne;
        const int row = row0 + r;
        double a = 0.0, b = 0.0;
        if (row < g.R) {
            if (MODE == MODE_FWD) {
                const int f = row / my;
                const long long o = f * g.fs + (long long)(row - f * my + 1) * g.nx + 1;
                const bool hs = sub != nullptr && f < sub_batches;
                const double x1 = src[o + p] - (hs ? sub[o + p] : 0.0);
                if (p < no) {
                    const double x2 = src[o + n - 1 - p] - (hs ? sub[o + n - 1 - p] : 0.0);
                    a = x1 + x2;
                    b = x1 - x2;
                } else {
                    a = x1;   // middle point of an odd-length transform
                }
            } else {
                const double* s = spec + (long long)row * g.lds;
                a = s[p];
                if (p < no) b = s[ne + p];
            }
        }
        As[p * TR + r] = a;
        if (p < no) Bs[p * TR + r] = b;
    }
    __syncthreads();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int half = warp / NW, wi = warp % NW, cw = wi % CWC, rg = wi / CWC;
    const int t = c0 + cw * 32 + lane;                   // < ldw: the tables' rows are zero-padded
    const int K = half == 0 ? ne : no;
    const double* __restrict__ W = (half == 0 ? W1 : W2) + t;
    const double* __restrict__ X = (half == 0 ? As : Bs) + rg * R;
    double acc[R];
#pragma unroll
    for (int i = 0; i < R; ++i) acc[i] = 0.0;
    if constexpr (PF) {
        static_assert(R == 1, "one row a warp");
        double wc[8], wn[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) wc[u] = u < K ? __ldg(W + (size_t)u * g.ldw) : 0.0;
        for (int k0 = 0; k0 < K; k0 += 8) {
#pragma unroll
            for (int u = 0; u < 8; ++u) wn[u] = k0 + 8 + u < K ? __ldg(W + (size_t)(k0 + 8 + u) * g.ldw) : 0.0;
            if (k0 + 8 <= K) {
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    acc[0] = fma(X[(k0 + u) * TR], wc[u], acc[0]);
            } else {
                // the last K % 8 as 4 + 2 + 1 (a predicated-off FMA would take its slot)
                int k = k0;
                const int rem = K - k0;
                if (rem & 4) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        acc[0] = fma(X[(k + u) * TR], wc[u], acc[0]);
                        wc[u] = wc[u + 4];
                    }
                    k += 4;
                }
                if (rem & 2) {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        acc[0] = fma(X[(k + u) * TR], wc[u], acc[0]);
                        wc[u] = wc[u + 2];
                    }
                    k += 2;
                }
                if (rem & 1) acc[0] = fma(X[k * TR], wc[0], acc[0]);
                break;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) wc[u] = wn[u];
        }
    } else {
#pragma unroll 8
        for (int k = 0; k < K; ++k) {
            const double w = __ldg(W + (size_t)k * g.ldw);
#pragma unroll
            for (int i = 0; i < R; ++i) acc[i] = fma(X[k * TR + i], w, acc[i]);
        }
    }

    if (MODE == MODE_FWD) {
        if (t < K) {
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int row = row0 + rg * R + i;
                if (row < g.R) spec[(long long)row * g.lds + (half == 0 ? 0 : ne) + t] = acc[i];
            }
        }
    } else {
        // y[p] = A + B, y[n-1-p] = A - B: the odd-half warps hand over B
        __shared__ double ex[NW][R][32];
        if (half == 1) {
#pragma unroll
            for (int i = 0; i < R; ++i) ex[wi][i][lane] = acc[i];
        }
        __syncthreads();
        if (half == 0 && t < ne) {
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int row = row0 + rg * R + i;
                if (row >= g.R) break;
                const int f = row / my, j = row - f * my + 1;
                const long long base = f * g.fs + (long long)j * g.nx + 1;
                const double B = t < no ? ex[wi][i][lane] : 0.0;
                const double ys[2] = {acc[i] + B, acc[i] - B};
                const int ps[2] = {t, n - 1 - t};
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (u == 1 && t >= no) break;
                    const long long o = base + ps[u];
                    if (EPI == EPI_H) out[o] = ys[u] + ((add != nullptr && f < add_batches) ? add[o] : 0.0);
                    else out[o] = (mask[j * g.nx + 1 + ps[u]] == 3) ? ys[u] + add[o] : 0.0;
                }
            }
        }
    }
}

// Chunked Thomas algorithm. Both sweeps are first-order linear recurrences
// with the multiplier alpha_j = -a*m_j: forward d_j = m_j F_j + alpha_j
// d_{j-1}, backward x_j = d_j + alpha_j x_{j+1}. A row piece runs from a zero
// carry while accumulating the product of its alphas; the true values follow
// by adding carry * partial product. |alpha| < 1 (diagonal dominance), so
// the products only shrink.
// CW spectral columns per CTA; the warp's lanes are CW columns x (32/CW)
// row pieces, so a CTA holds nw*(32/CW) pieces of CH rows per column. Each
// thread keeps its piece (values and multipliers) in registers and runs both
// Thomas sweeps locally (the recurrences are affine, so a piece is summarised
// by its end value and the product of its multipliers). The pieces of a
// column are then combined by a scan of the affine maps (d, P) o (d', P') =
// (d + P d', P P'): a shuffle scan over the warp's 32/CW pieces, then the
// warp totals through shared memory; every piece applies the carry it
// receives. Eight columns per CTA: 1024 CTAs for 16 fields of 512^2, 128 for
// one 1024^2 field.
// LEAN caps the registers at 80 (16-row pieces in float32 otherwise take
// ~124): three 256-thread CTAs fit an SM instead of two (a schedule choice,
// picked by timing). 8-row pieces are capped at 64 registers, so two CTAs
// of up to 512 threads fit an SM.
template <typename T, int CW, int CH, bool LEAN = false>
__global__ void __maxnreg__(LEAN ? 80 : (CH <= 8 ? 64 : 128))
tridiag_chunked_kernel(T* __restrict__ spec, const T* __restrict__ trim, int my, int n, int lds, T a)
{
    constexpr int SUB = 32 / CW;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int nw = blockDim.y;
    T* wD = reinterpret_cast<T*>(smem_raw);         // [nw][CW] warp totals: end value
    T* wP = wD + (size_t)nw * CW;                   // [nw][CW] warp totals: product
    const int f = blockIdx.y;
    const int lane = threadIdx.x, w = threadIdx.y;
    const int c = lane % CW;
    const int sp = lane / CW;                       // piece within the warp
    const int pc = w * SUB + sp;
    const int t = blockIdx.x * CW + c;
    const bool col_ok = t < n;
    T* S = spec + (long long)f * my * lds + t;
    const T* M = trim + t;
    const int j0 = pc * CH;
    const int cnt = col_ok ? max(0, min(CH, my - j0)) : 0;
    T x[CH], al[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i) {
        const bool v = i < cnt;
        x[i] = v ? S[(long long)(j0 + i) * lds] : T(0);
        al[i] = v ? __ldg(M + (long long)(j0 + i) * lds) : T(0);
    }

    // forward sweep, piece-local: d_j = m_j F_j + (-a m_j) d_{j-1}
    T d = T(0), P = T(1);
#pragma unroll
    for (int i = 0; i < CH; ++i) {
        if (i < cnt) {
            const T m = al[i];
            al[i] = -a * m;
            d = m * x[i] + al[i] * d;
            x[i] = d;
            P *= al[i];
        }
    }
    {
        // inclusive scan over the pieces of the warp (lanes CW apart)
        T sd = d, sP = P;
#pragma unroll
        for (int o = 1; o < SUB; o <<= 1) {
            const T od = __shfl_up_sync(0xffffffffu, sd, o * CW);
            const T oP = __shfl_up_sync(0xffffffffu, sP, o * CW);
            if (sp >= o) {
                sd = sd + sP * od;
                sP = sP * oP;
            }
        }
        if (sp == SUB - 1) {
            wD[w * CW + c] = sd;
            wP[w * CW + c] = sP;
        }
        __syncthreads();
        // carry into this warp: the warps before it, in order
        T cw = T(0);
        for (int v = 0; v < w; ++v) cw = wD[v * CW + c] + wP[v * CW + c] * cw;
        // end value of the previous piece
        const T pd = __shfl_up_sync(0xffffffffu, sd, CW);
        const T pP = __shfl_up_sync(0xffffffffu, sP, CW);
        const T cin = sp == 0 ? cw : pd + pP * cw;
        if (pc > 0) {
            T pr = T(1);
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                if (i < cnt) {
                    pr *= al[i];
                    x[i] += pr * cin;
                }
            }
        }
    }
    __syncthreads();   // the warp totals are read before they are rewritten

    // backward sweep, piece-local from the piece end: x_j = d_j + (-a m_j) x_{j+1}
    T xr = T(0);
    P = T(1);
#pragma unroll
    for (int i = CH - 1; i >= 0; --i) {
        if (i < cnt) {
            xr = x[i] + al[i] * xr;
            x[i] = xr;
            P *= al[i];
        }
    }
    {
        // inclusive scan from the last piece of the warp down to the first
        T sd = xr, sP = P;
#pragma unroll
        for (int o = 1; o < SUB; o <<= 1) {
            const T od = __shfl_down_sync(0xffffffffu, sd, o * CW);
            const T oP = __shfl_down_sync(0xffffffffu, sP, o * CW);
            if (sp + o < SUB) {
                sd = sd + sP * od;
                sP = sP * oP;
            }
        }
        if (sp == 0) {
            wD[w * CW + c] = sd;
            wP[w * CW + c] = sP;
        }
        __syncthreads();
        T cw = T(0);
        for (int v = nw - 1; v > w; --v) cw = wD[v * CW + c] + wP[v * CW + c] * cw;
        const T nd = __shfl_down_sync(0xffffffffu, sd, CW);
        const T nP = __shfl_down_sync(0xffffffffu, sP, CW);
        const T cin = sp == SUB - 1 ? cw : nd + nP * cw;
        if (pc < nw * SUB - 1) {
            T pr = T(1);
#pragma unroll
            for (int i = CH - 1; i >= 0; --i) {
                if (i < cnt) {
                    pr *= al[i];
                    x[i] += pr * cin;
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < CH; ++i)
        if (i < cnt) S[(long long)(j0 + i) * lds] = x[i];
}

// Rows of a piece of the float64 tridiagonal kernel with tables, and the tallest field
// it takes (16 warps of 4 pieces, 128 registers a thread).
constexpr int TRI_TAB_ROWS = 8, TRI_TAB_MAX = 16 * 4 * TRI_TAB_ROWS;

// Those tables, from the Thomas multipliers, at plan creation (columns behind n are never
// read): [4][my][lds] multipliers, alphas and their products within a piece, from its
// start and from its end. A 512^2 plan takes 6.7 ms with the tables formed on the host,
// 3.7 here.
__global__ void tridiag_tables_kernel(const double* __restrict__ trim, double* __restrict__ tab, int my, int n, int lds,
                                      double a)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int j0 = blockIdx.y * TRI_TAB_ROWS, j1 = min(j0 + TRI_TAB_ROWS, my);
    if (t >= n) return;
    const long long pl = (long long)my * lds;
    double pr = 1.0;
    for (int j = j0; j < j1; ++j) {
        const long long o = (long long)j * lds + t;
        const double m = trim[o], al = -a * m;
        tab[o] = m;
        tab[pl + o] = al;
        pr *= al;
        tab[2 * pl + o] = pr;
    }
    pr = 1.0;
    for (int j = j1 - 1; j >= j0; --j) {
        const long long o = (long long)j * lds + t;
        pr *= -a * trim[o];
        tab[3 * pl + o] = pr;
    }
}

// The float64 form of the chunked kernel with its data-independent products from
// tables: alpha_j, and the products of the alphas from a piece's start to j (pf) and
// from j to its end (pb), formed in the order the sweeps form them. 5 FP64
// instructions a row instead of 10, in pieces of 8 rows: one SM quarter issues a
// warp's FP64 instruction in 75 clocks, so a small grid's time is the instructions of
// one warp. 4 x 256^2: 6.1 us (11.4 without the tables), one 128^2 field 4.3 us (10.9).
template <int CW, int CH>
__global__ void __launch_bounds__(512)
tridiag_tab_kernel(double* __restrict__ spec, const double* __restrict__ tab, int my, int n, int lds)
{
    constexpr int SUB = 32 / CW;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int nw = blockDim.y;
    double* wD = reinterpret_cast<double*>(smem_raw);   // [nw][CW] warp totals: end value
    double* wP = wD + (size_t)nw * CW;                  // [nw][CW] warp totals: product
    const int lane = threadIdx.x, w = threadIdx.y;
    const int c = lane % CW, sp = lane / CW;
    const int pc = w * SUB + sp, j0 = pc * CH;
    const int t = blockIdx.x * CW + c;
    const int cnt = t < n ? max(0, min(CH, my - j0)) : 0;
    const long long plane = (long long)my * lds;
    double* S = spec + blockIdx.y * plane + (long long)j0 * lds + t;
    const double* A = tab + (long long)j0 * lds + t;   // m, then alpha, pf, pb
    double x[CH], al[CH], pf[CH], pb[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i) {
        const bool v = i < cnt;
        const long long o = (long long)i * lds;
        x[i] = v ? S[o] : 0.0;
        pf[i] = v ? __ldg(A + o) : 0.0;                // m, until the forward sweep has used it
        al[i] = v ? __ldg(A + plane + o) : 0.0;
        pb[i] = v ? __ldg(A + 3 * plane + o) : 0.0;
    }
    // (rows beyond the column stay 0 in every array, so no sweep is predicated)
    double d = 0.0;
#pragma unroll
    for (int i = 0; i < CH; ++i) {
        d = pf[i] * x[i] + al[i] * d;
        x[i] = d;
    }
#pragma unroll
    for (int i = 0; i < CH; ++i) pf[i] = i < cnt ? __ldg(A + 2 * plane + (long long)i * lds) : 0.0;
    double P = cnt > 0 ? __ldg(A + 2 * plane + (long long)(cnt - 1) * lds) : 1.0;
    {
        double sd = d, sP = P;
#pragma unroll
        for (int o = 1; o < SUB; o <<= 1) {
            const double od = __shfl_up_sync(0xffffffffu, sd, o * CW);
            const double oP = __shfl_up_sync(0xffffffffu, sP, o * CW);
            if (sp >= o) {
                sd = sd + sP * od;
                sP = sP * oP;
            }
        }
        if (sp == SUB - 1) {
            wD[w * CW + c] = sd;
            wP[w * CW + c] = sP;
        }
        __syncthreads();
        double cw = 0.0;
        for (int v = 0; v < w; ++v) cw = wD[v * CW + c] + wP[v * CW + c] * cw;
        const double pd = __shfl_up_sync(0xffffffffu, sd, CW);
        const double pP = __shfl_up_sync(0xffffffffu, sP, CW);
        const double cin = sp == 0 ? cw : pd + pP * cw;
#pragma unroll
        for (int i = 0; i < CH; ++i) x[i] += pf[i] * cin;
        if (cnt < CH) {   // an infinite carry times 0
#pragma unroll
            for (int i = 0; i < CH; ++i) x[i] = i < cnt ? x[i] : 0.0;
        }
    }
    __syncthreads();   // the warp totals are read before they are rewritten
    double xr = 0.0;
#pragma unroll
    for (int i = CH - 1; i >= 0; --i) {
        xr = x[i] + al[i] * xr;
        x[i] = xr;
    }
    {
        double sd = xr, sP = cnt > 0 ? pb[0] : 1.0;
#pragma unroll
        for (int o = 1; o < SUB; o <<= 1) {
            const double od = __shfl_down_sync(0xffffffffu, sd, o * CW);
            const double oP = __shfl_down_sync(0xffffffffu, sP, o * CW);
            if (sp + o < SUB) {
                sd = sd + sP * od;
                sP = sP * oP;
            }
        }
        if (sp == 0) {
            wD[w * CW + c] = sd;
            wP[w * CW + c] = sP;
        }
        __syncthreads();
        double cw = 0.0;
        for (int v = nw - 1; v > w; --v) cw = wD[v * CW + c] + wP[v * CW + c] * cw;
        const double nd = __shfl_down_sync(0xffffffffu, sd, CW);
        const double nP = __shfl_down_sync(0xffffffffu, sP, CW);
        const double cin = sp == SUB - 1 ? cw : nd + nP * cw;
#pragma unroll
        for (int i = 0; i < CH; ++i)
            if (i < cnt) S[(long long)i * lds] = x[i] + pb[i] * cin;
    }
}

// Same recurrences directly on the spectral buffer, for column blocks too tall
// for shared memory (float64 at the largest grids).
template <typename T>
__global__ void __launch_bounds__(32)
tridiag_global_kernel(T* __restrict__ spec, const T* __restrict__ trim, int my, int n, int lds, T a)
{
    const int f = blockIdx.y;
    const int t = blockIdx.x * 32 + threadIdx.x;
    if (t >= n) return;
    T* S = spec + (long long)f * my * lds + t;
    const T* M = trim + t;
    T d = S[0] * __ldg(M);
    S[0] = d;
    for (int j = 1; j < my; ++j) {
        d = (S[(long long)j * lds] - a * d) * __ldg(M + (long long)j * lds);
        S[(long long)j * lds] = d;
    }
    T x = d;
    for (int j = my - 2; j >= 0; --j) {
        x = S[(long long)j * lds] - a * __ldg(M + (long long)j * lds) * x;
        S[(long long)j * lds] = x;
    }
}

// ---------------------------------------------------------------------------
// Float64 DST-I by FFT
//
// The FP64 rate of this part is a small fraction of its FP32 / tensor rate, so
// the O(n^2) dense transform above costs ~3 ms a field at n ~ 1000 even at
// the FP64 peak; an FFT does the same transform in O(n log n). Two real rows
// a, b are packed as z = a + i b into their odd extension of length
// L = 2(n+1): z_0 = z_{n+1} = 0, z_{p+1} = a_p + i b_p, z_{L-1-p} = -z_{p+1}.
// The DFT of a real odd sequence is purely imaginary,
//   A_m = -2i sum_p a_p sin(pi (p+1) m / (n+1)),
// so Z = A + i B gives both rows at once: DST_a(m) = -Im Z_m / 2 and
// DST_b(m) = Re Z_m / 2, times sqrt(2/(n+1)) for the orthonormal form. The
// FFT is a Stockham autosort (each stage reads v_r = x[j + r L/R], applies the
// twiddles e^{-2 pi i k r / (Ns R)} with k = j mod Ns, takes the length-R DFT
// and writes y[(j/Ns) Ns R + k + r Ns]; the output is in natural order) with
// radix 4, 2, 3 and 5 stages and direct stages of other odd radices,
// ping-ponging between two shared-memory buffers.
// The oddness halves every stage. After the stages of product Ns the buffer holds
// rows j < T = L/Ns of the DFTs B[j][k] of the subsequences z_{j + q T}, and
//   B[T - j][k] = -e^{2 pi i k / Ns} B[j][Ns - k],   B[0][Ns - k] = -B[0][k],
// so a stage forms rows j <= T/2 alone (of row 0 the first half), and reads a row
// beyond T/2 as its mirror image, whose factor makes the twiddle another entry of
// the table: -conj(tw[k (R - r)]). (Even radices come first among the small ones:
// an odd T has one row that mirrors itself, an even T two.)
// The orthonormal DST-I is its own inverse, so the inverse pass is the same
// transform from the parity-split spectral rows to the field.
// ---------------------------------------------------------------------------
struct FftGeom {
    int L, N, n, ne, my, nx, R, lds, nst, pp;
    long long fs;
    double scale;        // sqrt(2/N) / 2
    int rad[24];
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// -i * a
__device__ __forceinline__ double2 cmi(double2 a) { return make_double2(a.y, -a.x); }

template <int R> struct Dft;
template <> struct Dft<2> {
    static __device__ __forceinline__ void run(double2 (&v)[2])
    {
        const double2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    }
};
template <> struct Dft<4> {
    static __device__ __forceinline__ void run(double2 (&v)[4])
    {
        const double2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
        const double2 c = cadd(v[1], v[3]), d = cmi(csub(v[1], v[3]));
        v[0] = cadd(a, c);
        v[2] = csub(a, c);
        v[1] = cadd(b, d);
        v[3] = csub(b, d);
    }
};
template <> struct Dft<3> {
    // y1,2 = v0 - (v1+v2)/2 -/+ i (sqrt(3)/2) (v1 - v2)
    static __device__ __forceinline__ void run(double2 (&v)[3])
    {
        constexpr double S3 = 0.86602540378443864676;   // sqrt(3)/2
        const double2 t = cadd(v[1], v[2]);
        const double2 m = make_double2(v[0].x - 0.5 * t.x, v[0].y - 0.5 * t.y);
        const double2 d = cmi(csub(v[1], v[2]));
        const double2 e = make_double2(S3 * d.x, S3 * d.y);
        v[0] = cadd(v[0], t);
        v[1] = cadd(m, e);
        v[2] = csub(m, e);
    }
};
template <> struct Dft<5> {
    // pairs r, 5-r: t1 = v1+v4, t2 = v2+v3, d1 = v1-v4, d2 = v2-v3;
    // y1,4 = v0 + c1 t1 + c2 t2 -/+ i (s1 d1 + s2 d2)
    // y2,3 = v0 + c2 t1 + c1 t2 -/+ i (s2 d1 - s1 d2)
    static __device__ __forceinline__ void run(double2 (&v)[5])
    {
        constexpr double C1 = 0.30901699437494742410;    // cos(2 pi / 5)
        constexpr double C2 = -0.80901699437494742410;   // cos(4 pi / 5)
        constexpr double S1 = 0.95105651629515357212;    // sin(2 pi / 5)
        constexpr double S2 = 0.58778525229247312917;    // sin(4 pi / 5)
        const double2 t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]);
        const double2 d1 = cmi(csub(v[1], v[4])), d2 = cmi(csub(v[2], v[3]));
        const double2 a1 = make_double2(v[0].x + C1 * t1.x + C2 * t2.x, v[0].y + C1 * t1.y + C2 * t2.y);
        const double2 a2 = make_double2(v[0].x + C2 * t1.x + C1 * t2.x, v[0].y + C2 * t1.y + C1 * t2.y);
        const double2 b1 = make_double2(S1 * d1.x + S2 * d2.x, S1 * d1.y + S2 * d2.y);
        const double2 b2 = make_double2(S2 * d1.x - S1 * d2.x, S2 * d1.y - S1 * d2.y);
        v[0] = cadd(v[0], cadd(t1, t2));
        v[1] = cadd(a1, b1);
        v[4] = csub(a1, b1);
        v[2] = cadd(a2, b2);
        v[3] = csub(a2, b2);
    }
};

// x with its sign flipped where neg (integers: an FP64 negation takes an issue slot)
__device__ __forceinline__ double flip(double x, bool neg)
{
    return __hiloint2double(__double2hiint(x) ^ (neg ? (int)0x80000000 : 0), __double2loint(x));
}

// A stage of a small radix over the rows j <= T/2 (T = L/(Ns R) output rows).
// 4 x 256^2 (510 = 17 2 3 5): 19.0 us a pass, 27.8 with whole stages.
template <int R>
__device__ __forceinline__ void fft_stage(const double2* __restrict__ in, double2* __restrict__ out,
                                          const double2* __restrict__ tw, int L, int Ns, int pp)
{
    const int T = L / (Ns * R), Ti = T * R;      // output and input rows; tw[m T] = e^{-2 pi i m / (Ns R)}
    const int n0 = Ns / 2 + 1;                   // butterflies of row 0
    const int nb = n0 + (T / 2) * Ns;
    for (int idx = threadIdx.x; idx < pp * nb; idx += blockDim.x) {
        const int q = idx / nb;
        int k = idx - q * nb, j = 0;
        if (k >= n0) {
            k -= n0;
            j = k / Ns;
            k -= j * Ns;
            ++j;
        }
        const double2* I = in + (long long)q * L;
        double2* O = out + (long long)q * L;
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = j + r * T;
            const bool up = 2 * row > Ti;
            v[r] = I[up ? (Ti - row) * Ns + (k ? Ns - k : 0) : row * Ns + k];
            if (r == 0) continue;                // row 0 .. T/2 is never beyond Ti/2
            if (Ns > 1) {
                double2 w = __ldg(tw + (long long)k * (up ? R - r : r) * T);
                w.x = flip(w.x, up);
                v[r] = cmul(v[r], w);
            } else {
                v[r] = make_double2(flip(v[r].x, up), flip(v[r].y, up));
            }
        }
        Dft<R>::run(v);
        const int base = j * Ns * R + k;
#pragma unroll
        for (int r = 0; r < R; ++r) O[base + r * Ns] = v[r];
        if (j == 0) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int m = Ns * R - k - r * Ns;
                if (m < Ns * R) O[m] = make_double2(flip(v[r].x, true), flip(v[r].y, true));
            }
        }
    }
}

// The rows beyond T/2 from their mirror images, for a direct odd stage that is not
// the first (it works in place on whole columns).
__device__ __forceinline__ void fft_expand(double2* __restrict__ in, const double2* __restrict__ tw, int L, int Ns,
                                           int pp)
{
    const int T = L / Ns, nr = T - 1 - T / 2;    // rows T/2 + 1 .. T - 1
    for (int idx = threadIdx.x; idx < pp * nr * Ns; idx += blockDim.x) {
        const int qr = idx / Ns, k = idx - qr * Ns;
        const int row = T / 2 + 1 + qr % nr;
        double2* I = in + (long long)(qr / nr) * L;
        const double2 w = __ldg(tw + (long long)k * T);
        I[row * Ns + k] = cmul(I[(T - row) * Ns + (k ? Ns - k : 0)], make_double2(flip(w.x, true), w.y));
    }
    __syncthreads();
}

// A stage of any odd radix p >= 7 (a prime factor of n + 1), as a direct
// length-p DFT by pairs: with t_q = v_q + v_{p-q}, d_q = v_q - v_{p-q},
//   y_r, y_{p-r} = v_0 + sum_q cos(2 pi q r/p) t_q  -/+  i sum_q sin(2 pi q r/p) d_q.
// A first pass writes t_q and d_q over v_q and v_{p-q} in place (with the
// stage's twiddles); then one thread forms one output pair of one butterfly,
// 4 FP64 FMAs per q. The pass is bound by the FP64 pipe (2 FMA a clock and
// SM), not by the shared-memory reads of t and d.
// FIRST (Ns = 1): butterflies j <= T/2 alone. A later one works on whole columns
// (fft_expand before it).
// Measured: 4 x 256^2 (n + 1 = 3 5 17) 19.0 us a pass (dense float32-style tile
// 300 us), one 512^2 field (7 73) 105 us a solve, 291 us with dense products.
template <bool FIRST>
__device__ __forceinline__ void fft_stage_odd(double2* __restrict__ in, double2* __restrict__ out,
                                              const double2* __restrict__ tw, int L, int Ns, int pp, int p)
{
    const int T = L / p, h = p >> 1;
    const int tstep = FIRST ? 0 : L / (Ns * p);
    const int nb = FIRST ? T / 2 + 1 : T;      // butterflies computed (L is even and p odd: T is even)
    for (int idx = threadIdx.x; idx < pp * nb * h; idx += blockDim.x) {
        const int bq = idx / nb, j = idx - bq * nb;
        const int q = bq % h + 1;
        double2* I = in + (long long)(bq / h) * L + j;
        double2 a = I[q * T], b = I[(p - q) * T];
        if (!FIRST) {
            const int k = j % Ns;
            a = cmul(a, __ldg(tw + (long long)k * q * tstep));
            b = cmul(b, __ldg(tw + (long long)k * (p - q) * tstep));
        }
        I[q * T] = cadd(a, b);
        I[(p - q) * T] = csub(a, b);
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < pp * nb * (h + 1); idx += blockDim.x) {
        const int br = idx / nb, j = idx - br * nb;
        const int r = br % (h + 1);
        const double2* I = in + (long long)(br / (h + 1)) * L + j;
        double2* O = out + (long long)(br / (h + 1)) * L;
        double2 C = I[0], S = make_double2(0.0, 0.0);
        if (r == 0) {
            for (int q = 1; q <= h; ++q) C = cadd(C, I[q * T]);
        } else {
            int m = 0;
            for (int q = 1; q <= h; ++q) {
                m += r * T;                    // (q r mod p) T
                if (m >= L) m -= L;
                const double2 w = __ldg(tw + m);   // cos, -sin
                const double2 t = I[q * T], d = I[(p - q) * T];
                C.x = fma(w.x, t.x, C.x);
                C.y = fma(w.x, t.y, C.y);
                S.x = fma(w.y, d.x, S.x);
                S.y = fma(w.y, d.y, S.y);
            }
        }
        // S holds -sum sin d: y_r = C + i S, y_{p-r} = C - i S
        const double2 yr = make_double2(C.x - S.y, C.y + S.x), yp = make_double2(C.x + S.y, C.y - S.x);
        if (FIRST) {
            O[j * p + r] = yr;
            if (r) O[j * p + p - r] = yp;
        } else {
            const int k = j % Ns;
            const int base = (j / Ns) * Ns * p + k;
            O[base + r * Ns] = yr;
            if (r) O[base + (p - r) * Ns] = yp;
        }
    }
}

// One CTA: g.pp pairs of rows (2 g.pp consecutive rows of the R row list).
template <int MODE, int EPI>
__global__ void __launch_bounds__(256)
dst_fft_kernel(FftGeom g, const double2* __restrict__ tw, const double* __restrict__ src,
               const double* __restrict__ sub, int sub_batches, double* __restrict__ spec,
               double* __restrict__ out, const double* __restrict__ add, int add_batches,
               const int8_t* __restrict__ mask)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* b0 = reinterpret_cast<double2*>(smem_raw);
    double2* b1 = b0 + (size_t)g.pp * g.L;
    const int L = g.L, N = g.N, n = g.n;
    const int row_base = 2 * blockIdx.x * g.pp;

    auto load = [&](int row, int p) -> double {
        if (row >= g.R) return 0.0;
        if (MODE == MODE_FWD) {
            const int f = row / g.my;
            const int j = row - f * g.my + 1;
            const long long o = f * g.fs + (long long)j * g.nx + 1 + p;
            double x = src[o];
            if (sub != nullptr && f < sub_batches) x -= sub[o];
            return x;
        } else {
            const int t = (p & 1) ? g.ne + (p >> 1) : (p >> 1);
            return spec[(long long)row * g.lds + t];
        }
    };
    for (int idx = threadIdx.x; idx < g.pp * n; idx += blockDim.x) {
        const int q = idx / n;
        const int p = idx - q * n;
        const int ra = row_base + 2 * q;
        const double xa = load(ra, p), xb = load(ra + 1, p);
        double2* Z = b0 + (size_t)q * L;
        Z[p + 1] = make_double2(xa, xb);
        Z[L - 1 - p] = make_double2(-xa, -xb);
    }
    for (int q = threadIdx.x; q < g.pp; q += blockDim.x) {
        b0[(size_t)q * L] = make_double2(0.0, 0.0);
        b0[(size_t)q * L + N] = make_double2(0.0, 0.0);
    }
    __syncthreads();
    int Ns = 1;
    for (int s = 0; s < g.nst; ++s) {
        const int R = g.rad[s];
        switch (R) {
            case 4: fft_stage<4>(b0, b1, tw, L, Ns, g.pp); break;
            case 2: fft_stage<2>(b0, b1, tw, L, Ns, g.pp); break;
            case 3: fft_stage<3>(b0, b1, tw, L, Ns, g.pp); break;
            case 5: fft_stage<5>(b0, b1, tw, L, Ns, g.pp); break;
            default:
                if (Ns == 1) fft_stage_odd<true>(b0, b1, tw, L, Ns, g.pp, R);
                else {
                    fft_expand(b0, tw, L, Ns, g.pp);
                    fft_stage_odd<false>(b0, b1, tw, L, Ns, g.pp, R);
                }
                break;
        }
        __syncthreads();
        double2* t = b0; b0 = b1; b1 = t;
        Ns *= R;
    }
    for (int idx = threadIdx.x; idx < g.pp * n; idx += blockDim.x) {
        const int q = idx / n;
        const int k = idx - q * n;
        const double2 Zm = b0[(size_t)q * L + k + 1];
        const double ys[2] = {-Zm.y * g.scale, Zm.x * g.scale};
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int row = row_base + 2 * q + u;
            if (row >= g.R) continue;
            if (MODE == MODE_FWD) {
                const int t = (k & 1) ? g.ne + (k >> 1) : (k >> 1);
                spec[(long long)row * g.lds + t] = ys[u];
            } else {
                const int f = row / g.my;
                const int j = row - f * g.my + 1;
                const long long o = f * g.fs + (long long)j * g.nx + 1 + k;
                if (EPI == EPI_H) {
                    double y = ys[u];
                    if (add != nullptr && f < add_batches) y += add[o];
                    out[o] = y;
                } else {
                    const int mi = j * g.nx + 1 + k;
                    out[o] = (mask[mi] == 3) ? ys[u] + add[o] : 0.0;
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
size_t spec_bytes(const vd_qg1l_plan* p, int nf)
{
    return size_t(nf) * p->dst.my * p->dst.lds * elem_size(p->d.dtype);
}

// Measured cost of an FP64 instruction of the FFT form over one of the dense
// form (index arithmetic, barriers between stages).
constexpr double FFT_OVER_DENSE = 1.3;

template <typename T>
static int upload(const std::vector<double>& h, void** d)
{
    std::vector<T> tmp(h.begin(), h.end());
    VD_CUDA_TRY(cudaMalloc(d, tmp.size() * sizeof(T)));
    VD_CUDA_TRY(cudaMemcpy(*d, tmp.data(), tmp.size() * sizeof(T), cudaMemcpyHostToDevice));
    return VD_OK;
}

// FFT radices for L = 2(n+1): the odd primes above 5 first, largest first (the
// first stage's odd symmetry halves its direct sums), then radix 4, 2, 3, 5.
// False when the buffers do not fit shared memory or the dense form needs
// fewer FP64 operations. Both forms are bound by the FP64 pipe, so the line is
// drawn on FP64 instructions a row: ne^2 + no^2 FMAs dense; for the FFT, half of
// L times the per-point cost of its stages (a row pair shares a transform).
// Lengths that factor into 2, 3, 5 always take the FFT. Measured solves, FFT /
// dense: n + 1 = 63 27 / 24 us, 127 50 / 34, 159 37 / 42, 191 (7 fields) 283 /
// 140, 255 (4 fields) 69 / 152, 447 156 / 194, 1023 279 / 1839; the rule picks
// the faster one of each. (These are with whole small stages, as the costs below
// count them: half stages take 52 us at 255 and 248 at 1023, and halving the costs
// would move only lengths of n <= 73, where launches are most of either time.)
static bool fft_factor(int L, std::vector<int>& rad)
{
    rad.clear();
    if (L < 4 || size_t(2) * L * sizeof(double2) > 200 * 1024) return false;
    int m = L;
    std::vector<int> small;
    while (m % 4 == 0) { small.push_back(4); m /= 4; }
    while (m % 2 == 0) { small.push_back(2); m /= 2; }
    while (m % 3 == 0) { small.push_back(3); m /= 3; }
    while (m % 5 == 0) { small.push_back(5); m /= 5; }
    for (int f = 7; m > 1; f += 2) {
        if (f * f > m) f = m;
        while (m % f == 0) { rad.push_back(f); m /= f; }
    }
    std::reverse(rad.begin(), rad.end());
    const bool odd_primes = !rad.empty();
    rad.insert(rad.end(), small.begin(), small.end());
    if (rad.size() > 24) return false;
    if (!odd_primes) return true;
    double per = 0.0;
    for (size_t i = 0; i < rad.size(); ++i) {
        const int p = rad[i], h = p / 2;
        if (p > 5) per += (i == 0 ? 2.0 * h * h / p + 4.0 : 4.0 * h * h / p + 6.0);
        else per += p == 4 ? 7.0 : p == 2 ? 4.0 : p == 3 ? 8.0 : 12.0;
    }
    const double no = (L / 2 - 1) / 2, ne = (L / 2 - 1) - no;
    return per * L / 2 * FFT_OVER_DENSE < ne * ne + no * no;
}

static int build_fft_tables(DSTTables& t)
{
    const int L = 2 * (t.n + 1);
    std::vector<int> rad;
    if (!fft_factor(L, rad)) return VD_OK;
    std::vector<double> tw(size_t(2) * L);
    for (int m = 0; m < L; ++m) {
        // e^{-2 pi i m / L} in float64 on the host
        const double a = 2.0 * M_PI * double(m) / double(L);
        tw[2 * m] = std::cos(a);
        tw[2 * m + 1] = -std::sin(a);
    }
    int rc;
    if ((rc = upload<double>(tw, &t.fft_tw))) return rc;
    t.fft_L = L;
    t.fft_nst = (int)rad.size();
    for (size_t i = 0; i < rad.size(); ++i) t.fft_rad[i] = rad[i];
    return VD_OK;
}

int build_dst_tables(vd_qg1l_plan* p)
{
    DSTTables& t = p->dst;
    const int n = p->d.nx - 2;
    const int my = p->d.ny - 2;
    t.n = n;
    t.my = my;
    t.no = n / 2;
    t.ne = n - t.no;
    t.ncol_tiles = (t.ne + DST_NC - 1) / DST_NC;
    t.kpad = ((t.ne + DST_KC - 1) / DST_KC) * DST_KC;
    t.ldw = t.ncol_tiles * DST_NC;
    t.lds = ((n + 3) / 4) * 4;

    const double scale = std::sqrt(2.0 / (n + 1));
    const long long period = 2LL * (n + 1);   // sin(pi*m/(n+1)) has period 2(n+1) in m
    auto s = [&](long long m) {
        m %= period;
        return scale * std::sin(M_PI * double(m) / double(n + 1));
    };
    std::vector<double> wodd(size_t(t.kpad) * t.ldw, 0.0), woddT(wodd.size(), 0.0),
        weven(wodd.size(), 0.0);
    for (int a = 0; a < t.ne; ++a)
        for (int b = 0; b < t.ne; ++b) {
            const double v = s((long long)(a + 1) * (2 * b + 1));
            wodd[size_t(a) * t.ldw + b] = v;
            woddT[size_t(b) * t.ldw + a] = v;
        }
    for (int a = 0; a < t.no; ++a)
        for (int b = 0; b < t.no; ++b)
            weven[size_t(a) * t.ldw + b] = s((long long)(a + 1) * (2 * b + 2));

    // Thomas multipliers per spectral column (parity-split order)
    const double gf = p->d.g / p->d.f;
    const double gfc2 = p->d.g * p->d.f / (p->d.c * p->d.c);
    const double dx = p->d.dx, dy = p->d.dy;
    const double a = gf / (dy * dy);
    t.tri_a = a;
    std::vector<double> trim(size_t(my) * t.lds, 0.0);
    for (int col = 0; col < n; ++col) {
        const int k = col < t.ne ? 2 * col : 2 * (col - t.ne) + 1;   // 0-based wavenumber
        const double mu = 2.0 * (std::cos(M_PI / (p->d.nx - 1) * (k + 1)) - 1.0) / (dx * dx);
        const double bk = gf * (-2.0 / (dy * dy) + mu) - gfc2;
        double c_prev = 0.0;
        for (int j = 0; j < my; ++j) {
            const double m = 1.0 / (bk - a * c_prev);
            trim[size_t(j) * t.lds + col] = m;
            c_prev = a * m;
        }
    }
    int rc;
    if (p->d.dtype == VD_F64 && (rc = build_fft_tables(t))) return rc;
    if (p->d.dtype == VD_F32) {
        if ((rc = upload<float>(wodd, &t.Wodd))) return rc;
        if ((rc = upload<float>(woddT, &t.WoddT))) return rc;
        if ((rc = upload<float>(weven, &t.Weven))) return rc;
        if ((rc = upload<float>(trim, &t.trim))) return rc;
    } else {
        if ((rc = upload<double>(wodd, &t.Wodd))) return rc;
        if ((rc = upload<double>(woddT, &t.WoddT))) return rc;
        if ((rc = upload<double>(weven, &t.Weven))) return rc;
        if ((rc = upload<double>(trim, &t.trim))) return rc;
        if (my <= TRI_TAB_MAX) {
            VD_CUDA_TRY(cudaMalloc(&t.tri_tab, 4 * trim.size() * sizeof(double)));
            tridiag_tables_kernel<<<dim3((n + 127) / 128, (my + TRI_TAB_ROWS - 1) / TRI_TAB_ROWS), 128>>>(
                (const double*)t.trim, (double*)t.tri_tab, my, n, t.lds, a);
            VD_LAUNCH_CHECK();
            VD_CUDA_TRY(cudaStreamSynchronize(0));
        }
    }
    return VD_OK;
}

void free_dst_tables(vd_qg1l_plan* p)
{
    cudaFree(p->dst.Wodd);
    cudaFree(p->dst.WoddT);
    cudaFree(p->dst.Weven);
    cudaFree(p->dst.trim);
    if (p->dst.tri_tab) cudaFree(p->dst.tri_tab);
    cudaFree(p->dst.fft_tw);
}

template <typename T, int TR>
static cudaError_t set_smem_attrs()
{
    const int maxb = 227 * 1024;
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(dst_gemm_kernel<T, TR, MODE_FWD, EPI_H>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, maxb))) return e;
    if ((e = cudaFuncSetAttribute(dst_gemm_kernel<T, TR, MODE_INV, EPI_H>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, maxb))) return e;
    return cudaFuncSetAttribute(dst_gemm_kernel<T, TR, MODE_INV, EPI_ADJQ>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, maxb);
}

template <int R, int CWC, int RG = 4 / CWC, bool PF = false>
static cudaError_t set_smem_dense64()
{
    const int maxb = 200 * 1024;   // plus the exchange tile in static shared memory
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(dst_dense64_kernel<R, CWC, RG, PF, MODE_FWD, EPI_H>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, maxb))) return e;
    if ((e = cudaFuncSetAttribute(dst_dense64_kernel<R, CWC, RG, PF, MODE_INV, EPI_H>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, maxb))) return e;
    return cudaFuncSetAttribute(dst_dense64_kernel<R, CWC, RG, PF, MODE_INV, EPI_ADJQ>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, maxb);
}

// The y-direction tridiagonal solves of nf fields: 8 columns per CTA,
// pieces of 16 rows (32 for fields of 1025-2048 rows; 8, in up to 32 warps,
// as a schedule choice for fields of up to 1024 rows) in at most 16 warps;
// taller fields fall back to one sequential thread per column. (Measured on
// GB300 against 32- and 16-column groups, shared-memory staging and a
// warp-shuffle chain of the pieces: this form is the fastest or tied at both
// 16 x 510^2 and 1 x 1022^2.)
template <typename T>
static int launch_tridiag(const vd_qg1l_plan* p, int nf, T* spec, cudaStream_t st)
{
    const DSTTables& t = p->dst;
    const T a = (T)t.tri_a;
    constexpr int CW = 8, SUB = 32 / CW;
    const dim3 grid((t.n + CW - 1) / CW, nf);
    const int nw8 = ((t.my + 7) / 8 + SUB - 1) / SUB;
    const int nw16 = ((t.my + 15) / 16 + SUB - 1) / SUB;
    const int nw32 = ((t.my + 31) / 32 + SUB - 1) / SUB;
    const bool want32 = p->sched.tridiag_rows == 32 && nw32 <= 16;
    const bool want8 = p->sched.tridiag_rows == 8 && nw8 <= 32;
    if constexpr (sizeof(T) == 8) {
        // the table form, unless the schedule asks for another piece length
        if (t.tri_tab && (p->sched.tridiag_rows == 0 || p->sched.tridiag_rows == TRI_TAB_ROWS)) {
            tridiag_tab_kernel<CW, TRI_TAB_ROWS><<<grid, dim3(32, nw8), 2 * nw8 * CW * sizeof(T), st>>>(
                spec, (const double*)t.tri_tab, t.my, t.n, t.lds);
            VD_LAUNCH_CHECK();
            return VD_OK;
        }
    }
    if (want8) {
        tridiag_chunked_kernel<T, CW, 8><<<grid, dim3(32, nw8), 2 * nw8 * CW * sizeof(T), st>>>(
            spec, (const T*)t.trim, t.my, t.n, t.lds, a);
    } else if (nw16 <= 16 && !want32 && p->sched.tridiag_lean == 1 && sizeof(T) == 4) {
        tridiag_chunked_kernel<T, CW, 16, true><<<grid, dim3(32, nw16), 2 * nw16 * CW * sizeof(T), st>>>(
            spec, (const T*)t.trim, t.my, t.n, t.lds, a);
    } else if (nw16 <= 16 && !want32) {
        tridiag_chunked_kernel<T, CW, 16><<<grid, dim3(32, nw16), 2 * nw16 * CW * sizeof(T), st>>>(
            spec, (const T*)t.trim, t.my, t.n, t.lds, a);
    } else if (nw32 <= 16) {
        tridiag_chunked_kernel<T, CW, 32><<<grid, dim3(32, nw32), 2 * nw32 * CW * sizeof(T), st>>>(
            spec, (const T*)t.trim, t.my, t.n, t.lds, a);
    } else {
        tridiag_global_kernel<T><<<dim3((t.n + 31) / 32, nf), 32, 0, st>>>(spec, (const T*)t.trim, t.my, t.n,
                                                                           t.lds, a);
    }
    VD_LAUNCH_CHECK();
    return VD_OK;
}

static PerDeviceOnce g_attr_once;

static cudaError_t configure_kernels()
{
    return g_attr_once.run([]() -> cudaError_t {
        cudaError_t e = cudaSuccess;
        if (!e) e = set_smem_attrs<float, 16>();
        if (!e) e = set_smem_attrs<float, 32>();
        if (!e) e = set_smem_attrs<float, 64>();
        if (!e) e = set_smem_dense64<1, 2>();
        if (!e) e = set_smem_dense64<1, 2, 2, true>();
        if (!e) e = set_smem_dense64<1, 2, 1, true>();
        if (!e) e = set_smem_dense64<2, 2>();
        if (!e) e = set_smem_dense64<4, 2>();
        if (!e) e = set_smem_dense64<2, 4>();
        if (!e) e = set_smem_dense64<4, 4>();
        const int maxb = 227 * 1024;
        if (!e) e = cudaFuncSetAttribute(dst_fft_kernel<MODE_FWD, EPI_H>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, maxb);
        if (!e) e = cudaFuncSetAttribute(dst_fft_kernel<MODE_INV, EPI_H>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, maxb);
        if (!e) e = cudaFuncSetAttribute(dst_fft_kernel<MODE_INV, EPI_ADJQ>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, maxb);
        return e;
    });
}

template <typename T, int TR>
static int launch_pair(const vd_qg1l_plan* p, const GemmGeom& g, const SolveArgs& a,
                       T* spec, cudaStream_t st, bool fwd)
{
    const DSTTables& t = p->dst;
    constexpr int NT = GemmShape<TR>::NT;
    const size_t smem = gemm_smem_elems<T, TR>(g.kpad) * sizeof(T);
    dim3 grid(t.ncol_tiles, (g.R + TR - 1) / TR);
    if (fwd) {
        dst_gemm_kernel<T, TR, MODE_FWD, EPI_H><<<grid, NT, smem, st>>>(
            g, (const T*)t.Wodd, (const T*)t.Weven, (const T*)a.src, (const T*)a.sub,
            a.sub_batches, spec, nullptr, nullptr, 0, nullptr);
    } else if (a.epi == EPI_H) {
        dst_gemm_kernel<T, TR, MODE_INV, EPI_H><<<grid, NT, smem, st>>>(
            g, (const T*)t.WoddT, (const T*)t.Weven, nullptr, nullptr, 0, spec, (T*)a.out,
            (const T*)a.add, a.add_batches, p->d_mask);
    } else {
        dst_gemm_kernel<T, TR, MODE_INV, EPI_ADJQ><<<grid, NT, smem, st>>>(
            g, (const T*)t.WoddT, (const T*)t.Weven, nullptr, nullptr, 0, spec, (T*)a.out,
            (const T*)a.add, a.add_batches, p->d_mask);
    }
    VD_LAUNCH_CHECK();
    return VD_OK;
}

template <int R, int CWC, int RG, bool PF>
static int launch_dense64_rg(const vd_qg1l_plan* p, const GemmGeom& g, const SolveArgs& a, double* spec,
                             cudaStream_t st, bool fwd)
{
    const DSTTables& t = p->dst;
    constexpr int TR = R * RG, NC = 32 * CWC, NT = 64 * CWC * RG;
    const size_t smem = (size_t)t.n * TR * sizeof(double);
    // one dimension: the row tiles of a large batch exceed the 65535 blocks of y and z
    const dim3 grid((unsigned)((t.ne + NC - 1) / NC) * (unsigned)((g.R + TR - 1) / TR));
    const double *Wo = (const double*)t.Wodd, *WoT = (const double*)t.WoddT, *We = (const double*)t.Weven;
    if (fwd)
        dst_dense64_kernel<R, CWC, RG, PF, MODE_FWD, EPI_H><<<grid, NT, smem, st>>>(
            g, Wo, We, (const double*)a.src, (const double*)a.sub, a.sub_batches, spec, nullptr, nullptr, 0, nullptr);
    else if (a.epi == EPI_H)
        dst_dense64_kernel<R, CWC, RG, PF, MODE_INV, EPI_H><<<grid, NT, smem, st>>>(
            g, WoT, We, nullptr, nullptr, 0, spec, (double*)a.out, (const double*)a.add, a.add_batches, p->d_mask);
    else
        dst_dense64_kernel<R, CWC, RG, PF, MODE_INV, EPI_ADJQ><<<grid, NT, smem, st>>>(
            g, WoT, We, nullptr, nullptr, 0, spec, (double*)a.out, (const double*)a.add, a.add_batches, p->d_mask);
    VD_LAUNCH_CHECK();
    return VD_OK;
}

// Row groups a CTA: 4 / CWC (8 warps), or one where that leaves SMs without a CTA and
// twice the CTAs still fit one wave (a scheduler's time is its warps' FMAs). W is
// prefetched up to four warps a scheduler: solves of one 126, 190, 222 and 382-mode
// field with / without: 18.4 / 27.0 us (and one row a CTA), 36.5 / 40.7, 41.2 / 46.1 and
// 116.3 / 115.1.
template <int R, int CWC>
static int launch_dense64_rc(const vd_qg1l_plan* p, const GemmGeom& g, const SolveArgs& a, double* spec,
                             cudaStream_t st, bool fwd)
{
    if constexpr (R == 1) {
        const long long ctas = (long long)((p->dst.ne + 32 * CWC - 1) / (32 * CWC)) * g.R;   // at one row a CTA
        if (ctas <= 152) return launch_dense64_rg<R, CWC, 1, true>(p, g, a, spec, st, fwd);
        if (2LL * ((p->dst.ne + 31) / 32) * g.R <= 4 * 608)
            return launch_dense64_rg<R, CWC, 4 / CWC, true>(p, g, a, spec, st, fwd);
    }
    return launch_dense64_rg<R, CWC, 4 / CWC, false>(p, g, a, spec, st, fwd);
}

// Rows a warp: as many as leave about four warps to each of the 608 schedulers
// (R FMAs share one W load); column groups a CTA: enough to cover the columns.
static int launch_dense64(const vd_qg1l_plan* p, const GemmGeom& g, const SolveArgs& a, double* spec,
                          cudaStream_t st, bool fwd)
{
    const int cols = (p->dst.ne + 31) / 32;
    const long long w1 = 2LL * cols * g.R;               // warps at one row each
    const int R = w1 >= 4 * 608 * 4 ? 4 : w1 >= 2 * 608 * 4 ? 2 : 1;
    if (cols == 1) {
        if (R == 4) return launch_dense64_rc<4, 1>(p, g, a, spec, st, fwd);
        if (R == 2) return launch_dense64_rc<2, 1>(p, g, a, spec, st, fwd);
        return launch_dense64_rc<1, 1>(p, g, a, spec, st, fwd);
    }
    if (cols == 2 || R == 1) {
        if (R == 4) return launch_dense64_rc<4, 2>(p, g, a, spec, st, fwd);
        if (R == 2) return launch_dense64_rc<2, 2>(p, g, a, spec, st, fwd);
        return launch_dense64_rc<1, 2>(p, g, a, spec, st, fwd);
    }
    if (R == 4) return launch_dense64_rc<4, 4>(p, g, a, spec, st, fwd);
    return launch_dense64_rc<2, 4>(p, g, a, spec, st, fwd);
}

// The float64 FFT pass over g.R rows: pairs of rows per CTA chosen for about
// two CTAs per SM-wave slot and at most ~100 KB of shared memory per CTA.
static int launch_fft(const vd_qg1l_plan* p, const GemmGeom& g, const SolveArgs& a, double* spec,
                      cudaStream_t st, bool fwd)
{
    const DSTTables& t = p->dst;
    FftGeom fg;
    fg.L = t.fft_L; fg.N = t.n + 1; fg.n = t.n; fg.ne = t.ne; fg.my = t.my; fg.nx = g.nx;
    fg.R = g.R; fg.lds = t.lds; fg.nst = t.fft_nst; fg.fs = g.fs;
    fg.scale = 0.5 * std::sqrt(2.0 / double(t.n + 1));
    for (int i = 0; i < 24; ++i) fg.rad[i] = t.fft_rad[i];
    const int pairs = (g.R + 1) / 2;
    const size_t per_pair = size_t(2) * t.fft_L * sizeof(double2);
    int pp = std::max(1, std::min<int>(8, int((100 * 1024) / per_pair)));
    pp = std::max(1, std::min(pp, pairs / (2 * 152)));
    fg.pp = pp;
    const size_t smem = per_pair * pp;
    const dim3 grid((pairs + pp - 1) / pp);
    const double2* tw = (const double2*)t.fft_tw;
    if (fwd) {
        dst_fft_kernel<MODE_FWD, EPI_H><<<grid, 256, smem, st>>>(fg, tw, (const double*)a.src,
                                                                 (const double*)a.sub, a.sub_batches, spec,
                                                                 nullptr, nullptr, 0, nullptr);
    } else if (a.epi == EPI_H) {
        dst_fft_kernel<MODE_INV, EPI_H><<<grid, 256, smem, st>>>(fg, tw, nullptr, nullptr, 0, spec, (double*)a.out,
                                                                 (const double*)a.add, a.add_batches, p->d_mask);
    } else {
        dst_fft_kernel<MODE_INV, EPI_ADJQ><<<grid, 256, smem, st>>>(fg, tw, nullptr, nullptr, 0, spec,
                                                                    (double*)a.out, (const double*)a.add,
                                                                    a.add_batches, p->d_mask);
    }
    VD_LAUNCH_CHECK();
    return VD_OK;
}

// Rows per CTA: the largest tile that still gives about two waves of CTAs on
// the 152 SMs and fits shared memory.
static int pick_tr(const vd_qg1l_plan* p, int R)
{
    const DSTTables& t = p->dst;
    if (p->sched.fma_rows) return p->sched.fma_rows;
    const int cand[3] = {64, 32, 16};
    for (int c : cand) {
        const size_t smem = (size_t(2) * t.kpad * c + size_t(std::max(2 * DST_KC * DST_NC, c * DST_NC))) * sizeof(float);
        if (smem > 200 * 1024) continue;
        const long long ctas = (long long)t.ncol_tiles * ((R + c - 1) / c);
        if (ctas >= 2 * 152) return c;
    }
    return 16;
}

// Whether a length with an FFT takes the dense form all the same: the rows are so few
// that it runs as one wave of one-row CTAs, a warp a scheduler, and a half sum of up to
// 120 FMAs is shorter than the FFT's chain of stages and barriers. Solves of one field,
// dense / FFT: 40 x 46 11.7 / 21.0 us, 64^2 + 1 13.0 / 20.3, 96^2 16.2 / 23.5, 128^2 + 1
// 18.4 / 22.9, 52 x 193 22.1 / 24.1, 40 x 241 25.0 / 26.1, 40 x 257 26.0 / 24.9, 24 x 385
// 34.4 / 28.4.
static bool dense64_few(const vd_qg1l_plan* p, const GemmGeom& g)
{
    if (p->dst.ne > 120) return false;
    const int cols = (p->dst.ne + 31) / 32, cwc = cols == 1 ? 1 : 2;
    return (long long)((cols + cwc - 1) / cwc) * g.R <= 152;
}

// One x-direction pass: float32 on the tensor cores or CUDA-core FMA, float64
// as FFT or dense products.
template <typename T>
static int dst_pass(const vd_qg1l_plan* p, int nf, const GemmGeom& g, const SolveArgs& a, T* spec, cudaStream_t st,
                    bool fwd)
{
    if constexpr (sizeof(T) == 4) {
        if (use_tc(p, nf)) return dst_pass_tc(p, nf, a, spec, fwd, st);
        const int tr = pick_tr(p, g.R);
        if (tr == 64) return launch_pair<T, 64>(p, g, a, spec, st, fwd);
        if (tr == 32) return launch_pair<T, 32>(p, g, a, spec, st, fwd);
        return launch_pair<T, 16>(p, g, a, spec, st, fwd);
    } else {
        if (p->dst.fft_L && !dense64_few(p, g)) return launch_fft(p, g, a, spec, st, fwd);
        return launch_dense64(p, g, a, spec, st, fwd);
    }
}

template <typename T>
int helmholtz_solve(const vd_qg1l_plan* p, int nf, const SolveArgs& a, T* spec, cudaStream_t st)
{
    if (configure_kernels() != cudaSuccess) return VD_ERR_CUDA;
    const DSTTables& t = p->dst;
    GemmGeom g;
    g.n = t.n; g.ne = t.ne; g.no = t.no; g.my = t.my; g.nx = p->d.nx;
    g.fs = (long long)p->d.ny * p->d.nx;
    g.R = nf * t.my;
    g.kpad = t.kpad; g.ldw = t.ldw; g.lds = t.lds;
    int rc;
    if constexpr (sizeof(T) == 4) {
        bool done = false;
        if (use_tc(p, nf) && (rc = dst_solve_tc(p, nf, a, spec, &done, st))) return rc;
        if (done) return dst_pass<T>(p, nf, g, a, spec, st, false);
    }
    if ((rc = dst_pass<T>(p, nf, g, a, spec, st, true))) return rc;
    if ((rc = launch_tridiag<T>(p, nf, spec, st))) return rc;
    return dst_pass<T>(p, nf, g, a, spec, st, false);
}

template int helmholtz_solve<float>(const vd_qg1l_plan*, int, const SolveArgs&, float*, cudaStream_t);
template int helmholtz_solve<double>(const vd_qg1l_plan*, int, const SolveArgs&, double*, cudaStream_t);

// The x-direction DST-I pass alone (forward: field interior -> spectral rows;
// inverse: spectral rows -> field interior).
template <typename T>
int dst_x_only(const vd_qg1l_plan* p, int nf, const T* field, T* spec, int inverse, T* out, cudaStream_t st)
{
    if (configure_kernels() != cudaSuccess) return VD_ERR_CUDA;
    const DSTTables& t = p->dst;
    GemmGeom g;
    g.n = t.n; g.ne = t.ne; g.no = t.no; g.my = t.my; g.nx = p->d.nx;
    g.fs = (long long)p->d.ny * p->d.nx;
    g.R = nf * t.my;
    g.kpad = t.kpad; g.ldw = t.ldw; g.lds = t.lds;
    SolveArgs a;
    a.src = field; a.sub = nullptr; a.sub_batches = 0;
    a.out = out; a.add = nullptr; a.add_batches = 0; a.epi = EPI_H;
    if (inverse == 2) {            // adjoint epilogue: out = M3 * (x + field)
        a.src = nullptr;
        a.add = field; a.add_batches = nf; a.epi = EPI_ADJQ;
    }
    return dst_pass<T>(p, nf, g, a, spec, st, !inverse);
}

// The y-direction tridiagonal solve alone, in place on spectral rows.
template <typename T>
int tridiag_only(const vd_qg1l_plan* p, int nf, T* spec, cudaStream_t st)
{
    if (configure_kernels() != cudaSuccess) return VD_ERR_CUDA;
    return launch_tridiag<T>(p, nf, spec, st);
}

template int tridiag_only<float>(const vd_qg1l_plan*, int, float*, cudaStream_t);
template int tridiag_only<double>(const vd_qg1l_plan*, int, double*, cudaStream_t);
template int dst_x_only<float>(const vd_qg1l_plan*, int, const float*, float*, int, float*, cudaStream_t);
template int dst_x_only<double>(const vd_qg1l_plan*, int, const double*, double*, int, double*, cudaStream_t);

}  // namespace vd
