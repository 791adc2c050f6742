// Gaussian space-time reduced basis: phi = G(t) X and adX += G(t)^T adphi.
//
// Reference: mapping/src/basis.py, Basis_gauss3d (1170-1555) and Basis_multi
// (4039-4135). The reference stores each component's space part as a CSC
// matrix Gauss_xy [nphys x Nx] and its time part as one weight per
// (time centre, basis time); operg is Gauss_xy . (sum over active time
// centres of g_it X[it, :]).
//
// Here the grid is rectilinear (x/longitude per column, y/latitude per row),
// so every footprint factorises: a centre (row j of the lattice, centre i of
// that row) contributes wy_j(y) * wx_{j,i}(x) at grid point (y, x), where
// wy_j(y) = mywindow((y - lat_j)/km2deg / sigma_D) and wx the same in x with
// the cos(lat_j) stretch (basis.py:1403-1419). The product is then two banded
// passes instead of a sparse matrix:
//   x pass  T[r][x]  = sum_i wx_{r,i}(x) * (sum_a g_a X[it_a, cb_r + i])   (r: lattice row)
//   y pass  phi[y][x] = land ? 0 : sum_g sum_j wy_{g,j}(y) T[row(g, j)][x]  (g: group of components)
// and the transpose runs them backwards:
//   y^T     U[r][x]  = sum_y wy_r(y) * (land ? 0 : adphi[y][x])
//   x^T     adX[it_a, cb_r + i] += g_a * sum_x wx_{r,i}(x) U[r][x]
// Every output is written by one thread (no atomics): results are
// deterministic. Tables are built on the host in float64 with the
// reference's formulas (including NumPy's arange/linspace value sequences),
// so footprint membership and weights match the reference's CSC entries.
#include "vd_internal.cuh"
#include "vd_basis_host.h"
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <new>
#include <tuple>
#include <vector>

namespace {

using namespace vd::basis_host;

struct HostComp {
    vd_gauss3d_params p;
    double norm_fact = 1.0;
    std::vector<double> enst;        // time centres
    std::vector<double> rows_lat;    // lattice rows (ENSLAT1)
    std::vector<int> row_n;          // centres per lattice row
    std::vector<long long> row_cb;   // first centre index of each row
    std::vector<double> enslat, enslon;
    long long Nx = 0;                // space centres
    long long boff = 0;              // offset of the component in X
    double window(double x) const { return p.flux ? mywindow_flux(x) : mywindow(x); }
};

}  // namespace

struct vd_basis_plan {
    int ny = 0, nx = 0, dtype = VD_F32, geographic = 0, host_only = 0;
    int ncomp = 0, ntime = 0;
    long long nbasis = 0;
    int R = 0;          // lattice rows over all groups
    int KX = 0;         // ELL width of the x table
    int ngrp = 0;       // groups of components on the same space lattice
    int NA = 0;         // max active time centres per (time, component)
    int gzT = 1;        // blocks along a row's centres of the transposed x pass
    bool longY = false, longYT = false;   // y lists of eight entries and more
    std::vector<HostComp> comps;
    std::vector<double> times;
    // time weights [ntime][ncomp][NA]
    std::vector<int> tact_n, tact_it;
    std::vector<double> tact_g;
    // device tables (one allocation)
    void* dev = nullptr;
    // pointers into dev
    const int32_t *row_grp, *row_pat, *row_n, *row_lg, *fx_i, *xr, *yl_ptr, *yl_row, *ty_ptr, *ty_row, *tx_ptr,
        *tx_col, *pat_cbase, *te_ptr;
    const long long *row_cb, *te_off;
    const void *fx_w, *yl_w, *ty_w, *tx_w, *te_w;
    const int8_t* land;
};

namespace vd {

template <typename T>
struct BasisDev {
    int ny, nx, R, KX, ngrp;
    const int32_t *row_grp, *row_pat, *row_n, *row_lg, *fx_i, *xr, *yl_ptr, *yl_row, *ty_ptr, *ty_row, *tx_ptr,
        *tx_col, *pat_cbase, *te_ptr;
    const long long *row_cb, *te_off;
    const T *fx_w, *yl_w, *ty_w, *tx_w, *te_w;
    const int8_t* land;
};

template <typename T>
BasisDev<T> dev_view(const vd_basis_plan* p)
{
    BasisDev<T> d;
    d.ny = p->ny; d.nx = p->nx; d.R = p->R; d.KX = p->KX; d.ngrp = p->ngrp;
    d.row_grp = p->row_grp; d.row_pat = p->row_pat; d.row_n = p->row_n; d.row_lg = p->row_lg;
    d.fx_i = p->fx_i; d.xr = p->xr; d.yl_ptr = p->yl_ptr; d.yl_row = p->yl_row; d.ty_ptr = p->ty_ptr;
    d.ty_row = p->ty_row; d.tx_ptr = p->tx_ptr; d.tx_col = p->tx_col; d.pat_cbase = p->pat_cbase;
    d.te_ptr = p->te_ptr; d.row_cb = p->row_cb; d.te_off = p->te_off;
    d.fx_w = (const T*)p->fx_w; d.yl_w = (const T*)p->yl_w; d.ty_w = (const T*)p->ty_w;
    d.tx_w = (const T*)p->tx_w; d.te_w = (const T*)p->te_w;
    d.land = p->land;
    return d;
}

// Components on the same space lattice (equal sigma_D and facns: the usual set of
// time scales per space scale) form a group: their coefficients are summed over
// the active time centres of all of them before the x pass, and G^T's space
// products are formed once. Rows, y tables and the workspace are per group; the
// active (component, time centre) entries of a basis time are one list per group.
//
// The passes are bound by load latency (the fields stay in L2), so every list is
// read eight entries at a time: the index loads (the same for all threads) and then
// the field loads of a batch are in flight together.
template <typename T, int U, typename F>
__device__ __forceinline__ void list_batch(T& acc, int e, int e1, const int32_t* __restrict__ idx,
                                           const T* __restrict__ w, F&& load)
{
    int j[U];
    T c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const bool on = e + u < e1;
        j[u] = on ? __ldg(idx + e + u) : -1;
        c[u] = on ? __ldg(w + e + u) : T(0);
    }
    T v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = j[u] >= 0 ? load(j[u]) : T(0);
#pragma unroll
    for (int u = 0; u < U; ++u) acc += c[u] * v[u];
}
// LONG: lists of eight entries and more on average; short ones do with fewer registers
// (more warps an SM). The rest of a list is padded to four entries in float32; in
// float64, bound by the FP64 pipe, it is taken as 4 + 2 + 1.
template <typename T, bool LONG, typename F>
__device__ __forceinline__ T list_sum(int e, int e1, const int32_t* __restrict__ idx, const T* __restrict__ w, F&& load)
{
    T acc = T(0);
    if constexpr (LONG)
        for (; e1 - e >= 8; e += 8) list_batch<T, 8>(acc, e, e1, idx, w, load);
    if constexpr (sizeof(T) == 4) {
        for (; e < e1; e += 4) list_batch<T, 4>(acc, e, e1, idx, w, load);
    } else {
        for (; e1 - e >= 4; e += 4) list_batch<T, 4>(acc, e, e1, idx, w, load);
        if (e1 - e >= 2) {
            list_batch<T, 2>(acc, e, e1, idx, w, load);
            e += 2;
        }
        if (e < e1) list_batch<T, 1>(acc, e, e1, idx, w, load);
    }
    return acc;
}

// x pass of G: one thread per (group row r, column x, window b). The block first
// sums over the group's entries the coefficients of the centres that its columns
// reach (xr), warps taking every fourth entry, 128 centres at a time. float32, 9
// components in 3 groups at 1024^2 3.9 us (7.8 a component at a time); 8 windows of
// 512^2, centres 5.3 km apart on 5 km columns, 22 us (32, and 107 with the sums of whole
// rows of centres in every block).
constexpr int BX_NT = 128, BX_Z = 128;

template <typename T>
__global__ void __launch_bounds__(BX_NT)
k_basis_xpass(BasisDev<T> d, int k, const T* __restrict__ X, long long ldX, T* __restrict__ Tw)
{
    __shared__ T zp[4][BX_Z];
    const int x = blockIdx.x * BX_NT + threadIdx.x;
    const int r = blockIdx.y, b = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pat = d.row_pat[r], g = d.row_grp[r];
    const int lo = d.xr[2 * (pat * gridDim.x + blockIdx.x)], hi = d.xr[2 * (pat * gridDim.x + blockIdx.x) + 1];
    const int f1 = d.te_ptr[k * d.ngrp + g + 1], f0 = d.te_ptr[k * d.ngrp + g];
    const T* Xr = X + (long long)b * ldX + d.row_cb[r];
    const long long e0 = x < d.nx ? ((long long)pat * d.nx + x) * d.KX : 0;
    T acc = T(0);
    for (int i0 = lo; i0 < hi; i0 += BX_Z) {
        T z[BX_Z / 32] = {};
#pragma unroll 4
        for (int f = f0 + warp; f < f1; f += 4) {
            const T* p = Xr + __ldg(d.te_off + f) + i0 + lane;
            const T w = __ldg(d.te_w + f);
#pragma unroll
            for (int u = 0; u < BX_Z / 32; ++u)
                if (i0 + 32 * u + lane < hi) z[u] += w * p[32 * u];
        }
        if (i0 > lo) __syncthreads();
#pragma unroll
        for (int u = 0; u < BX_Z / 32; ++u) zp[warp][32 * u + lane] = z[u];
        __syncthreads();
        auto sum = [&](int i) { return (zp[0][i] + zp[1][i]) + (zp[2][i] + zp[3][i]); };
        if constexpr (sizeof(T) == 8) {          // once a centre: an FP64 addition costs more than a barrier
            zp[0][threadIdx.x] = sum(threadIdx.x);
            __syncthreads();
        }
        if (x < d.nx)
            for (int e = 0; e < d.KX; ++e) {
                const int i = d.fx_i[e0 + e] - i0;
                if (i + i0 < 0) break;
                if (i >= 0 && i < BX_Z) acc += d.fx_w[e0 + e] * (sizeof(T) == 8 ? zp[0][i] : sum(i));
            }
    }
    if (x < d.nx) Tw[((long long)b * d.R + r) * d.nx + x] = acc;
}

// y pass of G: one thread per (y, x, b), summing every group in order. 9 components at
// 1024^2 in float32 10.7 us (40 with a loop per component; 11.8 with the list staged in
// shared memory, whose barriers cost short lists 8 %).
template <typename T, bool LONG>
__global__ void __launch_bounds__(BX_NT)
k_basis_ypass(BasisDev<T> d, const T* __restrict__ Tw, T* __restrict__ phi, int accumulate)
{
    const int x = blockIdx.x * BX_NT + threadIdx.x;
    const int y = blockIdx.y, b = blockIdx.z;
    if (x >= d.nx) return;
    const T* Tb = Tw + (long long)b * d.R * d.nx + x;
    T acc = list_sum<T, LONG>(d.yl_ptr[y], d.yl_ptr[y + 1], d.yl_row, d.yl_w, [&](int j) { return Tb[(long long)j * d.nx]; });
    const long long o = ((long long)b * d.ny + y) * d.nx + x;
    if (d.land && d.land[(long long)y * d.nx + x]) acc = T(0);
    phi[o] = accumulate ? phi[o] + acc : acc;
}

// y pass of G^T: U[r][x] = sum_y wy adphi (land masked out). LONG: the block stages the
// list in shared memory, 128 entries at a time (two loads less an entry and thread: 9
// components at 1024^2 8.4 us for 11.8; with 8 entries 6.8 for 7.6 at 8 x 512^2, with 3
// entries 14.5 for 11.0, so that short lists are read directly).
template <typename T, bool LONG>
__global__ void __launch_bounds__(BX_NT)
k_basisT_ypass(BasisDev<T> d, const T* __restrict__ adphi, T* __restrict__ Uw)
{
    const int x = blockIdx.x * BX_NT + threadIdx.x;
    const int r = blockIdx.y, b = blockIdx.z;
    const T* a = adphi + (long long)b * d.ny * d.nx + x;
    const int8_t* land = d.land ? d.land + x : nullptr;
    const int e0 = d.ty_ptr[r], e1 = d.ty_ptr[r + 1];
    T acc = T(0);
    if constexpr (LONG) {
        __shared__ int y_s[BX_NT];
        __shared__ T w_s[BX_NT];
        for (int e = e0; e < e1; e += BX_NT) {
            const int n = min(BX_NT, e1 - e);
            __syncthreads();
            if (threadIdx.x < n) {
                y_s[threadIdx.x] = d.ty_row[e + threadIdx.x];
                w_s[threadIdx.x] = d.ty_w[e + threadIdx.x];
            }
            __syncthreads();
            if (x < d.nx) {
                if (land) {
#pragma unroll 8
                    for (int u = 0; u < n; ++u) {
                        const long long o = (long long)y_s[u] * d.nx;
                        const T v = a[o];
                        acc += w_s[u] * (land[o] ? T(0) : v);
                    }
                } else {
#pragma unroll 8
                    for (int u = 0; u < n; ++u) acc += w_s[u] * a[(long long)y_s[u] * d.nx];
                }
            }
        }
        if (x >= d.nx) return;
    } else {
        if (x >= d.nx) return;
        if (land)
            acc = list_sum<T, false>(e0, e1, d.ty_row, d.ty_w, [&](int y) {
                const long long o = (long long)y * d.nx;
                const T v = a[o];
                return land[o] ? T(0) : v;
            });
        else
            acc = list_sum<T, false>(e0, e1, d.ty_row, d.ty_w, [&](int y) { return a[(long long)y * d.nx]; });
    }
    Uw[((long long)b * d.R + r) * d.nx + x] = acc;
}

// x pass of G^T. A block forms the space products of a run of centres of row r, each
// by 2^lg lanes over the centre's consecutive columns (up to eight a lane), and adds
// them to the coefficients of every entry, centres along the lanes. With a warp a centre
// everywhere the few columns of a fine lattice left its lanes idle and its additions
// were scattered: 8 x 512^2, centres 5.3 km apart on 5 km columns, 315 us, here 24; 9
// components at 1024^2 9.2 us, here 5.7.
__host__ __device__ constexpr int bxT_centres(int lg) { return lg < 4 ? BX_NT >> lg : 8; }   // of a block

template <typename T>
__global__ void __launch_bounds__(BX_NT)
k_basisT_xpass(BasisDev<T> d, int k, const T* __restrict__ Uw, T* __restrict__ adX, long long ldX)
{
    __shared__ T ss[BX_NT];
    const int r = blockIdx.x, b = blockIdx.y, lg = d.row_lg[r], nc = bxT_centres(lg);
    const int i0 = blockIdx.z * nc, n = min(nc, d.row_n[r] - i0);
    if (n <= 0) return;
    const int g = d.row_grp[r], f0 = d.te_ptr[k * d.ngrp + g], f1 = d.te_ptr[k * d.ngrp + g + 1];
    const T* U = Uw + ((long long)b * d.R + r) * d.nx;
    T* A = adX + (long long)b * ldX + d.row_cb[r] + i0;
    const int base = d.pat_cbase[d.row_pat[r]] + i0;
    const int lanes = 1 << lg, lane = threadIdx.x & (lanes - 1);
    for (int i = threadIdx.x >> lg; i < nc; i += BX_NT >> lg) {
        T s = T(0);
        if (i < n) {
            const int e1 = d.tx_ptr[base + i + 1];
#pragma unroll 4
            for (int e = d.tx_ptr[base + i] + lane; e < e1; e += lanes) s += d.tx_w[e] * U[d.tx_col[e]];
        }
        for (int o = lanes >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) ss[i] = s;
    }
    __syncthreads();
    const int i = threadIdx.x & (nc - 1), step = lg < 4 ? 1 << lg : BX_NT / 8;      // = BX_NT / nc
    if (i >= n) return;
    A += i;
    const T s = ss[i];
    for (int f = f0 + threadIdx.x / nc; f < f1; f += 4 * step) {     // four loads in flight
        T* o[4];
        T v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (f + u * step < f1) {
                o[u] = A + __ldg(d.te_off + f + u * step);
                v[u] = *o[u] + __ldg(d.te_w + f + u * step) * s;
            }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (f + u * step < f1) *o[u] = v[u];
    }
}

}  // namespace vd

namespace {

struct Tables {
    std::vector<int32_t> row_grp, row_pat, row_n, row_lg, fx_i, xr, yl_ptr, yl_row, ty_ptr, ty_row, tx_ptr, tx_col,
        pat_cbase, te_ptr;
    std::vector<long long> row_cb, te_off;
    std::vector<double> fx_w, yl_w, ty_w, tx_w, te_w;
};

// Lattice, time weights and banded tables of every component.
int build_host(vd_basis_plan* p, const vd_basis_grid* g, const vd_gauss3d_params* cp, Tables& tb)
{
    const int ny = g->ny, nx = g->nx;
    const bool geo = g->geographic != 0;
    const double k = geo ? 1.0 / 110 : 1.0;
    std::vector<double> xc(g->xc_host, g->xc_host + nx), yc(g->yc_host, g->yc_host + ny);
    for (double v : xc) if (!std::isfinite(v)) return VD_ERR_ARG;
    for (double v : yc) if (!std::isfinite(v)) return VD_ERR_ARG;
    const double LON_MIN = *std::min_element(xc.begin(), xc.end());
    double LON_MAX = *std::max_element(xc.begin(), xc.end());
    const double LAT_MIN = *std::min_element(yc.begin(), yc.end());
    const double LAT_MAX = *std::max_element(yc.begin(), yc.end());
    if (LON_MAX < LON_MIN) LON_MAX += 360.;
    p->times.assign(g->time_host, g->time_host + g->ntime);
    const double TMIN = *std::min_element(p->times.begin(), p->times.end());
    const double TMAX = *std::max_element(p->times.begin(), p->times.end());
    auto cosd = [&](double lat) { return geo ? std::cos(lat * M_PI / 180.) : 1.0; };
    auto wrap = [&](double d) { return geo ? pymod(d + 180, 360) - 180 : d; };

    // x-pattern dedup: rows of one component with the same lattice share tables
    std::map<std::tuple<int, double, double, long, double>, int> pat_of;
    std::vector<std::vector<std::vector<std::pair<int, double>>>> pat_cols;  // [pat][x] -> (i, w)
    std::vector<int> pat_n;

    long long boff = 0;
    int rowoff = 0;
    std::vector<int> leads, lead_of, grp_row0;   // leading component of every group / component; first rows
    p->comps.resize(p->ncomp);
    for (int c = 0; c < p->ncomp; ++c) {
        HostComp& hc = p->comps[c];
        hc.p = cp[c];
        const vd_gauss3d_params& q = cp[c];
        if (!(q.sigma_D > 0) || !(q.sigma_T > 0) || !(q.facns > 0) || !(q.facnlt > 0)) return VD_ERR_ARG;
        if (q.has_time_spinup && !(q.time_spinup != 0)) return VD_ERR_ARG;
        if (q.normalize_fact) {                                   // basis.py:1278-1283
            const int num = 50;
            const double step = (q.sigma_T - (-q.sigma_T)) / (num - 1);
            double tt[num], tmp = 0.0, mx = 0.0;
            for (int i = 0; i < num; ++i) tt[i] = (double)i * step + (-q.sigma_T);
            tt[num - 1] = q.sigma_T;
            for (int i = 0; i < num - 1; ++i) {
                tmp = tmp + hc.window(tt[i] / q.sigma_T) * (tt[i + 1] - tt[i]);
                mx = std::max(mx, tmp);
            }
            hc.norm_fact = mx;
        }
        // space lattice (basis.py:1303-1316)
        const double dlat = q.sigma_D / q.facns * k;
        const double lat0 = LAT_MIN - pymod(LAT_MIN, dlat) - q.sigma_D * (1 - 1. / q.facns) * k;
        const double lat1 = LAT_MAX + 1.5 * dlat;
        hc.rows_lat = np_arange(lat0, lat1, dlat);
        hc.boff = boff;
        int lead = c;
        for (int q2 = 0; q2 < c; ++q2)
            if (p->comps[q2].p.sigma_D == q.sigma_D && p->comps[q2].p.facns == q.facns) { lead = q2; break; }
        if (lead == c) {
            leads.push_back(c);
            grp_row0.push_back(rowoff);
            rowoff += (int)hc.rows_lat.size();
        }
        lead_of.push_back(lead);
        long long cb = 0;
        for (double la : hc.rows_lat) {
            const double cl = cosd(la);
            const double dlon = q.sigma_D / q.facns / cl * k;
            const double lon0 = LON_MIN - pymod(LON_MIN, dlon) - q.sigma_D * (1 - 1. / q.facns) / cl * k;
            const double lon1 = LON_MAX + dlon * 1.5;
            std::vector<double> lons = np_arange(lon0, lon1, dlon);
            const int n = (int)lons.size();
            auto key = std::make_tuple(lead, lon0, dlon, (long)n, cl);
            int pat = -1;
            auto it = pat_of.find(key);
            if (c != lead) {
                // the group's rows are the leading component's
            } else if (it != pat_of.end()) {
                pat = it->second;
            } else {
                pat = (int)pat_cols.size();
                pat_of[key] = pat;
                std::vector<std::vector<std::pair<int, double>>> cols((size_t)nx);
                for (int x = 0; x < nx; ++x)
                    for (int i = 0; i < n; ++i) {
                        const double xx = wrap(xc[x] - lons[i]) / k * cl;
                        if (std::fabs(xx) <= q.sigma_D) cols[x].push_back({i, mywindow(xx / q.sigma_D)});
                    }
                pat_cols.push_back(std::move(cols));
                pat_n.push_back(n);
            }
            if (c == lead) {
                tb.row_grp.push_back((int32_t)leads.size() - 1);
                tb.row_pat.push_back(pat);
                tb.row_n.push_back(n);
                tb.row_cb.push_back(cb);
            }
            hc.row_n.push_back(n);
            hc.row_cb.push_back(cb);
            for (double lo : lons) {
                hc.enslat.push_back(la);
                hc.enslon.push_back(lo);
            }
            cb += n;
        }
        hc.Nx = cb;
        // time lattice (basis.py:1320-1321)
        hc.enst = np_arange(-q.sigma_T * (1 - 1. / q.facnlt), (TMAX - TMIN) + 1.5 * q.sigma_T / q.facnlt,
                            q.sigma_T / q.facnlt);
        boff += (long long)hc.enst.size() * hc.Nx;
    }
    p->nbasis = boff;
    p->R = rowoff;
    p->ngrp = (int)leads.size();

    // x tables (ELL per pattern column, the centres that a block of columns reaches,
    // CSR per pattern centre)
    int KX = 1;
    for (auto& pc : pat_cols)
        for (auto& col : pc) KX = std::max(KX, (int)col.size());
    p->KX = KX;
    const int P = (int)pat_cols.size();
    tb.fx_i.assign((size_t)P * nx * KX, -1);
    tb.fx_w.assign((size_t)P * nx * KX, 0.0);
    tb.tx_ptr.push_back(0);
    for (int pt = 0; pt < P; ++pt) {
        tb.pat_cbase.push_back((int)tb.tx_ptr.size() - 1);
        std::vector<std::vector<std::pair<int, double>>> by_centre((size_t)pat_n[pt]);
        for (int x = 0; x < nx; ++x) {
            const auto& col = pat_cols[pt][x];
            if (x % vd::BX_NT == 0) {
                tb.xr.push_back(INT32_MAX);
                tb.xr.push_back(0);
            }
            int32_t *lo = &tb.xr[tb.xr.size() - 2], *hi = lo + 1;
            for (size_t e = 0; e < col.size(); ++e) {
                *lo = std::min<int32_t>(*lo, col[e].first);
                *hi = std::max<int32_t>(*hi, col[e].first + 1);
                tb.fx_i[((size_t)pt * nx + x) * KX + e] = col[e].first;
                tb.fx_w[((size_t)pt * nx + x) * KX + e] = col[e].second;
                by_centre[col[e].first].push_back({x, col[e].second});
            }
        }
        for (auto& lst : by_centre) {
            for (auto& pr : lst) {
                tb.tx_col.push_back(pr.first);
                tb.tx_w.push_back(pr.second);
            }
            tb.tx_ptr.push_back((int32_t)tb.tx_col.size());
        }
    }

    // lanes a centre in the transposed x pass: up to eight columns each
    for (size_t r = 0; r < tb.row_pat.size(); ++r) {
        const int pt = tb.row_pat[r], n = tb.row_n[r], cb = tb.pat_cbase[pt];
        const int cols = n ? (tb.tx_ptr[cb + n] - tb.tx_ptr[cb]) / n : 0;
        int lg = 0;
        while (lg < 5 && (8 << lg) < cols) ++lg;
        tb.row_lg.push_back(lg);
        p->gzT = std::max(p->gzT, (n + vd::bxT_centres(lg) - 1) / vd::bxT_centres(lg));
    }

    // y tables (CSR per grid row over all groups, CSR per lattice row)
    std::vector<std::vector<std::vector<std::pair<int, double>>>> ycols((size_t)p->ngrp);
    for (int c = 0; c < p->ngrp; ++c) {
        const HostComp& hc = p->comps[leads[c]];
        ycols[c].resize((size_t)ny);
        for (int y = 0; y < ny; ++y)
            for (int j = 0; j < (int)hc.rows_lat.size(); ++j) {
                const double yy = (yc[y] - hc.rows_lat[j]) / k;
                if (std::fabs(yy) <= hc.p.sigma_D) ycols[c][y].push_back({j, mywindow(yy / hc.p.sigma_D)});
            }
    }
    for (int y = 0; y < ny; ++y) {
        tb.yl_ptr.push_back((int32_t)tb.yl_row.size());
        for (int c = 0; c < p->ngrp; ++c)
            for (const auto& e : ycols[c][y]) {
                tb.yl_row.push_back(grp_row0[c] + e.first);
                tb.yl_w.push_back(e.second);
            }
    }
    tb.yl_ptr.push_back((int32_t)tb.yl_row.size());
    p->longY = tb.yl_row.size() >= 8 * (size_t)ny;
    p->longYT = tb.yl_row.size() >= 8 * (size_t)p->R;
    tb.ty_ptr.push_back(0);
    for (int c = 0; c < p->ngrp; ++c) {
        const int nr = (int)p->comps[leads[c]].rows_lat.size();
        std::vector<std::vector<std::pair<int, double>>> by_row((size_t)nr);
        for (int y = 0; y < ny; ++y) {
            const auto& l = ycols[c][y];
            for (size_t e = 0; e < l.size(); ++e) by_row[l[e].first].push_back({y, l[e].second});
        }
        for (auto& lst : by_row) {
            for (auto& pr : lst) {
                tb.ty_row.push_back(pr.first);
                tb.ty_w.push_back(pr.second);
            }
            tb.ty_ptr.push_back((int32_t)tb.ty_row.size());
        }
    }

    // time weights per (basis time, component) (basis.py:1423-1446)
    std::vector<std::vector<std::pair<int, double>>> act((size_t)p->ntime * p->ncomp);
    int NA = 1;
    for (int kt = 0; kt < p->ntime; ++kt) {
        const double t = p->times[kt];
        for (int c = 0; c < p->ncomp; ++c) {
            const HostComp& hc = p->comps[c];
            auto& lst = act[(size_t)kt * p->ncomp + c];
            for (int it = 0; it < (int)hc.enst.size(); ++it) {
                const double dt = t - hc.enst[it];
                if (std::fabs(dt) < hc.p.sigma_T) {
                    double fact = hc.window(dt / hc.p.sigma_T);
                    if (hc.p.normalize_fact) fact /= hc.norm_fact;
                    if (hc.p.has_time_spinup && t < hc.p.time_spinup)
                        fact *= (1 - hc.window(t / hc.p.time_spinup));
                    if (fact != 0) lst.push_back({it, fact});
                }
            }
            NA = std::max(NA, (int)lst.size());
        }
    }
    p->NA = NA;
    p->tact_n.assign((size_t)p->ntime * p->ncomp, 0);
    p->tact_it.assign((size_t)p->ntime * p->ncomp * NA, 0);
    p->tact_g.assign((size_t)p->ntime * p->ncomp * NA, 0.0);
    for (size_t s = 0; s < act.size(); ++s) {
        p->tact_n[s] = (int)act[s].size();
        for (size_t a = 0; a < act[s].size(); ++a) {
            p->tact_it[s * NA + a] = act[s][a].first;
            p->tact_g[s * NA + a] = act[s][a].second;
        }
    }
    // the active entries of (basis time, group): offset of the time centre in X, weight
    for (int kt = 0; kt < p->ntime; ++kt)
        for (int l : leads) {
            tb.te_ptr.push_back((int32_t)tb.te_off.size());
            for (int c = 0; c < p->ncomp; ++c)
                if (lead_of[c] == l)
                    for (const auto& a : act[(size_t)kt * p->ncomp + c]) {
                        tb.te_off.push_back(p->comps[c].boff + (long long)a.first * p->comps[c].Nx);
                        tb.te_w.push_back(a.second);
                    }
        }
    tb.te_ptr.push_back((int32_t)tb.te_off.size());
    return VD_OK;
}

template <typename T>
int upload(vd_basis_plan* p, const Tables& tb, const int8_t* land_host)
{
    Packer pk;
    const size_t o_row_grp = pk.add(tb.row_grp), o_row_pat = pk.add(tb.row_pat), o_row_n = pk.add(tb.row_n),
                 o_row_lg = pk.add(tb.row_lg), o_fx_i = pk.add(tb.fx_i), o_xr = pk.add(tb.xr),
                 o_yl_ptr = pk.add(tb.yl_ptr), o_yl_row = pk.add(tb.yl_row), o_ty_ptr = pk.add(tb.ty_ptr),
                 o_ty_row = pk.add(tb.ty_row), o_tx_ptr = pk.add(tb.tx_ptr), o_tx_col = pk.add(tb.tx_col),
                 o_pat_cbase = pk.add(tb.pat_cbase), o_te_ptr = pk.add(tb.te_ptr), o_row_cb = pk.add(tb.row_cb),
                 o_te_off = pk.add(tb.te_off), o_fx_w = pk.add_as<T>(tb.fx_w), o_yl_w = pk.add_as<T>(tb.yl_w),
                 o_ty_w = pk.add_as<T>(tb.ty_w), o_tx_w = pk.add_as<T>(tb.tx_w), o_te_w = pk.add_as<T>(tb.te_w);
    size_t o_land = 0;
    bool any_land = false;
    std::vector<int8_t> land;
    if (land_host) {
        land.assign(land_host, land_host + (size_t)p->ny * p->nx);
        for (int8_t v : land) any_land |= (v != 0);
        if (any_land) o_land = pk.add(land);
    }
    VD_CUDA_TRY(cudaMalloc(&p->dev, pk.blob.size()));
    VD_CUDA_TRY(cudaMemcpy(p->dev, pk.blob.data(), pk.blob.size(), cudaMemcpyHostToDevice));
    unsigned char* b = (unsigned char*)p->dev;
    p->row_grp = (const int32_t*)(b + o_row_grp);
    p->row_pat = (const int32_t*)(b + o_row_pat);
    p->row_n = (const int32_t*)(b + o_row_n);
    p->row_lg = (const int32_t*)(b + o_row_lg);
    p->fx_i = (const int32_t*)(b + o_fx_i);
    p->xr = (const int32_t*)(b + o_xr);
    p->yl_ptr = (const int32_t*)(b + o_yl_ptr);
    p->yl_row = (const int32_t*)(b + o_yl_row);
    p->ty_ptr = (const int32_t*)(b + o_ty_ptr);
    p->ty_row = (const int32_t*)(b + o_ty_row);
    p->tx_ptr = (const int32_t*)(b + o_tx_ptr);
    p->tx_col = (const int32_t*)(b + o_tx_col);
    p->pat_cbase = (const int32_t*)(b + o_pat_cbase);
    p->te_ptr = (const int32_t*)(b + o_te_ptr);
    p->row_cb = (const long long*)(b + o_row_cb);
    p->te_off = (const long long*)(b + o_te_off);
    p->fx_w = b + o_fx_w;
    p->yl_w = b + o_yl_w;
    p->ty_w = b + o_ty_w;
    p->tx_w = b + o_tx_w;
    p->te_w = b + o_te_w;
    p->land = any_land ? (const int8_t*)(b + o_land) : nullptr;
    return VD_OK;
}

size_t ws_bytes(const vd_basis_plan* p, int batch)
{
    return (size_t)batch * p->R * p->nx * (p->dtype == VD_F64 ? 8 : 4);
}

}  // namespace

extern "C" vd_status vd_basis_plan_create(vd_basis_plan** out, const vd_basis_grid* g, int ncomp,
                                          const vd_gauss3d_params* comps)
{
    if (!out || !g || !comps || ncomp < 1) return VD_ERR_ARG;
    *out = nullptr;
    if (g->ny < 1 || g->nx < 1 || !g->xc_host || !g->yc_host || g->ntime < 1 || !g->time_host) return VD_ERR_ARG;
    if (g->dtype != VD_F32 && g->dtype != VD_F64) return VD_ERR_ARG;
    for (int i = 0; i < g->ntime; ++i)
        if (!std::isfinite(g->time_host[i])) return VD_ERR_ARG;
    vd_basis_plan* p = new (std::nothrow) vd_basis_plan();
    if (!p) return VD_ERR_ARG;
    p->ny = g->ny; p->nx = g->nx; p->dtype = g->dtype; p->geographic = g->geographic;
    p->host_only = g->host_only; p->ncomp = ncomp; p->ntime = g->ntime;
    Tables tb;
    int st = build_host(p, g, comps, tb);
    if (st == VD_OK && (p->R > 65535 || p->ny > 65535)) st = VD_ERR_UNSUPPORTED;
    if (st == VD_OK && !p->host_only)
        st = p->dtype == VD_F64 ? upload<double>(p, tb, g->land_host) : upload<float>(p, tb, g->land_host);
    if (st != VD_OK) {
        if (p->dev) cudaFree(p->dev);
        delete p;
        return st;
    }
    *out = p;
    return VD_OK;
}

extern "C" vd_status vd_basis_plan_destroy(vd_basis_plan* p)
{
    if (!p) return VD_ERR_ARG;
    if (p->dev) cudaFree(p->dev);
    delete p;
    return VD_OK;
}

extern "C" long long vd_basis_nbasis(const vd_basis_plan* p) { return p ? p->nbasis : 0; }

extern "C" vd_status vd_basis_component(const vd_basis_plan* p, int c, long long* offset, int* nt, int* ns)
{
    if (!p || c < 0 || c >= p->ncomp) return VD_ERR_ARG;
    if (offset) *offset = p->comps[c].boff;
    if (nt) *nt = (int)p->comps[c].enst.size();
    if (ns) *ns = (int)p->comps[c].Nx;
    return VD_OK;
}

extern "C" vd_status vd_basis_lattice(const vd_basis_plan* p, int c, double* enst, double* enslat, double* enslon)
{
    if (!p || c < 0 || c >= p->ncomp) return VD_ERR_ARG;
    const HostComp& hc = p->comps[c];
    if (enst) std::copy(hc.enst.begin(), hc.enst.end(), enst);
    if (enslat) std::copy(hc.enslat.begin(), hc.enslat.end(), enslat);
    if (enslon) std::copy(hc.enslon.begin(), hc.enslon.end(), enslon);
    return VD_OK;
}

extern "C" vd_status vd_basis_q(const vd_basis_plan* p, double* q)
{
    if (!p || !q) return VD_ERR_ARG;
    for (const HostComp& hc : p->comps) {
        const double v = hc.p.sigma_Q / std::sqrt(hc.p.facns * hc.p.facnlt);
        std::fill(q + hc.boff, q + hc.boff + (long long)hc.enst.size() * hc.Nx, v);
    }
    return VD_OK;
}

extern "C" vd_status vd_basis_time_weights(const vd_basis_plan* p, int k, int c, int* count, int* it, double* w)
{
    if (!p || !count || k < 0 || k >= p->ntime || c < 0 || c >= p->ncomp) return VD_ERR_ARG;
    const size_t s = (size_t)k * p->ncomp + c;
    *count = p->tact_n[s];
    for (int a = 0; a < p->tact_n[s]; ++a) {
        if (it) it[a] = p->tact_it[s * p->NA + a];
        if (w) w[a] = p->tact_g[s * p->NA + a];
    }
    return VD_OK;
}

extern "C" size_t vd_basis_workspace_bytes(const vd_basis_plan* p, int batch)
{
    if (!p || batch < 1) return 0;
    return ws_bytes(p, batch);
}

namespace {

template <typename T>
int project(const vd_basis_plan* p, int B, int k, const T* X, long long ldX, T* phi, int acc, T* ws,
            cudaStream_t st)
{
    const vd::BasisDev<T> d = vd::dev_view<T>(p);
    const unsigned gx = (unsigned)((p->nx + vd::BX_NT - 1) / vd::BX_NT);
    vd::k_basis_xpass<T><<<dim3(gx, p->R, B), vd::BX_NT, 0, st>>>(d, k, X, ldX, ws);
    VD_LAUNCH_CHECK();
    if (p->longY) vd::k_basis_ypass<T, true><<<dim3(gx, p->ny, B), vd::BX_NT, 0, st>>>(d, ws, phi, acc);
    else vd::k_basis_ypass<T, false><<<dim3(gx, p->ny, B), vd::BX_NT, 0, st>>>(d, ws, phi, acc);
    VD_LAUNCH_CHECK();
    return VD_OK;
}

template <typename T>
int project_T(const vd_basis_plan* p, int B, int k, const T* adphi, T* adX, long long ldX, T* ws,
              cudaStream_t st)
{
    const vd::BasisDev<T> d = vd::dev_view<T>(p);
    const unsigned gx = (unsigned)((p->nx + vd::BX_NT - 1) / vd::BX_NT);
    if (p->longYT) vd::k_basisT_ypass<T, true><<<dim3(gx, p->R, B), vd::BX_NT, 0, st>>>(d, adphi, ws);
    else vd::k_basisT_ypass<T, false><<<dim3(gx, p->R, B), vd::BX_NT, 0, st>>>(d, adphi, ws);
    VD_LAUNCH_CHECK();
    vd::k_basisT_xpass<T><<<dim3(p->R, B, p->gzT), vd::BX_NT, 0, st>>>(d, k, ws, adX, ldX);
    VD_LAUNCH_CHECK();
    return VD_OK;
}

int check_call(const vd_basis_plan* p, int B, int k, long long ldX, const void* a, const void* b, void* ws,
               size_t wsb)
{
    if (!p || p->host_only || !p->dev) return VD_ERR_ARG;
    if (B < 1 || B > 65535 || k < 0 || k >= p->ntime || !a || !b || !ws) return VD_ERR_ARG;
    if (B > 1 && ldX < p->nbasis) return VD_ERR_ARG;
    if (wsb < ws_bytes(p, B)) return VD_ERR_WORKSPACE;
    return VD_OK;
}

}  // namespace

extern "C" vd_status vd_basis_project(const vd_basis_plan* p, int B, int k, const void* X, long long ldX,
                                      void* phi, int accumulate, void* ws, size_t wsb, void* stream)
{
    const int st = check_call(p, B, k, ldX, X, phi, ws, wsb);
    if (st != VD_OK) return st;
    if (p->dtype == VD_F64)
        return project<double>(p, B, k, (const double*)X, ldX, (double*)phi, accumulate, (double*)ws,
                               (cudaStream_t)stream);
    return project<float>(p, B, k, (const float*)X, ldX, (float*)phi, accumulate, (float*)ws,
                          (cudaStream_t)stream);
}

extern "C" vd_status vd_basis_project_T(const vd_basis_plan* p, int B, int k, const void* adphi, void* adX,
                                        long long ldX, void* ws, size_t wsb, void* stream)
{
    const int st = check_call(p, B, k, ldX, adphi, adX, ws, wsb);
    if (st != VD_OK) return st;
    if (p->dtype == VD_F64)
        return project_T<double>(p, B, k, (const double*)adphi, (double*)adX, ldX, (double*)ws,
                                 (cudaStream_t)stream);
    return project_T<float>(p, B, k, (const float*)adphi, (float*)adX, ldX, (float*)ws, (cudaStream_t)stream);
}
