// x-direction DST-I passes on the 5th-generation tensor cores (tcgen05, sm_103a)
// for float32 plans; the forward pass solves the y-direction tridiagonal systems
// in its epilogue.
//
// Each pass is two dense half-size products per row block (even/odd split, see
// vd_dst.cu), formed transposed: the UMMA's M dimension runs over 128 modes
// (forward) or positions (inverse) of the DST half matrix, its N dimension over
// a block of RB rows of one field. A thread of the epilogue therefore owns one
// mode and a run of rows in tensor memory (TMEM, fp32 accumulators):
//   - the tridiagonal solve along y is a recurrence along its own registers; the
//     RB-row blocks of a field form a cluster and exchange the carries of their
//     pieces through distributed shared memory;
//   - a warp holds 32 consecutive modes or positions of a row, so rows are
//     stored straight from registers, coalesced, with no staging tile.
// The K loop of the largest shape (128 rows, two groups) is bound by the SM's
// shared-memory port: a chunk's 24 MMAs read 8 KB of operands each, its rows and
// matrix add 96 KB of writes, 292 KB at 128 bytes a clock = 1.15 us, as measured.
// Every CTA reads its own matrix chunks (64 KB of them at most, from L2); handing a
// cluster's CTAs one shared copy took as long or longer (an inverse pass 20.0 us
// without it and 20.7 with it at 16 x 512^2, 17.0 and 17.8 at 1024^2, 10.8 and 11.3
// at 6 x 287x410; the fused forward pass within 1 %).
// Measured inversions (the row-major form with a separate solve in brackets, us): 16 x 512^2 52 (64),
// 1024^2 43 (54), 6 x 287x410 27 (62), 12 x 192^2 18 (28), 128^2 15 (24).
// A CTA holds MG = 1 or 2 groups of 128 modes (positions) of one parity of the
// same rows (MG * RB <= 256 TMEM columns), and 1 CTA runs per SM.
// Float32 accuracy comes from the 3xTF32 split: x = x_hi + x_lo with
// x_hi = tf32(x), and x.w ~= x_hi.w_hi + x_hi.w_lo + x_lo.w_hi (the dropped
// x_lo.w_lo term is ~2^-22 relative).
//
// Pipeline (per K chunk of 32 = one 128-byte swizzle row of fp32):
//   warps 0-15 build the row chunk (butterfly or copy of the input rows, hi/lo
//              split; RB/16 rows each) in the 128B-swizzled K-major layout and
//              arrive on fullA;
//   thread 0   also issues the bulk copies (cp.async.bulk) of the
//              pre-swizzled hi/lo chunks of the DST half matrix (fullB);
//   warp 16    owns the TMEM allocation; its lane 0 issues 3 x 4 MMAs per
//              chunk and group and commits to `empty` to recycle the stage;
//   warps 0-15 finally run the epilogue; in the inverse pass the two CTAs of a
//              cluster (odd-k and even-k sums of the same rows) each send the
//              other the half of its rows that it will write.
// Every mbarrier wait is bounded (2 s of %globaltimer); a timeout sets a bit
// in a device flag (vd_device_error) and the CTA finishes without hanging.
#include "vd_internal.cuh"
#include <algorithm>
#include <vector>
#include <cmath>
#include <cstring>
#include <mutex>
#include <type_traits>

namespace vd {

__device__ int g_tc_error = 0;

namespace tc {

constexpr int GM = 128;                // UMMA M: modes or positions of a group
constexpr int KCH = 32;
constexpr int NPW = 16;                // producer / epilogue warps
constexpr int NPROD = NPW * 32;
constexpr int NTHREADS = NPROD + 32;   // + warp NPW: TMEM owner and MMA issuer
constexpr int MAX_STAGES = 6;
constexpr int TMEM_COLS = 256;
constexpr uint32_t G_TILE = GM * KCH * 4;           // 16 KB: one group's hi or lo chunk of the half matrix
constexpr size_t SMEM_MAX = 227 * 1024;             // largest dynamic request of any launch (static: ~200 bytes)
constexpr size_t SMEM_ONE = 120 * 1024;             // smallest: one CTA per SM (a CTA waits for its cluster peers)
constexpr size_t SMEM_STATIC = 512;
constexpr int MAX_NR = 8;                           // row blocks of a field in one cluster

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t gtimer()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait on the phase of parity `parity`.
// The timer is read once every 64 polls.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int code)
{
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = gtimer();
    for (uint32_t it = 1;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 63u) == 0 && gtimer() - t0 > 2000000000ull) {
            atomicOr(&g_tc_error, code);
            return false;
        }
    }
}

// Distributed shared memory of the cluster.
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// Every thread of the cluster arrives; shared-memory writes before the barrier
// are visible to the peer CTAs after it.
__device__ __forceinline__ void cluster_arrive()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster_v2(uint32_t addr, float a, float b)
{
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish()
{
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void mma_tf32(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accum)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(dtmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum));
}
__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

// NC consecutive fp32 columns of this thread's TMEM lane.
template <int NC>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float (&v)[NC])
{
    uint32_t r[NC];
    if constexpr (NC == 4) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3])
                     :
                     : "memory");
    }
    if constexpr (NC == 8) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                       "=r"(r[7])
                     : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                       "+r"(r[7])
                     :
                     : "memory");
    }
    if constexpr (NC == 16) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                       "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
                       "=r"(r[14]), "=r"(r[15])
                     : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                       "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]),
                       "+r"(r[14]), "+r"(r[15])
                     :
                     : "memory");
    }
    if constexpr (NC == 32) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
                     "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                       "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
                       "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
                       "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
                       "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                     : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                       "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]),
                       "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]),
                       "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]),
                       "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                     :
                     : "memory");
    }
#pragma unroll
    for (int i = 0; i < NC; ++i) v[i] = __uint_as_float(r[i]);
}
template <int NC>
__device__ __forceinline__ void tmem_st(uint32_t taddr, const float (&v)[NC])
{
    uint32_t r[NC];
#pragma unroll
    for (int i = 0; i < NC; ++i) r[i] = __float_as_uint(v[i]);
    if constexpr (NC == 8) {
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                     ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                     : "memory");
    }
    if constexpr (NC == 16) {
        asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                     ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                       "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
                       "r"(r[15])
                     : "memory");
    }
    if constexpr (NC == 32) {
        asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,"
                     "%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                     ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                       "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
                       "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
                       "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
                       "r"(r[29]), "r"(r[30]), "r"(r[31])
                     : "memory");
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ float tf32_rna(float x)
{
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 bytes apart (SBO), descriptor version 1.
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t saddr)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1u << 16) | ((uint64_t)(1024u >> 4) << 32) |
           ((uint64_t)1u << 46) | ((uint64_t)2u << 61);
}

// Instruction descriptor of kind::tf32: fp32 accumulate, tf32 A and B, both
// K-major, N>>3 at bit 17, M>>4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_tf32(int M, int N)
{
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// byte offset of fp32 element (r, k) in a [rows][32] 128B-swizzled tile
__host__ __device__ constexpr uint32_t swz(int r, int k)
{
    return (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((((k >> 2) ^ (r & 7)) & 7) << 4) + (k & 3) * 4);
}

}  // namespace tc

constexpr int MAX_NE = 2048;

// Images: per parity (forward) or job (inverse), per K chunk, the hi then the
// lo part of the whole [Ntot][32] swizzled operand, so that the rows of any
// group of 128 are one contiguous range.
struct TcTab {
    int kch;                         // K chunks of 32
    int Ntot;                        // operand rows: ne rounded up to a multiple of 16
    long long fwd_base[2];           // forward image offsets (floats) per parity
    long long inv_base[2];           // inverse image offsets (floats) per job
    int nst;                         // pipeline stages of this launch (<= MAX_STAGES)
};

struct TcGeom {
    int n, ne, no, my, nx;
    long long fs;
    int lds;
    int nr;                          // row blocks of a field (fused forward pass)
    int rows;                        // interior rows of all fields
};

using namespace tc;

// Shared-memory plan of a launch: nst stages of
//   rows hi | rows lo | matrix hi | matrix lo      (every part 1024-byte aligned)
// then the forward pass's first carry exchange (peers may write it while this CTA
// is still in its K loop; the second one reuses the stages).
template <int RPW, int MG>
struct TcShape {
    static constexpr int RB = RPW * NPW;                 // rows of a block
    static constexpr uint32_t ROWS = RB * KCH * 4;       // bytes of one row chunk (hi or lo)
    static constexpr uint32_t MAT = MG * G_TILE;
    static constexpr uint32_t STAGE = 2 * ROWS + 2 * MAT;
    static constexpr int PC = MG * RB / 4;               // TMEM columns of an epilogue warp: a piece of PC rows
    static constexpr int NPC = 4 / MG;                   // pieces of a block
    static constexpr int DEPTH = RPW >= 8 ? 2 : RPW == 4 ? 3 : 4;       // register buffers of prefetched chunks
    static constexpr size_t exch_bytes(int nr) { return (size_t)MG * GM * NPC * nr * 8; }
    // inverse epilogue: received sums, then the staged rows
    static constexpr size_t INV_EPI = (size_t)(RB / 2) * (MG * GM + 2 * (MG * GM + 8)) * 4;
};

// The K loop shared by both passes: D[group][mode lane][row column] = half matrix
// x rows. `fwd`: butterflied interior rows of a field, else spectral rows.
template <int RPW, int MG, bool FWD>
struct TcLoop {
    using Sh = TcShape<RPW, MG>;
    uint32_t sbase, bar0, tmem;
    int stages, kch;

    __device__ __forceinline__ uint32_t rows_hi(int s) const { return sbase + s * Sh::STAGE; }
    __device__ __forceinline__ uint32_t mat_hi(int s) const { return rows_hi(s) + 2 * Sh::ROWS; }
    __device__ __forceinline__ uint32_t full_a(int s) const { return bar0 + 8u * s; }
    __device__ __forceinline__ uint32_t full_b(int s) const { return bar0 + 8u * (stages + s); }
    __device__ __forceinline__ uint32_t empty(int s) const { return bar0 + 8u * (2 * stages + s); }
    __device__ __forceinline__ uint32_t accf() const { return bar0 + 8u * (3 * stages); }

    __device__ __forceinline__ void init_barriers() const
    {
        for (int s = 0; s < stages; ++s) {
            mbar_init(full_a(s), NPROD);
            mbar_init(full_b(s), 1);
            mbar_init(empty(s), 1);
        }
        mbar_init(accf(), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }

    // Warp w fills rows [RPW w, RPW (w+1)); lane l handles K index k0 + l, so
    // every global load is one coalesced 128-byte row. rows + off(i) (block-uniform
    // pointer, 32-bit offset) is the warp's i-th row (element 0 of the transform,
    // or of the job's spectral half), `sub` likewise, or null (only where sub_on(i));
    // `nv` of the warp's rows exist, the others are zero. `half` 0 takes sums, 1
    // differences of mirrored elements.
    // side(c) runs beside chunk c.
    template <typename Off, typename On, typename Side>
    __device__ __forceinline__ void produce(const float* __restrict__ rows, const float* __restrict__ sub, Off&& roff,
                                            On&& sub_on, int nv, int n, int lim, int no, int half,
                                            const float* __restrict__ img, int ntot, uint32_t b_bytes,
                                            Side&& side) const
    {
        constexpr int DEPTH = Sh::DEPTH;
        const int tid = threadIdx.x, lane = tid & 31, r0 = (tid >> 5) * RPW;
        float x1[DEPTH][RPW], x2[DEPTH][RPW];
        auto load = [&](int c, float (&a)[RPW], float (&b)[RPW]) {
            const int p = c * KCH + lane;
            const bool v1 = p < lim, v2 = FWD && p < no;
#pragma unroll
            for (int i = 0; i < RPW; ++i) {
                const bool v = i < nv;
                a[i] = v && v1 ? __ldg(rows + (roff(i) + p)) : 0.f;
                if (FWD) b[i] = v && v2 ? __ldg(rows + (roff(i) + (n - 1 - p))) : 0.f;
            }
        };
        // background PV to subtract, loaded one chunk ahead
        float s1[FWD ? RPW : 1], s2[FWD ? RPW : 1];
        auto load_sub = [&](int c) {
            if constexpr (FWD) {
                const int p = c * KCH + lane;
#pragma unroll
                for (int i = 0; i < RPW; ++i) {
                    const bool v = i < nv && sub_on(i);
                    s1[i] = v && p < lim ? __ldg(sub + (roff(i) + p)) : 0.f;
                    s2[i] = v && p < no ? __ldg(sub + (roff(i) + (n - 1 - p))) : 0.f;
                }
            }
        };
        // byte offset of (row r0 + i, k = lane) in the swizzled [RB][32] tile
        uint32_t off[RPW];
#pragma unroll
        for (int i = 0; i < RPW; ++i) off[i] = swz(r0 + i, lane);
        int ps = 0;
        uint32_t pu = 0;
        auto process = [&](int c, float (&a)[RPW], float (&b)[RPW]) {
            if (FWD && sub) {
#pragma unroll
                for (int i = 0; i < RPW; ++i) {
                    a[i] -= s1[i];
                    b[i] -= s2[i];
                }
                if (c + 1 < kch) load_sub(c + 1);
            }
            const int s = ps;
            const uint32_t u = pu;
            if (++ps == stages) {
                ps = 0;
                ++pu;
            }
            if (c >= stages) mbar_wait(empty(s), (u - 1) & 1, 1);
            if (tid == 0) {
                mbar_arrive_expect_tx(full_b(s), 2 * b_bytes);
                const float* blk = img + (size_t)c * 2 * ntot * KCH;
                bulk_g2s(mat_hi(s), blk, b_bytes, full_b(s));
                bulk_g2s(mat_hi(s) + Sh::MAT, blk + (size_t)ntot * KCH, b_bytes, full_b(s));
            }
            const uint32_t ah = rows_hi(s), al = ah + Sh::ROWS;
#pragma unroll
            for (int i = 0; i < RPW; ++i) {
                // the middle element of an odd-length transform has no mirror (b = 0)
                const float val = FWD ? (half == 0 ? a[i] + b[i] : a[i] - b[i]) : a[i];
                const float h = tf32_rna(val);
                const float l = tf32_rna(val - h);
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(ah + off[i]), "f"(h) : "memory");
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(al + off[i]), "f"(l) : "memory");
            }
            fence_async_smem();
            mbar_arrive(full_a(s));
        };
        if (FWD && sub) load_sub(0);
#pragma unroll
        for (int d = 0; d < DEPTH; ++d)
            if (d < kch) load(d, x1[d], x2[d]);
        for (int c0 = 0; c0 < kch; c0 += DEPTH) {
#pragma unroll
            for (int d = 0; d < DEPTH; ++d) {
                const int c = c0 + d;
                if (c < kch) {
                    process(c, x1[d], x2[d]);
                    if (c + DEPTH < kch) load(c + DEPTH, x1[d], x2[d]);
                    side(c);
                }
            }
        }
    }

    // One thread issues every MMA: `ng` groups of 128 matrix rows.
    __device__ __forceinline__ void issue(int ng) const
    {
        const uint32_t idesc = idesc_tf32(GM, Sh::RB);
        int s = 0;
        uint32_t u = 0;
        for (int c = 0; c < kch; ++c) {
            mbar_wait(full_a(s), u & 1, 2);
            mbar_wait(full_b(s), u & 1, 2);
            tc_fence_after();
#pragma unroll
            for (int g = 0; g < MG; ++g) {
                if (g >= ng) break;
                const uint32_t d = tmem + g * Sh::RB;
#pragma unroll
                for (int kk = 0; kk < KCH / 8; ++kk) {
                    const uint64_t xh = sdesc_sw128(rows_hi(s) + kk * 32);
                    const uint64_t xl = sdesc_sw128(rows_hi(s) + Sh::ROWS + kk * 32);
                    const uint64_t wh = sdesc_sw128(mat_hi(s) + g * G_TILE + kk * 32);
                    const uint64_t wl = sdesc_sw128(mat_hi(s) + Sh::MAT + g * G_TILE + kk * 32);
                    mma_tf32(d, wh, xh, idesc, (c > 0 || kk > 0) ? 1u : 0u);
                    mma_tf32(d, wl, xh, idesc, 1u);
                    mma_tf32(d, wh, xl, idesc, 1u);
                }
            }
            // nobody waits for the last use of a stage
            if (c + stages < kch) mma_commit(empty(s));
            if (++s == stages) {
                s = 0;
                ++u;
            }
        }
        mma_commit(accf());
    }
};

// Forward pass. FUSE: the epilogue solves the tridiagonal systems and writes the
// solved spectrum, else the plain one. Grid: x = row blocks (FUSE: nr blocks of
// every field, a cluster; else blocks of the consecutive interior rows of all
// fields), y = groups of MG * 128 modes x parity.
//
// Tridiagonal solve (see vd_dst.cu): forward d_j = m_j (F_j - a d_{j-1}), backward
// x_j = d_j - a m_j x_{j+1}. A thread owns one mode and a piece of PC rows. Each
// sweep first runs over the piece from a zero carry, only for its end value and
// the product of its multipliers (the recurrence is affine in the carry); the
// pieces of a mode swap these through the cluster's shared memory, every thread
// folds those before its own into its carry, and the sweep runs again from it.
template <int RPW, int MG, bool FUSE>
__global__ void __launch_bounds__(NTHREADS, 1)
dst_tc_fwd_kernel(TcGeom g, TcTab tab, const float* __restrict__ img, const float* __restrict__ src,
                  const float* __restrict__ sub, int sub_batches, const int* __restrict__ bg_on,
                  float* __restrict__ spec, const float* __restrict__ trim, float a)
{
    using Sh = TcShape<RPW, MG>;
    constexpr int RB = Sh::RB, PC = Sh::PC, NPC = Sh::NPC;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bars[3 * MAX_STAGES + 1];
    __shared__ uint32_t tmem_base_sh;
    TcLoop<RPW, MG, true> L;
    L.sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    L.bar0 = smem_u32(&bars[0]);
    L.stages = tab.nst;
    L.kch = tab.kch;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int f = FUSE ? blockIdx.x / g.nr : 0, rb = blockIdx.x - f * g.nr;
    const int nrows = FUSE ? g.my : g.rows;              // rows that the blocks rb = 0, 1, ... cover
    const int half = blockIdx.y & 1, t_first = (blockIdx.y >> 1) * MG * GM;
    const int wrows = min(MG * GM, tab.Ntot - t_first);

    constexpr uint32_t COLS = FUSE ? 2 * TMEM_COLS : TMEM_COLS;   // the multipliers lie behind the accumulators
    if (warp == NPW) {
        tmem_alloc(smem_u32(&tmem_base_sh), COLS);
        tmem_relinquish();
    }
    if (tid == 0) L.init_barriers();
    __syncwarp();
    if constexpr (FUSE) cluster_arrive();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    L.tmem = tmem_base_sh;

    const int sp = warp & 3, hc = warp >> 2;
    const uint32_t tcol = L.tmem + ((uint32_t)(sp * 32) << 16) + hc * PC;    // this warp's piece
    const int grp = hc / NPC, pc = hc - grp * NPC;
    const int mode = grp * GM + sp * 32 + lane, t = t_first + mode;
    const int lim = half == 0 ? g.ne : g.no, col = (half == 0 ? 0 : g.ne) + t;
    const int j0 = rb * RB + pc * PC;                                        // first row of the piece
    const bool live = warp < NPW && t < lim;
    bool ok = true;
    if (warp < NPW) {
        const int r0 = rb * RB + warp * RPW, nv = min(RPW, nrows - r0);
        const long long o = f * g.fs;
        // the piece's multipliers go to TMEM 8 rows at a time beside the K loop
        float mb[8];
        auto side = [&](int c) {
            if constexpr (FUSE) {
                if (c >= 1 && c <= PC / 8) tmem_st<8>(tcol + TMEM_COLS + 8 * (c - 1), mb);
                if (c < PC / 8) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int j = j0 + 8 * c + i;
                        mb[i] = live && j < g.my ? __ldg(trim + (long long)j * g.lds + col) : 0.f;
                    }
                }
            }
        };
        const float* bimg = img + (half ? tab.fwd_base[1] : tab.fwd_base[0]) + (size_t)t_first * KCH;
        const uint32_t b_bytes = (uint32_t)wrows * KCH * 4;
        if constexpr (FUSE) {
            const unsigned first = (unsigned)((r0 + 1) * g.nx + 1), pitch = (unsigned)g.nx;
            L.produce(src + o, sub != nullptr && f < sub_batches && (!bg_on || bg_on[f]) ? sub + o : nullptr,
                      [&](int i) { return first + i * pitch; }, [](int) { return true; }, nv, g.n, lim, g.no, half,
                      bimg, tab.Ntot, b_bytes, side);
        } else {
            unsigned ro[RPW];                            // rows may run on into the next field
            unsigned on = 0;
#pragma unroll
            for (int i = 0; i < RPW; ++i) {
                const int r = min(r0 + i, nrows - 1), fi = r / g.my;
                ro[i] = (unsigned)(fi * g.fs + (long long)(r - fi * g.my + 1) * g.nx + 1);
                on |= (unsigned)(sub != nullptr && fi < sub_batches && (!bg_on || bg_on[fi])) << i;
            }
            L.produce(src, on ? sub : nullptr, [&](int i) { return ro[i]; }, [&](int i) { return (on >> i & 1u) != 0; }, nv, g.n,
                      lim, g.no, half, bimg, tab.Ntot, b_bytes, side);
        }
        if (FUSE)
            for (int c = L.kch; c <= PC / 8; ++c) side(c);
        ok = mbar_wait(L.accf(), 0, 4);
        __syncwarp();
        tc_fence_after();
    } else if (lane == 0) {
        L.issue((wrows + GM - 1) / GM);
    }
    __syncwarp();

    constexpr int NB = PC < 16 ? PC : 16;                // columns of a TMEM access
    float* const srow = spec + ((long long)f * g.my + j0) * g.lds + col;
    const int rows = live && ok ? nrows - j0 : 0;        // rows of the piece to write
    if constexpr (!FUSE) {
        if (warp < NPW) {
#pragma unroll
            for (int b = 0; b < PC; b += NB) {
                float v[NB];
                tmem_ld<NB>(tcol + b, v);
#pragma unroll
                for (int i = 0; i < NB; ++i)
                    if (b + i < rows) srow[(unsigned)((b + i) * g.lds)] = v[i];
            }
        }
    } else {
        const int npieces = g.nr * NPC, q = rb * NPC + pc;
        const uint32_t ex_row = (uint32_t)(MG * GM) * 8u, ex_own = (uint32_t)(q * MG * GM + mode) * 8u;
        const uint32_t ex[2] = {L.sbase + (uint32_t)tab.nst * Sh::STAGE, L.sbase};
        auto push = [&](uint32_t buf, float d, float P) {
            for (int r = 0; r < g.nr; ++r) st_cluster_v2(mapa_shared(buf + ex_own, (uint32_t)r), d, P);
        };
        auto fold = [&](uint32_t buf, int k, float c) {
            float d, P;
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(d), "=f"(P)
                         : "r"(buf + (uint32_t)k * ex_row + (uint32_t)mode * 8u));
            return fmaf(P, c, d);
        };
        const uint32_t mcol = tcol + TMEM_COLS;
        float d = 0.f, P = 1.f;
        cluster_wait();                  // every CTA of the cluster has started: its shared memory can be written
        if (warp < NPW) {
#pragma unroll
            for (int b = 0; b < PC; b += NB) {
                float v[NB], m[NB];
                tmem_ld<NB>(mcol + b, m);
                tmem_ld<NB>(tcol + b, v);
#pragma unroll
                for (int i = 0; i < NB; ++i) {
                    d = m[i] * fmaf(-a, d, v[i]);
                    P *= -a * m[i];
                }
            }
            push(ex[0], d, P);
        }
        cluster_arrive();
        cluster_wait();
        if (warp < NPW) {
            d = 0.f;
            for (int k = 0; k < q; ++k) d = fold(ex[0], k, d);
#pragma unroll
            for (int b = 0; b < PC; b += NB) {
                float v[NB], m[NB];
                tmem_ld<NB>(mcol + b, m);
                tmem_ld<NB>(tcol + b, v);
#pragma unroll
                for (int i = 0; i < NB; ++i) {
                    d = m[i] * fmaf(-a, d, v[i]);
                    v[i] = d;
                }
                tmem_st<NB>(tcol + b, v);
            }
            float x = 0.f;
            P = 1.f;
#pragma unroll
            for (int b = PC - NB; b >= 0; b -= NB) {
                float v[NB], m[NB];
                tmem_ld<NB>(mcol + b, m);
                tmem_ld<NB>(tcol + b, v);
#pragma unroll
                for (int i = NB - 1; i >= 0; --i) {
                    const float al = -a * m[i];
                    x = fmaf(al, x, v[i]);
                    P *= al;
                }
            }
            push(ex[1], x, P);
        }
        cluster_arrive();
        cluster_wait();
        if (warp < NPW) {
            float x = 0.f;
            for (int k = npieces - 1; k > q; --k) x = fold(ex[1], k, x);
#pragma unroll
            for (int b = PC - NB; b >= 0; b -= NB) {
                float v[NB], m[NB];
                tmem_ld<NB>(mcol + b, m);
                tmem_ld<NB>(tcol + b, v);
#pragma unroll
                for (int i = NB - 1; i >= 0; --i) {
                    x = fmaf(-a * m[i], x, v[i]);
                    if (b + i < rows) srow[(unsigned)((b + i) * g.lds)] = x;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == NPW) {
        tc_fence_after();
        tmem_dealloc(L.tmem, COLS);
    }
}

// Inverse pass. Grid: x = fields x row blocks x 2 jobs (a cluster of two CTAs:
// rank 0 the odd-k half A of the spectrum, rank 1 the even-k half B), y = groups
// of MG * 128 positions. x[p] = A + B and x[n-1-p] = A - B: the A CTA writes the
// first half of the block's rows, the B CTA the second, each after receiving the
// other's sums of those rows in its (free) pipeline stages. Rows go through
// shared memory once more so that they leave as aligned float4s: the interior
// starts one element into a row, and 128-byte stores off their lines cost the
// epilogue 8 us instead of 3 at 16 x 512^2.
template <int RPW, int MG, int EPI>
__global__ void __launch_bounds__(NTHREADS, 1)
dst_tc_inv_kernel(TcGeom g, TcTab tab, const float* __restrict__ img, const float* __restrict__ spec,
                  float* __restrict__ out, const float* __restrict__ add, int add_batches,
                  const int* __restrict__ bg_on, const int8_t* __restrict__ mask)
{
    using Sh = TcShape<RPW, MG>;
    constexpr int RB = Sh::RB, HR = RB / 2;
    constexpr int PH = MG * HR / 4;          // rows of an epilogue warp in one half of the block
    constexpr int NPH = 4 / MG;              // such pieces a half and group
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bars[3 * MAX_STAGES + 1];
    __shared__ uint32_t tmem_base_sh;
    TcLoop<RPW, MG, false> L;
    L.sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    L.bar0 = smem_u32(&bars[0]);
    L.stages = tab.nst;
    L.kch = tab.kch;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int job = blockIdx.x & 1, blk = blockIdx.x >> 1;
    const int p_first = blockIdx.y * MG * GM;
    const int wrows = min(MG * GM, tab.Ntot - p_first);

    if (warp == NPW) {
        tmem_alloc(smem_u32(&tmem_base_sh), TMEM_COLS);
        tmem_relinquish();
    }
    if (tid == 0) L.init_barriers();
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    L.tmem = tmem_base_sh;

    const int sp = warp & 3, hc = warp >> 2;
    const int grp = hc / NPH, pc = hc - grp * NPH;
    const uint32_t tlane = L.tmem + ((uint32_t)(sp * 32) << 16) + grp * RB + pc * PH;
    const int pl = grp * GM + sp * 32 + lane;      // position p_first + pl
    bool ok = true;
    if (warp < NPW) {
        const int r0 = blk * RB + warp * RPW, nv = min(RPW, g.rows - r0);
        const unsigned first = (unsigned)(r0 * g.lds + (job == 0 ? 0 : g.ne)), pitch = (unsigned)g.lds;
        L.produce(spec, nullptr, [&](int i) { return first + i * pitch; }, [](int) { return false; }, nv, g.n,
                  job == 0 ? g.ne : g.no, g.no, 0,
                  img + (job ? tab.inv_base[1] : tab.inv_base[0]) + (size_t)p_first * KCH, tab.Ntot,
                  (uint32_t)wrows * KCH * 4, [](int) {});
        ok = mbar_wait(L.accf(), 0, 4);
        __syncwarp();
        tc_fence_after();
    } else if (lane == 0) {
        L.issue((wrows + GM - 1) / GM);
    }
    __syncwarp();

    // [group, row of the half][128 positions] floats at the start of the stages
    const uint32_t xoff = (uint32_t)((grp * HR + pc * PH) * GM + sp * 32 + lane) * 4u;
    cluster_arrive();
    cluster_wait();                           // both CTAs are past their K loops
    if (warp < NPW) {
        float v[PH];
        tmem_ld<PH>(tlane + (job == 0 ? HR : 0), v);
        const uint32_t dst = mapa_shared(L.sbase + xoff, cluster_rank() ^ 1u);
#pragma unroll
        for (int i = 0; i < PH; ++i) st_cluster_f32(dst + (uint32_t)i * GM * 4u, v[i]);
    }
    cluster_arrive();
    cluster_wait();
    // Staged rows behind the received sums: per row the columns [c1, c1 + n1) of
    // x[p] and [c2, c2 + n2) of the mirrored x[n-1-p] (field columns), each from
    // its column rounded down to a multiple of 4, so that a float4 of shared
    // memory is one of a field whose rows are 16-byte aligned.
    constexpr int SEG = MG * GM + 8, XFL = MG * HR * GM;
    const int n1 = min(MG * GM, g.ne - p_first), n2 = min(MG * GM, g.no - p_first);
    const int c1 = 1 + p_first, c2 = g.n - p_first - n2 + 1;
    if (warp < NPW) {
        float v[PH];
        tmem_ld<PH>(tlane + (job == 0 ? 0 : HR), v);
        const uint32_t st = L.sbase + (uint32_t)(XFL + pc * PH * 2 * SEG) * 4u;
        const uint32_t s1 = st + (uint32_t)(pl + (c1 & 3)) * 4u;
        const uint32_t s2 = st + (uint32_t)(SEG + n2 - 1 - pl + (c2 & 3)) * 4u;
        const bool v1 = pl < n1, v2 = pl < n2;
#pragma unroll
        for (int i = 0; i < PH; ++i) {
            float w;
            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(w) : "r"(L.sbase + xoff + (uint32_t)i * GM * 4u));
            const float A = job == 0 ? v[i] : w, B = job == 0 ? w : v[i];
            if (v1) asm volatile("st.shared.f32 [%0], %1;" ::"r"(s1 + (uint32_t)i * 2 * SEG * 4u), "f"(v2 ? A + B : A) : "memory");
            if (v2) asm volatile("st.shared.f32 [%0], %1;" ::"r"(s2 + (uint32_t)i * 2 * SEG * 4u), "f"(A - B) : "memory");
        }
        asm volatile("bar.sync 1, %0;" ::"n"(NPROD) : "memory");
        if (ok) {
            const int jb = blk * RB + job * HR, rows = min(HR, g.rows - jb);
            const bool vec = (g.nx & 3) == 0 && (((uintptr_t)out | (uintptr_t)add) & 15) == 0;
            // row r of the half: start in the fields, in the mask, and whether it takes the addend
            struct Row { long long o; const int8_t* mk; bool ha; };
            auto locate = [&](int r) {
                const int f = (jb + r) / g.my, j = jb + r - f * g.my + 1;
                return Row{f * g.fs + (long long)j * g.nx, mask + (long long)j * g.nx,
                           add != nullptr && (EPI != EPI_H || (f < add_batches && (!bg_on || bg_on[f])))};
            };
            const float* stage = reinterpret_cast<const float*>(smem_raw) + ((L.sbase - smem_u32(smem_raw)) >> 2) + XFL;
            auto value = [&](const float x, float ad, int8_t mk) {
                return EPI == EPI_ADJQ ? (mk == 3 ? x + ad : 0.f) : x + ad;
            };
            const int cs[2] = {c1, c2}, ce[2] = {c1 + n1, c2 + n2};
            if (vec) {
                // whole float4s of the segments, then their ragged ends; the
                // addend and mask of the next row are loaded ahead
                float4 ad[2][2 * MG];
                char4 m4[2][2 * MG];
                auto fetch = [&](int r, float4 (&a4)[2 * MG], char4 (&k4)[2 * MG]) {
                    const Row R = locate(min(r, rows - 1));
#pragma unroll
                    for (int k = 0; k < 2 * MG; ++k) {
                        const int c = ((cs[k / MG] + 3) & ~3) + 4 * lane + 128 * (k % MG);
                        const bool on = r < rows && c + 4 <= ce[k / MG];
                        a4[k] = on && R.ha ? *reinterpret_cast<const float4*>(add + R.o + c)
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
                        if (EPI == EPI_ADJQ)
                            k4[k] = on ? *reinterpret_cast<const char4*>(R.mk + c) : make_char4(0, 0, 0, 0);
                    }
                };
                auto store = [&](int r, const float4 (&a4)[2 * MG], const char4 (&k4)[2 * MG]) {
                    const Row R = locate(r);
#pragma unroll
                    for (int k = 0; k < 2 * MG; ++k) {
                        const float* sr = stage + (r * 2 + k / MG) * SEG - (cs[k / MG] & ~3);   // by field column
                        const int c = ((cs[k / MG] + 3) & ~3) + 4 * lane + 128 * (k % MG);
                        if (c + 4 <= ce[k / MG]) {
                            float4 x = *reinterpret_cast<const float4*>(sr + c);
                            x.x = value(x.x, a4[k].x, k4[k].x);
                            x.y = value(x.y, a4[k].y, k4[k].y);
                            x.z = value(x.z, a4[k].z, k4[k].z);
                            x.w = value(x.w, a4[k].w, k4[k].w);
                            *reinterpret_cast<float4*>(out + R.o + c) = x;
                        }
                    }
                    // ragged ends: lanes 0-3 / 4-7 the first / last columns of
                    // the first segment, 8-15 those of the second
                    const int sg = lane >> 3 & 1, cb = cs[sg], cl = ce[sg];
                    const int q0 = (cb + 3) & ~3, q1 = cl & ~3;
                    const int c = (lane & 4) ? q1 + (lane & 3) : cb + (lane & 3);
                    if (lane < 16 && c < cl && ((lane & 4) ? c >= q0 : c < q0))
                        out[R.o + c] = value(stage[(r * 2 + sg) * SEG - (cb & ~3) + c], R.ha ? add[R.o + c] : 0.f,
                                             EPI == EPI_ADJQ ? R.mk[c] : (int8_t)3);
                };
                if (warp < rows) fetch(warp, ad[0], m4[0]);
                for (int r = warp; r < rows; r += 2 * NPW) {
                    fetch(r + NPW, ad[1], m4[1]);
                    store(r, ad[0], m4[0]);
                    fetch(r + 2 * NPW, ad[0], m4[0]);
                    if (r + NPW < rows) store(r + NPW, ad[1], m4[1]);
                }
            } else {
                for (int r = warp; r < rows; r += NPW) {
                    const Row R = locate(r);
#pragma unroll
                    for (int sg = 0; sg < 2; ++sg) {
                        const float* sr = stage + (r * 2 + sg) * SEG - (cs[sg] & ~3);
#pragma unroll 4
                        for (int c = cs[sg] + lane; c < ce[sg]; c += 32)
                            out[R.o + c] = value(sr[c], R.ha ? add[R.o + c] : 0.f,
                                                 EPI == EPI_ADJQ ? R.mk[c] : (int8_t)3);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == NPW) {
        tc_fence_after();
        tmem_dealloc(L.tmem, TMEM_COLS);
    }
}

// ---------------------------------------------------------------------------
// Host side: pre-swizzled hi/lo images of the half matrices
// ---------------------------------------------------------------------------
static float tf32_rna_host(float x)
{
    uint32_t b;
    std::memcpy(&b, &x, 4);
    if ((b & 0x7f800000u) != 0x7f800000u) {
        b += 0x1000u;
        b &= 0xFFFFE000u;
    }
    float r;
    std::memcpy(&r, &b, 4);
    return r;
}

struct TcPlanData {
    float* img;
    TcTab tab;
};

int build_tc_images(vd_qg1l_plan* p)
{
    const DSTTables& t = p->dst;
    const int n = t.n, ne = t.ne, no = t.no;
    TcPlanData* d = new TcPlanData();
    std::memset(&d->tab, 0, sizeof(TcTab));
    TcTab& tab = d->tab;
    tab.kch = (ne + KCH - 1) / KCH;
    if (ne > MAX_NE) { delete d; return VD_ERR_UNSUPPORTED; }
    const double scale = std::sqrt(2.0 / (n + 1));
    const long long period = 2LL * (n + 1);
    auto S = [&](long long m) { m %= period; return scale * std::sin(M_PI * double(m) / double(n + 1)); };
    // B operands as [N row][K] functions
    auto fwd_odd = [&](int tt, int pp) { return (tt < ne && pp < ne) ? S((long long)(pp + 1) * (2 * tt + 1)) : 0.0; };
    auto fwd_even = [&](int tt, int pp) { return (tt < no && pp < no) ? S((long long)(pp + 1) * (2 * tt + 2)) : 0.0; };
    auto inv_odd = [&](int pp, int tt) { return (pp < ne && tt < ne) ? S((long long)(pp + 1) * (2 * tt + 1)) : 0.0; };
    auto inv_even = [&](int pp, int tt) { return (pp < no && tt < no) ? S((long long)(pp + 1) * (2 * tt + 2)) : 0.0; };

    std::vector<float> img;
    auto emit = [&](auto fn, int row0, int N) {
        const long long off = (long long)img.size();
        for (int c = 0; c < tab.kch; ++c) {
            std::vector<float> hi(size_t(N) * KCH, 0.f), lo(size_t(N) * KCH, 0.f);
            for (int r = 0; r < N; ++r)
                for (int k = 0; k < KCH; ++k) {
                    const float v = (float)fn(row0 + r, c * KCH + k);
                    const float h = tf32_rna_host(v);
                    const float l = tf32_rna_host(v - h);
                    const uint32_t o = swz(r, k) / 4;
                    hi[o] = h;
                    lo[o] = l;
                }
            img.insert(img.end(), hi.begin(), hi.end());
            img.insert(img.end(), lo.begin(), lo.end());
        }
        return off;
    };
    tab.Ntot = ((ne + 15) / 16) * 16;
    tab.fwd_base[0] = emit(fwd_odd, 0, tab.Ntot);
    tab.fwd_base[1] = emit(fwd_even, 0, tab.Ntot);
    tab.inv_base[0] = emit(inv_odd, 0, tab.Ntot);
    tab.inv_base[1] = emit(inv_even, 0, tab.Ntot);
    if (cudaMalloc(&d->img, img.size() * sizeof(float)) != cudaSuccess) { delete d; return VD_ERR_CUDA; }
    if (cudaMemcpy(d->img, img.data(), img.size() * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaFree(d->img);
        delete d;
        return VD_ERR_CUDA;
    }
    p->dst.tc = d;
    return VD_OK;
}

void free_tc_images(vd_qg1l_plan* p)
{
    TcPlanData* d = (TcPlanData*)p->dst.tc;
    if (!d) return;
    cudaFree(d->img);
    delete d;
    p->dst.tc = nullptr;
}

static PerDeviceOnce g_tc_once;

// Calls fn(integral constants RPW, MG) of a launch shape.
template <typename F>
static auto tc_shape(int rb, int mg, F&& fn)
{
    if (mg == 2) {
        if (rb == 128) return fn(std::integral_constant<int, 8>(), std::integral_constant<int, 2>());
        if (rb == 64) return fn(std::integral_constant<int, 4>(), std::integral_constant<int, 2>());
        return fn(std::integral_constant<int, 2>(), std::integral_constant<int, 2>());
    }
    if (rb == 128) return fn(std::integral_constant<int, 8>(), std::integral_constant<int, 1>());
    if (rb == 64) return fn(std::integral_constant<int, 4>(), std::integral_constant<int, 1>());
    return fn(std::integral_constant<int, 2>(), std::integral_constant<int, 1>());
}

// Clusters of 1..MAX_NR CTAs (one CTA per SM) that run at once on each device.
static int g_tc_clusters[PerDeviceOnce::kMaxDevices][MAX_NR + 1];

static cudaError_t tc_configure()
{
    return g_tc_once.run([]() -> cudaError_t {
        cudaError_t e = cudaSuccess;
        auto set = [&](const void* k) {
            if (!e) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(SMEM_MAX - SMEM_STATIC));
        };
        for (int rb : {32, 64, 128})
            for (int mg : {1, 2})
                tc_shape(rb, mg, [&](auto R, auto M) {
                    set((const void*)dst_tc_fwd_kernel<R(), M(), true>);
                    set((const void*)dst_tc_fwd_kernel<R(), M(), false>);
                    set((const void*)dst_tc_inv_kernel<R(), M(), EPI_H>);
                    set((const void*)dst_tc_inv_kernel<R(), M(), EPI_ADJQ>);
                });
        int dev = 0;
        if (!e) e = cudaGetDevice(&dev);
        for (int c = 1; c <= MAX_NR && !e; ++c) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)c);
            cfg.blockDim = dim3(NTHREADS);
            cfg.dynamicSmemBytes = SMEM_MAX - SMEM_STATIC;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = (unsigned)c;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            e = cudaOccupancyMaxActiveClusters(&g_tc_clusters[dev][c], dst_tc_fwd_kernel<8, 2, true>, &cfg);
        }
        return e;
    });
}

// Batches are limited to 2^31 elements (the other float32 kernels' offsets).
bool tc_fits(const vd_qg1l_plan* p, int nf)
{
    const DSTTables& t = p->dst;
    const long long fs = (long long)p->d.ny * p->d.nx;
    return (long long)nf * fs < (1LL << 31) && (long long)nf * t.my * t.lds < (1LL << 31);
}

struct TcPick { int rb, mg; double us; };

// Rows and groups of a CTA: the shape with the least estimated time. A CTA's time
// is a fixed part that grows with the values it stores and its K chunks, whose
// cost grows with the rows it splits and the products it issues (microseconds,
// fitted to single-wave launches at 128^2 to 1024^2: a forward pass measured 16.7
// at 16 x 512^2 with 128 rows and two groups; 16.0 at 1024^2 with 64 rows and one
// group, 22.3 with 128 and one, 25.3 with 128 and two); clusters beyond those that
// run at once take further waves. `fuse`: the blocks of a field are one cluster,
// and the epilogue also solves.
static TcPick tc_pick(const vd_qg1l_plan* p, int nf, bool fwd, bool fuse)
{
    const DSTTables& t = p->dst;
    const int forced = fwd ? p->sched.tc_group_fwd : p->sched.tc_group_inv;
    int dev = 0;
    cudaGetDevice(&dev);
    const int kch = (t.ne + KCH - 1) / KCH;
    auto cost = [&](int rb, int mg) {
        const int nr = (t.my + rb - 1) / rb, groups = (t.ne + GM * mg - 1) / (GM * mg);
        if (fuse && nr > MAX_NR) return 1e30;
        const int csz = fuse ? nr : fwd ? 1 : 2;
        const long long blocks = fuse ? (long long)nf * nr : ((long long)nf * t.my + rb - 1) / rb;
        const long long clusters = (2LL * blocks * groups + csz - 1) / csz;
        const int at_once = std::max(1, g_tc_clusters[dev][csz]);
        const double fixed = (fwd ? 3.0 + 0.019 * rb * mg : 4.5 + 0.025 * rb * mg) + (fuse ? 3.5 : 0.0);
        const double chunk = 0.55 + 0.0031 * rb + (rb >= 128 ? 0.16 : 0.3) * (mg - 1) + (fuse ? 0.1 : 0.0);
        return double((clusters + at_once - 1) / at_once) * (fixed + kch * chunk);
    };
    TcPick best{128, 1, 1e30};
    for (int rb : {128, 64, 32})
        for (int mg : {1, 2}) {
            if (mg == 2 && t.ne <= GM) continue;
            const double c = cost(rb, mg);
            if (c < best.us) best = TcPick{rb, mg, c};
        }
    if (forced) {
        const int rb = forced >= 4 ? 128 : forced == 2 ? 64 : 32, mg = forced == 8 ? 2 : 1;
        const double c = cost(rb, mg);
        if (c < 1e29) best = TcPick{rb, mg, c};
    }
    return best;
}

// Whether the forward pass also solves the tridiagonal systems: not for fields
// whose row blocks exceed a cluster, nor where the plain pass with its freer shape
// and the separate solve (measured 3.5 us and 3.1 us per million points) are
// cheaper: single tall fields (1024^2: 16 + 6 us against 27 us fused; at
// 16 x 512^2 22 us fused against 17 + 16).
static bool tc_fusable(const vd_qg1l_plan* p, int nf)
{
    const DSTTables& t = p->dst;
    const TcPick f = tc_pick(p, nf, true, true);
    return f.us < 1e29 && f.us < tc_pick(p, nf, true, false).us + 4.5 + 3.1e-6 * nf * t.my * (double)t.n;
}

static int tc_launch_fwd(const vd_qg1l_plan* p, int nf, const SolveArgs& a, float* spec, bool fuse, cudaStream_t st)
{
    const TcPlanData* d = (const TcPlanData*)p->dst.tc;
    const DSTTables& t = p->dst;
    const TcPick c = tc_pick(p, nf, true, fuse);
    TcGeom g;
    g.n = t.n; g.ne = t.ne; g.no = t.no; g.my = t.my; g.nx = p->d.nx;
    g.fs = (long long)p->d.ny * p->d.nx;
    g.lds = t.lds;
    g.nr = fuse ? (t.my + c.rb - 1) / c.rb : 1;
    g.rows = nf * t.my;
    const cudaError_t e = tc_shape(c.rb, c.mg, [&](auto R, auto M) {
        using Sh = TcShape<R(), M()>;
        TcTab tab = d->tab;
        const size_t exch = fuse ? Sh::exch_bytes(g.nr) : 0;
        tab.nst = (int)std::min<size_t>(MAX_STAGES, (SMEM_MAX - SMEM_STATIC - 1024 - exch) / Sh::STAGE);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(fuse ? nf * g.nr : (g.rows + Sh::RB - 1) / Sh::RB), 2 * ((t.ne + GM * M() - 1) / (GM * M())));
        cfg.blockDim = dim3(NTHREADS);
        cfg.dynamicSmemBytes = std::max(SMEM_ONE, tab.nst * (size_t)Sh::STAGE + exch + 1024);
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = fuse ? (unsigned)g.nr : 1u;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        const float *src = (const float*)a.src, *sub = (const float*)a.sub, *trim = (const float*)t.trim;
        const float ta = (float)t.tri_a;
        return fuse ? cudaLaunchKernelEx(&cfg, dst_tc_fwd_kernel<R(), M(), true>, g, tab, (const float*)d->img, src,
                                         sub, a.sub_batches, a.bg_on, spec, trim, ta)
                    : cudaLaunchKernelEx(&cfg, dst_tc_fwd_kernel<R(), M(), false>, g, tab, (const float*)d->img, src,
                                         sub, a.sub_batches, a.bg_on, spec, trim, ta);
    });
    if (e != cudaSuccess) return VD_ERR_CUDA;
    VD_LAUNCH_CHECK();
    return VD_OK;
}

static int tc_launch_inv(const vd_qg1l_plan* p, int nf, const SolveArgs& a, const float* spec, cudaStream_t st)
{
    const TcPlanData* d = (const TcPlanData*)p->dst.tc;
    const DSTTables& t = p->dst;
    const TcPick c = tc_pick(p, nf, false, false);
    TcGeom g;
    g.n = t.n; g.ne = t.ne; g.no = t.no; g.my = t.my; g.nx = p->d.nx;
    g.fs = (long long)p->d.ny * p->d.nx;
    g.lds = t.lds;
    g.nr = 1;
    g.rows = nf * t.my;
    const cudaError_t e = tc_shape(c.rb, c.mg, [&](auto R, auto M) {
        using Sh = TcShape<R(), M()>;
        TcTab tab = d->tab;
        tab.nst = (int)std::min<size_t>(MAX_STAGES, (SMEM_MAX - SMEM_STATIC - 1024) / Sh::STAGE);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2u * (unsigned)((g.rows + Sh::RB - 1) / Sh::RB), (t.ne + GM * M() - 1) / (GM * M()));
        cfg.blockDim = dim3(NTHREADS);
        cfg.dynamicSmemBytes =
            std::max(SMEM_ONE, std::max<size_t>(tab.nst * (size_t)Sh::STAGE, Sh::INV_EPI) + 1024);
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 2;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        return a.epi == EPI_H ? cudaLaunchKernelEx(&cfg, dst_tc_inv_kernel<R(), M(), EPI_H>, g, tab,
                                                   (const float*)d->img, spec, (float*)a.out, (const float*)a.add,
                                                   a.add_batches, a.bg_on, (const int8_t*)p->d_mask)
                              : cudaLaunchKernelEx(&cfg, dst_tc_inv_kernel<R(), M(), EPI_ADJQ>, g, tab,
                                                   (const float*)d->img, spec, (float*)a.out, (const float*)a.add,
                                                   a.add_batches, a.bg_on, (const int8_t*)p->d_mask);
    });
    if (e != cudaSuccess) return VD_ERR_CUDA;
    VD_LAUNCH_CHECK();
    return VD_OK;
}

// One x-direction pass on the tensor cores (forward: fields -> spec,
// inverse: spec -> out with the epilogue of `a`).
int dst_pass_tc(const vd_qg1l_plan* p, int nf, const SolveArgs& a, float* spec, bool fwd, cudaStream_t st)
{
    if (!p->dst.tc || !tc_fits(p, nf)) return VD_ERR_UNSUPPORTED;
    if (tc_configure() != cudaSuccess) return VD_ERR_CUDA;
    return fwd ? tc_launch_fwd(p, nf, a, spec, false, st) : tc_launch_inv(p, nf, a, spec, st);
}

// Forward pass and tridiagonal solve in one kernel; *done says whether the
// field's rows fit (else nothing was launched).
int dst_solve_tc(const vd_qg1l_plan* p, int nf, const SolveArgs& a, float* spec, bool* done, cudaStream_t st)
{
    if (!p->dst.tc || !tc_fits(p, nf)) return VD_ERR_UNSUPPORTED;
    if (tc_configure() != cudaSuccess) return VD_ERR_CUDA;
    *done = tc_fusable(p, nf);
    if (!*done) return VD_OK;
    return tc_launch_fwd(p, nf, a, spec, true, st);
}

}  // namespace vd

extern "C" vd_status vd_device_error(int* flags, int reset)
{
    if (!flags) return VD_ERR_ARG;
    VD_CUDA_TRY(cudaMemcpyFromSymbol(flags, vd::g_tc_error, sizeof(int)));
    if (reset) {
        const int zero = 0;
        VD_CUDA_TRY(cudaMemcpyToSymbol(vd::g_tc_error, &zero, sizeof(int)));
    }
    return (vd_status)vd::qg_tile_error(flags, reset);
}
