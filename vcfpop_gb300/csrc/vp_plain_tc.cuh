// The plain form's two contractions over 2-bit biallelic diploid genotypes on
// the tensor cores (sm_103a), for one chain: the no-admixture likelihood
// LL[i, k] (UpdateQNoAdmix, src/structure.cpp:902-932) and the allele counts
// Ni (UpdateZNoAdmix, src/structure.cpp:1257-1348).
//
// Both multiply a matrix of genotype counts 0, 1, 2 by a narrow matrix (the
// clusters), so the counts are never stored: builder warps decode 2-bit words
// in registers and write them straight into tensor memory (tcgen05.st), where
// tcgen05.mma reads its A operand; the narrow B operand comes through shared
// memory. A ring of A stages in tensor memory lets the decoding run ahead of
// the MMAs. Every wait is bounded: on time-out the CTA records an error in its
// chain's control block (read with the chain's results), waits for the copies
// and MMAs in flight, frees its tensor memory and returns.
#pragma once
#include "vp_admix.cuh"
#include "vp_tc.cuh"

namespace vp {
namespace ptc {

using tc::mbar_expect_tx;
using tc::mbar_init;
using tc::mma_commit;
using tc::mbar_wait;
using tc::smem_u32;

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// A from tensor memory; one-byte floats (the formats are in idesc)
__device__ __forceinline__ void mma_f8_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d),
        "r"(a), "l"(bdesc), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void tmem_st16(uint32_t t, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(t),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[j]);
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t bar_done(uint32_t bar, uint32_t parity) {
    uint32_t d;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(d)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return d;
}
// Waits on a phase of the barrier at shared address bar, by a thread or by a
// whole warp, which takes one way. The first poll is the common case and all
// that is inlined: a stage's waits and arrivals are a chain of dependent
// instructions on few warps, and their length sets the kernels' pace. A wait
// that runs out (abort[1] polls), or finds that another warp's has (abort[0]),
// ends the CTA's work (false).
__device__ __noinline__ bool bar_wait_long(uint32_t bar, uint32_t parity, bool warp, volatile int* abort, int* err, int code) {
    const int limit = abort[1];
    for (int it = 0; it < limit; ++it) {
        const uint32_t d = bar_done(bar, parity);
        if (warp ? __all_sync(0xffffffffu, d) : d) return true;
        if ((it & 255) == 255 && (warp ? __any_sync(0xffffffffu, *abort) : *abort)) return false;
    }
    *abort = 1;
    atomicExch(err, code);
    return false;
}
__device__ __forceinline__ bool thread_wait(uint32_t bar, uint32_t parity, volatile int* abort, int* err, int code) {
    return bar_done(bar, parity) || bar_wait_long(bar, parity, false, abort, err, code);
}
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort, int* err, int code) {
    return __all_sync(0xffffffffu, bar_done(bar, parity)) || bar_wait_long(bar, parity, true, abort, err, code);
}
// polls of a wait; few where a diagnostic has the waits run out (DevChain::stall)
__device__ __forceinline__ int poll_limit(const DevChain& c) { return c.stall ? 1 << 12 : (int)tc::SPIN_LIMIT; }
// a place in a ring of ST stages: its index and how often it has come round
template <int ST>
struct Ring {
    int s = 0;
    uint32_t round = 0;
    __device__ __forceinline__ void step(int d = 1) {
        s += d;
        if (s >= ST) { s -= ST; ++round; }
    }
};

// ---- the likelihood, exact ------------------------------------------------
// ln p is taken to about 2^-29 of its value (ln_split) in units of 2^-29, in
// seven digits to base 32, exact in e4m3 as the copies 0, 1, 2 are (ln_digits).
// A digit is at most 352 in magnitude (in the logarithm of a zero frequency; at
// most 64 else, 16 from p = 1e-14 up), so a locus adds at most 2 x 352 to its
// sum, and the FP32 accumulator holds whole numbers up to 2^24: the sums of 2^14
// loci are exact whatever the order of the adds, and the digits combine in
// 64-bit integers. What rounds is a copy's logarithm.
// LL against float64, rms relative, and the FP32 stream's on the same inputs:
// frequencies from Beta(1/2, 1/2) 3e-12 to 4e-12 and 1.7e-9 to 4.0e-9, from a 1/x
// spectrum 1e-11 and 3.3e-9, around 1%, 0.1%, 0.01% and 0.001% 7e-12 to 3.4e-11 and
// 2.7e-9 to 5.9e-9 (N = 512 and 1,000, L = 32,000 and 100,000, K = 3, 6 and 10).
constexpr int LL_LOCI = 32;                        // loci of a stage: 64 A bytes (copies of allele 1 and 0 of each)
constexpr int LL_MAXST = (1 << 14) / LL_LOCI;
constexpr int LL_M = 256;                          // individuals per CTA: two 128-row tiles share a B stage
constexpr int LL_TEAM = 8;                         // builder warps of a stage: one per 32 individuals
constexpr int LL_BW = 2 * LL_TEAM;                 // two teams take alternate stages
constexpr int LL_THREADS = (LL_BW + 2) * 32;       // the builders, the MMA warp, the B producer
constexpr int LL_TCK = 32;                         // most clusters
constexpr int LL_PF = 4;                           // stages of genotype words in flight
__host__ __device__ constexpr int ll_rows(int K) {   // B rows: seven digits a cluster, a compiled width
    return K <= 4 ? 32 : K <= 6 ? 48 : K <= 11 ? 80 : K <= 16 ? 112 : 224;
}
// tensor memory: two accumulators of NB columns, then stages of 2 x 16 columns;
// half of it (two CTAs per SM) where that leaves three stages
template <int NB>
struct LlShape {
    static constexpr int COLS = NB <= 80 ? 256 : 512;
    static constexpr int FIT = (COLS - 2 * NB) / 32;
    static constexpr int ST = FIT > 4 ? 4 : FIT;
    static_assert(ST >= 2, "two stages");
};

// e4m3 bytes of a code's copies of allele 1 (0, 1, 2, missing 0) and of allele 0
// (2, 1, 0, 0)
constexpr uint32_t E4_A1 = 0x00403800u, E4_A0 = 0x00003840u;
// 16 calls of one word to 32 bytes: four registers of copies of allele 1, four
// of allele 0; register b's byte e is call 8 (b / 2) + (b & 1) + 2 e
// (the codes at the selector's nibbles after one shift)
__device__ __forceinline__ void calls_to_e4m3(uint32_t w, uint32_t* r) {
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const uint32_t sel = (w >> (16 * (b >> 1) + 2 * (b & 1))) & 0x3333u;
        r[b] = __byte_perm(E4_A1, 0u, sel);
        r[4 + b] = __byte_perm(E4_A0, 0u, sel);
    }
}

// the FP32 stream's table from the frequencies, by thread t of nt
__device__ __noinline__ void fill_lt(const DevChain& c, int64_t t, int64_t nt) {
    const int64_t L = c.D.L;
    for (; t < (int64_t)c.K * L; t += nt) {
        const int k = (int)(t / L);
        const int64_t l = t - k * L;
        write_lt(c, k, l, c.Freq + (int64_t)k * c.D.KT + 2 * l, 2);
    }
}

// CTA: LL_M individuals x the stages of its chunk (grid.y). The dependent
// instructions of a stage (copies, shuffles, byte permutes, waits, a store) set
// the pace: halving the MMAs or the ring changed nothing, so two teams of
// builders take alternate stages and a wait's first poll is all that is inlined.
// N = 10,000 x L = 60,000, K = 10: 149 us (680 for the FP32 stream; 271 with f16
// digits and a team, 232 with one-byte digits, 180 with the words copied
// ahead, in shorter runs); ALU pipe 60%, issue 66%, tensor pipe 29%, DRAM 1.1 TB/s. Lane n of a
// builder warp is individual n / 2 of the warp's first genotype word or of its
// second, by n's last bit (the in-register transpose's order).
template <int NB>
__global__ void __launch_bounds__(LL_THREADS, NB <= 80 ? 2 : 1) k_loglik_tc(const DevChain* chains, const int4* map = nullptr) {
    using S = LlShape<NB>;
    constexpr int ST = S::ST;
    constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(NB >> 3) << 17) | (8u << 24);   // e4m3 x e4m3 -> f32, 128 rows
    __shared__ __align__(1024) unsigned char sB[ST][NB * 64];
    __shared__ __align__(16) uint32_t sW[LL_BW][LL_PF][LL_LOCI][2];
    __shared__ uint64_t full[ST], fullB[ST], empty[ST], accum;
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort[2];
    const VBlock vb = vblock(map);
    const DevChain& c = chains[vb.z];
    if (map && run_over(c)) return;
    const int m = c.ctl->m;
    if (!ll_tc_at(c, m)) {
        if (ll_tc_turn(c, m))
            fill_lt(c, ((int64_t)vb.y * vb.gx + vb.x) * LL_THREADS + threadIdx.x, (int64_t)vb.gx * c.tcchunk * LL_THREADS);
        return;
    }
    const DevData& D = c.D;
    const int K = c.K;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nst = (int)((D.L + LL_LOCI - 1) / LL_LOCI), per = c.tcper;
    const int st0 = vb.y * per, n = min(nst, st0 + per) - st0;
    if (n <= 0) return;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) { mbar_init(&full[s], 8); mbar_init(&fullB[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(&accum, 1);
        s_abort[0] = 0;
        s_abort[1] = poll_limit(c);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == LL_BW) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(S::COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = s_tmem, ring = tmem + 2 * NB;
    int* err = &c.ctl->err;
    const uint32_t full0 = smem_u32(&full[0]), fullB0 = smem_u32(&fullB[0]), empty0 = smem_u32(&empty[0]);
    if (warp < LL_BW) {
        const int team = warp / LL_TEAM, tile = (warp >> 2) & 1, q = warp & 3;
        const int ib = vb.x * LL_M + (warp % LL_TEAM) * 32;
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        const BitTranspose tr(lane);
        // the warp's two genotype words of a stage's loci (lane = locus), copied
        // asynchronously LL_PF stages ahead; zeros past the last locus, where
        // the digits are zero too, and past the last word
        const int64_t l0 = (int64_t)st0 * LL_LOCI + lane;
        const bool wok = (ib >> 4) < D.Nw;
        const uint32_t* gp = D.g2 + l0 * D.Nw + (ib >> 4);
        auto fetch = [&](int u) {        // the team's u-th stage
            const int it = 2 * u + team;
            const bool ok = wok && it < n && l0 + (int64_t)it * LL_LOCI < D.L;
            cp_async8(&sW[warp][u % LL_PF][lane][0], ok ? gp + (int64_t)it * LL_LOCI * D.Nw : D.g2, ok);
            cp_async_commit();
        };
        for (int u = 0; u < LL_PF - 1; ++u) fetch(u);
        Ring<ST> r_;
        r_.step(team);
        for (int u = 0, it = team; it < n; ++u, it += 2, r_.step(2)) {
            const int s = r_.s;
            fetch(u + LL_PF - 1);        // into the buffer that the stage before was read from
            cp_async_wait<LL_PF - 1>();
            __syncwarp();
            const uint32_t* sw = &sW[warp][u % LL_PF][0][0];
            const uint32_t w0 = sw[lane], w1 = sw[32 + lane];
            __syncwarp();
            uint32_t r[16];
            calls_to_e4m3(tr.codes(w0), r);
            calls_to_e4m3(tr.codes(w1), r + 8);
            if (r_.round && !warp_wait(empty0 + 8 * s, (r_.round & 1) ^ 1, s_abort, err, 11)) break;
            fence_after();
            tmem_st16(ring + lanes + (uint32_t)(s * 32 + tile * 16), r);
            wait_st();
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
        cp_async_wait<0>();
        // the digits' sums of this lane's individual
        const bool got = warp_wait(smem_u32(&accum), 0, s_abort, err, 12) && !*(volatile int*)s_abort;
        fence_after();
        const int i = ib + (lane >> 1) + 16 * (lane & 1);
        double* out = c.LLp + ((int64_t)vb.y * D.N + i) * K;
#pragma unroll 1
        for (int k = team; k < K; k += 2) {
            float v[8];
            tmem_ld8(tmem + lanes + (uint32_t)(tile * NB + 7 * k), v);
            if (!got || i >= D.N) continue;
            long long t = 0;
#pragma unroll
            for (int j = 6; j >= 0; --j) t = t * 32 + __float2int_rn(v[j]);
            out[k] = (double)t * LL_UNIT;
        }
    } else if (warp == LL_BW) {
        if (lane == 0) {
            const uint64_t d0 = tc::sw_desc(smem_u32(&sB[0][0]), 64);
            Ring<ST> r_;
            for (int it = 0; it < n; ++it, r_.step()) {
                const int s = r_.s;
                if (!thread_wait(fullB0 + 8 * s, r_.round & 1, s_abort, err, 15) || !thread_wait(full0 + 8 * s, r_.round & 1, s_abort, err, 13)) break;
                fence_after();
                const uint64_t bd = d0 + (uint64_t)((s * NB * 64) >> 4);
#pragma unroll
                for (int t = 0; t < 2; ++t)
#pragma unroll
                    for (int kk = 0; kk < 2; ++kk)
                        mma_f8_ts(tmem + (uint32_t)(t * NB), ring + (uint32_t)(s * 32 + t * 16 + kk * 8), bd + (uint64_t)(kk * 2),
                                   IDESC, (it | kk) ? 1u : 0u);
                mma_commit(&empty[s]);
            }
            // also when a wait has run out: it arrives once the MMAs issued are done,
            // and tensor memory is not given back before
            mma_commit(&accum);
            mbar_wait(&accum, 0);
        }
    } else if (lane == 0) {
        const uint32_t tx = NB * 64 + c.stall;
        const char* src = reinterpret_cast<const char*>(c.ltd) + (int64_t)st0 * (NB * 64);
        int issued = 0;
        Ring<ST> r_;
        for (int it = 0; it < n; ++it, r_.step()) {
            const int s = r_.s;
            if (r_.round && !thread_wait(empty0 + 8 * s, (r_.round & 1) ^ 1, s_abort, err, 14)) break;
            mbar_expect_tx(&fullB[s], tx);
            bulk_load(&sB[s][0], src + (int64_t)it * (NB * 64), NB * 64, &fullB[s]);
            issued = it + 1;
        }
        // every copy issued has landed before the CTA may exit
        for (int it = issued > ST ? issued - ST : 0; it < issued; ++it) mbar_wait(&fullB[it % ST], (it / ST) & 1, s_abort[1]);
    }
    fence_before();
    __syncthreads();
    if (warp == LL_BW) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::COLS));
    }
}

// ---- the counts -----------------------------------------------------------
// Per CTA 128 loci (one a lane of a team of four builder warps); stages of 128
// individuals. A call is one e5m2 byte: its copies of allele 1, or CT_MISS for
// a missing call, so that one matrix gives both counts: over at most CT_GROUP
// stages a cluster's sum is copies + CT_MISS x missing calls with copies below
// CT_MISS, a whole number below 2^24, and so exact. Two accumulators alternate
// between groups; the builders take one apart while the MMAs fill the other.
// B is the one-hot matrix of the labels, written once per sweep by k_onehot as
// the shared-memory image of the stages (a warp of each CTA building it set the
// kernel's pace: 172 us against 125), with the clusters' sizes: copies of
// allele 0 are 2 (size - missing) - copies of allele 1.
// Bound, as the likelihood, by the builders' and waits' dependent instructions.
// N = 10,000 x L = 60,000, K = 10: 93 us against 307 for the bit-plane kernel's
// population counts (125 with one team of builders and longer waits).
constexpr int CT_IND = 128, CT_M = 128, CT_BW = 8;   // two teams of four builder warps take alternate stages
constexpr int CT_THREADS = (CT_BW + 3) * 32;         // the builders, MMA, B producer, cluster sizes
constexpr int CT_PITCH = 48;                         // bytes of a staged row: 32 and a 16-byte pad (odd chunks)
constexpr int DRAIN_AT = 7;                          // stage of a group after which the group before is taken apart
constexpr int CT_MISS = 1 << 12, CT_GROUP = (CT_MISS - 1) / (2 * CT_IND);   // 15 stages: 3,840 copies
static_assert((int64_t)CT_MISS * CT_GROUP * CT_IND + CT_MISS < (1 << 24), "exact sums");
__host__ __device__ constexpr int ct_rows(int K) { return K <= 16 ? 16 : 32; }
template <int NB>
struct CtShape {
    static constexpr int COLS = 256, FIT = (COLS - 2 * NB) / 32, ST = FIT > 4 ? 4 : FIT;
    static constexpr int PF = NB == 16 ? 3 : 2;      // a team's stages of genotype words in flight
};
// e5m2 bytes by code: 0, 1, 2, 4096
constexpr uint32_t E5_CODE = 0x6C403C00u, E5_ONE = 0x3Cu;
// The one-hot image: per stage ct_rows(K) rows of 128 bytes with the 16-byte
// chunks of row k exchanged by k mod 8 (the 128-byte swizzle); byte 16 w + 4 u +
// e of a row is individual 16 w + 8 (u / 2) + (u & 1) + 2 e (the builders'
// order). Behind the stages the sizes, [stage][row]. One block per stage.
__global__ void __launch_bounds__(CT_IND) k_onehot(const DevChain* chains, int force, const int4* map = nullptr) {
    const VBlock vb = vblock(map);
    const DevChain& c = chains[vb.z];
    if (map && counts_over(c)) return;
    if (!force && !binaryq_at(c, c.ctl->m)) return;
    const int N = c.D.N, NB = ct_rows(c.K), t = threadIdx.x;
    __shared__ uint16_t z[CT_IND];
    __shared__ int nk[32];
    if (t < NB) nk[t] = 0;
    const int i = vb.x * CT_IND + t;
    z[t] = i < N ? c.Z[i] : 0xFFFF;
    __syncthreads();
    // a label set from outside may be any number: one without a row is in no
    // cluster, here and in the rows below (as in k_count_packed)
    if (z[t] < NB) atomicAdd(&nk[z[t]], 1);
    // thread t: words t & 31 of rows t / 32, t / 32 + 4, ...
    const int w = t & 31, i0 = 16 * (w >> 2) + 8 * ((w >> 1) & 1) + (w & 1);
    uint32_t* B = reinterpret_cast<uint32_t*>(c.oh + (int64_t)vb.x * NB * 128);
    for (int k = t >> 5; k < NB; k += CT_IND / 32) {
        uint32_t v = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) v |= z[i0 + 2 * e] == k ? E5_ONE << (8 * e) : 0u;
        B[k * 32 + (((w >> 2) ^ (k & 7)) << 2) + (w & 3)] = v;
    }
    __syncthreads();
    const int n = (N + CT_IND - 1) / CT_IND;
    if (t < NB) reinterpret_cast<int*>(c.oh + (int64_t)n * NB * 128)[vb.x * NB + t] = nk[t];
}
template <int NB>
__global__ void __launch_bounds__(CT_THREADS, NB == 16 ? 2 : 1) k_count_tc(const DevChain* chains, int force, const int4* map = nullptr) {
    using S = CtShape<NB>;
    constexpr int ST = S::ST, PF = S::PF;
    // e5m2 x e5m2 -> f32, 128 rows
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NB >> 3) << 17) | (8u << 24);
    __shared__ __align__(1024) unsigned char sB[ST][NB * 128];
    __shared__ __align__(16) unsigned char sG[CT_BW][PF][32 * CT_PITCH];
    __shared__ uint64_t full[ST], fullB[ST], empty[ST], dfull[2], dempty[2], drained;
    __shared__ int s_nk[NB];
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort[2];
    const VBlock vb = vblock(map);
    const DevChain& c = chains[vb.z];
    if (map && counts_over(c)) return;
    if (!force && !binaryq_at(c, c.ctl->m)) return;
    const DevData& D = c.D;
    const int K = c.K;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = (D.N + CT_IND - 1) / CT_IND, ngr = (n + CT_GROUP - 1) / CT_GROUP;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) { mbar_init(&full[s], 4); mbar_init(&fullB[s], 1); mbar_init(&empty[s], 1); }
        for (int d = 0; d < 2; ++d) { mbar_init(&dfull[d], 1); mbar_init(&dempty[d], 4); }
        mbar_init(&drained, 1);
        s_abort[0] = 0;
        s_abort[1] = poll_limit(c);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == CT_BW) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(S::COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = s_tmem, ring = tmem + 2 * NB;
    int* err = &c.ctl->err;
    const uint32_t full0 = smem_u32(&full[0]), fullB0 = smem_u32(&fullB[0]), empty0 = smem_u32(&empty[0]);
    const uint32_t dfull0 = smem_u32(&dfull[0]), dempty0 = smem_u32(&dempty[0]);
    int a1[NB], ms[NB];          // this lane's locus: copies of allele 1 and missing calls by cluster
    if (warp < CT_BW) {
        const int team = warp >> 2;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        const int64_t lw = (int64_t)vb.x * CT_M + (warp & 3) * 32;
#pragma unroll
        for (int k = 0; k < NB; ++k) { a1[k] = 0; ms[k] = 0; }
        // a stage's 8 words of this warp's 32 rows, by 16-byte asynchronous
        // copies PF - 1 of the team's stages ahead; a row's words past its end
        // (and rows past the last locus) are filled with zeros, whose individuals
        // have no label
        const int ch = lane & 1;
        const uint32_t* gp = D.g2 + (lw + (lane >> 1)) * D.Nw + ch * 4;
        const bool ok0 = lw + (lane >> 1) < D.L, ok1 = lw + 16 + (lane >> 1) < D.L;
        unsigned char* dst = &sG[warp][0][(lane >> 1) * CT_PITCH + ch * 16];
        auto fetch = [&](int u) {            // the team's u-th stage
            const int w = (2 * u + team) * 8;
            const bool in = w + ch * 4 < D.Nw;
            unsigned char* d = dst + (u % PF) * (32 * CT_PITCH);
            cp_async16(d, in && ok0 ? gp + w : D.g2, in && ok0);
            cp_async16(d + 16 * CT_PITCH, in && ok1 ? gp + 16 * (int64_t)D.Nw + w : D.g2, in && ok1);
            cp_async_commit();
        };
        auto drain = [&](int g) {
            if (!warp_wait(dfull0 + 8 * (g & 1), (g >> 1) & 1, s_abort, err, 22)) return false;
            fence_after();
#pragma unroll
            for (int b = 0; b < NB; b += 16) {
                float v[16];
                tc::tmem_ld16(tmem + lanes + (uint32_t)((g & 1) * NB + b), v);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int x = __float2int_rn(v[j]);
                    a1[b + j] += x & (CT_MISS - 1);
                    ms[b + j] += x >> 12;
                }
            }
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&dempty[g & 1]);
            return true;
        };
        bool run = true;
        for (int u = 0; u < PF - 1; ++u) fetch(u);
        Ring<ST> r_;
        r_.step(team);
        int since = team;                    // stages since the group began
        for (int u = 0, it = team; it < n; ++u, it += 2, r_.step(2)) {
            const int s = r_.s;
            fetch(u + PF - 1);            // into the buffer that the stage before was read from
            cp_async_wait<PF - 1>();
            __syncwarp();
            const unsigned char* my = &sG[warp][u % PF][lane * CT_PITCH];
            const uint4 x = *reinterpret_cast<const uint4*>(my), y = *reinterpret_cast<const uint4*>(my + 16);
            __syncwarp();
            const uint32_t wd[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
            if (r_.round && !warp_wait(empty0 + 8 * s, (r_.round & 1) ^ 1, s_abort, err, 21)) { run = false; break; }
            fence_after();
            const uint32_t a = ring + lanes + (uint32_t)(s * 32);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t r[16];
#pragma unroll
                for (int v = 0; v < 4; ++v)
#pragma unroll
                    for (int b = 0; b < 4; ++b)
                        // codes b', b' + 2, b' + 4, b' + 6 of a half word (b' = b & 1, the half by b >> 1)
                        r[4 * v + b] = __byte_perm(E5_CODE, 0u, (wd[4 * h + v] >> (16 * (b >> 1) + 2 * (b & 1))) & 0x3333u);
                tmem_st16(a + 16 * h, r);
            }
            wait_st();
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
            // the first team takes a group apart halfway through the next, when
            // its MMAs are long done
            if (team == 0 && since >= DRAIN_AT && since < DRAIN_AT + 2 && it > CT_GROUP && !drain(it / CT_GROUP - 1)) {
                run = false;
                break;
            }
            since = since + 2 >= CT_GROUP ? since + 2 - CT_GROUP : since + 2;
        }
        cp_async_wait<0>();
        // groups not yet taken apart
        if (team == 0) {
            const int last = ((n - 1) & ~1), g = last / CT_GROUP, r = last - g * CT_GROUP;    // the team's last stage
            for (int d = max(0, r >= DRAIN_AT ? g : g - 1); d < ngr && run; ++d) run = drain(d);
        }
        if (!run) a1[0] = -1;                // nothing is written
    } else if (warp == CT_BW) {
        if (lane == 0) {
            const uint64_t d0 = tc::sw_desc(smem_u32(&sB[0][0]), 128);
            Ring<ST> r_;
            Ring<CT_GROUP> g_;
            for (int it = 0; it < n; ++it, r_.step(), g_.step()) {
                const int s = r_.s, g = (int)g_.round;
                const bool first = g_.s == 0;
                if ((first && g >= 2 && !thread_wait(dempty0 + 8 * (g & 1), ((g >> 1) & 1) ^ 1, s_abort, err, 25)) ||
                    !thread_wait(fullB0 + 8 * s, r_.round & 1, s_abort, err, 26) || !thread_wait(full0 + 8 * s, r_.round & 1, s_abort, err, 23))
                    break;
                fence_after();
                const uint64_t bd = d0 + (uint64_t)((s * NB * 128) >> 4);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    mma_f8_ts(tmem + (uint32_t)((g & 1) * NB), ring + (uint32_t)(s * 32 + kk * 8), bd + (uint64_t)(kk * 2), IDESC,
                              !first || kk ? 1u : 0u);
                mma_commit(&empty[s]);
                if (g_.s == CT_GROUP - 1 || it == n - 1) mma_commit(&dfull[g & 1]);
            }
            // as the likelihood's accum: the MMAs issued are done before tensor memory goes
            mma_commit(&drained);
            mbar_wait(&drained, 0);
        }
    } else if (warp == CT_BW + 1) {
        if (lane == 0) {
            const uint32_t tx = NB * 128 + c.stall;
            int issued = 0;
            Ring<ST> r_;
            for (int it = 0; it < n; ++it, r_.step()) {
                const int s = r_.s;
                if (r_.round && !thread_wait(empty0 + 8 * s, (r_.round & 1) ^ 1, s_abort, err, 24)) break;
                mbar_expect_tx(&fullB[s], tx);
                bulk_load(&sB[s][0], c.oh + (int64_t)it * (NB * 128), NB * 128, &fullB[s]);
                issued = it + 1;
            }
            // every copy issued has landed before the CTA may exit
            for (int it = issued > ST ? issued - ST : 0; it < issued; ++it) mbar_wait(&fullB[it % ST], (it / ST) & 1, s_abort[1]);
        }
    } else if (lane < NB) {
        const int* nk = reinterpret_cast<const int*>(c.oh + (int64_t)n * NB * 128);
        int t = 0;
#pragma unroll 8
        for (int it = 0; it < n; ++it) t += nk[it * NB + lane];
        s_nk[lane] = t;
    }
    fence_before();
    __syncthreads();
    if (warp == CT_BW) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::COLS));
    }
    if (warp < 4 && a1[0] >= 0) {
        const int64_t l = (int64_t)vb.x * CT_M + warp * 32 + lane;
        int2* N2 = reinterpret_cast<int2*>(c.Ni);
        if (l < D.L)
#pragma unroll
            for (int k = 0; k < NB; ++k)
                if (k < K) N2[(int64_t)k * D.L + l] = make_int2(2 * (s_nk[k] - ms[k]) - a1[k], a1[k]);
    }
}

}  // namespace ptc
}  // namespace vp
