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
// chain's control block (read with the chain's results), waits for what is in
// flight, frees its tensor memory and returns.
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
// a wait that gives up when any warp of the CTA has
__device__ __forceinline__ bool ring_wait(uint64_t* bar, uint32_t parity, volatile int* abort, int* err, int code) {
    if (mbar_wait(bar, parity)) return !*abort;
    *abort = 1;
    atomicExch(err, code);
    return false;
}
// the same for a whole warp, which takes one way
__device__ __forceinline__ bool warp_ring_wait(uint64_t* bar, uint32_t parity, volatile int* abort, int* err, int code) {
    int ok = 0;
    if ((threadIdx.x & 31) == 0) ok = ring_wait(bar, parity, abort, err, code);
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

// ---- the likelihood, exact ------------------------------------------------
// ln p is taken as a whole number of 2^-24 units (|ln p| < 2^10, so 34 bits) in
// seven digits to base 32, each a whole number of at most 16 in magnitude and
// so exact in e4m3, as the copies 0, 1, 2 are. A call adds at most 2 x 16 to a
// digit's sum and the FP32 accumulator holds whole numbers up to 2^24, so the
// sums of up to 2^19 loci are exact whatever the order of the adds, and the
// digits combine in 64-bit integers. What rounds is the logarithm itself (FP32,
// as in the FP32 forms) and its unit, an FP32 ulp of 0.5 to 1: against 64 bits
// LL is 2.5e-9 off, where the FP32 stream is 3.1e-9 to 5.7e-9 off (N = 512 to
// 2,000, L = 4,096 to 60,000, K = 3 to 16).
constexpr int LL_LOCI = 32;                        // loci of a stage: 64 A bytes (copies of allele 1 and 0 of each)
constexpr int LL_MAXST = (1 << 19) / LL_LOCI;
constexpr int LL_M = 256;                          // individuals per CTA: two 128-row tiles share a B stage
constexpr int LL_THREADS = 320;                    // eight builder warps, the MMA warp, the B producer
constexpr int LL_TCK = 32;                         // most clusters
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

// CTA: LL_M individuals x the stages of its chunk (grid.y). Lane n of a
// builder warp is individual n / 2 of the warp's first genotype word or of its
// second, by n's last bit (the in-register transpose's order).
template <int NB>
__global__ void __launch_bounds__(LL_THREADS, NB <= 80 ? 2 : 1) k_loglik_tc(const DevChain* chains, const int4* map = nullptr) {
    using S = LlShape<NB>;
    constexpr int ST = S::ST;
    constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(NB >> 3) << 17) | (8u << 24);   // e4m3 x e4m3 -> f32, 128 rows
    __shared__ __align__(1024) unsigned char sB[ST][NB * 64];
    __shared__ uint64_t full[ST], fullB[ST], empty[ST], accum;
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    const VBlock vb = vblock(map);
    const DevChain& c = chains[vb.z];
    if (map && run_over(c)) return;
    if (!ll_tc_at(c, c.ctl->m)) return;
    const DevData& D = c.D;
    const int K = c.K;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nst = (int)((D.L + LL_LOCI - 1) / LL_LOCI), per = c.tcper;
    const int st0 = vb.y * per, n = min(nst, st0 + per) - st0;
    if (n <= 0) return;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) { mbar_init(&full[s], 8); mbar_init(&fullB[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(&accum, 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(S::COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = s_tmem, ring = tmem + 2 * NB;
    int* err = &c.ctl->err;
    if (warp < 8) {
        const int tile = warp >> 2, q = warp & 3;
        const int ib = vb.x * LL_M + warp * 32;
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        const BitTranspose tr(lane);
        auto word = [&](int st, int h) {
            const int64_t l = (int64_t)(st0 + st) * LL_LOCI + 16 * h + (lane >> 1);
            const int w = (ib >> 4) + (lane & 1);
            return l < D.L && w < D.Nw ? __ldg(D.g2 + l * D.Nw + w) : 0xFFFFFFFFu;
        };
        uint32_t w0 = word(0, 0), w1 = word(0, 1);
        for (int it = 0; it < n; ++it) {
            const int s = it % ST;
            uint32_t r[16];
            calls_to_e4m3(tr.codes(w0), r);
            calls_to_e4m3(tr.codes(w1), r + 8);
            if (it + 1 < n) {
                w0 = word(it + 1, 0);
                w1 = word(it + 1, 1);
            }
            if (it >= ST && !warp_ring_wait(&empty[s], ((it / ST) & 1) ^ 1, &s_abort, err, 11)) break;
            fence_after();
            tmem_st16(ring + lanes + (uint32_t)(s * 32 + tile * 16), r);
            wait_st();
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
        // the digits' sums of this lane's individual
        const bool got = warp_ring_wait(&accum, 0, &s_abort, err, 12);
        fence_after();
        const int i = ib + (lane >> 1) + 16 * (lane & 1);
        long long* out = reinterpret_cast<long long*>(c.LLp) + ((int64_t)vb.y * D.N + i) * K;
#pragma unroll 1
        for (int k = 0; k < K; ++k) {
            float v[8];
            tmem_ld8(tmem + lanes + (uint32_t)(tile * NB + 7 * k), v);
            if (!got || i >= D.N) continue;
            long long t = 0;
#pragma unroll
            for (int j = 6; j >= 0; --j) t = t * 32 + __float2int_rn(v[j]);
            out[k] = t;
        }
    } else if (warp == 8) {
        if (lane == 0) {
            const uint64_t d0 = tc::sw_desc(smem_u32(&sB[0][0]), 64);
            for (int it = 0; it < n; ++it) {
                const int s = it % ST;
                if (!ring_wait(&full[s], (it / ST) & 1, &s_abort, err, 13) || !ring_wait(&fullB[s], (it / ST) & 1, &s_abort, err, 15)) break;
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
            mma_commit(&accum);
        }
    } else if (lane == 0) {
        const char* src = reinterpret_cast<const char*>(c.ltd) + (int64_t)st0 * (NB * 64);
        int issued = 0;
        for (int it = 0; it < n; ++it) {
            const int s = it % ST;
            if (it >= ST && !ring_wait(&empty[s], ((it / ST) & 1) ^ 1, &s_abort, err, 14)) break;
            if (*(volatile int*)&s_abort) break;
            mbar_expect_tx(&fullB[s], NB * 64);
            bulk_load(&sB[s][0], src + (int64_t)it * (NB * 64), NB * 64, &fullB[s]);
            issued = it + 1;
        }
        // every copy issued has landed before the CTA may exit
        for (int it = issued > ST ? issued - ST : 0; it < issued; ++it) mbar_wait(&fullB[it % ST], (it / ST) & 1);
    }
    fence_before();
    __syncthreads();
    if (warp == 8) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::COLS));
    }
}

// ---- the counts -----------------------------------------------------------
// Per CTA 128 loci (one a lane of four builder warps); stages of 128
// individuals. A call is one e5m2 byte: its copies of allele 1, or CT_MISS for
// a missing call, so that one matrix gives both counts: over at most CT_GROUP
// stages a cluster's sum is copies + CT_MISS x missing calls with copies below
// CT_MISS, a whole number below 2^24, and so exact. Two accumulators alternate
// between groups; the builders take one apart while the MMAs fill the other.
// B is the one-hot matrix of the labels, built in shared memory by its own
// warp, which also counts the clusters' sizes: copies of allele 0 are
// 2 (size - missing) - copies of allele 1.
// Bound by the MMAs' reads of A from tensor memory (128 cycles per 128 rows x
// 32 bytes whatever the clusters' count, as in the likelihood).
constexpr int CT_IND = 128, CT_M = 128, CT_THREADS = 192;
constexpr int CT_PITCH = 80;                         // bytes of a staged row: 64 and a 16-byte pad (odd chunks)
constexpr int CT_MISS = 1 << 12, CT_GROUP = (CT_MISS - 1) / (2 * CT_IND);   // 15 stages: 3,840 copies
static_assert((int64_t)CT_MISS * CT_GROUP * CT_IND + CT_MISS < (1 << 24), "exact sums");
__host__ __device__ constexpr int ct_rows(int K) { return K <= 16 ? 16 : 32; }
template <int NB>
struct CtShape {
    static constexpr int COLS = 256, FIT = (COLS - 2 * NB) / 32, ST = FIT > 4 ? 4 : FIT;
};
// e5m2 bytes by code: 0, 1, 2, 4096
constexpr uint32_t E5_CODE = 0x6C403C00u, E5_ONE = 0x3Cu;
template <int NB>
__global__ void __launch_bounds__(CT_THREADS, 2) k_count_tc(const DevChain* chains, int force, const int4* map = nullptr) {
    using S = CtShape<NB>;
    constexpr int ST = S::ST;
    // e5m2 x e5m2 -> f32, 128 rows
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NB >> 3) << 17) | (8u << 24);
    __shared__ __align__(1024) unsigned char sB[ST][NB * 128];
    __shared__ __align__(16) unsigned char sG[2][CT_M * CT_PITCH];
    __shared__ uint64_t full[ST], empty[ST], dfull[2], dempty[2];
    __shared__ int s_nk[NB];
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    const VBlock vb = vblock(map);
    const DevChain& c = chains[vb.z];
    if (map && run_over(c)) return;
    if (!force && !binaryq_at(c, c.ctl->m)) return;
    const DevData& D = c.D;
    const int K = c.K;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = (D.N + CT_IND - 1) / CT_IND, ngr = (n + CT_GROUP - 1) / CT_GROUP;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) { mbar_init(&full[s], 5); mbar_init(&empty[s], 1); }
        for (int d = 0; d < 2; ++d) { mbar_init(&dfull[d], 1); mbar_init(&dempty[d], 4); }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < NB) s_nk[threadIdx.x] = 0;
    if (warp == 4) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(S::COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = s_tmem, ring = tmem + 2 * NB;
    int* err = &c.ctl->err;
    int a1[NB], ms[NB];          // this lane's locus: copies of allele 1 and missing calls by cluster
    if (warp < 4) {
        const uint32_t lanes = (uint32_t)(warp * 32) << 16;
        const int64_t lw = (int64_t)vb.x * CT_M + warp * 32;
#pragma unroll
        for (int k = 0; k < NB; ++k) { a1[k] = 0; ms[k] = 0; }
        // this warp's 32 rows, 16 words (256 individuals) at a time, by 16-byte
        // asynchronous copies one piece ahead; a row's words past its end (and
        // rows past the last locus) are filled with zeros, whose individuals
        // have no label
        auto fetch = [&](int g) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int row = 8 * u + (lane >> 2), ch = lane & 3, w = g * 16 + ch * 4;
                const bool ok = lw + row < D.L && w < D.Nw;
                cp_async16(&sG[g & 1][(warp * 32 + row) * CT_PITCH + ch * 16], ok ? D.g2 + (lw + row) * D.Nw + w : D.g2, ok);
            }
            cp_async_commit();
        };
        auto drain = [&](int g) {
            if (!warp_ring_wait(&dfull[g & 1], (g >> 1) & 1, &s_abort, err, 22)) return false;
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
        const int np = (n + 1) / 2;
        fetch(0);
        bool run = true;
        for (int g = 0; g < np && run; ++g) {
            if (g + 1 < np) {
                fetch(g + 1);
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncwarp();
            const unsigned char* my = &sG[g & 1][(warp * 32 + lane) * CT_PITCH];
            for (int j = 0; j < 2; ++j) {
                const int it = g * 2 + j, s = it % ST;
                if (it >= n) break;
                const uint4 x = *reinterpret_cast<const uint4*>(my + 32 * j), y = *reinterpret_cast<const uint4*>(my + 32 * j + 16);
                const uint32_t wd[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
                if (it >= ST && !warp_ring_wait(&empty[s], ((it / ST) & 1) ^ 1, &s_abort, err, 21)) { run = false; break; }
                fence_after();
                const uint32_t a = ring + lanes + (uint32_t)(s * 32);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t r[16];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll
                        for (int b = 0; b < 4; ++b)
                            // codes b', b' + 2, b' + 4, b' + 6 of a half word (b' = b & 1, the half by b >> 1)
                            r[4 * u + b] = __byte_perm(E5_CODE, 0u, (wd[4 * h + u] >> (16 * (b >> 1) + 2 * (b & 1))) & 0x3333u);
                    tmem_st16(a + 16 * h, r);
                }
                wait_st();
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[s]);
                // once a group is built the one before it, long finished, is taken apart
                if (it % CT_GROUP == CT_GROUP - 1 && it / CT_GROUP > 0 && !drain(it / CT_GROUP - 1)) { run = false; break; }
            }
            __syncwarp();   // the piece's rows are rewritten two pieces on
        }
        cp_async_wait<0>();
        // groups not yet taken apart: the one before the last (unless the last
        // was full and did it) and the last
        const int full_groups = n / CT_GROUP;
        for (int g = max(0, full_groups - 1); g < ngr && run; ++g) run = drain(g);
        if (!run) {
            // an abort: the MMAs issued must have ended before tensor memory goes
            mbar_wait(&dfull[(ngr - 1) & 1], ((ngr - 1) >> 1) & 1);
            a1[0] = -1;
        }
    } else if (warp == 4) {
        if (lane == 0) {
            const uint64_t d0 = tc::sw_desc(smem_u32(&sB[0][0]), 128);
            bool run = true;
            for (int it = 0; it < n && run; ++it) {
                const int s = it % ST, g = it / CT_GROUP;
                const bool first = it % CT_GROUP == 0;
                if (first && g >= 2 && !ring_wait(&dempty[g & 1], ((g >> 1) & 1) ^ 1, &s_abort, err, 25)) { run = false; break; }
                if (!ring_wait(&full[s], (it / ST) & 1, &s_abort, err, 23)) { run = false; break; }
                fence_after();
                const uint64_t bd = d0 + (uint64_t)((s * NB * 128) >> 4);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    mma_f8_ts(tmem + (uint32_t)((g & 1) * NB), ring + (uint32_t)(s * 32 + kk * 8), bd + (uint64_t)(kk * 2), IDESC,
                              !first || kk ? 1u : 0u);
                mma_commit(&empty[s]);
                if (it % CT_GROUP == CT_GROUP - 1 || it == n - 1) mma_commit(&dfull[g & 1]);
            }
            if (!run) {
                mma_commit(&dfull[0]);
                mma_commit(&dfull[1]);
            }
        }
    } else {
        // B: row k, byte position p of the stage's 128 individuals. Lane j
        // writes positions 4 j .. 4 j + 3 of every row; position 4 u + e of a
        // word's 16 (u the decoded register, e its byte) is individual
        // 8 (u >> 1) + (u & 1) + 2 e of the word.
        const int wd = lane >> 2, u = lane & 3;
        const int i0 = 16 * wd + 8 * (u >> 1) + (u & 1);
        for (int it = 0; it < n; ++it) {
            const int s = it % ST;
            int z[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = it * CT_IND + i0 + 2 * e;
                z[e] = i < D.N ? (int)c.Z[i] : -1;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (z[e] >= 0) atomicAdd(&s_nk[z[e]], 1);
            if (it >= ST && !warp_ring_wait(&empty[s], ((it / ST) & 1) ^ 1, &s_abort, err, 24)) break;
            uint32_t* B = reinterpret_cast<uint32_t*>(&sB[s][0]);
#pragma unroll 4
            for (int k = 0; k < NB; ++k) {
                uint32_t v = 0;
#pragma unroll
                for (int e = 0; e < 4; ++e) v |= z[e] == k ? E5_ONE << (8 * e) : 0u;
                // 128-byte swizzle: the 16-byte chunk of row k moves by k mod 8
                B[k * 32 + (((lane >> 2) ^ (k & 7)) << 2) + (lane & 3)] = v;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 4) {
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
