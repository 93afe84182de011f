// Per-copy label draws of the admixture model on 2-bit biallelic diploid data
// (UpdateZAdmix, src/structure.cpp:1350-1487) with counter streams.
#pragma once
#include "vp_kernels.cuh"

namespace vp {

// loci of a slice: the Philox streams of the label draws are per slice
constexpr int PZ_LC = ZA_LC;
static_assert(PZ_LC == 16, "a slice's codes of one individual fill a word");

// two FP32 values in one 64-bit register pair, and the packed operations on
// them (each half rounds as the scalar instruction does)
typedef unsigned long long f2x;
__device__ __forceinline__ f2x f2_pack(float a, float b) {
    f2x r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_unpack(f2x v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2x f2_fma(f2x a, f2x b, f2x c) {
    f2x r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2x f2_mul(f2x a, f2x b) {
    f2x r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2x f2_add(f2x a, f2x b) {
    f2x r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// transpose of a 32 x 32 bit matrix held as one word a lane: bit p of lane n
// becomes bit n of lane p
struct BitTranspose {
    uint32_t s16, s8, k4, k2, k1;   // byte selectors of the two outer steps, kept bits of the inner ones
    int r4, r2, r1;                 // left rotations of the partner's word
    __device__ __forceinline__ explicit BitTranspose(int lane) {
        s16 = lane & 16 ? 0x3276u : 0x5410u;
        s8 = lane & 8 ? 0x3715u : 0x6240u;
        k4 = lane & 4 ? 0xF0F0F0F0u : 0x0F0F0F0Fu;
        k2 = lane & 2 ? 0xCCCCCCCCu : 0x33333333u;
        k1 = lane & 1 ? 0xAAAAAAAAu : 0x55555555u;
        r4 = lane & 4 ? 28 : 4;
        r2 = lane & 2 ? 30 : 2;
        r1 = lane & 1 ? 31 : 1;
    }
    // the outer four steps: a 16 x 16 transpose of two-bit elements in the
    // even lanes and one in the odd lanes (element p of lane 2 n + w becomes
    // element n of lane 2 p + w)
    __device__ __forceinline__ uint32_t codes(uint32_t x) const {
        x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 16), s16);
        x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 8), s8);
        uint32_t y = __shfl_xor_sync(0xffffffffu, x, 4);
        x = (x & k4) | (__funnelshift_l(y, y, r4) & ~k4);
        y = __shfl_xor_sync(0xffffffffu, x, 2);
        return (x & k2) | (__funnelshift_l(y, y, r2) & ~k2);
    }
    __device__ __forceinline__ uint32_t operator()(uint32_t x) const {
        x = codes(x);
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, 1);
        return (x & k1) | (__funnelshift_l(y, y, r1) & ~k1);
    }
};

// the words with label k among the bit planes p[0..3] of 32 labels
template <int KM>
__device__ __forceinline__ uint32_t label_mask(const uint32_t* p, int k) {
    uint32_t m = k & 1 ? p[0] : ~p[0];
    if (KM > 2) m &= k & 2 ? p[1] : ~p[1];
    if (KM > 4) m &= k & 4 ? p[2] : ~p[2];
    if (KM > 8) m &= k & 8 ? p[3] : ~p[3];
    return m;
}

// lane's word of slice s for the warp's 32 individuals from ib: locus lane / 2,
// the first genotype word in even lanes, the second in odd ones (missing codes
// past the last locus and word)
__device__ __forceinline__ uint32_t slice_word(const DevData& D, int s, int ib, int lane) {
    const int64_t l = (int64_t)s * PZ_LC + (lane >> 1);
    const int w = (ib >> 4) + (lane & 1);
    return l < D.L && w < D.Nw ? __ldg(D.g2 + l * D.Nw + w) : 0xFFFFFFFFu;
}

// 16-byte chunks (two clusters' frequency pairs) of a table row, an odd count:
// the four codes' rows of a locus then start in different banks
template <int KM>
__host__ __device__ constexpr int pz_chunks() { return ((KM + 1) / 2) | 1; }

// Label draws of every copy, one lane per individual, a warp of 32
// individuals walking the slices of the CTA's locus range (grid.y).
//
// The same draws as k_update_z_admix_ctr, bit for bit: one Philox stream per
// (individual, slice), two draws per locus, prefix sums of q_k p_k by fused
// multiply-adds in cluster order, and the first cluster whose cumulative
// weight exceeds the uniform times the total. The prefix sums do not
// decrease, so that cluster is the number of clusters (but the last) whose
// threshold the uniform reaches.
//
// What bounds it is instruction issue, so the work per copy is cut down to
// the draw itself:
//  - the staged table holds, for each code of a locus, the pair (frequency of
//    the first copy's allele, of the second's) of every cluster, so that one
//    16-byte load brings two clusters of both copies and packed FP32
//    instructions serve both copies at once;
//  - a warp reads the slice's 32 genotype words (16 loci x 32 individuals),
//    one a lane, and transposes them in registers, so that each lane holds
//    its individual's 16 codes in one word;
//  - labels go four bits each into a word (eight copies), the words become
//    bit planes of a slice's 32 copies, and a lane's copies per cluster are
//    one population count a cluster and slice;
//  - for the counts per locus the planes are transposed across the warp (bit
//    n = lane n), lane p then holds one copy slot of one locus for the 32
//    individuals, and copies of an allele with label k are one population
//    count against the genotype words' own bit planes (lane n is individual
//    n / 2 of the first genotype word or of the second, by n's last bit, so
//    that the planes interleave as the words do).
// Counts of both alleles share a word of the CTA's histogram (16 bits each: a
// CTA adds at most 2 x 256 per slice), which goes to Ni as 64-bit additions of
// the two neighbouring counts. One barrier a slice: table and histogram are
// double-buffered.
//
// Measured, us a launch against k_update_z_admix_ctr on the same calls: N = 2,000 x
// L = 50,000, K = 5 1,030 -> 375; N = 4,999 x L = 40,009, K = 11 3,700 -> 1,160;
// N = 300 x L = 3,000, K = 4 32 -> 17. At K = 5 issue is 76% active, the ALU
// pipe 62%, the multiplier pipe (Philox) 55%. Round keys read from shared
// memory instead of added up gave 1.7%, 2 or 4 CTAs per SM instead of 3 lost 1%.
constexpr int PZ_MAXK = 16;
constexpr int PZ_MAXT = 256;
// INIT: the initial labels (InitAdmix, as k_init_admix_ctr: a Philox stream a
// call, draws modulo K) with the same counting, for the padded cluster count
// only. N = 2,000 x L = 50,000, K = 5 801 -> 311 us, N = 4,999 x L =
// 40,009, K = 11 1,676 -> 631 us against k_init_admix_ctr, which adds every copy
// to shared histograms.
template <int KM, bool EXACT, bool INIT = false>
__global__ void __launch_bounds__(PZ_MAXT, KM <= 6 || INIT ? 3 : 2) k_z_admix_pk(const DevChain* chains, int force,
                                                                        const int4* map = nullptr) {
    constexpr int CH = pz_chunks<KM>();
    constexpr int NPL = KM <= 2 ? 1 : KM <= 4 ? 2 : KM <= 8 ? 3 : 4;      // bit planes of a label
    constexpr int NF = (PZ_LC * KM + 127) / 128;                          // staged frequencies a thread (128 threads or more)
    __shared__ __align__(16) float2 sF[INIT ? 1 : 2][INIT ? 1 : PZ_LC][4][CH * 2];
    __shared__ uint32_t hs[2][KM][PZ_LC];
    __shared__ double sh[32];
    const VBlock vb = vblock(map);
    const DevChain& c = chains[vb.z];
    if (map && run_over(c)) return;
    const DevData& D = c.D;
    const int K = EXACT ? KM : c.K, m = c.ctl->m;
    if (!INIT && !force && binaryq_at(c, m)) return;
    const int lane = threadIdx.x & 31, T = blockDim.x;
    const int ib = vb.x * T + (threadIdx.x & ~31);
    const int i = ib + (lane >> 1) + 16 * (lane & 1);
    const bool live = i < D.N;
    const uint32_t lives = __ballot_sync(0xffffffffu, live);
    const int nsl = (int)((D.L + PZ_LC - 1) / PZ_LC);
    const int s0 = vb.y * c.pz_slices, s1 = min(nsl, s0 + c.pz_slices);
    f2x q[KM];
    int32_t mi[KM];
#pragma unroll
    for (int k = 0; k < KM; ++k) {
        const float v = (!INIT && live && (EXACT || k < K)) ? c.Q[(int64_t)i * K + k] : 0.f;
        q[k] = f2_pack(v, v);
        mi[k] = 0;
    }
    // this lane's copy slot after the transpose: copy j of the group of four
    // loci g sits in nibble 7 - j of the group's word and at bit 3 - g of the
    // nibble once the four groups' planes are merged
    const int slot = 7 - (lane >> 2), pl = 4 * (3 - (lane & 3)) + (slot >> 1);
    const bool second = slot & 1;
    const BitTranspose tr(lane);
    const bool rec = !INIT && (force || record_at(c, m));
    float ls = 0.f, lc = 0.f;                       // Kahan sum of ln(sum_k q_k p)
    const float minf = (float)VP_MIN_FREQ;
    const f2x kmin = f2_pack((float)(VP_MIN_FREQ * K), (float)(VP_MIN_FREQ * K));
    const uint2 key = make_uint2((uint32_t)c.seed, (uint32_t)(c.seed >> 32));
    const uint32_t ca = ST_ZSLICE | ((uint32_t)m << 4);
    const float2* F2 = reinterpret_cast<const float2*>(c.Freq);
    float2 fn[NF];
    auto load_f = [&](int s) {
#pragma unroll
        for (int u = 0; u < NF; ++u) {
            const int j = threadIdx.x + u * T, k = j >> 4;
            const int64_t l = (int64_t)s * PZ_LC + (j & 15);
            fn[u] = j < PZ_LC * K && l < D.L ? __ldg(F2 + (int64_t)k * D.L + l) : make_float2(0.f, 0.f);
        }
    };
    auto store_f = [&](int buf) {
#pragma unroll
        for (int u = 0; u < NF; ++u) {
            const int j = threadIdx.x + u * T;
            if (j < PZ_LC * KM) {
                float2(*r)[CH * 2] = sF[buf][j & 15];
                const int k = j >> 4;
                r[0][k] = make_float2(fn[u].x, fn[u].x);
                r[1][k] = fn[u];
                r[2][k] = make_float2(fn[u].y, fn[u].y);
            }
        }
    };
    if (s0 >= s1) return;
    if constexpr (!INIT)
        for (int j = threadIdx.x; j < 2 * PZ_LC * CH * 2; j += T)
            sF[j / (PZ_LC * CH * 2)][j / (CH * 2) % PZ_LC][3][j % (CH * 2)] = make_float2(0.f, 0.f);
    for (int j = threadIdx.x; j < 2 * KM * PZ_LC; j += T) (&hs[0][0][0])[j] = 0;
    if constexpr (!INIT) {
        load_f(s0);
        store_f(0);
    }
    const uint32_t modm = INIT ? (uint32_t)min(0x100000000ull / (uint32_t)K, 0xFFFFFFFFull) : 0;
    uint32_t wn = slice_word(D, s0, ib, lane);
    __syncthreads();
    int buf = 0;
    for (int s = s0; s < s1; ++s, buf ^= 1) {
        const uint32_t w = wn;
        uint32_t gw = tr.codes(w);
        if (!live) gw = 0xFFFFFFFFu;
        if (s + 1 < s1) {
            wn = slice_word(D, s + 1, ib, lane);
            if constexpr (!INIT) load_f(s + 1);
        }
        uint32_t P[NPL];
#pragma unroll
        for (int b = 0; b < NPL; ++b) P[b] = 0;
#pragma unroll 1
        for (int g = 0; g < 4; ++g) {
            uint32_t Z = 0;
            if constexpr (INIT) {
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const uint4 rb = Philox::round10(make_uint4(ST_INITADM, (uint32_t)(s * PZ_LC + 4 * g + v), (uint32_t)i, 0), key);
                    // x mod K: the quotient from 2^32 / K rounded down is at most one short
                    uint32_t za = rb.x - __umulhi(rb.x, modm) * K, zb = rb.y - __umulhi(rb.y, modm) * K;
                    za = min(za, za - K);
                    zb = min(zb, zb - K);
                    Z = (((Z << 4) | za) << 4) | zb;
                }
            } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4 rb = Philox::round10(make_uint4(ca, (uint32_t)s, (uint32_t)i, (uint32_t)(2 * g + h)), key);
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    const uint32_t code = gw & 3u;
                    gw >>= 2;
                    const float4* row = reinterpret_cast<const float4*>(&sF[buf][4 * g + 2 * h + v][code][0]);
                    f2x pre[KM], sx = 0;
#pragma unroll
                    for (int k = 0; k < KM; k += 2) {
                        const float4 f = row[k >> 1];
                        sx = f2_fma(q[k], f2_pack(f.x, f.y), sx);
                        pre[k] = sx;
                        if (k + 1 < KM) {
                            sx = f2_fma(q[k + 1], f2_pack(f.z, f.w), sx);
                            pre[k + 1] = sx;
                        }
                    }
                    // uniforms ((x >> 8) + 1) / 2^24: every step exact
                    const float ua = fmaf((float)((v ? rb.z : rb.x) >> 8), 1.f / 16777216.f, 1.f / 16777216.f);
                    const float ub = fmaf((float)((v ? rb.w : rb.y) >> 8), 1.f / 16777216.f, 1.f / 16777216.f);
                    float ta, tb;
                    f2_unpack(f2_mul(f2_pack(ua, ub), f2_add(sx, kmin)), ta, tb);
                    uint32_t za = 0, zb = 0;
#pragma unroll
                    for (int k = 0; k < KM - 1; ++k) {
                        if (!EXACT && k >= K - 1) break;
                        float pa, pb;
                        f2_unpack(pre[k], pa, pb);
                        if (!(ta < __fmaf_rn((float)(k + 1), minf, pa))) ++za;
                        if (!(tb < __fmaf_rn((float)(k + 1), minf, pb))) ++zb;
                    }
                    Z = (((Z << 4) | za) << 4) | zb;
                    if (rec && code != 3u) {
                        float xa, xb;
                        f2_unpack(sx, xa, xb);
                        const float y = (logf(xa) + logf(xb)) - lc, t = ls + y;
                        lc = (t - ls) - y;
                        ls = t;
                    }
                }
            }
            }
#pragma unroll
            for (int b = 0; b < NPL; ++b) P[b] = (P[b] << 1) | ((Z >> b) & 0x11111111u);
        }
        // this lane's locus for the counts: its two genotype words' planes, bit
        // n = lane n's individual
        const uint32_t w0 = __shfl_sync(0xffffffffu, w, 2 * pl), w1 = __shfl_sync(0xffffffffu, w, 2 * pl + 1);
        const uint32_t LO = (w0 & 0x55555555u) | ((w1 << 1) & 0xAAAAAAAAu);
        const uint32_t HI = ((w0 >> 1) & 0x55555555u) | (w1 & 0xAAAAAAAAu);
        const uint32_t MS = (LO & HI) | ~lives;
        const uint32_t A1 = (second ? LO ^ HI : HI & ~LO) & ~MS, A0 = ~(A1 | MS);
        const uint32_t typed = ~tr(MS);                  // this lane's typed copies
#pragma unroll
        for (int k = 0; k < KM; ++k)
            if (EXACT || k < K) mi[k] += __popc(label_mask<KM>(P, k) & typed);
        uint32_t R[NPL];
#pragma unroll
        for (int b = 0; b < NPL; ++b) R[b] = tr(P[b]);
#pragma unroll
        for (int k = 0; k < KM; ++k) {
            if (!EXACT && k >= K) break;
            const uint32_t mk = label_mask<KM>(R, k);
            const uint32_t n = (uint32_t)__popc(mk & A0) | ((uint32_t)__popc(mk & A1) << 16);
            atomicAdd(&hs[buf][k][pl], n);
        }
        if constexpr (!INIT)
            if (s + 1 < s1) store_f(buf ^ 1);
        __syncthreads();
        unsigned long long* N2 = reinterpret_cast<unsigned long long*>(c.Ni);
        for (int j = threadIdx.x; j < PZ_LC * K; j += T) {
            uint32_t* h = &hs[buf][j >> 4][j & 15];
            const uint32_t n = *h;
            if (!n) continue;
            *h = 0;
            atomicAdd(N2 + (int64_t)(j >> 4) * D.L + (int64_t)s * PZ_LC + (j & 15),
                      (unsigned long long)(n & 0xFFFFu) | ((unsigned long long)(n >> 16) << 32));
        }
    }
    if (live)
#pragma unroll
        for (int k = 0; k < KM; ++k)
            if ((EXACT || k < K) && mi[k]) atomicAdd(&c.Mi[(int64_t)i * K + k], mi[k]);
    if constexpr (!INIT) {
        const double t = block_sum((double)ls - (double)lc, sh);
        if (threadIdx.x == 0) c.lnlp[vb.y * vb.gx + vb.x] = t;
    }
}

// The Metropolis log ratios (UpdateQMetro, src/structure.cpp:1006-1086) on 2-bit
// genotypes: per individual the sum over its copies of
// ln(sum_k q'_k p / sum_k q_k p), one partial per locus range (grid.y) in
// metrop. The staged table and packed FP32 operations of k_z_admix_pk give the
// four weighted sums of a call. Their logarithms are not taken one by one: the
// products of the numerators and of the denominators are carried as a mantissa
// in [1, 2) and an integer exponent each, and one logarithm of the mantissas'
// ratio closes a range, which rounds less than a sum of FP32 logarithms (two
// roundings of 2^-24 a copy against a rounding at the running sum's size). A
// call with a product outside 2^-100 to 2^28 adds its logarithms singly, so that
// zeros, infinities and NaNs come out as they do from the terms.
// Issue-bound: N = 2,000 x L = 50,000, K = 5 593 -> 157 us a launch, N = 4,999 x
// L = 40,009, K = 11 1,586 -> 570 us (against k_metro_ratio on the same calls).
template <int KM, bool EXACT>
__global__ void __launch_bounds__(PZ_MAXT, KM <= 11 ? 3 : 2) k_metro_pk(const DevChain* chains, int force, const int4* map = nullptr) {
    constexpr int CH = pz_chunks<KM>();
    constexpr int NF = (PZ_LC * KM + 127) / 128;
    __shared__ __align__(16) float2 sF[2][PZ_LC][4][CH * 2];
    const VBlock vb = vblock(map);
    const DevChain& c = chains[vb.z];
    if (map && run_over(c)) return;
    const DevData& D = c.D;
    const int K = EXACT ? KM : c.K, m = c.ctl->m;
    if (!force && !metro_turn(c, m)) return;
    const int T = blockDim.x, lane = threadIdx.x & 31, ib = vb.x * T + (threadIdx.x & ~31);
    const int i = ib + (lane >> 1) + 16 * (lane & 1);
    const bool live = i < D.N;
    const BitTranspose tr(lane);
    const int nsl = (int)((D.L + PZ_LC - 1) / PZ_LC);
    const int s0 = vb.y * c.pz_slices, s1 = min(nsl, s0 + c.pz_slices);
    if (s0 >= s1) return;
    f2x q1[KM], q0[KM];
#pragma unroll
    for (int k = 0; k < KM; ++k) {
        const bool on = live && (EXACT || k < K);
        const float a = on ? c.Qprop[(int64_t)i * K + k] : 0.f, b = on ? c.Q[(int64_t)i * K + k] : 0.f;
        q1[k] = f2_pack(a, a);
        q0[k] = f2_pack(b, b);
    }
    const float2* F2 = reinterpret_cast<const float2*>(c.Freq);
    auto stage = [&](int s, int buf) {
#pragma unroll
        for (int u = 0; u < NF; ++u) {
            const int j = threadIdx.x + u * T, k = j >> 4;
            if (j >= PZ_LC * KM) break;
            const int64_t l = (int64_t)s * PZ_LC + (j & 15);
            const float2 f = k < K && l < D.L ? __ldg(F2 + (int64_t)k * D.L + l) : make_float2(0.f, 0.f);
            float2(*r)[CH * 2] = sF[buf][j & 15];
            r[0][k] = make_float2(f.x, f.x);
            r[1][k] = f;
            r[2][k] = make_float2(f.y, f.y);
        }
    };
    // an odd cluster count leaves one column unwritten, read and not used;
    // the missing code's rows are read and not used too
    float R1 = 1.f, R0 = 1.f, single = 0.f;
    int ex = 0;
    auto normalise = [](float& r) {
        const uint32_t b = __float_as_uint(r);
        r = __uint_as_float((b & 0x007FFFFFu) | 0x3F800000u);
        return (int)(b >> 23) - 127;
    };
    stage(s0, 0);
    uint32_t wn = slice_word(D, s0, ib, lane);
    __syncthreads();
    int buf = 0;
    for (int s = s0; s < s1; ++s, buf ^= 1) {
        uint32_t gw = tr.codes(wn);
        if (s + 1 < s1) {
            wn = slice_word(D, s + 1, ib, lane);
            stage(s + 1, buf ^ 1);
        }
#pragma unroll 4
        for (int ll = 0; ll < PZ_LC; ++ll) {
            const uint32_t code = gw & 3u;
            gw >>= 2;
            const float4* row = reinterpret_cast<const float4*>(&sF[buf][ll][code][0]);
            f2x x1 = 0, x0 = 0;
#pragma unroll
            for (int k = 0; k < KM; k += 2) {
                const float4 f = row[k >> 1];
                const f2x fa = f2_pack(f.x, f.y), fb = f2_pack(f.z, f.w);
                x1 = f2_fma(q1[k], fa, x1);
                x0 = f2_fma(q0[k], fa, x0);
                if (k + 1 < KM) {
                    x1 = f2_fma(q1[k + 1], fb, x1);
                    x0 = f2_fma(q0[k + 1], fb, x0);
                }
            }
            float a1, b1, a0, b0;
            f2_unpack(x1, a1, b1);
            f2_unpack(x0, a0, b0);
            const float p1 = a1 * b1, p0 = a0 * b0;
            // 2^-100 <= p < 2^28, 128 exponents, by the bits
            constexpr uint32_t LO = 27u << 23;
            const bool fine = (((__float_as_uint(p1) - LO) | (__float_as_uint(p0) - LO)) & 0xC0000000u) == 0;
            if (code != 3u) {
                if (fine) {
                    R1 *= p1;
                    R0 *= p0;
                    ex += normalise(R1) - normalise(R0);
                } else {
                    single += logf(a1 / a0);
                    single += logf(b1 / b0);
                }
            }
        }
        __syncthreads();
    }
    if (live)
        c.metrop[(int64_t)vb.y * D.N + i] = (double)ex * 0.693147180559945309 + (double)logf(R1 / R0) + (double)single;
}

// Label draws per copy of the byte layout (any ploidy and allele count), up to
// 16 clusters, on the same streams and with the same operations a copy as
// k_update_z_admix_ctr: one lane per individual (in ascending ploidy with mixed
// ploidy), 256 individuals per CTA. A call is two or three aligned loads; the staged
// frequencies of an allele are whole 16-byte chunks, an odd count, so that a
// copy's weights take a quarter of the loads; the label is the number of
// thresholds that the uniform reaches, its count goes to the lane's own column
// of a shared array and to the slice's shared histogram. The Philox block is
// formed when the warp's draw index enters it (mixed ploidy skips some).
// N = 1,500 x L = 8,000, ploidy 2, 4 and 6, 2-8 alleles, K = 8: 295 -> 278 us
// (256 with calls padded to 8 bytes, a third more device memory).
// Issue-bound (59% active, 131 instructions a warp's copy); loading the
// calls four loci ahead or taking 16 to 64 CTAs per SM made no difference.
constexpr int ZG_T = 256, ZG_G = 4;
static_assert(ZA_LC % ZG_G == 0, "whole groups a slice");
__host__ __device__ constexpr int zg_stride(int km) { return 4 * (((km + 3) / 4) | 1); }   // floats of an allele's row
template <int KM, bool EXACT, bool WIDE = false>
__global__ void __launch_bounds__(ZG_T, KM <= 8 ? 3 : 2) k_z_admix_gen(const DevChain* chains, int force, const int4* map = nullptr) {
    constexpr int FS = zg_stride(KM);
    extern __shared__ __align__(16) unsigned char smraw[];
    const VBlock vb = vblock(map);
    const DevChain& c = chains[vb.z];
    if (map && run_over(c)) return;
    const DevData& D = c.D;
    const int K = EXACT ? KM : c.K, m = c.ctl->m, MK = D.maxK;
    if (!force && binaryq_at(c, m)) return;
    __shared__ double sh[32];
    const int nbins = K * MK, t = threadIdx.x, vmax = D.vmax;
    float* sF = reinterpret_cast<float*>(smraw);                                 // [ZA_LC][MK][FS]
    int32_t* hs = reinterpret_cast<int32_t*>(sF + ZA_LC * MK * FS);              // [ZA_LC][K][MK]
    int32_t* ms = hs + ZA_LC * nbins + t;                                        // [K][ZG_T]
    const int slot = vb.x * ZG_T + t;
    const bool live = slot < D.N;
    const int i = live && D.perm ? D.perm[slot] : slot;
    float q[KM];
#pragma unroll
    for (int k = 0; k < KM; ++k) {
        q[k] = (live && (EXACT || k < K)) ? c.Q[(int64_t)i * K + k] : 0.f;
        if (EXACT || k < K) ms[k * ZG_T] = 0;
    }
    const int64_t lb0 = (int64_t)vb.y * c.zadm_lc, lb1 = min(D.L, lb0 + c.zadm_lc);
    float ls = 0.f, lc = 0.f;  // Kahan sum of ln(sum_k q_k p)
    const bool rec = force || record_at(c, m);
    const float minf = (float)VP_MIN_FREQ, kmin = (float)(VP_MIN_FREQ * K);
    const uint2 key = make_uint2((uint32_t)c.seed, (uint32_t)(c.seed >> 32));
    const uint32_t ca = ST_ZSLICE | ((uint32_t)m << 4);
    // a call's bytes: copy a in byte a, 0xFF past the last one, anything from byte
    // vmax on (WIDE: 16 bytes). Calls start anywhere: a call is put together from
    // the aligned words that hold it, two up to 6 bytes and at 8, else three (the
    // array is longer than its calls by GB_PAD bytes for the last one's).
    const uint8_t* gp = D.gb + (size_t)i * vmax;
    const size_t row = (size_t)D.N * vmax;
    const bool third = WIDE || vmax == 7;
    auto call = [&](int64_t l, uint64_t& lo, uint64_t& hi) {
        lo = hi = ~0ull;
        if (!live || l >= lb1) return;
        const uintptr_t g = (uintptr_t)(gp + l * row);
        const uint32_t* w = reinterpret_cast<const uint32_t*>(g & ~(uintptr_t)3);
        const uint32_t sh = 8 * (uint32_t)g, w1 = __ldg(w + 1), w2 = third ? __ldg(w + 2) : 0u;   // shifts by sh mod 32
        lo = __funnelshift_r(__ldg(w), w1, sh) | ((uint64_t)__funnelshift_r(w1, w2, sh) << 32);
        if constexpr (WIDE) hi = w2 >> (sh & 31);
    };
    // the calls of ZG_G loci are loaded while the ones before are drawn
    uint64_t nlo[ZG_G], nhi[ZG_G];
#pragma unroll
    for (int u = 0; u < ZG_G; ++u) call(lb0 + u, nlo[u], nhi[u]);
    for (int64_t l0 = lb0; l0 < lb1; l0 += ZA_LC) {
        const int nl = (int)min((int64_t)ZA_LC, lb1 - l0);
        __syncthreads();
        for (int j = t; j < ZA_LC * MK * FS; j += ZG_T) {
            const int k = j % FS, a = (j / FS) % MK, ll = j / (FS * MK);
            float v = 0.f;
            if (ll < nl && k < K && a < D.k[l0 + ll]) v = __ldg(c.Freq + (int64_t)k * D.KT + D.off[l0 + ll] + a);
            sF[j] = v;
        }
        for (int j = t; j < ZA_LC * nbins; j += ZG_T) hs[j] = 0;
        __syncthreads();
        int block = -1;
        uint4 rb = make_uint4(0, 0, 0, 0);
        for (int lg = 0; lg < nl; lg += ZG_G) {
          uint64_t clo[ZG_G], chi[ZG_G];
#pragma unroll
          for (int u = 0; u < ZG_G; ++u) {
            clo[u] = nlo[u];
            chi[u] = nhi[u];
            call(l0 + lg + ZG_G + u, nlo[u], nhi[u]);
          }
#pragma unroll
          for (int u = 0; u < ZG_G; ++u) {
            const int ll = lg + u;
            if (ll >= nl) break;
            const uint64_t lo = clo[u], hi = chi[u];
            // allele indices are below 64: a copy past the last has its high bit set
            const uint64_t e0 = lo & 0x8080808080808080ull, e1 = hi & 0x8080808080808080ull;
            const int n = min(vmax, e0 ? (__ffsll((long long)e0) - 1) >> 3 : WIDE && e1 ? 8 + ((__ffsll((long long)e1) - 1) >> 3) : WIDE ? 16 : 8);
            const int nw = (int)__reduce_max_sync(0xffffffffu, (unsigned)n);
            float lacc = 0.f;
            for (int a = 0; a < nw; ++a) {
                const int pos = ll * vmax + a;
                if ((pos >> 2) != block) {
                    block = pos >> 2;
                    rb = Philox::round10(make_uint4(ca, (uint32_t)(l0 / ZA_LC), (uint32_t)i, (uint32_t)block), key);
                }
                const uint32_t x = pos & 2 ? (pos & 1 ? rb.w : rb.z) : (pos & 1 ? rb.y : rb.x);
                if (a < n) {
                    const int al = (int)((!WIDE || a < 8 ? lo >> (8 * a) : hi >> (8 * (a - 8))) & 63u);
                    const float4* f = reinterpret_cast<const float4*>(sF + (ll * MK + al) * FS);
                    float sx = 0.f, pre[KM];
#pragma unroll
                    for (int k = 0; k < KM; k += 4) {
                        const float4 v = f[k >> 2];
                        sx = __fmaf_rn(q[k], v.x, sx);
                        pre[k] = sx;
                        if (k + 1 < KM) { sx = __fmaf_rn(q[k + 1], v.y, sx); pre[k + 1] = sx; }
                        if (k + 2 < KM) { sx = __fmaf_rn(q[k + 2], v.z, sx); pre[k + 2] = sx; }
                        if (k + 3 < KM) { sx = __fmaf_rn(q[k + 3], v.w, sx); pre[k + 3] = sx; }
                    }
                    if (rec) lacc += logf(sx);
                    const float tt = Philox::to_uniformf(x) * (sx + kmin);
                    int z = 0;
#pragma unroll
                    for (int k = 0; k < KM - 1; ++k)
                        if ((EXACT || k < K - 1) && !(tt < __fmaf_rn((float)(k + 1), minf, pre[k]))) ++z;
                    atomicAdd(&ms[z * ZG_T], 1);
                    atomicAdd(&hs[ll * nbins + z * MK + al], 1);
                }
            }
            const float y = lacc - lc, sum = ls + y;
            lc = (sum - ls) - y;
            ls = sum;
          }
        }
        __syncthreads();
        for (int j = t; j < nl * nbins; j += ZG_T) {
            const int v = hs[j];
            if (!v) continue;
            const int a = j % MK, k = (j / MK) % K, ll = j / nbins;
            atomicAdd(&c.Ni[(int64_t)k * D.KT + D.off[l0 + ll] + a], v);
        }
    }
    if (live)
#pragma unroll
        for (int k = 0; k < KM; ++k)
            if (EXACT || k < K) {
                const int v = ms[k * ZG_T];
                if (v) atomicAdd(&c.Mi[(int64_t)i * K + k], v);
            }
    const double tot = block_sum((double)ls - (double)lc, sh);
    if (t == 0) c.lnlp[vb.y * vb.gx + vb.x] = tot;
}

}  // namespace vp
