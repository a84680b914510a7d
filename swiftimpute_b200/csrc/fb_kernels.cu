// fb_kernels.cu — fused emission / forward-backward / posterior epilogue.
//
// Model (the reference's recurrences, restated in linear space):
//   emission   E_m[k] = exp(GL[a(h0_k) + a(h1_k)])         emission.cu:35-54
//              GL is {0, -999, -999}-style (imputer.cpp:244-295): slots whose
//              pair sum equals the call get 1, the others e^-999 (= 0 here);
//              a call no slot matches scales every slot by e^-999 alike.
//   transition T = c + delta * I, c = exp(log10 switch),   transition.cu:98-115
//              c + delta = exp(log10 stay) (log10 values fed to natural-log
//              recursions, logsumexp.cuh:67-70).
//   forward    alpha_m = E_m . (T^T alpha_{m-1})             forward_backward.cu:92-131
//   backward   beta_m  = e^-999 + T (E_{m+1} . beta_{m+1})   forward_backward.cu:221-241
//              The e^-999 term is the LOG_ZERO seed of every logsumexp2
//              chain; beta is never rescaled in the reference, so the term
//              matters once beta decays near e^-999. beta's absolute scale is
//              therefore tracked exactly as 2^Kb * e^(-999 nb); when the floor
//              dominates the unit switches to e^-999 itself.
//   posterior  P_m(k) = softmax(log alpha + log beta)       sampling.cu:80-100
// FP32 values, exact power-of-two rescaling every marker (no rounding from
// the rescale), the floor term computed from the integer scale in FP64.
//
// One thread carries one target chain with all L slots in registers (the
// transition is rank-1 plus diagonal, so a step is O(L), not O(L^2)). Markers
// are cut into segments of C:
//   fb_ends_kernel     the two recursions over all markers, forward and backward
//                      at the same time, leaving alpha and beta at the segments'
//                      ends (HBM);
//   fb_segment_kernel  every segment on its own, all at once: alpha recomputed
//                      from its start into shared memory, beta walked back from
//                      its end, and dosage, P(hap=1) and haplotypes written.
// Without room for beta's ends (the caller's HBM budget, the allocation-free
// entry point's fixed array) one CTA takes its chains' segments one after the
// other, forward and then back (fb_segment_kernel with kAll), with the same
// results. Inputs and outputs of a segment are staged in shared memory so global
// traffic is coalesced row segments.
#include "philox.cuh"
#include "si_internal.hpp"
#include "slots.cuh"

#include <type_traits>

namespace si {
namespace {

struct FbArgs {
    const uint8_t* geno;
    const SlotMasks* masks;
    const SlotMasks* smasks;  // per-target [M][B] (target-aware selection), else null
    const uint8_t* raw;
    const LinTrans* trans;
    uint32_t B, M, L, C, nseg;
    int sampling;
    float tie_eps;
    uint64_t seed, sid_base;
    float* ckpt;          // alpha at the segments' last markers [nseg - 1][LM][B]
    float* bckpt;         // beta at the segments' first markers but the first's [nseg - 1][LM][B], or null
    int2* bunit;          // its unit {Kb, nb} [nseg - 1][B]
    float* dosage;
    float* hprob;
    uint8_t* haps;
};

__device__ __forceinline__ int exp2_of(float x) {  // floor(log2 x) for positive normal x
    return ((__float_as_int(x) >> 23) & 0xff) - 127;
}
__device__ __forceinline__ float pow2_neg(int e) {  // 2^-e, |e| <= 126
    return __int_as_float((127 - e) << 23);
}

// exact int -> double on the FP64 pipe: 2^52 + 2^31 + x has x + 2^31 in its low word
__device__ __forceinline__ double i2d(int x) {
    return __hiloint2double(0x43300000, (int)((uint32_t)x ^ 0x80000000u)) - 4503601774854144.0;
}

template <int LM>
__device__ __forceinline__ void forward_step(float (&al)[LM], float& S, uint32_t em, LinTrans tr, bool first) {
    if (first) {
#pragma unroll
        for (int k = 0; k < LM; ++k) al[k] = ((em >> k) & 1u) ? 1.0f : 0.0f;
    } else {
        const float sc = pow2_neg(exp2_of(S));
        const float cS = tr.c * (S * sc);
        const float dl = tr.delta * sc;
#pragma unroll
        for (int k = 0; k < LM; ++k) al[k] = ((em >> k) & 1u) ? fmaf(dl, al[k], cS) : 0.0f;
    }
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < LM; ++k) s += al[k];
    S = s;
}

// Offset of the slot masks in a CTA's shared memory, behind the alpha tile
// [C][LM][T], the dosage rows [T][C + 1] and, for P(hap=1), its rows [T][2 C + 1].
__host__ __device__ constexpr size_t mask_offset(uint32_t LM, uint32_t T, uint32_t C, bool hprob) {
    return ((size_t)C * LM * T * 4 + (size_t)T * (C + 1) * 4 + (hprob ? (size_t)T * (2 * C + 1) * 4 : 0) + 15) & ~size_t(15);
}

// Bound by latency at few warps an SM (the alpha tile is most of a chain's 1.3 KB
// of shared memory at C = 32, 0.65 at 16): 1,000 x 20,000 at L = 8 takes 1.20 ms
// with segments of 32 markers, 0.76 with 16 and no room kept for an unwanted P(hap=1).
// kAll: the CTA runs the whole chain, forward first; else segment blockIdx.x /
// tiles alone, from the ends that fb_ends_kernel left.
template <int LM, bool kAll>
__global__ void __launch_bounds__(128) fb_segment_kernel(FbArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t T = blockDim.x, C = a.C;
    const uint32_t GS = C + 4;          // code row stride (bytes)
    const uint32_t DS = C + 1;          // dosage row stride (floats)
    const uint32_t HS = 2 * C + 1;      // hprob row stride (floats)
    const uint32_t PS = C + 4;          // hap row stride (bytes, per phase)
    float* abuf = reinterpret_cast<float*>(smem);                       // [C][LM][T]
    float* dbuf = abuf + (size_t)C * LM * T;                            // [T][DS]
    float* hbuf = dbuf + (size_t)T * DS;                                // [T][HS] (P(hap=1) only)
    SlotMasks* mseg = reinterpret_cast<SlotMasks*>(smem + mask_offset(LM, T, C, a.hprob != nullptr));  // [C]
    LinTrans* tseg = reinterpret_cast<LinTrans*>(mseg + C);             // [C]
    uint8_t* gbuf = reinterpret_cast<uint8_t*>(tseg + C);               // [T][GS]
    uint8_t* pbuf = gbuf + (size_t)T * GS;                              // [T][2][PS]

    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5, nwarps = T >> 5;
    const uint32_t tiles = (a.B + T - 1) / T;
    const uint32_t s0 = (kAll ? blockIdx.x : blockIdx.x % tiles) * T;
    const uint32_t s = s0 + t;
    const bool live = s < a.B;
    const uint32_t M = a.M, L = a.L;
    const uint32_t lmask = (L >= 32) ? 0xffffffffu : ((1u << L) - 1u);

    // stage codes, masks and transitions of markers [m0, m0 + cl)
    auto stage = [&](uint32_t m0, uint32_t cl) {
        for (uint32_t r = warp; r < T; r += nwarps) {
            const uint32_t sr = s0 + r;
            if (sr < a.B && lane < cl) gbuf[r * GS + lane] = a.geno[(uint64_t)sr * M + m0 + lane];
        }
        for (uint32_t i = t; i < cl; i += T) {
            if (!a.smasks) mseg[i] = a.masks[m0 + i];
            tseg[i] = a.trans[m0 + i];
        }
    };
    // the slot masks of marker m (staged at i): per marker, or this target's own
    auto mask_at = [&](uint32_t i, uint32_t m) {
        if (!a.smasks) return mseg[i];
        return live ? a.smasks[(uint64_t)m * a.B + s] : SlotMasks{0u, 0u, 0u, 0u};
    };

    float al[LM];
    float S = 0.f;

    // ---------------- forward: checkpoints at segment ends ----------------
    for (uint32_t j = 0; kAll && j < a.nseg; ++j) {
        const uint32_t m0 = j * C, cl = min(C, M - m0);
        __syncthreads();
        stage(m0, cl);
        __syncthreads();
        for (uint32_t i = 0; i < cl; ++i) {
            uint32_t sh;
            const uint32_t em = emission_mask(gbuf[t * GS + i], mask_at(i, m0 + i), lmask, &sh);
            forward_step<LM>(al, S, em, tseg[i], m0 + i == 0);
        }
        if (live && j + 1 < a.nseg) {
#pragma unroll
            for (int k = 0; k < LM; ++k) a.ckpt[((uint64_t)j * LM + k) * a.B + s] = al[k];
        }
    }

    // ---------------- backward with fused posterior epilogue ----------------
    float be[LM];
    int Kb = 0, nb = 0;                  // |beta| = 2^Kb * e^(-999 nb) * be
    uint32_t em_next = 0, sh_next = 0;   // emission of marker m + 1
    LinTrans tr_next = {0.f, 0.f};       // transition into marker m + 1
    const float keep = 1.0f - a.tie_eps;

    const int jfirst = kAll ? (int)a.nseg - 1 : (int)(blockIdx.x / tiles), jlast = kAll ? 0 : jfirst;
    if (!kAll && jfirst + 1 < (int)a.nseg) {
        // beta at the next segment's first marker, and that marker's emission and transition
        const uint32_t mn = (uint32_t)(jfirst + 1) * C;
#pragma unroll
        for (int k = 0; k < LM; ++k) be[k] = live ? a.bckpt[((uint64_t)jfirst * LM + k) * a.B + s] : 0.f;
        const int2 u = live ? a.bunit[(uint64_t)jfirst * a.B + s] : make_int2(0, 0);
        Kb = u.x;
        nb = u.y;
        const SlotMasks mk = !a.smasks ? a.masks[mn] : live ? a.smasks[(uint64_t)mn * a.B + s] : SlotMasks{0u, 0u, 0u, 0u};
        em_next = emission_mask(live ? a.geno[(uint64_t)s * M + mn] : 3u, mk, lmask, &sh_next);
        tr_next = a.trans[mn];
    }
    for (int jj = jfirst; jj >= jlast; --jj) {
        const uint32_t j = (uint32_t)jj;
        const uint32_t m0 = j * C, cl = min(C, M - m0);
        __syncthreads();
        stage(m0, cl);
        __syncthreads();
        // recompute alpha over the segment
        if (j > 0) {
            S = 0.f;
#pragma unroll
            for (int k = 0; k < LM; ++k) {
                al[k] = live ? a.ckpt[((uint64_t)(j - 1) * LM + k) * a.B + s] : 0.f;
                S += al[k];
            }
            if (!live) S = 1.f;
        }
        for (uint32_t i = 0; i < cl; ++i) {
            uint32_t sh;
            const uint32_t em = emission_mask(gbuf[t * GS + i], mask_at(i, m0 + i), lmask, &sh);
            forward_step<LM>(al, S, em, tseg[i], m0 + i == 0);
#pragma unroll
            for (int k = 0; k < LM; ++k) abuf[((size_t)i * LM + k) * T + t] = al[k];
        }
        // beta walk and epilogue
        for (int ii = (int)cl - 1; ii >= 0; --ii) {
            const uint32_t i = (uint32_t)ii, m = m0 + i;
            if (m == M - 1) {
#pragma unroll
                for (int k = 0; k < LM; ++k) be[k] = ((lmask >> k) & 1u) ? 1.0f : 0.0f;
                Kb = 0; nb = 0;
            } else {
                float w[LM];
                float sw = 0.f;
#pragma unroll
                for (int k = 0; k < LM; ++k) { w[k] = ((em_next >> k) & 1u) ? be[k] : 0.0f; sw += w[k]; }
                // beta_m = e^-999 + U * (c sw + delta w), U = 2^Kb e^(-999 (nb + sh)): the
                // floor in units of U is exp(farg)
                const double farg = 999.0 * (double)(nb + (int)sh_next - 1) - (double)Kb * 0.69314718055994530942;
                if (farg > 0.0) {
                    // the floor dominates: switch the unit to e^-999 (Kb = 0, nb = 1),
                    // beta_m = e^-999 (1 + exp(-farg) (c sw + delta w))
                    const float g = expf(-(float)fmin(farg, 100.0));
                    const float cs = tr_next.c * sw;
#pragma unroll
                    for (int k = 0; k < LM; ++k)
                        be[k] = ((lmask >> k) & 1u) ? fmaf(g, fmaf(tr_next.delta, w[k], cs), 1.0f) : 0.0f;
                    Kb = 0;
                    nb = 1;
                } else {
                    const float F = farg > -104.0 ? expf((float)farg) : 0.0f;
                    const float base = fmaf(tr_next.c, sw, F);  // common part of every slot, >= c
                    const int e = exp2_of(base);
                    const float sc = pow2_neg(e);
                    const float b2 = base * sc;
                    const float dl = tr_next.delta * sc;
#pragma unroll
                    for (int k = 0; k < LM; ++k) be[k] = ((lmask >> k) & 1u) ? fmaf(dl, w[k], b2) : 0.0f;
                    Kb += e;
                    nb += (int)sh_next;
                }
            }
            // posterior at m
            const SlotMasks mk = mask_at(i, m);
            float p[LM];
            float tot = 0.f, q0 = 0.f, q1 = 0.f, pmax = 0.f;
#pragma unroll
            for (int k = 0; k < LM; ++k) {
                p[k] = abuf[((size_t)i * LM + k) * T + t] * be[k];
                tot += p[k];
                q0 += ((mk.a0 >> k) & 1u) ? p[k] : 0.f;
                q1 += ((mk.a1 >> k) & 1u) ? p[k] : 0.f;
                pmax = fmaxf(pmax, p[k]);
            }
            uint32_t pick = 0;
            if (a.sampling == SI_SAMPLE_ARGMAX) {
                const float thr = pmax * keep;
                pick = LM;
#pragma unroll
                for (int k = LM - 1; k >= 0; --k) pick = (p[k] >= thr) ? (uint32_t)k : pick;
                if (pick >= LM) pick = 0;
            } else {
                const float target = cell_uniform(a.seed, a.sid_base + s, m) * tot;
                float cum = 0.f;
                uint32_t last_nz = 0;
                pick = LM;
#pragma unroll
                for (int k = 0; k < LM; ++k) {
                    cum += p[k];
                    if (p[k] > 0.f) last_nz = (uint32_t)k;
                    if (pick == LM && target < cum) pick = (uint32_t)k;
                }
                if (pick == LM) pick = last_nz;
            }
            const float inv = 1.0f / tot;
            dbuf[t * DS + i] = (q0 + q1) * inv;
            if (a.hprob) {
                hbuf[t * HS + 2 * i] = q0 * inv;
                hbuf[t * HS + 2 * i + 1] = q1 * inv;
            }
            const uint32_t hv = slot_alleles(mk, a.raw, fb_lmax(L), m, pick);
            pbuf[(t * 2 + 0) * PS + i] = (uint8_t)(hv & 0xffu);
            pbuf[(t * 2 + 1) * PS + i] = (uint8_t)(hv >> 8);
            // this marker's emission/transition drive beta_{m-1}
            uint32_t sh;
            em_next = emission_mask(gbuf[t * GS + i], mk, lmask, &sh);
            sh_next = sh;
            tr_next = tseg[i];
        }
        __syncthreads();
        // flush the segment's outputs as coalesced row segments
        for (uint32_t r = warp; r < T; r += nwarps) {
            const uint32_t sr = s0 + r;
            if (sr >= a.B) continue;
            const uint64_t row = (uint64_t)sr * M + m0;
            if (lane < cl) {
                if (a.dosage) a.dosage[row + lane] = dbuf[r * DS + lane];
                if (a.haps) {
                    a.haps[(uint64_t)sr * 2 * M + m0 + lane] = pbuf[(r * 2 + 0) * PS + lane];
                    a.haps[(uint64_t)sr * 2 * M + M + m0 + lane] = pbuf[(r * 2 + 1) * PS + lane];
                }
            }
            if (a.hprob)
                for (uint32_t l = lane; l < 2 * cl; l += 32) a.hprob[row * 2 + l] = hbuf[r * HS + l];
        }
    }
}

// ---------------------------------------------------------------- the chains

// markers per staged block: two blocks of 32 slots' factors stay under 48 KB
__host__ __device__ constexpr uint32_t ends_block(uint32_t LM) { return LM <= 16 ? 8u : 4u; }
constexpr uint32_t kEndsChunk = 32;                        // codes of a row staged at a time
constexpr uint32_t kEndsPrep = 4;                          // warps that prepare a chain warp's steps
constexpr uint32_t kEndsThreads = 32 * (1 + kEndsPrep);

// A marker as a step needs it: the emission over the lane's slots as 0/1 factors,
// whether no slot matches the call, and the transition into it.
template <int LM>
struct EndsStage {
    float4 mask[ends_block(LM)][LM / 4][32];
    uint32_t sh[ends_block(LM)][32];
    LinTrans tr[ends_block(LM)];
};

// One chain per lane; a CTA runs the forward (even blocks) or the backward (odd
// blocks) recursion of 32 samples over all markers, in warp 0. The arithmetic and
// its order are those of fb_segment_kernel.
// Bound: the dependent recursion (a sum over the slots a marker, and backward the
// floor), one warp's markers one after the other. So the other warps stage the
// rows' codes (coalesced, a chunk ahead) and prepare each marker's record, and the
// chain warp does nothing else than step: a masked update (an emission bit is a
// factor 0 or 1, exact), the slots' sum in slot order and the rescale.
// 1,000 chains x 20,000 markers on a per-gap map, L = 8: 2.19 ms here and 0.76 in
// fb_segment_kernel, 27.7 when one thread walked each chain three times in one
// kernel; a backward step takes 213 cycles, a forward one 167 (clock64). Not kept:
// two preparing warps that waited for each block's slot masks (3.44 ms), a vote
// and a branch for chains whose floor dominates (2.67).
template <int LM, bool kFull>
__global__ void __launch_bounds__(kEndsThreads) fb_ends_kernel(FbArgs a) {
    constexpr uint32_t KB = ends_block(LM), H = LM / 2, Q4 = LM / 4, kRow = kEndsChunk + 4;
    __shared__ __align__(16) EndsStage<LM> stage[2];
    __shared__ uint8_t codes[2][32 * kRow];  // by chunk parity
    __shared__ float4 nibble[16];            // four emission bits as factors
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool forward = (blockIdx.x & 1u) == 0;
    const uint32_t s0 = (blockIdx.x >> 1) * 32, s = s0 + lane;
    const bool live = s < a.B;
    const uint32_t M = a.M, C = a.C;
    const uint32_t lmask = (a.L >= 32) ? 0xffffffffu : ((1u << a.L) - 1u);
    // iteration i takes block blk(i) of KB markers, forward ascending, backward descending
    const uint32_t NB = (M + KB - 1) / KB;
    auto blk = [&](uint32_t i) { return forward ? i : NB - 1 - i; };
    if (threadIdx.x < 16)
        nibble[threadIdx.x] = make_float4(threadIdx.x & 1u ? 1.f : 0.f, threadIdx.x & 2u ? 1.f : 0.f,
                                          threadIdx.x & 4u ? 1.f : 0.f, threadIdx.x & 8u ? 1.f : 0.f);

    if (warp > 0) {
        constexpr uint32_t kRows = 32 / kEndsPrep, JP = KB / kEndsPrep, kPer = kEndsChunk / KB;
        uint8_t got[kRows];  // this lane's column of this warp's rows, on their way
        auto load = [&](uint32_t chunk) {
            const uint32_t m = chunk * kEndsChunk + lane;
#pragma unroll
            for (uint32_t r = 0; r < kRows; ++r) {
                const uint32_t sr = s0 + (warp - 1) * kRows + r;
                got[r] = (sr < a.B && m < M) ? a.geno[(uint64_t)sr * M + m] : 3;
            }
        };
        auto put = [&](uint32_t chunk) {
#pragma unroll
            for (uint32_t r = 0; r < kRows; ++r) codes[chunk & 1u][((warp - 1) * kRows + r) * kRow + lane] = got[r];
        };
        // slot masks and transitions of the iteration to prepare next, on their way since the last one
        SlotMasks mk[JP];
        LinTrans tr = {0.f, 0.f};
        auto fetch = [&](uint32_t i) {
            if (i >= NB) return;
            const uint32_t b = blk(i);
#pragma unroll
            for (uint32_t jj = 0; jj < JP; ++jj) {
                const uint32_t m = min(b * KB + (warp - 1) * JP + jj, M - 1);
                mk[jj] = !a.smasks ? a.masks[m] : live ? a.smasks[(uint64_t)m * a.B + s] : SlotMasks{0u, 0u, 0u, 0u};
            }
            if (warp == 1 && lane < KB) tr = a.trans[min(b * KB + lane, M - 1)];
        };
        auto prepare = [&](uint32_t i) {
            const uint32_t b = blk(i), chunk = b / kPer;
            EndsStage<LM>& S = stage[i & 1u];
            if (warp == 1 && lane < KB) S.tr[lane] = tr;
#pragma unroll
            for (uint32_t jj = 0; jj < JP; ++jj) {
                const uint32_t j = (warp - 1) * JP + jj;
                const uint32_t g = codes[chunk & 1u][lane * kRow + (b % kPer) * KB + j];
                uint32_t sh;
                const uint32_t em = emission_mask(g, mk[jj], lmask, &sh);
                S.sh[j][lane] = sh;
#pragma unroll
                for (uint32_t q = 0; q < Q4; ++q) S.mask[j][q][lane] = nibble[(em >> (4 * q)) & 15u];
            }
            fetch(i + 1);
        };
        // the chunk after the current one in walking order is loaded when its first block is
        // prepared and put into shared memory when its last one is
        auto turn = [&](uint32_t i) {  // prepare iteration i's records
            const uint32_t b = blk(i), chunk = b / kPer, at = b % kPer;
            const bool first = i == 0 || at == (forward ? 0u : kPer - 1), last = at == (forward ? kPer - 1 : 0u);
            const uint32_t next = forward ? chunk + 1 : chunk - 1;
            const bool more = forward ? next * kEndsChunk < M : chunk > 0;
            if (first && more) load(next);
            prepare(i);
            if (last && more) put(next);
        };
        load(blk(0) / kPer);
        fetch(0);
        put(blk(0) / kPer);
        __syncthreads();
        turn(0);
        for (uint32_t i = 0; i < NB; ++i) {
            __syncthreads();  // records i are ready; records i - 1 have been read
            if (i + 1 < NB) turn(i + 1);
        }
        return;
    }

    auto masks = [&](const EndsStage<LM>& S, uint32_t j, float2 (&m)[H]) {
#pragma unroll
        for (uint32_t q = 0; q < Q4; ++q) {
            const float4 x = S.mask[j][q][lane];
            m[2 * q] = make_float2(x.x, x.y);
            m[2 * q + 1] = make_float2(x.z, x.w);
        }
    };
    auto slot_sum = [&](const float2 (&x)[H]) {  // in slot order
        float t = 0.f;
#pragma unroll
        for (uint32_t h = 0; h < H; ++h) {
            t += x[h].x;
            t += x[h].y;
        }
        return t;
    };
    auto pair = [](float x) { return make_float2(x, x); };
    float2 x[H];
    __syncthreads();
    if (forward) {
        float S = 0.f;
        uint32_t to_end = C;  // markers to the segment's end
        float* ck = a.ckpt + s;
        uint32_t segs = a.nseg - 1;  // ends to store
        for (uint32_t i = 0; i < NB; ++i) {
            __syncthreads();
            const EndsStage<LM>& R = stage[i & 1u];
            float2 m[H], mn[H];
            masks(R, 0, mn);
#pragma unroll
            for (uint32_t j = 0; j < KB; ++j) {
#pragma unroll
                for (uint32_t h = 0; h < H; ++h) m[h] = mn[h];
                if (j + 1 < KB) masks(R, j + 1, mn);
                if (i * KB + j < M) {
                    if (j == 0 && i == 0) {
#pragma unroll
                        for (uint32_t h = 0; h < H; ++h) x[h] = m[h];
                    } else {
                        const LinTrans tr = R.tr[j];
                        const float sc = __int_as_float(0x7f000000 - (__float_as_int(S) & 0x7f800000));
                        const float2 cS = pair(tr.c * (S * sc)), dl = pair(tr.delta * sc);
#pragma unroll
                        for (uint32_t h = 0; h < H; ++h)
                            x[h] = __ffma2_rn(__fmul2_rn(dl, m[h]), x[h], __fmul2_rn(cS, m[h]));
                    }
                    S = slot_sum(x);
                    if (--to_end == 0) {
                        to_end = C;
                        if (segs) {
                            --segs;
                            if (live) {
#pragma unroll
                                for (uint32_t h = 0; h < H; ++h) {
                                    ck[(uint64_t)(2 * h) * a.B] = x[h].x;
                                    ck[(uint64_t)(2 * h + 1) * a.B] = x[h].y;
                                }
                            }
                            ck += (uint64_t)LM * a.B;
                        }
                    }
                }
            }
        }
    } else {
        int Kb = 0, nb = 0;
        float2 one[H];  // the slots in use
#pragma unroll
        for (uint32_t h = 0; h < H; ++h) {
            one[h] = make_float2((lmask >> (2 * h)) & 1u ? 1.f : 0.f, (lmask >> (2 * h + 1)) & 1u ? 1.f : 0.f);
            x[h] = one[h];
        }
        auto store = [&](uint32_t seg) {  // beta at the first marker of segment seg + 1
            if (!live) return;
            float* ck = a.bckpt + (uint64_t)seg * LM * a.B + s;
#pragma unroll
            for (uint32_t h = 0; h < H; ++h) {
                ck[(uint64_t)(2 * h) * a.B] = x[h].x;
                ck[(uint64_t)(2 * h + 1) * a.B] = x[h].y;
            }
            a.bunit[(uint64_t)seg * a.B + s] = make_int2(Kb, nb);
        };
        uint32_t seg = a.nseg - 1, left = M - 1 - seg * C;  // the marker is `left` past the first one of segment seg
        if (left == 0 && seg > 0) store(seg - 1);
        for (uint32_t i = 0; i < NB; ++i) {
            __syncthreads();
            const EndsStage<LM>& R = stage[i & 1u];
            const uint32_t m0 = (NB - 1 - i) * KB;
            float2 m[H], mn[H];
            masks(R, KB - 1, mn);
            // kEdge: the block holds markers past the last one, or the first one
            auto steps = [&](auto kEdge) {
#pragma unroll
                for (uint32_t jj = 0; jj < KB; ++jj) {
                    const uint32_t j = KB - 1 - jj, mr = m0 + j;  // the step from marker mr to mr - 1
#pragma unroll
                    for (uint32_t h = 0; h < H; ++h) m[h] = mn[h];
                    if (j > 0) masks(R, j - 1, mn);
                    if (kEdge && (mr >= M || mr == 0)) continue;
                    const LinTrans tr = R.tr[j];
                    const uint32_t sh_next = R.sh[j][lane];
                    float2 w[H];
#pragma unroll
                    for (uint32_t h = 0; h < H; ++h) w[h] = __fmul2_rn(x[h], m[h]);
                    const float sw = slot_sum(w);
                    const double farg = 999.0 * i2d(nb + (int)sh_next - 1) - i2d(Kb) * 0.69314718055994530942;
                    const bool big = farg > 0.0;  // the floor dominates: the unit becomes e^-999
                    const float fa = (float)farg;
                    const float ex = expf(big ? -fminf(fa, 100.f) : fa);
                    const float F = farg > -104.0 ? ex : 0.f;
                    const float base = fmaf(tr.c, sw, F);
                    const int bits = __float_as_int(base) & 0x7f800000;
                    const float sc = __int_as_float(0x7f000000 - bits);  // 2^-e
                    // delta w + base in the new unit, or, the floor dominating, 1 + e^-farg (delta w + c sw):
                    // both as g (d w + c) + o
                    const float2 g2 = pair(big ? ex : 1.f), o2 = pair(big ? 1.f : 0.f);
                    const float2 d2 = pair(big ? tr.delta : tr.delta * sc), c2 = pair(big ? tr.c * sw : base * sc);
#pragma unroll
                    for (uint32_t h = 0; h < H; ++h) {
                        const float2 y = __ffma2_rn(g2, __ffma2_rn(d2, w[h], c2), o2);
                        x[h] = kFull ? y : __fmul2_rn(y, one[h]);
                    }
                    Kb = big ? 0 : Kb + (bits >> 23) - 127;
                    nb = big ? 1 : nb + (int)sh_next;
                    if (left == 0) {
                        left = C;
                        --seg;
                    }
                    if (--left == 0 && seg > 0) store(seg - 1);
                }
            };
            if (i == 0 || i + 1 == NB) steps(std::true_type{});
            else steps(std::false_type{});
        }
    }
}

template <int LM>
size_t smem_bytes(uint32_t T, uint32_t C, bool hprob = true) {
    return mask_offset(LM, T, C, hprob) + (size_t)C * (sizeof(SlotMasks) + sizeof(LinTrans)) +
           (size_t)T * (C + 4) + (size_t)T * 2 * (C + 4) + 16;
}

template <int LM, bool kAll>
cudaError_t launch_segments(const FbArgs& fa, uint32_t T, size_t sm, cudaStream_t s) {
    cudaError_t e = allow_smem(fb_segment_kernel<LM, kAll>);
    if (e != cudaSuccess) return e;
    const unsigned long long grid = (unsigned long long)((fa.B + T - 1) / T) * (kAll ? 1u : fa.nseg);
    if (grid > 0x7fffffffull) return cudaErrorInvalidConfiguration;
    fb_segment_kernel<LM, kAll><<<(uint32_t)grid, T, sm, s>>>(fa);
    return cudaGetLastError();
}

template <int LM>
cudaError_t launch_lm(const FbArgs& fa, uint32_t T, cudaStream_t s) {
    const size_t sm = smem_bytes<LM>(T, fa.C, fa.hprob != nullptr);
    if (sm > kMaxSmem) return cudaErrorInvalidValue;
    if (!fa.bckpt) return launch_segments<LM, true>(fa, T, sm, s);
    const uint32_t ctas = 2 * ((fa.B + 31) / 32);
    if (fa.L == LM) fb_ends_kernel<LM, true><<<ctas, kEndsThreads, 0, s>>>(fa);
    else fb_ends_kernel<LM, false><<<ctas, kEndsThreads, 0, s>>>(fa);
    const cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? e : launch_segments<LM, false>(fa, T, sm, s);
}

}  // namespace


size_t fb_smem_bytes(uint32_t L, uint32_t T, uint32_t C) {
    switch (fb_lmax(L)) {
        case 4: return smem_bytes<4>(T, C);
        case 8: return smem_bytes<8>(T, C);
        case 16: return smem_bytes<16>(T, C);
        default: return smem_bytes<32>(T, C);
    }
}

size_t fb_ckpt_bytes(uint32_t B, uint32_t M, uint32_t L, uint32_t C) {
    const uint32_t nseg = (M + C - 1) / C;
    return (size_t)(nseg > 1 ? nseg - 1 : 1) * fb_lmax(L) * B * sizeof(float);
}

// beta's ends: the vectors, then their units
size_t fb_back_bytes(uint32_t B, uint32_t M, uint32_t L, uint32_t C) {
    const uint32_t nseg = (M + C - 1) / C;
    return (size_t)(nseg > 1 ? nseg - 1 : 1) * (fb_lmax(L) * sizeof(float) + sizeof(int2)) * B;
}

bool fb_segments_fit(uint32_t B, uint32_t M, uint32_t C, uint32_t T) {
    return (unsigned long long)((B + T - 1) / T) * ((M + C - 1) / C) <= 0x7fffffffull;
}

cudaError_t launch_fb(const FbLaunch& l, cudaStream_t s) {
    FbArgs fa;
    fa.geno = l.geno; fa.masks = l.masks; fa.smasks = l.smasks; fa.raw = l.raw; fa.trans = l.trans;
    fa.B = l.B; fa.M = l.M; fa.L = l.L; fa.C = l.C; fa.nseg = (l.M + l.C - 1) / l.C;
    fa.sampling = l.sampling; fa.tie_eps = l.tie_eps; fa.seed = l.seed; fa.sid_base = l.sample_id_base;
    fa.ckpt = l.ckpt; fa.bckpt = fb_segments_fit(l.B, l.M, l.C, l.threads) ? l.bckpt : nullptr;
    fa.bunit = fa.bckpt ? (int2*)(fa.bckpt + (size_t)(fa.nseg > 1 ? fa.nseg - 1 : 1) * fb_lmax(l.L) * l.B) : nullptr;
    fa.dosage = l.dosage; fa.hprob = l.hprob; fa.haps = l.haps;
    if (l.C == 0 || l.C > 32 || l.threads == 0 || l.threads % 32 || l.threads > 128) return cudaErrorInvalidValue;
    switch (fb_lmax(l.L)) {
        case 4: return launch_lm<4>(fa, l.threads, s);
        case 8: return launch_lm<8>(fa, l.threads, s);
        case 16: return launch_lm<16>(fa, l.threads, s);
        default: return launch_lm<32>(fa, l.threads, s);
    }
}

}  // namespace si
