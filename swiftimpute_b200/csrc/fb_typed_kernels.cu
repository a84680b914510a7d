// fb_typed_kernels.cu — forward-backward over typed markers only.
//
// Same model as fb_kernels.cu (the reference's recurrences restated in linear
// space, with beta's e^-999 logsumexp floor), specialised to one transition
// for every gap (the reference reads matrix 0 for all gaps,
// forward_backward.cu:108,201,234,269). Untyped markers have emission 1 in
// every slot, and T = c 11^T + delta I, so a run of n untyped markers has a
// closed form (rho = delta + L c, q = delta / rho):
//   forward   alpha_{p+n}  ~  q^n a + sum(a) (1 - q^n) / L
//   backward  beta_{t-n}   ~  q^n w + sum(w) (1 - q^n) / L + e^-999 / U * G(n)
//             with w = E_t . beta_t at typed marker t, U its scale and
//             G(n) = sum_{k=1..n} rho^-k (the floor accumulated over the run).
// The sequential chain therefore steps over typed markers ("anchors") only,
// and every cell's posterior follows from its two bracketing anchors, so the
// per-cell work runs in parallel. Kernels:
//   anchor_count / anchor_scan / anchor_fill   per-sample anchor lists (marker 0
//                                              is always an anchor)
//   anchor_chain     one lane per sample and direction (all slots in
//                    registers): forward and backward over anchors; backward
//                    checkpoints every C anchors (a window), forward ones
//                    every K windows
//   anchor_posterior one lane per sample walks the markers of K windows:
//                    the window's backward records are rebuilt from its
//                    checkpoint, alpha is carried from anchor to anchor, and
//                    every marker's dosage, P(hap=1) and haplotypes are
//                    written through a shared-memory tile.
#include "fb_typed.hpp"
#include "philox.cuh"

#include <type_traits>

namespace si {
namespace {

__device__ __forceinline__ int exp2_of(float x) { return ((__float_as_int(x) >> 23) & 0xff) - 127; }
__device__ __forceinline__ float pow2_neg(int e) { return __int_as_float((127 - e) << 23); }

using Tabs = TypedTables;

// Per-sample view: a plain batch is B rows of M codes sharing reg0; an uneven
// batch reads its sample and region descriptors.
struct View {
    const uint8_t* geno;
    uint64_t out;
    uint64_t sid;
    uint32_t m0, len;
    TypedRegion r;
};

__device__ __forceinline__ View view_of(const TypedArgs& A, uint32_t s) {
    View v;
    if (A.samples) {
        const TypedSample d = A.samples[s];
        v.geno = A.geno + d.geno_off;
        v.out = d.out_off;
        v.sid = d.sample_id;
        v.m0 = d.m0;
        v.len = d.len;
        v.r = A.regions[d.region];
    } else {
        v.geno = A.geno + (uint64_t)s * A.M;
        v.out = (uint64_t)s * A.M;
        v.sid = A.sid_base + s;
        v.m0 = 0;
        v.len = A.M;
        v.r = A.reg0;
    }
    return v;
}

__device__ __forceinline__ uint32_t lmask_of(uint32_t L) { return L >= 32 ? 0xffffffffu : ((1u << L) - 1u); }

// {Q[n], S[n]}: table entry, or the closed form past the table
__device__ __forceinline__ float2 tabQS(const Tabs& t, uint32_t n) {
    if (n < t.NT) return __ldg(t.QS + n);
    const float qn = exp2f((float)n * t.log2q);
    return make_float2(qn, (1.0f - qn) * t.invL);
}
__device__ __forceinline__ double tabG(const Tabs& t, uint32_t n) {
    if (n < t.NT) return __ldg(t.G + n);
    if (t.regime == 0) return -(double)n * t.lr + log1p(-exp((double)n * t.lr)) - t.lgc;
    if (t.regime == 1) return log(-expm1(-(double)n * t.lr)) - t.lgc;
    return log((double)n);
}

// asynchronous global -> shared copies (cp.async); a thread waits for its own copies
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ---------------------------------------------------------------- anchor lists

constexpr uint32_t kWarpsPerBlock = 8;

// Rows of codes are read in 16-byte chunks on absolute 16-byte boundaries, so a
// row may start anywhere: with a = address % 16, chunk u (a multiple of 16)
// holds the codes u - a .. u - a + 15 of the row. Codes outside the row read
// as missing; nothing outside it is read.
__device__ __forceinline__ uint32_t row_shift(const uint8_t* g) { return (uint32_t)(reinterpret_cast<uintptr_t>(g) & 15u); }
__device__ __noinline__ uint4 row_edge(const uint8_t* g, uint32_t a, uint32_t u, uint32_t len) {
    uint32_t w[4] = {0x03030303u, 0x03030303u, 0x03030303u, 0x03030303u};
    if (u < len + a) {  // the row's first or last chunk
#pragma unroll
        for (uint32_t j = 0; j < 16; ++j)  // unrolled: the word index is a constant, w stays in registers
            if (u + j >= a && u + j - a < len)
                w[j >> 2] = (w[j >> 2] & ~(0xffu << (8 * (j & 3)))) | ((uint32_t)__ldg(g + (u + j - a)) << (8 * (j & 3)));
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ uint4 row_chunk(const uint8_t* g, uint32_t a, uint32_t u, uint32_t len) {
    if (u >= a && u - a + 16 <= len) return __ldg(reinterpret_cast<const uint4*>(g + (u - a)));
    return row_edge(g, a, u, len);
}

// bit 7 of each byte set where the code is below 3 (typed)
__device__ __forceinline__ uint32_t typed_bytes(uint32_t w) {
    return ~(((w | 0x80808080u) - 0x03030303u) | w) & 0x80808080u;
}

// bit j set when code j of the chunk is typed
__device__ __forceinline__ uint32_t typed_bits(uint4 c) {
    const uint32_t lo = __dp4a(typed_bytes(c.x) >> 7, 0x08040201u, __dp4a(typed_bytes(c.y) >> 7, 0x80402010u, 0u));
    const uint32_t hi = __dp4a(typed_bytes(c.z) >> 7, 0x08040201u, __dp4a(typed_bytes(c.w) >> 7, 0x80402010u, 0u));
    return lo | (hi << 8);
}

// Anchor counts per segment of kFillSeg markers from a chunk boundary (segment j
// of a row holds its codes j kFillSeg - a .. (j + 1) kFillSeg - a - 1, the last
// one the rest): a warp per (sample, segment), its eight 512-byte loads in flight
// together. Bound by reading the codes: 4,000 x 50,000 in 34 us, 5.9 TB/s (a copy,
// which also writes, measures 6.45); a warp per sample with one load ahead took 65.
__global__ void __launch_bounds__(32 * kWarpsPerBlock) anchor_count_kernel(TypedArgs A) {
    const unsigned long long gw = (unsigned long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t s = (uint32_t)(gw / A.nseg), seg = (uint32_t)(gw % A.nseg);
    if (s >= A.B) return;
    const View v = view_of(A, s);
    const uint32_t a = row_shift(v.geno);
    const uint32_t u0 = seg * kFillSeg;
    uint32_t n = 0;
    constexpr uint32_t kIt = kFillSeg / 512;
    uint4 c[kIt];
    if (u0 >= a && u0 + kFillSeg - a <= v.len) {  // the whole segment lies inside the row
        const uint4* p = reinterpret_cast<const uint4*>(v.geno + (u0 - a)) + lane;
#pragma unroll
        for (uint32_t i = 0; i < kIt; ++i) c[i] = __ldg(p + 32 * i);
    } else {
#pragma unroll
        for (uint32_t i = 0; i < kIt; ++i) c[i] = row_chunk(v.geno, a, u0 + 512 * i + 16 * lane, v.len);
    }
#pragma unroll
    for (uint32_t i = 0; i < kIt; ++i)
        n += __popc(typed_bytes(c[i].x) | (typed_bytes(c[i].y) >> 1) | (typed_bytes(c[i].z) >> 2) | (typed_bytes(c[i].w) >> 3));
    if (seg + 1 == A.nseg && lane == 0)  // at most 15 codes past the last segment's chunks
        n += __popc(typed_bits(row_chunk(v.geno, a, u0 + kFillSeg, v.len)));
    if (seg == 0 && lane == 0 && v.geno[0] >= 3) ++n;  // marker 0 is always an anchor
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0) A.segc[(size_t)seg * A.B + s] = n;
}

// The most anchors of any sample of group g, by one warp (lane = sample).
__device__ __forceinline__ uint32_t group_most(const uint32_t* __restrict__ segc, uint32_t nseg, uint32_t B, uint32_t g) {
    const uint32_t s = g * 32 + (threadIdx.x & 31);
    uint32_t x = 0;
    if (s < B) {
#pragma unroll 8
        for (uint32_t j = 0; j < nseg; ++j) x += __ldg(segc + (size_t)j * B + s);
    }
    return __reduce_max_sync(0xffffffffu, x);
}

__global__ void __launch_bounds__(128) anchor_group_kernel(const uint32_t* __restrict__ segc, uint32_t nseg, uint32_t B,
                                                           unsigned long long* __restrict__ aoff) {
    const uint32_t g = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (g >= (B + 31) / 32) return;  // whole warp
    const uint32_t x = group_most(segc, nseg, B, g);
    if ((threadIdx.x & 31) == 0) aoff[g] = x;
}

// Exclusive scans over the 32-sample groups of the interleaved lists, in one
// CTA: a group takes 32 x its most anchors and 32 x its most windows
// (ceil(count / C)). The groups' most anchors are summed up here, or stand in
// aoff (kGroups false) when anchor_group_kernel ran before: one SM reads the
// counts of more than kScanGroups groups slower than a second launch costs
// (313 groups x 13 segments: 43 us in one launch, 6 + 6 in two).
// Entry G holds the totals, also written with the most windows of any sample to
// host_totals[0..2] (mapped pinned host memory) when given: a copy would queue
// behind other device-to-host copies on the copy engine.
constexpr uint32_t kScanGroups = 64;
template <bool kGroups>
__global__ void __launch_bounds__(1024) anchor_scan_kernel(const uint32_t* __restrict__ segc, uint32_t nseg, uint32_t B,
                                                           uint32_t C, unsigned long long* __restrict__ aoff,
                                                           unsigned long long* __restrict__ woff,
                                                           unsigned long long* __restrict__ host_totals) {
    __shared__ unsigned long long sa[32], sw[32];
    __shared__ uint32_t smax[32];
    const uint32_t t = threadIdx.x, T = blockDim.x, lane = t & 31, warp = t >> 5;
    const uint32_t G = (B + 31) / 32;
    const uint32_t per = (G + T - 1) / T;
    const uint32_t g0 = min(G, t * per), g1 = min(G, g0 + per);
    if (kGroups) {
        for (uint32_t g = warp; g < G; g += T >> 5) {
            const uint32_t x = group_most(segc, nseg, B, g);
            if (lane == 0) aoff[g] = x;  // until its offset replaces it
        }
        __syncthreads();
    }
    auto group_max = [&](uint32_t g) { return (uint32_t)aoff[g]; };
    unsigned long long la = 0, lw = 0;
    uint32_t mx = 0;
    for (uint32_t g = g0; g < g1; ++g) {
        const uint32_t x = group_max(g);
        la += 32ull * x;
        lw += 32ull * ((x + C - 1) / C);
        mx = max(mx, x);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) smax[warp] = mx;
    unsigned long long ia = la, iw = lw;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long ya = __shfl_up_sync(0xffffffffu, ia, o), yw = __shfl_up_sync(0xffffffffu, iw, o);
        if (lane >= (uint32_t)o) { ia += ya; iw += yw; }
    }
    if (lane == 31) { sa[warp] = ia; sw[warp] = iw; }
    __syncthreads();
    if (warp == 0) {
        unsigned long long xa = lane < (T >> 5) ? sa[lane] : 0, xw = lane < (T >> 5) ? sw[lane] : 0;
        unsigned long long pa = xa, pw = xw;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long ya = __shfl_up_sync(0xffffffffu, pa, o), yw = __shfl_up_sync(0xffffffffu, pw, o);
            if (lane >= (uint32_t)o) { pa += ya; pw += yw; }
        }
        sa[lane] = pa - xa;
        sw[lane] = pw - xw;
        smax[lane] = __reduce_max_sync(0xffffffffu, lane < (T >> 5) ? smax[lane] : 0u);
    }
    __syncthreads();
    unsigned long long ra = sa[warp] + ia - la, rw = sw[warp] + iw - lw;
    for (uint32_t g = g0; g < g1; ++g) {
        const uint32_t x = group_max(g);
        aoff[g] = ra;
        woff[g] = rw;
        ra += 32ull * x;
        rw += 32ull * ((x + C - 1) / C);
    }
    if (t == T - 1) {
        aoff[G] = ra;
        woff[G] = rw;
        if (host_totals) {  // mapped host memory: the host reads the totals without a copy
            host_totals[0] = ra;
            host_totals[1] = rw;
            host_totals[2] = (smax[0] + C - 1) / C;
            __threadfence_system();
        }
    }
}

// Anchor lists: marker position (with the "no slot matches" flag, which
// scales every slot by e^-999, counted in beta's unit, in bit 31) and emission
// mask over the slots, in marker order; marker 0 is always an anchor. A CTA
// fills one segment of the 32 samples of a group, 512 markers of every row at a
// time: a warp takes four rows, each lane 16 codes of one, and puts the typed
// ones (a warp scan gives their places) into the row's list in shared memory;
// then the warps write entry after entry of all 32 rows, lane = row, so lanes
// at the same entry (samples of one array) write whole 128-byte lines of the
// interleaved lists. The next 512 codes of the rows are on their way meanwhile.
// A row's first entry of the segment is the sum of its earlier segments' counts.
// A batch of few groups is split further, A.split CTAs a segment: each counts the
// part of the segment before its own again.
// Bound by instruction issue (finding and placing the typed codes, about 110
// warp instructions per 512): 10,000 x 50,000 codes with 2,942 typed in 231 us, of
// which reading them once would be 78. A warp per group that walked its rows lane
// by lane took 300 us, and four to ten times as long where rows start off 16-byte
// boundaries (single-byte loads): the lists of 2,003 x 30,011 took 403 us in all
// and take 93, those of 1,500 x 6,007 302 and 56, those of one target 87 and 40
// (most of it the host's wait for the totals).
constexpr uint32_t kFillChunk = 512;
constexpr uint32_t kFillWarps = 8;
constexpr uint32_t kFillStride = kFillChunk + 2;  // list stride (entries): an odd number of words, no bank conflicts

__global__ void __launch_bounds__(32 * kFillWarps, 4) anchor_fill_kernel(TypedArgs A) {
    __shared__ uint16_t list[32][kFillStride];  // position in the chunk | code << 9
    __shared__ uint32_t cnt[32], part[kFillWarps][32];
    __shared__ uint4 rowd[32];  // {ptr lo, ptr hi, len, -}
    constexpr uint32_t kRows = 32 / kFillWarps;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t G = (A.B + 31) / 32;
    const uint32_t g = blockIdx.x % G, seg = blockIdx.x / G / A.split, sub = blockIdx.x / G % A.split;
    const uint32_t s = g * 32 + lane;  // lane = row
    View v{};
    uint32_t lim = 0;
    if (s < A.B) {
        v = view_of(A, s);
        lim = A.cap ? A.cap[s] : 0xffffffffu;
        uint32_t sum = 0;
        for (uint32_t j = warp; j < seg; j += kFillWarps) sum += A.segc[(size_t)j * A.B + s];
        part[warp][lane] = sum;
    }
    const uint32_t a = row_shift(v.geno);
    if (warp == 0) {
        const unsigned long long gp = reinterpret_cast<unsigned long long>(v.geno);
        rowd[lane] = make_uint4((uint32_t)gp, (uint32_t)(gp >> 32), s < A.B ? v.len : 0u, 0u);
    }
    __syncthreads();
    uint32_t at = 0;
    if (s < A.B) {
#pragma unroll
        for (uint32_t w = 0; w < kFillWarps; ++w) at += part[w][lane];
        if (warp == 0 && seg + 1 == A.nseg && sub == 0) {
            const uint32_t n = at + A.segc[(size_t)seg * A.B + s];
            if (n > lim) atomicOr(A.err, 1u);  // the job is cut to its capacity; the host reports it
            A.counts[s] = min(n, lim);
        }
    }
    const uint32_t ulast = __reduce_max_sync(0xffffffffu, s < A.B ? v.len + a : 0u);
    const uint32_t us = seg * kFillSeg, u0 = us + sub * (kFillSeg / A.split);
    const bool tail = seg + 1 == A.nseg && sub + 1 == A.split;
    const uint32_t u1 = tail ? ulast : min(u0 + kFillSeg / A.split, ulast);
    if (u0 >= u1) return;  // whole CTA: no row reaches this part
    const uint32_t lmask = lmask_of(v.r.L);
    const unsigned long long lb = A.aoff[g] + lane;
    const uint8_t* rp[kRows];
    uint32_t rl[kRows];
#pragma unroll
    for (uint32_t i = 0; i < kRows; ++i) {
        const uint4 d = rowd[warp * kRows + i];
        rp[i] = reinterpret_cast<const uint8_t*>(((unsigned long long)d.y << 32) | d.x);
        rl[i] = d.z;
    }
    uint4 cur[kRows];
    auto load = [&](uint32_t c0) {
#pragma unroll
        for (uint32_t i = 0; i < kRows; ++i) cur[i] = row_chunk(rp[i], row_shift(rp[i]), c0 + 16 * lane, rl[i]);
    };
    load(u0);
    if (sub) {  // the segment's markers before u0
#pragma unroll
        for (uint32_t i = 0; i < kRows; ++i) {
            uint32_t n = 0;
#pragma unroll 4
            for (uint32_t u = us + 16 * lane; u < u0; u += kFillChunk)
                n += __popc(typed_bits(row_chunk(rp[i], row_shift(rp[i]), u, rl[i])));
            if (us + lane == 0 && rl[i] && rp[i][0] >= 3) ++n;
            n = __reduce_add_sync(0xffffffffu, n);
            if (lane == 0) cnt[warp * kRows + i] = n;
        }
        __syncthreads();
        at += cnt[lane];
        __syncthreads();
    }
    for (uint32_t c0 = u0; c0 < u1; c0 += kFillChunk) {
        uint32_t bits[kRows], incl[kRows / 2];  // counts of two rows share a word (a chunk has at most 512)
#pragma unroll
        for (uint32_t i = 0; i < kRows; ++i) {
            bits[i] = typed_bits(cur[i]);
            if (c0 + lane == 0 && rl[i]) bits[i] |= 1u << row_shift(rp[i]);  // marker 0
        }
#pragma unroll
        for (uint32_t i = 0; i < kRows / 2; ++i) incl[i] = __popc(bits[2 * i]) | __popc(bits[2 * i + 1]) << 16;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
            for (uint32_t i = 0; i < kRows / 2; ++i) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl[i], o);
                if (lane >= (uint32_t)o) incl[i] += y;
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < kRows; ++i) {
            const uint4 x = cur[i];
            const uint32_t end = i & 1 ? incl[i / 2] >> 16 : incl[i / 2] & 0xffffu;
            if (lane == 31) cnt[warp * kRows + i] = end;
            uint16_t* to = &list[warp * kRows + i][end - __popc(bits[i])];
            for (uint32_t b = bits[i]; b; b &= b - 1) {
                const uint32_t j = __ffs(b) - 1;
                const uint32_t w = j < 8 ? (j < 4 ? x.x : x.y) : (j < 12 ? x.z : x.w);
                const uint32_t code = min((w >> (8 * (j & 3))) & 0xffu, 3u);
                *to++ = (uint16_t)(16 * lane + j | code << 9);
            }
        }
        if (c0 + kFillChunk < u1) load(c0 + kFillChunk);
        __syncthreads();
        const uint32_t n = cnt[lane], most = __reduce_max_sync(0xffffffffu, n);
#pragma unroll 2
        for (uint32_t k = warp; k < most; k += kFillWarps) {
            if (k < n && at + k < lim) {
                const uint32_t e = list[lane][k];
                const uint32_t m = c0 + (e & 511u) - a;
                uint32_t sh;
                const uint32_t em = emission_mask(e >> 9, v.r.masks[m], lmask, &sh);
                A.apos[lb + 32ull * (at + k)] = m | (sh ? kShiftBit : 0u);
                A.aem[lb + 32ull * (at + k)] = em;
            }
        }
        at += n;
        __syncthreads();  // the lists are read before they are refilled
    }
}

// ---------------------------------------------------------------- chain

template <int LM>
__device__ __forceinline__ float vsum(const float (&v)[LM]) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < LM; ++k) s += v[k];
    return s;
}

// Exact int -> double on the FP64 pipe: 2^52 + 2^31 + x has x + 2^31 in its
// low word, so one subtraction recovers x (a conversion instruction would use
// the special-function pipe, which the backward chain otherwise saturates).
__device__ __forceinline__ double i2d(int x) {
    return __hiloint2double(0x43300000, (int)((uint32_t)x ^ 0x80000000u)) - 4503601774854144.0;  // 2^52 + 2^31
}
__device__ __forceinline__ double u2d(uint32_t x) { return __hiloint2double(0x43300000, (int)x) - 4503599627370496.0; }

// sum over slot pairs, as a tree
template <uint32_t H>
__device__ __forceinline__ float vsum2(const float2 (&v)[H]) {
    float2 t[H];
#pragma unroll
    for (uint32_t h = 0; h < H; ++h) t[h] = v[h];
#pragma unroll
    for (uint32_t w = H / 2; w >= 1; w >>= 1)
#pragma unroll
        for (uint32_t h = 0; h < w; ++h) t[h] = __fadd2_rn(t[h], t[h + w]);
    return t[0].x + t[0].y;
}

// beta anchor at the last anchor (marker p): beta_{M-1} = 1, n = M-1-p untyped
// steps give the uniform value rho^n + e^-999 sum_{i<n} rho^i.
__device__ __forceinline__ double chain_end_logU(const Tabs& tb, uint32_t n) {
    if (n == 0) return 0.0;
    const double f = -999.0 + tabG(tb, n);
    return (double)n * tb.lr + (f > 30.0 ? f + log1p(exp(-f)) : log1p(exp(f)));
}

// One backward step of a window's rebuild over a run of n markers to the anchor
// with emission em (sh: no slot matches its call). The floor's log in units of
// U: fterm > 0, the floor dominates and the unit becomes U rho^n e^fterm;
// fterm <= -104, it is negligible. No branch: a warp's lanes differ in this.
template <int LM>
__device__ __forceinline__ void backward_step(const Tabs& tb, uint32_t n, float (&w)[LM], double& logU, uint32_t em,
                                              uint32_t sh) {
    const float2 qs = tabQS(tb, n);
    const float sw = vsum<LM>(w);
    const double fterm = -999.0 - logU + tabG(tb, n);
    const bool big = fterm > 0.0;
    const float ft = (float)fterm;
    const float ex = expf(big ? -fminf(ft, 100.f) : ft);
    const float xs = big ? ex : 1.f;                          // scale of the carried terms
    const float F = big ? 1.f : (fterm > -104.0 ? ex : 0.f);  // the floor term
    const float base = fmaf(xs * sw, qs.y, F);
    const float g = xs * qs.x;
#pragma unroll
    for (int k = 0; k < LM; ++k) w[k] = ((em >> k) & 1u) ? fmaf(g, w[k], base) : 0.f;
    const double dn = u2d(n);
    logU = big ? logU + fma(dn, tb.lr, fterm) : fma(dn, tb.lr, logU);
    logU -= sh ? 999.0 : 0.0;
    const float s = vsum<LM>(w);
    const int e = exp2_of(s);
    const float sc = pow2_neg(e);
#pragma unroll
    for (int k = 0; k < LM; ++k) w[k] *= sc;
    logU = fma(i2d(e), 0.69314718055994530942, logU);
}

template <int LM>
__device__ __forceinline__ void init_forward(float (&a)[LM], uint32_t em) {
#pragma unroll
    for (int k = 0; k < LM; ++k) a[k] = ((em >> k) & 1u) ? 1.f : 0.f;
}

// Steps per staged block: two blocks of a direction's records stay under 48 KB
// of shared memory, five CTAs an SM.
__host__ __device__ constexpr uint32_t chain_block(uint32_t LM) { return LM <= 8 ? 8u : 4u; }
constexpr uint32_t kChainPrep = 2;                            // warps that prepare a chain warp's steps
constexpr uint32_t kChainThreads = 32 * (1 + kChainPrep);
constexpr uint32_t kChainAhead = 3;                           // blocks of list entries in flight before the one prepared

// What a chain's step needs beyond its state, per lane: the emission over the
// slots as 0/1 factors, the run's {Q, S} and, backward, G(n) - 999 (the floor's
// log before the unit) and the unit's change n log rho - 999 shift.
template <int LM>
struct ChainStage {
    float4 mask[chain_block(LM)][LM / 4][32];
    float2 qs[chain_block(LM)][32];
    double g[chain_block(LM)][32];
    double c[chain_block(LM)][32];
};

// One chain per lane with all LM slots in registers; a CTA runs the forward
// (even blocks) or the backward (odd blocks) chains of a group of 32 samples,
// warp 0 the recursion, all lanes at the same anchor in a step.
// Bound: the dependent recursion, one warp's steps one after the other, so each
// instruction of that warp counts and it must not wait for memory. The CTA's
// other warps therefore prepare the steps: list entries come by cp.async blocks
// ahead, a block's table entries together, and finished records stand in shared
// memory (two blocks, one barrier a block). A step is then the masked slot
// update (an emission bit is a factor 0 or 1, exact), the sum over the slots and
// the power-of-two rescale and, backward, the unit's log and the floor, without
// a branch.
// A forward chain past its last anchor, and a backward chain before its first,
// step over records that mean nothing: nothing of theirs is stored, and a
// backward chain sets its state when its first anchor comes. Checkpoints:
// backward vector and the log of its unit at anchors k % C == 0 (window
// starts); forward vector at anchors k % (K C) == 0.
// Measured against one warp that loaded, looked up and stepped by itself (launch,
// CUDA events): 10,000 targets x 2,942 anchors, L = 8: 0.95 -> 0.59 ms; 2,003 x
// 1,876: 0.58 -> 0.27; one target of 329: 0.101 -> 0.055; 4,000 x 1,000 at L = 16:
// 0.39 -> 0.17; 1,500 x 601 at L = 32: 0.29 -> 0.19. A backward step alone takes
// 215 cycles (most of it the floor: FP64 difference, conversion, expf), a forward
// one 130. Not kept: one preparing warp (it set the pace: 0.96 ms), table entries
// by cp.async one by one (the same), factors looked up by the chain warp at L >= 16
// (0.19 and 0.22 ms), four preparing warps at L = 32 (0.20).
template <int LM>
__global__ void __launch_bounds__(kChainThreads, LM <= 16 ? 5 : 3) anchor_chain_kernel(TypedArgs A) {
    constexpr uint32_t KB = chain_block(LM), H = LM / 2, Q4 = LM / 4;
    __shared__ __align__(16) ChainStage<LM> stage[2];
    __shared__ __align__(16) uint32_t rpos[kChainAhead + 2][KB][32], rem[kChainAhead + 2][KB][32];  // list entries
    __shared__ float4 nibble[16];  // four emission bits as factors
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool forward = (blockIdx.x & 1u) == 0;
    const uint32_t s = (blockIdx.x >> 1) * 32 + lane;
    const bool live = s < A.B;
    // A lane past the batch's end takes the last sample's tables (gap 0 is in every
    // table; past an empty table each lookup would evaluate the FP64 closed form).
    const View v = view_of(A, live ? s : A.B - 1);
    uint32_t NA = 0;
    unsigned long long base = 0, wb = 0;
    if (live) {
        base = A.aoff[s >> 5];
        wb = A.woff[s >> 5] + lane;
        NA = A.counts[s];
    }
    const uint32_t NAw = __reduce_max_sync(0xffffffffu, NA);
    if (NAw == 0) return;  // every warp of the CTA
    const Tabs& tb = v.r.tabs;
    // Block b holds anchors [b KB, b KB + KB) of the group's lists. A forward chain steps
    // over anchors 1, 2, ... in blocks 0, 1, ...; a backward chain over NAw - 2, ... , 0
    // in blocks NB - 1, NB - 2, ... . Iteration i takes block blk(i).
    const uint32_t NB = (NAw + KB - 1) / KB;
    auto blk = [&](uint32_t i) { return forward ? i : NB - 1 - i; };
    if (threadIdx.x < 16)
        nibble[threadIdx.x] = make_float4(threadIdx.x & 1u ? 1.f : 0.f, threadIdx.x & 2u ? 1.f : 0.f,
                                          threadIdx.x & 4u ? 1.f : 0.f, threadIdx.x & 8u ? 1.f : 0.f);

    if (warp > 0) {
        const uint32_t* apos = A.apos + __shfl_sync(0xffffffffu, base, 0);  // the group's lists
        const uint32_t* aem = A.aem + __shfl_sync(0xffffffffu, base, 0);
        const uint32_t pt = threadIdx.x - 32;
        // block of iteration i: KB x 128 contiguous bytes of positions and of emissions
        auto fetch = [&](uint32_t i) {
            if (i < NB) {
                const uint32_t slot = i % (kChainAhead + 2), k0 = blk(i) * KB;
                for (uint32_t x = pt; x < KB * 8; x += 32 * kChainPrep)
                    if (k0 + x / 8 < NAw) {
                        cp_async16(&rpos[slot][0][0] + 4 * x, apos + 32ull * k0 + 4 * x);
                        cp_async16(&rem[slot][0][0] + 4 * x, aem + 32ull * k0 + 4 * x);
                    }
            }
            cp_async_commit();
        };
        // records of iteration i; a record's run lies between its anchor and the one before
        // it in list order (forward) or after it (backward), perhaps in a neighbour block
        auto prepare = [&](uint32_t i) {
            const uint32_t slot = i % (kChainAhead + 2), k0 = blk(i) * KB;
            const uint32_t before = (i + kChainAhead + 1) % (kChainAhead + 2);  // slot of iteration i - 1
            ChainStage<LM>& S = stage[i & 1u];
            constexpr uint32_t JP = KB / kChainPrep;
            uint32_t n[JP], nt[JP], em[JP], sh[JP];
            float2 qs[JP];
            double g[JP];
            bool past = false;
#pragma unroll
            for (uint32_t jj = 0; jj < JP; ++jj) {
                const uint32_t j = (warp - 1) * JP + jj, k = k0 + j;
                const uint32_t pe = rpos[slot][j][lane];
                uint32_t po;  // the neighbour's position
                if (forward) po = j ? rpos[slot][j - 1][lane] : rpos[before][KB - 1][lane];
                else po = j + 1 < KB ? rpos[slot][j + 1][lane] : rpos[before][0][lane];
                const bool ok = forward ? (k >= 1 && k < NA) : k + 1 < NA;
                n[jj] = ok ? (forward ? pe - po : po - pe) & ~kShiftBit : 0u;
                sh[jj] = pe >> 31;
                em[jj] = rem[slot][j][lane];
                past |= n[jj] >= tb.NT;
                nt[jj] = min(n[jj], tb.NT - 1);
            }
#pragma unroll
            for (uint32_t jj = 0; jj < JP; ++jj) {  // the block's table entries in flight together
                qs[jj] = __ldg(tb.QS + nt[jj]);
                g[jj] = forward ? 0.0 : __ldg(tb.G + nt[jj]);
            }
            if (past) {  // runs longer than the tables
#pragma unroll
                for (uint32_t jj = 0; jj < JP; ++jj)
                    if (n[jj] >= tb.NT) {
                        qs[jj] = tabQS(tb, n[jj]);
                        g[jj] = tabG(tb, n[jj]);
                    }
            }
#pragma unroll
            for (uint32_t jj = 0; jj < JP; ++jj) {
                const uint32_t j = (warp - 1) * JP + jj;
                S.qs[j][lane] = qs[jj];
                if (!forward) {
                    S.g[j][lane] = g[jj] - 999.0;
                    S.c[j][lane] = fma(u2d(n[jj]), tb.lr, sh[jj] ? -999.0 : 0.0);
                }
#pragma unroll
                for (uint32_t q = 0; q < Q4; ++q) S.mask[j][q][lane] = nibble[(em[jj] >> (4 * q)) & 15u];
            }
        };
        for (uint32_t i = 0; i <= kChainAhead; ++i) fetch(i);
        cp_async_wait_group<kChainAhead - 1>();  // the entries of iterations 0 and 1 have landed
        __syncthreads();
        prepare(0);
        for (uint32_t i = 0; i < NB; ++i) {
            cp_async_wait_group<kChainAhead - 1>();
            __syncthreads();  // records i are ready, with the entries of i + 1; records i - 1 have been read
            fetch(i + 1 + kChainAhead);  // into the slot of iteration i - 1
            if (i + 1 < NB) prepare(i + 1);
        }
        return;
    }

    struct Rec {
        float4 m[Q4];
        float2 q;
    };
    auto read = [&](const ChainStage<LM>& S, uint32_t j) {
        Rec r;
        r.q = S.qs[j][lane];
#pragma unroll
        for (uint32_t i = 0; i < Q4; ++i) r.m[i] = S.mask[j][i][lane];
        return r;
    };
    auto store = [&](float* dst, const float2 (&x)[H]) {
#pragma unroll
        for (uint32_t q = 0; q < Q4; ++q)
            reinterpret_cast<float4*>(dst)[q] = make_float4(x[2 * q].x, x[2 * q].y, x[2 * q + 1].x, x[2 * q + 1].y);
    };
    // the sum of xn and the power-of-two rescale that brings it into [1, 2): x = xn 2^-e
    auto rescale = [&](float2 (&x)[H], const float2 (&xn)[H], float& sum, int& bits) {
        const float s2 = vsum2<H>(xn);
        bits = __float_as_int(s2) & 0x7f800000;
        const float sc = __int_as_float(0x7f000000 - bits);
        const float2 S2 = make_float2(sc, sc);
#pragma unroll
        for (uint32_t h = 0; h < H; ++h) x[h] = __fmul2_rn(xn[h], S2);
        sum = s2 * sc;
    };
    // a step's update of the slot pairs: factor m_l (0 or 1) times (g x_l + b), summed and rescaled
    auto update = [&](float2 (&x)[H], const float4 (&m)[Q4], float g, float b, float& sum, int& bits) {
        const float2 G2 = make_float2(g, g), B2 = make_float2(b, b);
        float2 xn[H];
#pragma unroll
        for (uint32_t q = 0; q < Q4; ++q) {
            const float2 m0 = make_float2(m[q].x, m[q].y), m1 = make_float2(m[q].z, m[q].w);
            xn[2 * q] = __ffma2_rn(__fmul2_rn(G2, m0), x[2 * q], __fmul2_rn(B2, m0));
            xn[2 * q + 1] = __ffma2_rn(__fmul2_rn(G2, m1), x[2 * q + 1], __fmul2_rn(B2, m1));
        }
        rescale(x, xn, sum, bits);
    };
    auto emission = [&](float2 (&xn)[H], uint32_t em) {
#pragma unroll
        for (uint32_t h = 0; h < H; ++h)
            xn[h] = make_float2((em >> (2 * h)) & 1u ? 1.f : 0.f, (em >> (2 * h + 1)) & 1u ? 1.f : 0.f);
    };
    float2 x[H];
    float sx = 0.f;
    __syncthreads();
    if (forward) {
        // anchor 0's emission over uniform slots, then per anchor the run from the one before and its emission
        const uint32_t KC = A.K * A.C;
        float* ck = A.ckptF + wb * LM;  // the next checkpoint: every K-th window's entry
        const size_t ckstep = (size_t)32 * A.K * LM;
        float2 xn[H];
        emission(xn, NA > 0 ? A.aem[base + lane] : 1u);
        int bits;
        rescale(x, xn, sx, bits);
        if (NA > 0) store(ck, x);
        uint32_t next = KC;  // its anchor
        for (uint32_t i = 0; i < NB; ++i) {
            __syncthreads();
            const ChainStage<LM>& S = stage[i & 1u];
            Rec r = read(S, 0);
#pragma unroll
            for (uint32_t j = 0; j < KB; ++j) {
                Rec rn = r;
                if (j + 1 < KB) rn = read(S, j + 1);
                const uint32_t k = i * KB + j;
                if (j || i) {  // anchor 0 is the start
                    update(x, r.m, r.q.x, sx * r.q.y, sx, bits);
                    if (k == next) {
                        ck += ckstep;
                        next += KC;
                        if (k < NA) store(ck, x);
                    }
                }
                r = rn;
            }
        }
    } else {
        const uint32_t C = A.C;
        double logU = 0.0, logU0 = 0.0;
        uint32_t em0 = 1u;
        if (NA > 0) {
            const uint32_t pl = A.apos[base + lane + 32ull * (NA - 1)];
            logU0 = chain_end_logU(tb, v.len - 1 - (pl & ~kShiftBit)) - ((pl & kShiftBit) ? 999.0 : 0.0);
            em0 = A.aem[base + lane + 32ull * (NA - 1)];
        }
        emission(x, em0);
        sx = vsum2<H>(x);
        uint32_t left = (NAw - 1) % C;  // anchors to the next checkpoint, a multiple of C
        float* ckB = A.ckptB + (wb + 32ull * ((NAw - 1) / C)) * LM;  // its entries
        double* ckU = A.ckptU + wb + 32ull * ((NAw - 1) / C);
        const uint32_t first = __reduce_min_sync(0xffffffffu, NA);
        for (uint32_t i = 0; i < NB; ++i) {
            __syncthreads();
            const ChainStage<LM>& S = stage[i & 1u];
            const uint32_t k0 = (NB - 1 - i) * KB;
            Rec r = read(S, KB - 1);
            double g = S.g[KB - 1][lane], c = S.c[KB - 1][lane];
            // kStart: a chain of the group starts in this block
            auto steps = [&](auto kStart) {
#pragma unroll
                for (uint32_t jj = 0; jj < KB; ++jj) {
                    const uint32_t j = KB - 1 - jj, k = k0 + j;
                    Rec rn = r;
                    double gn = g, cn = c;
                    if (j > 0) {
                        rn = read(S, j - 1);
                        gn = S.g[j - 1][lane];
                        cn = S.c[j - 1][lane];
                    }
                    if (!kStart || k < NAw) {
                        // the floor's log in units of U: fterm > 0, the floor dominates and the unit
                        // becomes U rho^n e^fterm; fterm <= -104, it is negligible
                        const double fterm = g - logU;
                        const bool big = fterm > 0.0;
                        const float ex = expf(-fminf(fabsf((float)fterm), 104.f));
                        const float xs = big ? ex : 1.f;                          // scale of the carried terms
                        const float F = big ? 1.f : (fterm > -104.0 ? ex : 0.f);  // the floor term
                        int bits;
                        update(x, r.m, xs * r.q.x, fmaf(xs * sx, r.q.y, F), sx, bits);
                        logU = fma(i2d((bits >> 23) - 127), 0.69314718055994530942, (big ? g : logU) + c);
                        if (kStart && k + 1 >= NA) {  // at or before the chain's last anchor: its start
                            emission(x, em0);
                            sx = vsum2<H>(x);
                            logU = logU0;
                        }
                        if (left == 0) {
                            if (!kStart || k < NA) {
                                store(ckB, x);
                                *ckU = logU;
                            }
                            left = C;
                            ckB -= 32 * LM;
                            ckU -= 32;
                        }
                        --left;
                    }
                    r = rn;
                    g = gn;
                    c = cn;
                }
            };
            if (k0 + KB >= first) steps(std::true_type{});
            else steps(std::false_type{});
        }
    }
}

// ---------------------------------------------------------------- posterior
//
// One warp per (32 samples, group of K consecutive windows of C anchors); lane
// = sample (the warp's samples are one group of the interleaved lists). A lane
// walks its sample's markers of the group in tiles of 32 absolute markers:
//   group start: alpha from the forward checkpoint at the group's first anchor
//     (the chain writes one every K windows), and the first window's
//     backward records;
//   at an anchor (a typed marker, or marker 0): alpha steps over the run from
//     the previous anchor and takes the anchor's emission; the run starting
//     there takes its backward record, and at a window's first anchor the
//     window's records are rebuilt from the window's end checkpoint;
//   every marker: p_l = (Q[i] a'_l + S[i]) (X w'_l + Y), dosage, pick and
//     P(hap=1), two markers of a run per step.
// The backward record of the run [pos[k], pos[k+1]) holds
//   w'     the backward vector of anchor k+1 (E . beta), divided by its sum;
//   farg'  -999 - logU - ln(sum w), the log of beta's e^-999 floor in units of
//          w': -inf when the floor is negligible over the whole run, and the
//          run is "uniform" (w' = 0, beta constant) for the chain's last run
//          or where the floor dominates everywhere;
//   the run's end (pos[k+1], or the slice length) and anchor k+1's emission
//          mask, so an anchor step reads nothing from global memory.
// A window's inputs (its list entries and end checkpoint) are copied into a
// per-lane staging area with cp.async while the previous window is walked.
// With a' and w' of unit sum, a cell i markers after pos[k] and j = pos[k+1]
// - m before the next anchor has alpha_l ~ Q[i] a'_l + S[i] and beta_l ~
// Q[j] w'_l + S[j] (+ floor). Outputs are staged in a per-warp tile [32
// samples][32 markers] in shared memory and leave as row segments of 32
// consecutive markers.
//
// Two walks. If every sample of the CTA has the same anchors in the group (an
// array's sites; the kernel looks, one load an anchor), all its lanes step
// through the same markers: control and addresses are the warp's, the CTA stages
// the markers' slot data and the head of the run tables in shared memory, a tile
// ahead, and the floor is one branch-free form for all lanes. Otherwise every
// lane walks by itself. The arithmetic of a cell is the same, bit for bit.
// Bound: instruction issue. A pair of cells takes about 140 warp instructions at
// L = 8 (24 f32x2 operations for the slots, 15 for the sums, 47 for the argmax,
// 20 for the floor), an anchor about 300. Launch times, one walk for all before
// -> now: 10,000 x 50,000 (L = 8) 4.06 -> 2.35 ms (writing its 3 GB would take
// 0.47); 2,003 x 30,011 0.76 -> 0.41; 4,000 x 20,000 (L = 16) 1.27 -> 0.63; 1,500
// x 6,007 (L = 32, alleles only) 0.22 -> 0.16; one target x 1,644 98 -> 21 us;
// 131 x 7,919 with sites of their own (each lane by itself) 1.24 -> 0.22 ms.

// high word of farg' for a uniform run and for a negligible floor
constexpr uint32_t kInfHi = 0x7ff00000u;
constexpr uint32_t kNegInfHi = 0xfff00000u;

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float ex2_ftz(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// three-input maximum (sm_100)
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

template <int LM>
__device__ __forceinline__ float vmax(const float (&p)[LM]) {
    float m = p[0];
#pragma unroll
    for (int l = 1; l + 1 < LM; l += 2) m = max3(m, p[l], p[l + 1]);
    if (LM % 2 == 0) m = fmaxf(m, p[LM - 1]);
    return m;
}


// Argmax picks of two cells: the first slot with p >= (1 - eps) max; the
// sign of p - thr marks the slots below the threshold.
template <int LM>
__device__ __forceinline__ void pick_pair(const float2 (&p2)[LM], float keep, uint32_t& k0, uint32_t& k1) {
    float px[LM], py[LM];
#pragma unroll
    for (int l = 0; l < LM; ++l) { px[l] = p2[l].x; py[l] = p2[l].y; }
    const float2 thr2 = __fmul2_rn(make_float2(vmax<LM>(px), vmax<LM>(py)), make_float2(-keep, -keep));
    uint32_t bx = 0u, by = 0u;  // bit LM-1-l: slot l below the threshold
#pragma unroll
    for (int l = 0; l < LM; ++l) {
        const float2 d = __fadd2_rn(p2[l], thr2);
        bx = __funnelshift_l(__float_as_uint(d.x), bx, 1);
        by = __funnelshift_l(__float_as_uint(d.y), by, 1);
    }
    constexpr uint32_t kTop = LM >= 32 ? 1u : 1u << (32 - LM);  // slot l's bit at 31 - l, the bits below clear
    k0 = (uint32_t)__clz(~bx * kTop);
    k1 = (uint32_t)__clz(~by * kTop);
}

// x >> k, 0 for k = 32 (no slot picked)
__device__ __forceinline__ uint32_t shr(uint32_t x, uint32_t k) { return __funnelshift_rc(x, 0u, k); }

// Shared memory of one warp: backward records [C][LM/4][32] float4 and
// [C][32] {farg' lo, farg' hi, run end, end emission}; the dosage tile [32][36] f32, the allele tile [64][36] u8
// (rows 2r and 2r + 1: the two haplotypes of lane r) and, for P(hap=1),
// [32][34] f32x2; the staging area of the next window: end checkpoint
// [LM/4][32] float4 and [32] f64, list entries [C+1][32] positions and
// [C+1][32] emission masks.
__host__ __device__ constexpr size_t post_warp_bytes(uint32_t LM, uint32_t C, bool hprob) {
    return (size_t)C * LM * 128 + (size_t)C * 512 + 32 * 36 * 4 + 64 * 36 + (hprob ? 32 * 34 * 8 : 0) +
           (size_t)LM * 128 + 256 + 2 * ((size_t)C + 1) * 128;
}

// In front of the warps' parts, when A.stage: the head of the run tables (up and
// dg, kPostTab entries), two tiles of slot data (32 markers' masks and, where
// dosage is written, weights), and what warp 0 walks.
constexpr uint32_t kPostTab = 64;
// 32 slots' weights would take a CTA an SM: they are read where they lie
__host__ __device__ constexpr bool post_stage_weights(uint32_t LM, bool dos) { return dos && LM <= 16; }
__host__ __device__ constexpr size_t post_cta_bytes(uint32_t LM, bool dos) {
    return kPostTab * 48 + 2 * (32 * sizeof(SlotMasks) + (post_stage_weights(LM, dos) ? 32 * (size_t)LM * 8 : 0)) + 32;
}

struct Staging {
    float4* B;    // [LM/4][32] backward checkpoint at the window's end
    double* U;    // [32] its unit's log
    uint32_t* P;  // [C+1][32] list positions (with the shift bit) of anchors wC .. wC + C
    uint32_t* E;  // [C+1][32] their emission masks
};

// Issue the copies of window w's inputs into the lane's staging column.
template <int LM>
__device__ __forceinline__ void stage_window(const TypedArgs& A, const uint32_t* apos, const uint32_t* aem,
                                             unsigned long long wb, uint32_t NA, uint32_t w, const Staging& st,
                                             uint32_t lane) {
    const uint32_t C = A.C, k0 = w * C, k1 = min(k0 + C, NA);
    const uint32_t* p = apos + 32ull * k0;
    const uint32_t* e0 = aem + 32ull * k0;
    uint32_t* sp = st.P + lane;
    uint32_t* se = st.E + lane;
    if (C == 2 && k1 < NA) {
#pragma unroll
        for (uint32_t n = 0; n < 3; ++n) {
            cp_async4(sp + 32 * n, p + 32 * n);
            cp_async4(se + 32 * n, e0 + 32 * n);
        }
    } else {
        for (uint32_t n = min(k1, NA - 1) - k0 + 1; n; --n, p += 32, e0 += 32, sp += 32, se += 32) {
            cp_async4(sp, p);
            cp_async4(se, e0);
        }
    }
    if (k1 < NA) {
        const unsigned long long e = wb + 32ull * (w + 1);
        const float4* src = reinterpret_cast<const float4*>(A.ckptB + e * LM);
#pragma unroll
        for (uint32_t q = 0; q < LM / 4; ++q) cp_async16(st.B + q * 32 + lane, src + q);
        cp_async8(st.U + lane, A.ckptU + e);
    }
    cp_async_commit();
}

// The backward record of a run of n markers from the vector bv of its end
// anchor (at position pk, emission em) and the log of that vector's unit.
template <int LM>
__device__ __forceinline__ void write_record(const Tabs& tb, uint32_t n, const float (&bv)[LM], double logU, uint32_t pk,
                                             uint32_t em, float4* recW, uint4* recF) {
    const float sw = vsum<LM>(bv);
    const double farg = -999.0 - logU;
    const double f = farg - (double)logf(sw);
    uint32_t lo = (uint32_t)__double2loint(f), hi = (uint32_t)__double2hiint(f);
    if (farg + __ldg(tb.G + 1) > 60.0) { lo = 0u; hi = kInfHi; }       // floor dominates: beta uniform
    if (farg + tabG(tb, n) < -104.0) { lo = 0u; hi = kNegInfHi; }      // floor negligible over the run
    const float inv = hi == kInfHi ? 0.f : rcp_approx(sw);
#pragma unroll
    for (uint32_t q = 0; q < LM / 4; ++q)
        recW[q * 32] = make_float4(bv[4 * q] * inv, bv[4 * q + 1] * inv, bv[4 * q + 2] * inv, bv[4 * q + 3] * inv);
    *recF = make_uint4(lo, hi, pk, em);
}

// Backward records of window w (anchors [wC, min(wC + C, NA))) of one sample,
// rebuilt from the staged end checkpoint, into the lane's column of recW/recF.
template <int LM>
__device__ __forceinline__ void rebuild_window(const TypedArgs& A, const Tabs& tb, uint32_t NA, uint32_t len,
                                               uint32_t w, const Staging& st, float4* recW, uint4* recF,
                                               uint32_t lane) {
    constexpr uint32_t Q4 = LM / 4;
    cp_async_wait_all();
    const uint32_t C = A.C;
    const uint32_t k0 = w * C, k1 = min(k0 + C, NA);
    const uint32_t* P = st.P + lane;  // entry k at 32 (k - k0)
    const uint32_t* E = st.E + lane;
    recW += lane;
    recF += lane;
    float bv[LM];
    double logU;
    if (k1 < NA) {
#pragma unroll
        for (uint32_t q = 0; q < Q4; ++q) {
            const float4 x = st.B[q * 32 + lane];
            bv[4 * q] = x.x; bv[4 * q + 1] = x.y; bv[4 * q + 2] = x.z; bv[4 * q + 3] = x.w;
        }
        logU = st.U[lane];
    }
    if (C == 2 && k1 < NA) {  // the default window, without loops
        const uint32_t pa = P[0], pb = P[32], pc = P[64] & ~kShiftBit, eb = E[32];
        const uint32_t qb = pb & ~kShiftBit;
        write_record<LM>(tb, pc - qb, bv, logU, pc, E[64], recW + Q4 * 32, recF + 32);
        backward_step<LM>(tb, pc - qb, bv, logU, eb, pb >> 31);
        write_record<LM>(tb, qb - (pa & ~kShiftBit), bv, logU, qb, eb, recW, recF);
        return;
    }
    uint32_t r = k1 - k0;  // records left
    if (k1 == NA) {
        // the chain's last run: beta is uniform there
        const uint32_t pl = P[32 * (r - 1)];
        logU = chain_end_logU(tb, len - 1 - (pl & ~kShiftBit)) - ((pl & kShiftBit) ? 999.0 : 0.0);
        init_forward<LM>(bv, E[32 * (r - 1)]);
        --r;
#pragma unroll
        for (uint32_t q = 0; q < Q4; ++q) recW[(r * Q4 + q) * 32] = make_float4(0.f, 0.f, 0.f, 0.f);
        recF[r * 32] = make_uint4(0u, kInfHi, len, 0u);
    }
    for (; r; --r) {
        const uint32_t pk = P[32 * r] & ~kShiftBit, pb = P[32 * (r - 1)];
        const uint32_t n = pk - (pb & ~kShiftBit);
        write_record<LM>(tb, n, bv, logU, pk, E[32 * r], recW + (r - 1) * Q4 * 32, recF + (r - 1) * 32);
        if (r > 1) backward_step<LM>(tb, n, bv, logU, E[32 * (r - 1)], pb >> 31);
    }
}

// Barrier of the CTA's first n threads (whole warps), and whether x holds in all of them.
__device__ __forceinline__ void cta_barrier(uint32_t n) { asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory"); }
__device__ __forceinline__ bool cta_all(bool x, uint32_t n) {
    uint32_t r;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.and.pred q, 1, %2, p;\n selp.u32 %0, 1, 0, q;\n}"
                 : "=r"(r)
                 : "r"((uint32_t)x), "r"(n)
                 : "memory");
    return r != 0;
}

// Whether every lane's sample has the lane 0 sample's region, length and anchor
// count, and its anchor positions from k0 to the group's end k1.
template <bool kPlain>
__device__ __forceinline__ bool lanes_in_step(const TypedArgs& A, const View& v, uint32_t NA, uint32_t len, bool live,
                                              const uint32_t* apos, uint32_t k0, uint32_t k1) {
    constexpr uint32_t kAll = 0xffffffffu;
    const uint32_t NA0 = __shfl_sync(kAll, NA, 0);
    bool same = live && NA == NA0;
    if (!kPlain) {
        auto equal = [&](unsigned long long x) { return x == __shfl_sync(kAll, x, 0); };
        same = equal(reinterpret_cast<unsigned long long>(v.r.masks)) && same;
        same = equal(reinterpret_cast<unsigned long long>(v.r.tabs.QS)) && same;
        same = equal((unsigned long long)len << 32 | v.r.L) && same;
    }
    if (!__all_sync(kAll, same)) return false;
    k0 = __shfl_sync(kAll, k0, 0);
    k1 = min(__shfl_sync(kAll, k1, 0), NA0 - 1);
    for (uint32_t k = k0; k <= k1; k += 8) {
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            const uint32_t p = apos[32ull * min(k + j, k1)];
            same = ((p ^ __shfl_sync(kAll, p, 0)) & ~kShiftBit) == 0u && same;
        }
        if (!__all_sync(kAll, same)) return false;
    }
    return true;
}

// Warps an SM over registers: at L = 16 a plain batch runs 3 CTAs at 168 registers faster than
// 2 (4,000 x 20,000: 668 -> 625 us; launch_post_v has the exception).
template <int LM, bool kPlain>
constexpr int kPostCtas = LM <= 8 ? (kPlain ? 4 : 3) : LM == 16 && kPlain ? 3 : 2;

// kFull: every sample of the launch uses all LM slots (no active-slot masking).
// kFast: argmax picks, no P(hap=1). kPlain: every sample covers the whole
// panel with the launch's one region (read from the kernel parameters).
// kDos: dosage written (false only with kFast, for calls that return the
// phased alleles alone: no dosage sums and no g2 loads).
// A lane takes two consecutive cells of a run per step (an even marker and
// the next one) with f32x2 arithmetic across the two cells; a run's odd first
// marker or last marker takes a step alone (the second half is discarded).
// Tiles are aligned to absolute 32-marker columns, so a tile every lane of a
// warp fills completely leaves as 128-bit row segments.
template <int LM, bool kFull, bool kFast, bool kPlain, bool kDos, int kCtas>
__global__ void __launch_bounds__(128, kCtas)
    anchor_posterior_kernel(const __grid_constant__ TypedArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr uint32_t Q4 = LM / 4;
    constexpr uint32_t kAll = 0xffffffffu;
    constexpr bool kBcast = LM <= 16;  // a', w' held as (x, x) pairs: no per-step pairing moves
    uint32_t lane;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));  // kept in a register, not read again at each use
    const uint32_t warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t C = A.C, K = A.K;
    unsigned char* wbase = smem + (A.stage ? post_cta_bytes(LM, kDos) : 0) + (size_t)warp * post_warp_bytes(LM, C, !kFast);
    float4* recW = reinterpret_cast<float4*>(wbase);                     // [C][Q4][32]
    uint4* recF = reinterpret_cast<uint4*>(recW + (size_t)C * Q4 * 32);  // [C][32]
    float* tD = reinterpret_cast<float*>(recF + (size_t)C * 32);         // [32][36]
    uint8_t* tH = reinterpret_cast<uint8_t*>(tD + 32 * 36);              // [64][36]
    float2* tP = reinterpret_cast<float2*>(tH + 64 * 36);                // [32][34] (P(hap=1) only)
    Staging st;
    st.B = reinterpret_cast<float4*>(reinterpret_cast<unsigned char*>(tP) + (kFast ? 0 : 32 * 34 * 8));
    st.U = reinterpret_cast<double*>(st.B + Q4 * 32);
    st.P = reinterpret_cast<uint32_t*>(st.U + 32);
    st.E = st.P + (C + 1) * 32;

    // a warp takes A.rows samples (a divisor of 32): SW warps and SC CTAs of one window group
    const uint32_t SW = (A.B + A.rows - 1) / A.rows, SC = (SW + nw - 1) / nw;
    // A.parts warps share a window group's windows; each carries alpha from the group's first anchor
    const uint32_t Kp = K / A.parts;
    const unsigned long long grp = blockIdx.x / SC / A.parts;
    const unsigned long long first = grp * K + blockIdx.x / SC % A.parts * Kp;  // its first window
    const uint32_t w0cta = blockIdx.x % SC * nw;
    const uint32_t cta_threads = 32 * min(nw, SW - w0cta);  // the warps with samples
    if (w0cta + warp >= SW) return;  // whole warp
    const uint32_t row0 = (w0cta + warp) * A.rows, g = row0 / 32;
    // a lane past the warp's samples or the batch's end repeats one of them, and writes nothing
    const bool real = lane < A.rows && row0 + lane < A.B;
    const uint32_t s = min(row0 + (lane & (A.rows - 1)), A.B - 1);
    bool live = first < A.max_windows;
    View v{};
    if (!kPlain) v = view_of(A, s);
    const uint32_t NA = A.counts[s];
    const unsigned long long ab = A.aoff[g] + (s & 31u), wb = A.woff[g] + (s & 31u);
    const uint32_t NW = (NA + C - 1) / C;
    const uint32_t w0 = live ? (uint32_t)first : 0u;
    const uint32_t wend = min(w0 + Kp, NW);
    live = live && w0 < wend;
    const bool warp_live = __any_sync(kAll, live);
    if (!A.stage && !warp_live) return;  // whole warp

    const TypedRegion& R = kPlain ? A.reg0 : v.r;
    const uint32_t len = kPlain ? A.M : v.len;
    const unsigned long long out = kPlain ? (unsigned long long)s * A.M : v.out;
    const Tabs& tb = R.tabs;
    const uint32_t Lr = R.L;
    const uint32_t* apos = A.apos + ab;  // entry k at [32 k]
    const uint32_t* aem = A.aem + ab;
    const bool w_dos = kDos && A.dosage != nullptr, w_hap = A.haps != nullptr;
    const bool w_hp = !kFast && A.hprob != nullptr;
    const bool argmax = kFast || A.sampling == SI_SAMPLE_ARGMAX;
    const float keep = 1.0f - A.tie_eps;

    float2 a2[kBcast ? LM : 1], w2[kBcast ? LM : 1];  // (a'_l, a'_l), (w'_l, w'_l)
    float ap[kBcast ? 1 : LM], wp[kBcast ? 1 : LM];
#pragma unroll
    for (int l = 0; l < LM; ++l) {
        if constexpr (kBcast) { a2[l] = make_float2(0.f, 0.f); w2[l] = make_float2(0.f, 0.f); }
        else { ap[l] = 0.f; wp[l] = 0.f; }
    }
    auto A2 = [&](int l) { if constexpr (kBcast) return a2[l]; else return make_float2(ap[l], ap[l]); };
    auto W2 = [&](int l) { if constexpr (kBcast) return w2[l]; else return make_float2(wp[l], wp[l]); };
    auto a_of = [&](int l) { if constexpr (kBcast) return a2[l].x; else return ap[l]; };
    auto set_a = [&](int l, float x) { if constexpr (kBcast) a2[l] = make_float2(x, x); else ap[l] = x; };
    auto set_w = [&](int l, float x) { if constexpr (kBcast) w2[l] = make_float2(x, x); else wp[l] = x; };
    uint4 fr = make_uint4(0u, kNegInfHi, 0u, 0u);  // the current run's record: farg' lo, hi, end, end emission
    float2 FH = make_float2(0.f, 0.f), FL = make_float2(0.f, 0.f);  // a floor run's farg' as float hi + lo
    uint32_t p0 = 0, p1 = 0, m = 0, mend = 0;
    auto load_record = [&](uint32_t r) {
#pragma unroll
        for (uint32_t q = 0; q < Q4; ++q) {
            const float4 x = recW[(r * Q4 + q) * 32 + lane];
            set_w(4 * q, x.x); set_w(4 * q + 1, x.y); set_w(4 * q + 2, x.z); set_w(4 * q + 3, x.w);
        }
        fr = recF[r * 32 + lane];
        if ((fr.y & kInfHi) != kInfHi) {
            const double fa = __hiloint2double((int)fr.y, (int)fr.x);
            const float h = (float)fa, l = (float)(fa - (double)h);
            FH = make_float2(h, h);
            FL = make_float2(l, l);
        }
    };
    // alpha over a run ({Q, S} = qs) and the emission em of the anchor at its end
    auto alpha_step = [&](float2 qs, uint32_t em) {
        float x[LM];
#pragma unroll
        for (int l = 0; l < LM; ++l) x[l] = a_of(l);
        const float base = vsum<LM>(x) * qs.y;
#pragma unroll
        for (int l = 0; l < LM; ++l) x[l] = ((em >> l) & 1u) ? fmaf(qs.x, x[l], base) : 0.f;
        const float inv = rcp_approx(vsum<LM>(x));
#pragma unroll
        for (int l = 0; l < LM; ++l) set_a(l, x[l] * inv);
    };
    if (live) {
        stage_window<LM>(A, apos, aem, wb, NA, w0, st, lane);
        const float4* src = reinterpret_cast<const float4*>(A.ckptF + (wb + 32ull * grp * K) * LM);
        float x[LM];
#pragma unroll
        for (uint32_t q = 0; q < Q4; ++q) {
            const float4 y = src[q];
            x[4 * q] = y.x; x[4 * q + 1] = y.y; x[4 * q + 2] = y.z; x[4 * q + 3] = y.w;
        }
        const float inv = rcp_approx(vsum<LM>(x));
#pragma unroll
        for (int l = 0; l < LM; ++l) set_a(l, x[l] * inv);
        // alpha from the group's first anchor to this warp's
        const uint32_t ka = (uint32_t)grp * K * C, kb = w0 * C;
        uint32_t pa = apos[32ull * ka] & ~kShiftBit;
        for (uint32_t k = ka; k < kb; k += 4) {
            uint32_t pk[4], ek[4];
            float2 qk[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {  // four anchors' loads together
                const uint32_t kk = min(k + 1 + j, kb);
                pk[j] = apos[32ull * kk] & ~kShiftBit;
                ek[j] = aem[32ull * kk];
            }
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) qk[j] = tabQS(tb, pk[j] - (j ? pk[j - 1] : pa));
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
                if (k + 1 + j <= kb) alpha_step(qk[j], ek[j]);
            pa = pk[3];
        }
        p0 = pa;
        mend = wend * C < NA ? (apos[32ull * wend * C] & ~kShiftBit) : len;
        m = p0;
        rebuild_window<LM>(A, tb, NA, len, w0, st, recW, recF, lane);
        if (w0 + 1 < wend) stage_window<LM>(A, apos, aem, wb, NA, w0 + 1, st, lane);
        load_record(0);
        p1 = fr.z;
    }
    bool in_tab = p1 - p0 < tb.NT;  // every i, i+1, j, j-1 of the run index the pair tables

    const bool vec_ok = kPlain && (A.M & 3u) == 0 && !w_hp &&
                        (reinterpret_cast<uintptr_t>(A.dosage) & 15u) == 0 &&
                        (reinterpret_cast<uintptr_t>(A.haps) & 3u) == 0;
    // Write out the tile at absolute columns [tbase, tbase + 32): this lane
    // filled columns [tlo, thi).
    auto flush = [&](uint32_t tbase, uint32_t tlo, uint32_t thi, bool on) {
        __syncwarp();
        const bool has = on && real && thi > tlo;
        const uint32_t tb0 = __shfl_sync(kAll, tbase, 0);
        if (__all_sync(kAll, vec_ok && has && tlo == 0 && thi == 32 && tbase == tb0)) {
            // every lane filled the same whole tile: 128-bit rows of dosage, 32-bit rows of alleles
            const unsigned long long s0 = s - lane;
            const uint32_t r = lane >> 3, c = (lane & 7) * 4;  // four rows at a time
            if (w_dos) {
                float* to = A.dosage + (s0 + r) * A.M + tb0 + c;
                const float* from = tD + r * 36 + c;
#pragma unroll
                for (uint32_t it = 0; it < 8; ++it, to += 4ull * A.M)
                    *reinterpret_cast<float4*>(to) = *reinterpret_cast<const float4*>(from + it * 4 * 36);
            }
            if (w_hap) {  // rows 2 s, 2 s + 1 follow each other
                uint8_t* to = A.haps + (2 * s0 + r) * A.M + tb0 + c;
                const uint8_t* from = tH + r * 36 + c;
#pragma unroll
                for (uint32_t it = 0; it < 16; ++it, to += 4ull * A.M)
                    *reinterpret_cast<uint32_t*>(to) = *reinterpret_cast<const uint32_t*>(from + it * 4 * 36);
            }
        } else {
            for (uint32_t r = 0; r < 32; ++r) {
                if (!__shfl_sync(kAll, has, r)) continue;
                const unsigned long long ro = __shfl_sync(kAll, out, r);
                const uint32_t rl = __shfl_sync(kAll, len, r), at = __shfl_sync(kAll, tbase, r) + lane;
                const uint32_t lo = __shfl_sync(kAll, tlo, r), hi = __shfl_sync(kAll, thi, r);
                if (lane >= lo && lane < hi) {
                    if (w_dos) A.dosage[ro + at] = tD[r * 36 + lane];
                    if (w_hap) {
                        A.haps[2 * ro + at] = tH[(2 * r) * 36 + lane];
                        A.haps[2 * ro + rl + at] = tH[(2 * r + 1) * 36 + lane];
                    }
                    if (w_hp) reinterpret_cast<float2*>(A.hprob)[ro + at] = tP[r * 34 + lane];
                }
            }
        }
        __syncwarp();
    };

    // run coefficients of cells (mm, mm + 1): {Q_i, Q_i+1, S_i, S_i+1}, {Q_j, Q_j-1, S_j, S_j-1}
    auto coeffs = [&](uint32_t mm, float4& qa, float4& qb) {
        const uint32_t i = mm - p0, j = p1 - mm;
        if (in_tab) {
            qa = __ldg(tb.up + i);
            qb = __ldg(tb.dg + 2 * j);
        } else {
            const float2 x0 = tabQS(tb, i), x1 = tabQS(tb, i + 1), y0 = tabQS(tb, j), y1 = tabQS(tb, j - 1);
            qa = make_float4(x0.x, x1.x, x0.y, x1.y);
            qb = make_float4(y0.x, y1.x, y0.y, y1.y);
        }
    };

    // cells m (and m + 1 when two) of the current run, into tile columns c0 (, c0 + 1)
    auto cells = [&](uint32_t mm, bool two, const float4 qa, const float4 qb, uint32_t c0) {
        const uint32_t j = p1 - mm;
        float2 XX = make_float2(qb.x, qb.y), YY = make_float2(qb.z, qb.w);
        if (fr.y == kInfHi) {
            YY = make_float2(1.f, 1.f);  // uniform run: w' = 0, beta = 1
        } else if ((fr.y & kInfHi) != kInfHi) {
            // floor e^ft beside Q w' + S, ft = farg' + G(j); when it dominates (ft > 0) scale both by e^-ft
            float2 ft2;
            if (in_tab) {
                // (hi + hi) + (lo + lo) in FP32: where the floor is within reach of the carried
                // terms the high parts nearly cancel, and their sum is exact
                const float4 g = __ldg(tb.dg + 2 * j + 1);
                ft2 = __fadd2_rn(__fadd2_rn(FH, make_float2(g.x, g.y)), __fadd2_rn(FL, make_float2(g.z, g.w)));
            } else {
                const double fa = __hiloint2double((int)fr.y, (int)fr.x);
                ft2 = make_float2((float)(fa + tabG(tb, j)), (float)(fa + tabG(tb, j - 1)));
            }
            const float ft[2] = {ft2.x, ft2.y};
            float xx[2] = {XX.x, XX.y}, yy[2] = {YY.x, YY.y};
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const float e = exp2f(fminf(fabsf(ft[c]), 104.f) * -1.44269504088896341f);  // e^-|ft|
                const bool big = ft[c] > 0.f;
                const float xs = big ? e : 1.f;
                const float F = big ? 1.f : (ft[c] > -104.f ? e : 0.f);
                yy[c] = fmaf(yy[c], xs, F);
                xx[c] *= xs;
            }
            XX = make_float2(xx[0], xx[1]);
            YY = make_float2(yy[0], yy[1]);
        }
        const float2 QQ = make_float2(qa.x, qa.y), SS = make_float2(qa.z, qa.w);
        const SlotMasks mkA = R.masks[mm];
        const SlotMasks mkB = two ? R.masks[mm + 1] : mkA;
        const float4* g4 = reinterpret_cast<const float4*>(R.g2 + (size_t)mm * R.gs);
        float2 p2[LM];
#pragma unroll
        for (int l = 0; l < LM; ++l) {
            p2[l] = __fmul2_rn(__ffma2_rn(QQ, A2(l), SS), __ffma2_rn(XX, W2(l), YY));
            if (!kFull && (uint32_t)l >= Lr) p2[l] = make_float2(0.f, 0.f);
        }
        float2 t2[LM / 2];
#pragma unroll
        for (int l = 0; l < LM / 2; ++l) t2[l] = __fadd2_rn(p2[2 * l], p2[2 * l + 1]);
#pragma unroll
        for (int h = LM / 4; h >= 1; h >>= 1)
#pragma unroll
            for (int l = 0; l < h; ++l) t2[l] = __fadd2_rn(t2[l], t2[l + h]);
        const float2 tot2 = t2[0];
        float2 d2 = make_float2(0.f, 0.f);
#pragma unroll
        for (int q = 0; q < LM / 2; ++q) {
            if (kDos && (kFull || (uint32_t)(2 * q) < R.gs)) {
                const float4 gv = __ldg(g4 + q);
                d2 = __ffma2_rn(p2[2 * q], make_float2(gv.x, gv.y), d2);
                d2 = __ffma2_rn(p2[2 * q + 1], make_float2(gv.z, gv.w), d2);
            }
        }
        uint32_t pk[2];
        if (argmax) {
            pick_pair<LM>(p2, keep, pk[0], pk[1]);
        } else {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float pc[LM];
#pragma unroll
                for (int l = 0; l < LM; ++l) pc[l] = c ? p2[l].y : p2[l].x;
                const float tot = c ? tot2.y : tot2.x;
                const float target = cell_uniform(A.seed, kPlain ? A.sid_base + s : v.sid,
                                                  (kPlain ? 0u : v.m0) + mm + c) * tot;
                float cum = 0.f;
                uint32_t last_nz = 0, pick = LM;
#pragma unroll
                for (int l = 0; l < LM; ++l) {
                    cum += pc[l];
                    if (pc[l] > 0.f) last_nz = (uint32_t)l;
                    if (pick == LM && target < cum) pick = (uint32_t)l;
                }
                pk[c] = pick == LM ? last_nz : pick;
            }
        }
        const float2 inv2 = make_float2(rcp_approx(tot2.x), rcp_approx(tot2.y));
        const float2 dos2 = __fmul2_rn(d2, inv2);
        const uint32_t hA = slot_alleles(mkA, R.raw, R.gs, mm, pk[0]);
        if (two) {
            const uint32_t hB = slot_alleles(mkB, R.raw, R.gs, mm + 1, pk[1]);
            if constexpr (kDos) *reinterpret_cast<float2*>(tD + lane * 36 + c0) = dos2;
            *reinterpret_cast<uint16_t*>(tH + (2 * lane) * 36 + c0) = (uint16_t)((hA & 0xffu) | ((hB & 0xffu) << 8));
            *reinterpret_cast<uint16_t*>(tH + (2 * lane + 1) * 36 + c0) = (uint16_t)((hA >> 8) | (hB & 0xff00u));
            if (w_hp) {
                float q0[2] = {0.f, 0.f}, q1[2] = {0.f, 0.f};
#pragma unroll
                for (int l = 0; l < LM; ++l) {
                    q0[0] += ((mkA.a0 >> l) & 1u) ? p2[l].x : 0.f;
                    q1[0] += ((mkA.a1 >> l) & 1u) ? p2[l].x : 0.f;
                    q0[1] += ((mkB.a0 >> l) & 1u) ? p2[l].y : 0.f;
                    q1[1] += ((mkB.a1 >> l) & 1u) ? p2[l].y : 0.f;
                }
                *reinterpret_cast<float4*>(tP + lane * 34 + c0) =
                    make_float4(q0[0] * inv2.x, q1[0] * inv2.x, q0[1] * inv2.y, q1[1] * inv2.y);
            }
        } else {
            if constexpr (kDos) tD[lane * 36 + c0] = dos2.x;
            tH[(2 * lane) * 36 + c0] = (uint8_t)(hA & 0xffu);
            tH[(2 * lane + 1) * 36 + c0] = (uint8_t)(hA >> 8);
            if (w_hp) {
                float q0 = 0.f, q1 = 0.f;
#pragma unroll
                for (int l = 0; l < LM; ++l) {
                    q0 += ((mkA.a0 >> l) & 1u) ? p2[l].x : 0.f;
                    q1 += ((mkA.a1 >> l) & 1u) ? p2[l].x : 0.f;
                }
                tP[lane * 34 + c0] = make_float2(q0 * inv2.x, q1 * inv2.x);
            }
        }
    };

    // the next anchor: alpha steps over the current run and takes its emission, and the run starting
    // there becomes the current one
    uint32_t rec = 0, win = w0;  // the current run's record, its window
    auto anchor = [&](float2 qs) {
        const uint32_t em = fr.w;
        if (++rec == C) {
            rec = 0;
            ++win;
            rebuild_window<LM>(A, tb, NA, len, win, st, recW, recF, lane);
            if (win + 1 < wend) stage_window<LM>(A, apos, aem, wb, NA, win + 1, st, lane);
        }
        alpha_step(qs, em);
        load_record(rec);
    };

    // ---- lanes in step: every lane's sample has the same anchors (an array's sites). All control and
    // every address but the outputs' is then the warp's own, not a lane's.
    const bool in_step = warp_live && lanes_in_step<kPlain>(A, v, NA, len, live, apos, w0 * C, wend * C);
    // The warps of a CTA walk the same window group of neighbouring samples. If they are all in step, the CTA
    // keeps the markers' slot data and the head of the run tables in shared memory, a tile ahead: read from
    // global memory they missed L1 (28 KB beside this kernel's shared memory) two times out of three.
    bool staged = false;
    float4* sT = reinterpret_cast<float4*>(smem);                    // [kPostTab] up, [kPostTab][2] dg
    SlotMasks* sM = reinterpret_cast<SlotMasks*>(sT + 3 * kPostTab);  // [2][32]
    float4* sG = reinterpret_cast<float4*>(sM + 64);                 // [2][32][gs / 2]
    if (A.stage) {
        unsigned long long* what = reinterpret_cast<unsigned long long*>(smem + post_cta_bytes(LM, kDos) - 32);
        const unsigned long long mine[4] = {(unsigned long long)m << 32 | mend,
                                            reinterpret_cast<unsigned long long>(R.masks),
                                            reinterpret_cast<unsigned long long>(tb.QS), R.gs};
        if (threadIdx.x == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) what[i] = mine[i];
        }
        cta_barrier(cta_threads);
        bool same = in_step;
#pragma unroll
        for (int i = 0; i < 4; ++i) same = same && what[i] == mine[i];
        staged = cta_all(same, cta_threads);
        if (!warp_live) return;  // whole warp, of a CTA that does not stage
    }
    if (staged) {
        auto warp_value = [&](uint32_t x) { return __reduce_max_sync(kAll, x); };
        uint32_t um = warp_value(m), u0 = um, u1 = warp_value(p1);
        const uint32_t uend = warp_value(mend);
        const uint32_t rows = min(A.rows, A.B - row0);
        // the current run's floor on one form for every lane, so that a step needs no branch: -3e38
        // stands for a negligible floor (F = 0), 3e38 for a uniform run (X w' = 0 there, Y F + 1 = 1)
        auto one_form = [&] {
            if ((fr.y & kInfHi) == kInfHi) {
                const float h = fr.y == kInfHi ? 3e38f : -3e38f;
                FH = make_float2(h, h);
                FL = make_float2(0.f, 0.f);
            }
        };
        one_form();
        const float4* g2 = reinterpret_cast<const float4*>(R.g2);
        const uint32_t gq = kPlain ? LM / 2 : R.gs / 2;  // float4s of a marker's weights
        const bool has_raw = R.raw != nullptr;
        const SlotMasks* mrow = sM;  // the current tile's slot data
        const float4* grow = sG;
        float* const tDl = tD + lane * 36;
        uint8_t* const tHl = tH + 2 * lane * 36;
        auto stage_tile = [&](uint32_t t0, uint32_t b) {  // slot data of markers [t0, t0 + 32)
            if (t0 >= uend) return;
            const uint32_t nm = min(32u, len - t0);
            for (uint32_t x = threadIdx.x; x < nm; x += cta_threads) cp_async16(sM + 32 * b + x, R.masks + t0 + x);
            if constexpr (post_stage_weights(LM, kDos))
                for (uint32_t x = threadIdx.x; x < nm * gq; x += cta_threads)
                    cp_async16(sG + 32 * gq * b + x, g2 + (size_t)t0 * gq + x);
        };
        for (uint32_t x = threadIdx.x; x < 3 * kPostTab; x += cta_threads)
            cp_async16(sT + x, x < kPostTab ? tb.up + x : tb.dg + (x - kPostTab));
        stage_tile(um & ~31u, 0);
        // cells mm and mm + 1 (the second one discarded unless two) into columns c0, c0 + 1, from the run's
        // coefficients and the floor's log at them
        auto pair_at = [&](uint32_t mm, auto two, const float4 qa, const float4 qb, auto floor_log, uint32_t c0) {
            const SlotMasks mkA = mrow[c0];
            const SlotMasks mkB = two ? mrow[c0 + 1] : mkA;
            float2 XX = make_float2(qb.x, qb.y), YY = make_float2(qb.z, qb.w);
            // floor e^ft beside X w' + Y; when it dominates (ft > 0) both are scaled by e^-ft. e^-|ft| below the
            // smallest normal number reads 0: it is added to 1 or to Y >= 1e-30, which it would not change.
            const float2 ft = floor_log();
            const float e0 = ex2_ftz(fabsf(ft.x) * -1.44269504088896341f), e1 = ex2_ftz(fabsf(ft.y) * -1.44269504088896341f);
            const bool big0 = ft.x > 0.f, big1 = ft.y > 0.f;
            const float2 xs = make_float2(big0 ? e0 : 1.f, big1 ? e1 : 1.f);
            YY = __ffma2_rn(YY, xs, make_float2(big0 ? 1.f : e0, big1 ? 1.f : e1));
            XX = __fmul2_rn(XX, xs);
            const float2 QQ = make_float2(qa.x, qa.y), SS = make_float2(qa.z, qa.w);
            float2 p2[LM];
#pragma unroll
            for (int l = 0; l < LM; ++l) {
                p2[l] = __fmul2_rn(__ffma2_rn(QQ, A2(l), SS), __ffma2_rn(XX, W2(l), YY));
                if (!kFull && (uint32_t)l >= Lr) p2[l] = make_float2(0.f, 0.f);
            }
            float2 inv2 = make_float2(0.f, 0.f);
            float2 tot2 = inv2;
            if (kDos || !kFast) {
                float2 t2[LM / 2];
#pragma unroll
                for (int l = 0; l < LM / 2; ++l) t2[l] = __fadd2_rn(p2[2 * l], p2[2 * l + 1]);
#pragma unroll
                for (int h = LM / 4; h >= 1; h >>= 1)
#pragma unroll
                    for (int l = 0; l < h; ++l) t2[l] = __fadd2_rn(t2[l], t2[l + h]);
                tot2 = t2[0];
                inv2 = make_float2(rcp_approx(tot2.x), rcp_approx(tot2.y));
            }
            if constexpr (kDos) {
                float2 d2 = make_float2(0.f, 0.f);
#pragma unroll
                for (int q = 0; q < LM / 2; ++q) {
                    if (kFull || (uint32_t)(2 * q) < 2 * gq) {
                        float4 w;
                        if constexpr (post_stage_weights(LM, kDos)) w = grow[c0 * gq + q];
                        else w = __ldg(g2 + (size_t)mm * gq + q);
                        d2 = __ffma2_rn(p2[2 * q], make_float2(w.x, w.y), d2);
                        d2 = __ffma2_rn(p2[2 * q + 1], make_float2(w.z, w.w), d2);
                    }
                }
                const float2 dos2 = __fmul2_rn(d2, inv2);
                if (two) *reinterpret_cast<float2*>(tDl + c0) = dos2;
                else tDl[c0] = dos2.x;
            }
            uint32_t pk[2];
            if (argmax) {
                pick_pair<LM>(p2, keep, pk[0], pk[1]);
            } else {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const float target = cell_uniform(A.seed, kPlain ? A.sid_base + s : v.sid,
                                                      (kPlain ? 0u : v.m0) + mm + c) * (c ? tot2.y : tot2.x);
                    float cum = 0.f;
                    uint32_t last_nz = 0, pick = LM;
#pragma unroll
                    for (int l = 0; l < LM; ++l) {
                        const float pl = c ? p2[l].y : p2[l].x;
                        cum += pl;
                        if (pl > 0.f) last_nz = (uint32_t)l;
                        if (pick == LM && target < cum) pick = (uint32_t)l;
                    }
                    pk[c] = pick == LM ? last_nz : pick;
                }
            }
            // the picks' alleles: bytes {hap0 A, hap0 B, hap1 A, hap1 B}
            uint32_t hv;
            if (has_raw && (mkA.x | mkB.x) != 0u) {
                const uint32_t hA = slot_alleles(mkA, R.raw, R.gs, mm, pk[0]);
                const uint32_t hB = two ? slot_alleles(mkB, R.raw, R.gs, mm + 1, pk[1]) : 0u;
                hv = (hA & 0xffu) | (hB & 0xffu) << 8 | (hA >> 8) << 16 | (hB >> 8) << 24;
            } else if constexpr (LM <= 16) {
                hv = (shr(mkA.a0 | mkA.a1 << 16, pk[0]) & 0x10001u) + (shr(mkB.a0 | mkB.a1 << 16, pk[1]) & 0x10001u) * 256u;
            } else {
                hv = (shr(mkA.a0, pk[0]) & 1u) | (shr(mkB.a0, pk[1]) & 1u) << 8 | (shr(mkA.a1, pk[0]) & 1u) << 16 |
                     (shr(mkB.a1, pk[1]) & 1u) << 24;
            }
            if (two) {
                *reinterpret_cast<uint16_t*>(tHl + c0) = (uint16_t)hv;
                *reinterpret_cast<uint16_t*>(tHl + 36 + c0) = (uint16_t)(hv >> 16);
            } else {
                tHl[c0] = (uint8_t)hv;
                tHl[36 + c0] = (uint8_t)(hv >> 16);
            }
            if (w_hp) {
                float q0[2] = {0.f, 0.f}, q1[2] = {0.f, 0.f};
#pragma unroll
                for (int l = 0; l < LM; ++l) {
                    q0[0] += ((mkA.a0 >> l) & 1u) ? p2[l].x : 0.f;
                    q1[0] += ((mkA.a1 >> l) & 1u) ? p2[l].x : 0.f;
                    q0[1] += ((mkB.a0 >> l) & 1u) ? p2[l].y : 0.f;
                    q1[1] += ((mkB.a1 >> l) & 1u) ? p2[l].y : 0.f;
                }
                if (two)
                    *reinterpret_cast<float4*>(tP + lane * 34 + c0) =
                        make_float4(q0[0] * inv2.x, q1[0] * inv2.x, q0[1] * inv2.y, q1[1] * inv2.y);
                else tP[lane * 34 + c0] = make_float2(q0[0] * inv2.x, q1[0] * inv2.x);
            }
        };
        auto pair = [&](uint32_t mm, auto two, const float4* pu, const float4* pd, uint32_t c0) {
            const float4 qa = *pu, qb = pd[0], gv = pd[1];
            auto floor_log = [&] {
                return __fadd2_rn(__fadd2_rn(FH, make_float2(gv.x, gv.y)), __fadd2_rn(FL, make_float2(gv.z, gv.w)));
            };
            pair_at(mm, two, qa, qb, floor_log, c0);
        };
        uint32_t buf = 0;
        for (uint32_t utb = um & ~31u; um < uend; utb += 32, buf ^= 1u) {
            const uint32_t lo = um - utb, tend = min(utb + 32, uend);
            cp_async_wait_all();
            cta_barrier(cta_threads);  // this tile's slot data are there; the last tile's have been read
            stage_tile(utb + 32, buf ^ 1u);
            mrow = sM + 32 * buf;
            grow = sG + 32 * gq * buf;
            while (um < tend) {
                if (um == u1) {
                    anchor(tabQS(tb, u1 - u0));
                    u0 = u1;
                    u1 = warp_value(fr.z);
                    p0 = u0;
                    p1 = u1;
                    in_tab = u1 - u0 < tb.NT;
                    one_form();
                }
                const uint32_t e = min(u1, tend);
                if (u1 - u0 < tb.NT) {
                    const bool head = u1 - u0 < kPostTab;
                    const float4* pu = (head ? sT : tb.up) + (um - u0);
                    const float4* pd = (head ? sT + kPostTab : tb.dg) + 2 * (u1 - um);
                    if (um & 1u) {
                        pair(um, std::false_type{}, pu, pd, um - utb);
                        ++um, ++pu, pd -= 2;
                    }
                    for (; um + 1 < e; um += 2, pu += 2, pd -= 4) pair(um, std::true_type{}, pu, pd, um - utb);
                    if (um < e) {
                        pair(um, std::false_type{}, pu, pd, um - utb);
                        ++um;
                    }
                } else {  // a run longer than the tables: the closed form (an infinite farg' stays infinite)
                    const double fa = __hiloint2double((int)fr.y, (int)fr.x);
                    const bool floors = __any_sync(kAll, (fr.y & kInfHi) != kInfHi);
                    while (um < e) {
                        const bool two = (um & 1u) == 0u && um + 1 < e;
                        const uint32_t j = u1 - um;
                        float4 qa, qb;
                        coeffs(um, qa, qb);
                        auto floor_log = [&] {
                            return floors ? make_float2((float)(fa + tabG(tb, j)), (float)(fa + tabG(tb, j - 1))) : FH;
                        };
                        pair_at(um, two, qa, qb, floor_log, um - utb);
                        um += two ? 2u : 1u;
                    }
                }
            }
            if (vec_ok && lo == 0 && tend == utb + 32 && rows == 32) {
                flush(utb, 0, 32, true);
            } else {  // rows at any offset, one 32-marker segment after the other
                __syncwarp();
                const bool col = lane >= lo && utb + lane < tend;
                const unsigned long long od = out + utb + lane;
#pragma unroll 4
                for (uint32_t r = 0; r < rows; ++r) {
                    const unsigned long long rd = kPlain ? (unsigned long long)(row0 + r) * A.M + utb + lane
                                                         : __shfl_sync(kAll, od, r) - r + lane;
                    if (col) {
                        if (w_dos) A.dosage[rd] = tD[r * 36 + lane];
                        if (w_hp) reinterpret_cast<float2*>(A.hprob)[rd] = tP[r * 34 + lane];
                        if (w_hap) {
                            const unsigned long long rh = 2 * rd - utb - lane;  // 2 x the row's offset + the marker
                            A.haps[rh] = tH[(2 * r) * 36 + lane];
                            A.haps[rh + len] = tH[(2 * r + 1) * 36 + lane];
                        }
                    }
                }
                __syncwarp();
            }
        }
        return;
    }

    // ---- every lane by itself: lanes reach their anchors at different cells. A turn of the loop is the anchors of
    // those at one, or a step of cells for all. (Lanes that waited at an anchor until four of them were there, or none
    // had cells left in the tile, made the others' wait shorter but left the tile's last cells to few lanes: 9,000 x
    // 6,000, L = 8, whole calls, a site every 11 markers 2.23 ms against 2.21, every 40 2.35 against 2.22, every 200
    // 4.57 against 3.54. Anchors and a step in one turn came out of the compiler slower where L is not a power of two:
    // 9,000 x 3,000, L = 19, every 17: 4.24 ms against 3.46.)
    uint32_t tbase = m & ~31u;
    for (;;) {
        const bool on = live && m < mend;
        if (!__any_sync(kAll, on)) break;
        const uint32_t tend = min(tbase + 32, mend), tlo = on ? m - tbase : 32u;
        for (;;) {
            const bool more = on && m < tend, turn = more && m == p1;
            const uint32_t turns = __ballot_sync(kAll, turn), steps = __ballot_sync(kAll, more && !turn);
            if (!(turns | steps)) break;
            if (turns) {
                if (turn) {
                    anchor(tabQS(tb, p1 - p0));
                    p0 = p1;
                    p1 = fr.z;
                    in_tab = p1 - p0 < tb.NT;
                }
            } else if (more) {  // the next cells of the run, two per step when they pair up
                const uint32_t e = min(p1, tend);
                const bool two = (m & 1u) == 0u && m + 1 < e;
                float4 qa, qb;
                coeffs(m, qa, qb);
                cells(m, two, qa, qb, m - tbase);
                m += two ? 2u : 1u;
            }
        }
        flush(tbase, tlo, on ? m - tbase : 0u, on);
        tbase += 32;
    }
}

template <int LM, bool kFull, bool kFast, bool kPlain, bool kDos = true>
cudaError_t launch_post_v(const TypedArgs& a, cudaStream_t s) {
    const uint32_t T = a.threads;
    // the CTA's part is left out where it would not fit beside the windows
    size_t sm = (size_t)(T / 32) * post_warp_bytes(LM, a.C, !kFast);
    TypedArgs f = a;
    f.stage = sm + post_cta_bytes(LM, kDos) <= 227u * 1024u;
    if (f.stage) sm += post_cta_bytes(LM, kDos);
    const unsigned long long groups = ((unsigned long long)a.max_windows + a.K - 1) / a.K;
    // A batch of few warps has several share a window group, while that leaves at most two a scheduler (the
    // anchors before a warp's own cost it alpha steps alone): one target x 1,644 57 -> 21 us, 444 of them 60 ->
    // 33, 131 x 7,919 with sites of their own 548 -> 224 (296 with at most one warp a scheduler).
    f.parts = 1;
    while (f.parts < 8 && a.K % (2 * f.parts) == 0 && groups * f.parts * 2 * typed_groups(a.B) <= 8u * 148u) f.parts *= 2;
    const unsigned long long parts = groups * f.parts;
    // A batch of few warps gives each fewer samples, while that leaves at most two warps a scheduler:
    // lanes at their own sites wait for fewer others (131 x 7,919, a window group a warp: 0.79 ms with 32
    // samples a warp, 0.58 with 8, 0.55 with 4, 0.75 with 2), and lanes in step lose nothing (444 x 1,644: 64
    // us and 60).
    f.rows = 32;
    while (f.rows > 4 && parts * ((a.B + f.rows / 2 - 1) / (f.rows / 2)) <= 8u * 148u) f.rows /= 2;
    const unsigned long long grid = parts * (((a.B + f.rows - 1) / f.rows + T / 32 - 1) / (T / 32));
    if (grid == 0) return cudaSuccess;
    if (grid > 0x7fffffffull) return cudaErrorInvalidConfiguration;
    auto launch = [&](auto kernel) -> cudaError_t {
        // set outside stream capture only (a plan launches once before it is captured)
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        cudaError_t e = cudaStreamIsCapturing(s, &cs);
        if (e != cudaSuccess) return e;
        if (cs == cudaStreamCaptureStatusNone) {
            e = allow_smem(kernel);
            if (e != cudaSuccess) return e;
        }
        kernel<<<(uint32_t)grid, T, sm, s>>>(f);
        return cudaGetLastError();
    };
    // With 16 slots, argmax and dosage the third CTA's register bound spills. In step the CTA is worth it (3,000 x
    // 20,000, whole calls: 0.87 -> 0.82 ms); lanes by themselves wait for memory, which more warps do not hide (9,000 x
    // 6,000 with sites of their own, every 25 markers 2.79 -> 3.65 ms, every 60 2.84 -> 3.75, 131 targets 0.31 -> 0.35).
    // Samples of one array have equally long lists: three where every group's longest list is the batch's longest and
    // there are CTAs for it, else two.
    if constexpr (LM == 16 && kFull && kPlain && kFast && kDos)
        if (grid <= 2u * 148u || a.total_windows != 32ull * typed_groups(a.B) * a.max_windows)
            return launch(anchor_posterior_kernel<LM, kFull, kFast, kPlain, kDos, 2>);
    return launch(anchor_posterior_kernel<LM, kFull, kFast, kPlain, kDos, kPostCtas<LM, kPlain>>);
}

template <int LM, bool kFull>
cudaError_t launch_post(const TypedArgs& a, cudaStream_t s) {
    const bool fast = !a.hprob && a.sampling == SI_SAMPLE_ARGMAX;
    if (fast && !a.dosage)
        return a.samples ? launch_post_v<LM, kFull, true, false, false>(a, s)
                         : launch_post_v<LM, kFull, true, true, false>(a, s);
    if (!a.samples)
        return fast ? launch_post_v<LM, kFull, true, true>(a, s) : launch_post_v<LM, kFull, false, true>(a, s);
    return fast ? launch_post_v<LM, kFull, true, false>(a, s) : launch_post_v<LM, kFull, false, false>(a, s);
}

template <int LM>
cudaError_t launch_typed_lm(const TypedArgs& a, bool full, cudaStream_t s) {
    // a lane per chain; a CTA per direction of a group spreads the few chain warps evenly over the SMs
    const unsigned long long ctas = 2ull * ((a.B + 31) / 32);
    anchor_chain_kernel<LM><<<(uint32_t)ctas, kChainThreads, 0, s>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (a.ev_chain_done && (e = cudaEventRecord(a.ev_chain_done, s)) != cudaSuccess) return e;
    return full ? launch_post<LM, true>(a, s) : launch_post<LM, false>(a, s);
}

}  // namespace

// The window (anchors rebuilt from one checkpoint) fixes where rounding
// restarts, so it must not depend on the batch: one value for every L. The
// CTA size changes nothing numerically.
uint32_t typed_default_window(uint32_t) { return 2u; }
uint32_t typed_default_threads(uint32_t lmax) { return lmax <= 16 ? 128u : 64u; }

size_t typed_post_smem_bytes(uint32_t L, uint32_t T, uint32_t C) {
    return (size_t)(T / 32) * (post_warp_bytes(fb_lmax(L), C, true) + 1024);  // 1 KB a warp kept free
}

cudaError_t launch_anchor_count_only(const TypedArgs& a, cudaStream_t s) {
    const unsigned long long warps = (unsigned long long)a.B * a.nseg;
    const unsigned long long grid = (warps + kWarpsPerBlock - 1) / kWarpsPerBlock;
    if (grid > 0x7fffffffull) return cudaErrorInvalidConfiguration;
    anchor_count_kernel<<<(uint32_t)grid, kWarpsPerBlock * 32, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_anchor_lists_count(const TypedArgs& a, cudaStream_t s) {
    const cudaError_t e = launch_anchor_count_only(a, s);
    if (e != cudaSuccess) return e;
    const uint32_t G = typed_groups(a.B);
    if (G <= kScanGroups) {
        anchor_scan_kernel<true><<<1, 1024, 0, s>>>(a.segc, a.nseg, a.B, a.C, a.aoff, a.woff, a.host_totals);
    } else {
        anchor_group_kernel<<<(G + 3) / 4, 128, 0, s>>>(a.segc, a.nseg, a.B, a.aoff);
        anchor_scan_kernel<false><<<1, 1024, 0, s>>>(a.segc, a.nseg, a.B, a.C, a.aoff, a.woff, a.host_totals);
    }
    return cudaGetLastError();
}

cudaError_t launch_anchor_lists_fill(const TypedArgs& a, cudaStream_t s) {
    // split the segments while they would leave SMs without four CTAs (a small batch is a few chunks of latency)
    const unsigned long long parts = (unsigned long long)typed_groups(a.B) * a.nseg;
    TypedArgs f = a;
    f.split = 1;
    while (f.split < kFillSeg / kFillChunk && parts * f.split < 4 * 148) f.split *= 2;
    const unsigned long long grid = parts * f.split;
    if (grid == 0) return cudaSuccess;
    if (grid > 0x7fffffffull) return cudaErrorInvalidConfiguration;
    anchor_fill_kernel<<<(uint32_t)grid, 32 * kFillWarps, 0, s>>>(f);
    return cudaGetLastError();
}

// lmax: slots held per thread (every region's L <= lmax); the fast variant
// runs when every region uses exactly lmax slots.
cudaError_t launch_typed_fb(const TypedArgs& a, uint32_t lmax, bool all_full, cudaStream_t s) {
    switch (lmax) {
        case 4: return launch_typed_lm<4>(a, all_full, s);
        case 8: return launch_typed_lm<8>(a, all_full, s);
        case 16: return launch_typed_lm<16>(a, all_full, s);
        default: return launch_typed_lm<32>(a, all_full, s);
    }
}

}  // namespace si
