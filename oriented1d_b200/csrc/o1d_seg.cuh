// Segment kernels: the oriented convolution straight from NHWC tiles, on pairs of channels with packed
// fp32 arithmetic (fma.rn.f32x2).
//
// A tile (32 bytes of channels: 8 pairs of bf16 or 4 pairs of fp32 channels, 32 bytes being one DRAM
// sector) is brought into shared memory by TMA in its global layout and is never rearranged.  A thread
// owns one channel pair and a block of outputs, and streams the inputs that the block can see, each
// loaded once and used for every output it reaches:
//   rows, columns   28 positions of one line (14 on short lines): 58 loads for 868 packed FMAs (31 taps)
//   diagonals       14 positions along the diagonal:              34 loads for 294 (21 distinct taps)
//   slanted lines   3 lines x 8 positions:                       174 loads for 696 (29 taps on 11 lines)
// The line is a stride (pixel, row, or row +- pixel), so the eight orientations are three bodies.
// Weights sit in registers, one pair of floats per tap.
//
// Bound: neither memory nor the FMA pipe, but waits that three warps a scheduler do not cover.  56x56x96 bf16, batch 128: issue
// slots 44 % busy while an SM is active, half of them packed FMAs (which hold the pipe for two slots each); the
// largest stalls of a warp are instruction fetch (1.3 cycles an issue: the warps of a CTA run the bodies of
// different line kinds, 10-14 KB of straight code each), fixed latency (1.3) and the busy FMA pipe (0.8); 28 % of
// the SM cycles wait for the slowest CTA.  Useful operations are 19-22 % of the fp32 rate.
// Inputs take arbitrary positions inside the tile without special cases: those past the end of a line are
// clamped onto a pixel of zeros (TMA fills coordinates outside the tensor); whole left / right halves of a
// line's halo are skipped at the borders of the map.  One CTA of twelve warps per SM; the tile after next is
// loaded while the warps, each at its own pace, walk through the tasks of the current one.
//
// Lanes are ordered pair first, so that the lanes of a load cover whole 32-byte pixels of neighbouring
// lines (an odd pixel pitch keeps those in different banks) and the lanes of a store whole sectors.
// Channels of a chunk that lie on different lines form classes with tasks of their own; a pair whose two
// channels differ is computed once for each.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "o1d_common.cuh"
#include "o1d_lines.cuh"
#include "o1d_seg.h"

namespace o1d {
namespace seg {

constexpr int kWarps = 12, kThreads = 32 * kWarps;
constexpr int kTD = 14;                  // outputs of a thread along a diagonal
// lines x positions of a thread on slanted lines: an odd number of lines keeps neighbouring blocks in
// different banks (4 x 7: 6 wavefronts a load)
constexpr int kSR = 3, kST = 8;
constexpr int kMaxBuf = 4;
constexpr int kMaxCC = 32;               // channels of a chunk
constexpr int kPadBytes = 256;           // zeros in front of the tile
constexpr uint32_t kSpinLimit = 1u << 22;

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void add2(f32x2 &d, f32x2 a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }
__device__ __forceinline__ void fma2(f32x2 &d, f32x2 a, f32x2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait; on expiry raises the device flag and reports false.
__device__ __noinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int *err_flag) {
#pragma unroll 1
    for (uint32_t i = 0; i < kSpinLimit; i++)
        if (mbar_try_wait(bar, parity)) return true;
    *err_flag = 1;
    return false;
}
// One more warp is through with a buffer; true for the last of the kWarps, and the count starts over.  Acquire
// and release: every warp's reads of the buffer come before the refill that the last one issues.
__device__ __forceinline__ bool last_warp(int *count) {
    uint32_t before;
    asm volatile("atom.acq_rel.cta.shared::cta.inc.u32 %0, [%1], %2;" : "=r"(before) : "r"(smem_u32(count)), "n"(kWarps - 1) : "memory");
    return before == kWarps - 1;
}
__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void tma_prefetch_4d(const CUtensorMap *map, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];" ::"l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
template <int I, int N, class F> __device__ __forceinline__ void static_for(F &&f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        static_for<I + 1, N>(f);
    }
}

extern __shared__ __align__(1024) char g_smem[];

// One pixel's channel pair, as two floats (from a byte offset in shared memory), and back.
template <typename T> struct Pair;
template <> struct Pair<float> {
    static constexpr int kBytes = 8;
    static __device__ __forceinline__ f32x2 lds(int a) { return *reinterpret_cast<const f32x2 *>(g_smem + a); }
    static __device__ __forceinline__ f32x2 ldg_if(bool c, const float *p) {         // zero when !c
        f32x2 r;
        asm volatile("{.reg .pred q;\n setp.ne.u32 q, %2, 0;\n mov.b64 %0, 0;\n @q ld.global.nc.b64 %0, [%1];}" : "=l"(r) : "l"(p), "r"((uint32_t)c));
        return r;
    }
    static __device__ __forceinline__ void st(float *p, f32x2 v) { *reinterpret_cast<f32x2 *>(p) = v; }
};
template <> struct Pair<__nv_bfloat16> {
    static constexpr int kBytes = 4;
    static __device__ __forceinline__ f32x2 widen(uint32_t v) {
        return pack2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
    }
    static __device__ __forceinline__ f32x2 lds(int a) { return widen(*reinterpret_cast<const uint32_t *>(g_smem + a)); }
    static __device__ __forceinline__ f32x2 ldg_if(bool c, const __nv_bfloat16 *p) {
        uint32_t r;
        asm volatile("{.reg .pred q;\n setp.ne.u32 q, %2, 0;\n mov.b32 %0, 0;\n @q ld.global.nc.b32 %0, [%1];}" : "=r"(r) : "l"(p), "r"((uint32_t)c));
        return widen(r);
    }
    static __device__ __forceinline__ void st(__nv_bfloat16 *p, f32x2 v) {
        const float2 f = unpack2(v);
        uint32_t r;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(f.y), "f"(f.x));
        *reinterpret_cast<uint32_t *>(p) = r;
    }
};

// Order of a sum: taps ascending, one FMA each on top of the bias, as in the general and the direct kernels.  The
// tiled kernels add taps that fall on one pixel first, and walk canonical lines 3 and 4 from the last tap to the
// first: MERGED does the same (21 FMAs instead of 31 on a diagonal).  bf16 outputs and input gradients take the
// order, and so the bits, of the family that the layer would otherwise have (a bf16 network amplifies
// differences of the last bit to the size of its gradients' noise); fp32 ones are MERGED always.  The weight
// gradient has an order of its own: lanes, warps and CTAs, each in a fixed order.
//
// Frame of canonical line o: positions run along image columns (H), rows (V) or both (diagonals, from row to
// row), in the direction in which the taps ascend: base tap m of the line is met m-th.  Lines whose tap k
// ascends against the image axis are walked backwards (`mirrored`), and the base line's taps are
// point-symmetric, so all lines of a kind run the same code; sgn: direction of a slanted line's steps across.
enum : int { FR_H = 0, FR_V = 1, FR_D = 2 };
__host__ __device__ constexpr int frame_of(int o) { return (o == 0 || o == 1 || o == 7) ? FR_H : (o == 2 || o == 6) ? FR_D : FR_V; }
__host__ __device__ constexpr int kind_of(int o) { return (o == 0 || o == 4) ? KIND_AXIS : (o == 2 || o == 6) ? KIND_DIAG : KIND_SLANT; }
__host__ __device__ constexpr bool backwards(int o, bool tiled) { return tiled && (o == 3 || o == 4); }   // m = 30 - k
__host__ __device__ constexpr bool mirrored(int o, bool tiled) { return o > 1 && !backwards(o, tiled); }
__host__ __device__ constexpr int sgn_of(int o, bool tiled) { return ((o == 5 || o == 7) != mirrored(o, tiled)) ? -1 : 1; }
constexpr bool frames_consistent() {
    for (int o = 0; o < 8; o++)
        for (int m = 0; m < kMaxTaps; m++)
            for (int tiled = 0; tiled < 2; tiled++) {
                const int k = backwards(o, tiled) ? kMaxTaps - 1 - m : m, b = kind_of(o), fr = frame_of(o);
                const int dir = mirrored(o, tiled) ? -1 : 1;
                const int dh = kCanonDh[o][k], dw = kCanonDw[o][k];
                const int pos = fr == FR_H ? dw : dh;
                const int line = fr == FR_H ? dh : fr == FR_V ? dw : o == 2 ? dw + dh : dw - dh;
                if (dir * pos != kCanonDw[b][m]) return false;
                if (line != (b == KIND_SLANT ? sgn_of(o, tiled) * kCanonDh[1][m] : 0)) return false;
            }
    return true;
}
static_assert(frames_consistent(), "every canonical line must be a line (or a staircase of lines) of its frame");

// Taps of a block's input, a run of n stored taps.  MERGED: taps that fall on one pixel are stored as one.
struct Taps { int first, n; };
constexpr Taps slant_taps(int dr, int dp, int half, bool merged) {
    Taps f{0, 0};
    for (int t = kHalf - half; t <= kHalf + half; t++)
        if (kCanonDh[1][t] == dr && kCanonDw[1][t] == dp) {
            if (f.n == 0) f.first = t;
            f.n++;
        }
    if (merged && f.n == 3) f = {kHalf, 1};                     // the three centre taps share 15
    return f;
}
// j: position offset; merged diagonals are stored by position
template <int KIND, bool MERGED> constexpr Taps line_taps(int j, int half) {
    Taps f{kHalf + j, j >= -half && j <= half ? 1 : 0};
    if (KIND == KIND_DIAG && !MERGED) {
        f.n = 0;
        for (int t = kHalf - half; t <= kHalf + half; t++)
            if (kCanonDw[2][t] == j) {
                if (f.n == 0) f.first = t;
                f.n++;
            }
    }
    return f;
}
// Does input (rho, pi) reach any output of a slanted block?
constexpr bool slant_used(int rho, int pi, int half) {
    for (int r = 0; r < kSR; r++)
        for (int t = 0; t < kST; t++)
            if (slant_taps(rho - r, pi - t, half, true).n) return true;
    return false;
}
constexpr int slant_first(int rho, int half) {
    for (int pi = -13; pi < kST + 13; pi++) if (slant_used(rho, pi, half)) return pi;
    return 99;
}
constexpr int slant_last(int rho, int half) {
    for (int pi = kST + 13; pi >= -13; pi--) if (slant_used(rho, pi, half)) return pi;
    return -99;
}

// ---- bodies ----------------------------------------------------------------------------------------
// O: the block's outputs (or, for the weight gradient, the values of dy there); Wt: the weights (or the
// accumulators of their gradient), by stored tap.  Addresses are byte offsets in shared memory, of the
// lane's channel pair.  Inputs are visited in ascending position, one compare and one predicated add each: the
// address stays where it is while the position is before `first` or past `last`.
template <bool WG, int M, int NM> __device__ __forceinline__ void use(f32x2 &o, f32x2 (&w)[kMaxTaps], f32x2 x) {
    static_for<M, M + NM>([&](auto m_) {
        constexpr int m = decltype(m_)::value;
        if (WG) fma2(w[m], o, x); else fma2(o, w[m], x);
    });
}
// From position I to I + 1.
template <int I> __device__ __forceinline__ void step_from(int &a, int step, int first) {
    asm("{.reg .pred p;\n setp.le.s32 p, %2, %3;\n @p add.s32 %0, %0, %1;}" : "+r"(a) : "r"(step), "r"(first), "n"(I));
}
template <int I> __device__ __forceinline__ void step_to(int &a, int step, int last) {
    asm("{.reg .pred p;\n setp.gt.s32 p, %2, %3;\n @p add.s32 %0, %0, %1;}" : "+r"(a) : "r"(step), "r"(last), "n"(I));
}
template <int I> __device__ __forceinline__ void step_between(int &a, int step, int first, int last) {
    asm("{.reg .pred p;\n setp.le.s32 p, %2, %4;\n setp.gt.and.s32 p, %3, %4, p;\n @p add.s32 %0, %0, %1;}"
        : "+r"(a) : "r"(step), "r"(first), "r"(last), "n"(I));
}

// The same number, but not known to be: what is derived from it is derived anew.
__device__ __forceinline__ int anew(int v) {
    asm volatile("" : "+r"(v));
    return v;
}

// Line (KIND_AXIS, KIND_DIAG): a = address of the block's first position, step between positions.  A diagonal's
// first position may itself lie before `first` (never past `last`).  left / right: run the inputs before /
// behind the block.
template <typename T, int KIND, int R, int NO, bool WG, bool MERGED>
__device__ __forceinline__ void line_body(int a, int step, int first, int last, bool left, bool right, f32x2 (&O)[NO],
                                          f32x2 (&Wt)[kMaxTaps]) {
    constexpr int RP = KIND == KIND_DIAG ? kCanonDh[2][kHalf - R] : R;       // reach in positions
    auto input = [&](auto i_, f32x2 x) {            // position i relative to the first output
        constexpr int i = decltype(i_)::value;
        static_for<0, NO>([&](auto o_) {
            constexpr int o = decltype(o_)::value;
            constexpr Taps f = line_taps<KIND, MERGED>(i - o, KIND == KIND_DIAG && MERGED ? RP : R);
            if constexpr (f.n > 0) use<WG, f.first, f.n>(O[o], Wt, x);
        });
    };
    if (left) {
        int b = a + max(-RP, first) * step;
        static_for<-RP, 0>([&](auto i_) {
            input(i_, Pair<T>::lds(b));
            step_from<decltype(i_)::value>(b, step, first);
        });
    }
    if constexpr (KIND == KIND_DIAG) a += max(0, first) * step;
    static_for<0, NO>([&](auto i_) {
        input(i_, Pair<T>::lds(a));
        if constexpr (KIND == KIND_DIAG) step_between<decltype(i_)::value>(a, step, first, last);
        else step_to<decltype(i_)::value>(a, step, last);
    });
    if (right)
        static_for<NO, NO + RP>([&](auto i_) {
            input(i_, Pair<T>::lds(a));
            step_to<decltype(i_)::value>(a, step, last);
        });
}

// Slanted line: 3 lines (l0.., in direction sgn) x 8 positions.  base = address of line 0, first position of
// the block; lines outside [llo, lhi] read line lzero.  Taps ascend from the line furthest ahead to the last.
template <typename T, int HALF, bool WG, bool MERGED>
__device__ __forceinline__ void slant_body(int base, int lstep, int pstep, int l0, int sgn, int llo, int lhi, int lzero, int first,
                                           int last, f32x2 (&O)[kSR * kST], f32x2 (&Wt)[kMaxTaps]) {
    constexpr int D = kCanonDh[1][kHalf - HALF];     // reach in lines
    static_for<0, kSR + 2 * D>([&](auto r_) {
        constexpr int rho = kSR - 1 + D - decltype(r_)::value, p0 = slant_first(rho, HALF), p1 = slant_last(rho, HALF);
        int l = sgn > 0 ? l0 + rho : l0 + kSR - 1 - rho;
        l = l < llo || l > lhi ? lzero : l;
        int a = base + l * lstep + (p0 < 0 ? max(p0, first) : min(p0, last)) * pstep;
        static_for<p0, p1 + 1>([&](auto pi_) {
            constexpr int pi = decltype(pi_)::value;
            if constexpr (slant_used(rho, pi, HALF)) {
                const f32x2 x = Pair<T>::lds(a);
                static_for<0, kSR * kST>([&](auto o_) {
                    constexpr int o = decltype(o_)::value;
                    constexpr Taps f = slant_taps(rho - o / kST, pi - o % kST, HALF, MERGED);
                    if constexpr (f.n > 0) use<WG, f.first, f.n>(O[o], Wt, x);
                });
            }
            if constexpr (pi < 0) step_from<pi>(a, pstep, first);
            else step_to<pi>(a, pstep, last);
        });
    });
}

// ---- tables ----------------------------------------------------------------------------------------
constexpr int kMaxPairs = kMaxCC / 2;
// Pairs of one line that share a group of lanes: all of them, or half where that leaves fewer lanes idle.
__host__ __device__ constexpr int class_pairs(int m) { return 32 / m * m < 27 ? (m + 1) / 2 : m; }
struct Class {
    int canon, n, full;
    int warp0, warps;                        // weight gradient: warps that work on it
    int entry[kMaxPairs];
};        // entry: pair | channels of it (1 low, 2 high) << 4; full: all are 3
struct Tables {
    f32x2 w[32][kMaxPairs];                  // by stored tap and pair
    f32x2 bias[kMaxPairs];
    int ncls, ids[kMaxCC];
    Class cls[12];
};
// MERGED: taps summed into stored tap i of a line kind (three 5-bit numbers, 31 = none).
struct MergeTable { uint16_t src[3][32]; };
constexpr MergeTable make_merge() {
    MergeTable m{};
    for (int kind = 0; kind < 3; kind++)
        for (int i = 0; i < 32; i++) {
            int found[3] = {31, 31, 31}, n = 0;
            for (int t = 0; t < kMaxTaps; t++) {
                const int at = kind == KIND_SLANT ? (t == 14 || t == 16 ? 15 : t) : kCanonDw[kind][t] + kHalf;
                if (at == i) found[n++] = t;
            }
            for (int e = 0; e < 3; e++) m.src[kind][i] |= (uint16_t)(found[e] << (5 * e));
        }
    return m;
}
static __device__ const MergeTable g_merge = make_merge();
// MERGED: stored tap of each tap of a diagonal.
struct DiagTable { int8_t at[kMaxTaps]; __device__ int operator[](int t) const { return at[t]; } };
constexpr DiagTable make_diag() {
    DiagTable d{};
    for (int t = 0; t < kMaxTaps; t++) d.at[t] = (int8_t)(kCanonDw[2][t] + kHalf);
    return d;
}
static __device__ const DiagTable g_diag_at = make_diag();

// Weight of tap m (in the order of the sum) of channel c on canonical line id, the identity added to the
// centre tap (0 when the kernel is shorter than the line).
template <bool MERGED>
__device__ __forceinline__ float base_weight(const void *w, int wbf16, int c, int id, int m, const SegParams &p) {
    if (m >= kMaxTaps) return 0.f;
    const int k = (backwards(id, MERGED) != (p.flip != 0) ? kMaxTaps - 1 - m : m) - kHalf + p.K / 2;
    if (k < 0 || k >= p.K) return 0.f;
    const size_t at = (size_t)c * p.K + k;
    const float v = wbf16 ? __bfloat162float(((const __nv_bfloat16 *)w)[at]) : __ldg((const float *)w + at);
    return m == kHalf && p.identity ? v + 1.f : v;
}
// Tables of the chunk that starts at channel c0; ends in a barrier.
template <bool MERGED>
__device__ __noinline__ void build_tables(Tables *tab, const SegParams &p, const void *w, const void *bias, int wbf16,
                                          const int8_t *chan, int c0) {
    const int tid = threadIdx.x;
    if (tid < p.CC) tab->ids[tid] = c0 + tid < p.C ? (int)__ldg(chan + c0 + tid) : -1;
    if (tid < p.CC)
        reinterpret_cast<float *>(tab->bias)[tid] =
            !bias || c0 + tid >= p.C ? 0.f
            : wbf16 ? __bfloat162float(((const __nv_bfloat16 *)bias)[c0 + tid]) : __ldg((const float *)bias + c0 + tid);
    __syncthreads();
    if (w)
#pragma unroll 1
        for (int i = tid; i < p.CC * 32; i += kThreads) {
            const int c = i >> 5, t = i & 31, id = tab->ids[c];
            float v = 0.f;
            if (id >= 0) {
                const uint32_t src = MERGED ? g_merge.src[kind_of(id)][t] : t;
                v = base_weight<MERGED>(w, wbf16, c0 + c, id, src & 31, p);
                if (MERGED)
                    v = v + base_weight<MERGED>(w, wbf16, c0 + c, id, src >> 5 & 31, p) + base_weight<MERGED>(w, wbf16, c0 + c, id, src >> 10 & 31, p);
            }
            reinterpret_cast<float *>(&tab->w[t][c >> 1])[c & 1] = v;
        }
    if (tid == kThreads - 1) {
        int n = 0;
#pragma unroll 1
        for (int o = 0; o < 8; o++) {
            int m = 0;
#pragma unroll 1
            for (int q = 0; q < p.CC / 2; q++) m += tab->ids[2 * q] == o || tab->ids[2 * q + 1] == o;
            const int most = m ? class_pairs(m) : 0;
            int q = 0;
#pragma unroll 1
            while (m > 0) {
                Class *cl = &tab->cls[n++];
                cl->canon = o;
                cl->full = 1;
                cl->n = 0;
#pragma unroll 1
                for (; cl->n < most && m > 0; q++) {
                    const int mask = (tab->ids[2 * q] == o ? 1 : 0) | (tab->ids[2 * q + 1] == o ? 2 : 0);
                    if (!mask) continue;
                    cl->entry[cl->n++] = q | mask << 4;
                    m--;
                    if (mask != 3) cl->full = 0;
                }
            }
        }
        tab->ncls = n;
    }
    __syncthreads();
}

// Cycles of one task on a scheduler with three warps, for the division of the work: chunks among CTAs on the host,
// warps among classes here.  Measured in the forward kernel at 56x56x96, batch 128, one line kind at a time; they
// know nothing of the instruction fetches of a CTA whose warps run several kinds.
__host__ __device__ constexpr int task_cycles(int kind, int lt) {
    return kind == KIND_SLANT ? 4600 : kind == KIND_DIAG ? 2050 : lt == 28 ? 3600 : 1950;
}

// Weight gradient: the warps are dealt to the classes in proportion to their tasks' cost, so that a warp
// keeps its accumulators for all items of a segment.  One thread.
__device__ __noinline__ void deal_warps(Tables *tab, int imgs, int lenh, int lenw, int lt) {
    float cost[12], total = 0.f;
    int left = kWarps;
#pragma unroll 1
    for (int i = 0; i < tab->ncls; i++) {
        const Class &c = tab->cls[i];
        const int kind = kind_of(c.canon), fr = frame_of(c.canon), lpg = 32 / c.n;
        const int plen = fr == FR_H ? lenw : lenh, llen = fr == FR_H ? lenh : lenw;
        const int lines = kind == KIND_AXIS ? llen : kind == KIND_DIAG ? lenw + kTD - 1 : (llen + kSR - 1) / kSR;
        const int bl = kind == KIND_SLANT ? kST : kind == KIND_AXIS ? lt : kTD;
        cost[i] = (float)task_cycles(kind, lt) * ((imgs * lines + lpg - 1) / lpg) * ((plen + bl - 1) / bl);
        total += cost[i];
    }
#pragma unroll 1
    for (int i = 0; i < tab->ncls; i++) {
        tab->cls[i].warps = max(1, (int)(kWarps * cost[i] / total));
        left -= tab->cls[i].warps;
    }
#pragma unroll 1
    while (left != 0) {                      // one more to the slowest class, or one less from the fastest
        int at = -1;
#pragma unroll 1
        for (int i = 0; i < tab->ncls; i++) {
            const float v = cost[i] / tab->cls[i].warps, w = at < 0 ? 0.f : cost[at] / tab->cls[at].warps;
            if (left > 0 ? (at < 0 || v > w) : (tab->cls[i].warps > 1 && (at < 0 || v < w))) at = i;
        }
        tab->cls[at].warps += left > 0 ? 1 : -1;
        left += left > 0 ? -1 : 1;
    }
    int w = 0;
#pragma unroll 1
    for (int i = 0; i < tab->ncls; i++) { tab->cls[i].warp0 = w; w += tab->cls[i].warps; }
}

// Either channel of a pair, or both: predicated stores (branches would triple the code).
template <typename T> __device__ __forceinline__ void store_pair(T *p, f32x2 v, int mask) {
    const float2 f = unpack2(v);
    if constexpr (sizeof(T) == 4)
        asm volatile("{.reg .pred l, h;\n setp.ne.u32 l, %3, 0;\n setp.ne.u32 h, %4, 0;\n @l st.global.f32 [%0], %1;\n @h st.global.f32 [%0+4], %2;}"
                     ::"l"(p), "f"(f.x), "f"(f.y), "r"(mask & 1), "r"(mask & 2) : "memory");
    else
        asm volatile("{.reg .pred l, h;\n .reg .b16 a, b;\n setp.ne.u32 l, %3, 0;\n setp.ne.u32 h, %4, 0;\n cvt.rn.bf16.f32 a, %1;\n"
                     " cvt.rn.bf16.f32 b, %2;\n @l st.global.b16 [%0], a;\n @h st.global.b16 [%0+2], b;}"
                     ::"l"(p), "f"(f.x), "f"(f.y), "r"(mask & 1), "r"(mask & 2) : "memory");
}

// The block's dy, zero past the last `left` positions of the line.
template <typename T, int NO> __device__ __forceinline__ void load_line(const T *q, ptrdiff_t ps, f32x2 *O, int left) {
#pragma unroll
    for (int o = 0; o < NO; o++) {
        O[o] = Pair<T>::ldg_if(o < left, q);
        q += ps;
    }
}
// `left` outputs of a line (at most NO), ps elements apart.
template <typename T, int NO>
__device__ __forceinline__ void store_line(T *q, ptrdiff_t ps, const f32x2 *O, int left, bool all, int mask) {
    if (all) {
#pragma unroll
        for (int o = 0; o < NO; o++) {
            if (o < left) Pair<T>::st(q, O[o]);
            q += ps;
        }
    } else {
#pragma unroll
        for (int o = 0; o < NO; o++) {
            if (o < left) store_pair(q, O[o], mask);
            q += ps;
        }
    }
}

// ---- kernel ----------------------------------------------------------------------------------------
// Division of the work.  A part is 1 / kParts of an item's tasks.
//   CTAs per chunk (p.per_chunk): every chunk has a number of CTAs in proportion to its cost; they take its
//   items in turn, and the last, incomplete round by parts.  All chunks advance through the images at one
//   pace, so the chunks that share a pixel's DRAM bursts and L2 lines meet there.
//   Otherwise (too many chunks for that): the sequence runs, chunks, items, parts is cut into shares of
//   equal cost, one per CTA.
constexpr int kParts = 8;
struct Segment {                             // work of a CTA on one chunk
    int run, chunk;                          // chunk within the run
    int full, first, step;                   // items first, first + step, ...: `full` whole ones,
    int begin, end;                          // then the parts [begin, end) of the chunk
    __device__ __forceinline__ int count() const { return full + (end > begin ? (end + kParts - 1) / kParts - begin / kParts : 0); }
    __device__ __forceinline__ int item(int s) const { return s < full ? first + s * step : begin / kParts + s - full; }
};
struct Spot { int run, chunk, part; };
__device__ __forceinline__ Spot spot_of(const SegParams &p, long long at) {
    Spot s{0, 0, 0};
#pragma unroll 1
    for (; s.run < p.nruns; s.run++) {
        const SegRun &r = p.run[s.run];
        const long long chunk = (long long)r.cost * p.geo[r.geo].items * kParts, all = chunk * r.nchunks;
        if (at < all) {
            s.chunk = (int)(at / chunk);
            s.part = (int)((at - s.chunk * chunk) / r.cost);
            return s;
        }
        at -= all;
    }
    return s;                                // one past the end
}
__device__ __forceinline__ bool first_segment(const SegParams &p, Segment &g, Spot &at, const Spot &end, int cta) {
    if (p.per_chunk) {
        int b = cta;
        g.run = 0;
#pragma unroll 1
        while (b >= p.run[g.run].nchunks * p.run[g.run].ctas) { b -= p.run[g.run].nchunks * p.run[g.run].ctas; g.run++; }
        const int kc = p.run[g.run].ctas, items = p.geo[p.run[g.run].geo].items;
        g.chunk = b / kc;
        g.first = b - g.chunk * kc;
        g.step = kc;
        g.full = items / kc;
        const int base = g.full * kc * kParts, tail = items * kParts - base;
        g.begin = base + tail * g.first / kc;
        g.end = base + tail * (g.first + 1) / kc;
        return g.count() > 0;
    }
    g.full = g.first = g.step = 0;
    if (at.run > end.run || (at.run == end.run && (at.chunk > end.chunk || (at.chunk == end.chunk && at.part >= end.part)))) return false;
    g.run = at.run;
    g.chunk = at.chunk;
    g.begin = at.part;
    const bool here = at.run == end.run && at.chunk == end.chunk;
    g.end = here ? end.part : p.geo[p.run[at.run].geo].items * kParts;
    // where the next segment starts
    at.part = 0;
    if (here) at = end;
    else if (++at.chunk == p.run[at.run].nchunks) { at.chunk = 0; at.run++; }
    return at.run < p.nruns || g.run < p.nruns;
}

// R: reach of the taps (15, or 7 for kernels of up to 15 taps); LT: outputs of a thread along a line.
// MERGED: the tiled kernels' order of a sum (see above).
// WG = false: y = conv(x) + bias.  WG = true: y is dy, and each CTA leaves its share of the weight and bias
// gradients of its chunks in `partial` ([slot][channel of the chunk][32], by stored tap, the bias last).
template <typename T, int R, int LT, bool WG, bool MERGED>
__global__ void __launch_bounds__(kThreads, 1)
seg_kernel(const __grid_constant__ SegMaps maps, const __grid_constant__ SegMaps dy_maps, const void *__restrict__ wv,
           const void *__restrict__ biasv, int wbf16, const int8_t *__restrict__ chan, T *__restrict__ y,
           float *__restrict__ partial, int *__restrict__ err_flag, const __grid_constant__ SegParams p) {
    char *sm = g_smem;
    constexpr int PB = Pair<T>::kBytes;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    Tables *tab = reinterpret_cast<Tables *>(sm + p.off_tab);
    uint64_t *full = reinterpret_cast<uint64_t *>(sm + p.off_bar);
    int *cnt = reinterpret_cast<int *>(full + kMaxBuf);

    Segment g;
    Spot at{0, 0, 0}, end{0, 0, 0};
    if (!p.per_chunk) {
        at = spot_of(p, p.total_cost * blockIdx.x / gridDim.x);
        end = spot_of(p, p.total_cost * (blockIdx.x + 1) / gridDim.x);
    }
    bool more = first_segment(p, g, at, end, blockIdx.x);
    auto issue = [&](const Segment &g, int s, int buf) {          // item number s of the segment
        const SegGeo &ge = p.geo[p.run[g.run].geo];
        const int it = g.item(s), tiles = ge.nth * ge.ntw;
        int n0 = it * ge.G, th = 0, tw = 0;
        if (tiles > 1) {
            n0 = it / tiles;
            const int r = it - n0 * tiles;
            th = r / ge.ntw;
            tw = r - th * ge.ntw;
        }
        mbar_expect_tx(&full[buf], ge.tile_bytes);
        tma_load_4d(sm + p.off_tile + buf * ge.buf_bytes, &maps.m[p.run[g.run].geo], &full[buf],
                    (p.run[g.run].chunk0 + g.chunk) * p.CC, tw * ge.TW - ge.ow, th * ge.TH - ge.oh, n0);
        // dy is read straight from global memory, each value once: have it in L2 by then
        if (WG) tma_prefetch_4d(&dy_maps.m[p.run[g.run].geo], (p.run[g.run].chunk0 + g.chunk) * p.CC, tw * ge.TW, th * ge.TH, n0);
    };
    if (tid == 0) {
#pragma unroll 1
        for (int b = 0; b < kMaxBuf; b++) { mbar_init(&full[b], 1); cnt[b] = 0; }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < kPadBytes / 4; i += kThreads) reinterpret_cast<float *>(sm + p.off_tile - kPadBytes)[i] = 0.f;

    int turn = warp;                             // tasks until this warp's next one
    bool ok = true;
    uint32_t phase = 0;                          // parity of each buffer's barrier
#pragma unroll 1
    for (; more; more = !p.per_chunk && first_segment(p, g, at, end, blockIdx.x)) {
        const SegGeo &ge = p.geo[p.run[g.run].geo];
        const int c0 = (p.run[g.run].chunk0 + g.chunk) * p.CC, tiles = ge.nth * ge.ntw, row_bytes = ge.P * p.px, px = p.px;
        const int nitems = g.count();
        // The previous segment is done with tables and buffers.  What it stored there itself (pixels of zeros, where
        // its buffers ended; sums over the warps) comes before the copies issued below.
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
#pragma unroll 1
            for (int b = 0; b < ge.nbuf && b < nitems; b++) issue(g, b, b);
        }
        // the pixel in front of a buffer's tile is the previous buffer's last one: zeros
        for (int i = tid; i < ge.nbuf * 16; i += kThreads)
            if ((i & 15) * 4 < px)
                *reinterpret_cast<float *>(sm + p.off_tile + ((i >> 4) + 1) * ge.buf_bytes - px + (i & 15) * 4) = 0.f;
        build_tables<MERGED>(tab, p, wv, biasv, wbf16, chan, c0);
        int buf = 0, my_class = 0, stride = kWarps;
        f32x2 Wg[kMaxTaps], dbias = 0;           // weight gradient: the warp's accumulators
        if constexpr (WG) {
            if (tid == 0) deal_warps(tab, ge.G, ge.TH, ge.TW, LT);
            __syncthreads();
            while (warp >= tab->cls[my_class].warp0 + tab->cls[my_class].warps) my_class++;
            stride = tab->cls[my_class].warps;
            turn = warp - tab->cls[my_class].warp0;
#pragma unroll
            for (int i = 0; i < kMaxTaps; i++) Wg[i] = 0;
        }
#pragma unroll 1
        for (int s = 0; s < nitems; s++) {
            const int it = g.item(s);
            const int part0 = s < g.full ? 0 : max(g.begin - it * kParts, 0), part1 = s < g.full ? kParts : min(g.end - it * kParts, kParts);
            int n0 = it * ge.G, h0 = 0, w0 = 0, imgs = min(ge.G, p.N - n0);
            if (tiles > 1) {
                n0 = it / tiles;
                imgs = 1;
                const int r = it - n0 * tiles;
                h0 = r / ge.ntw;
                w0 = (r - h0 * ge.ntw) * ge.TW;
                h0 *= ge.TH;
            }
            const int lenh = min(ge.TH, p.H - h0), lenw = min(ge.TW, p.W - w0);       // outputs of this tile
            const int tbuf = p.off_tile + buf * ge.buf_bytes + ge.oh * row_bytes + ge.ow * px;
            if (ok) ok = mbar_wait(&full[buf], phase >> buf & 1, err_flag);
            phase ^= 1u << buf;
#pragma unroll 1
            for (int ci = WG ? my_class : 0; ci < (WG ? my_class + 1 : tab->ncls); ci++) {
                const Class *cl = &tab->cls[ci];
                const int id = cl->canon, np = cl->n, kind = kind_of(id), fr = frame_of(id);
                const int lpg = 32 / np;                                            // lines per group of lanes
                const int plen = fr == FR_H ? lenw : lenh, llen = fr == FR_H ? lenh : lenw;
                const int nlines = kind == KIND_AXIS ? llen : kind == KIND_DIAG ? lenw + kTD - 1 : (llen + kSR - 1) / kSR;
                const int bl = kind == KIND_SLANT ? kST : kind == KIND_AXIS ? LT : kTD, npb = (plen + bl - 1) / bl;
                const int nt = (imgs * nlines + lpg - 1) / lpg * npb, t0 = nt * part0 / kParts, t1 = nt * part1 / kParts;
                const int ln = lane / np, entry = cl->entry[lane - ln * np], pair = entry & 15, mask = entry >> 4;
                const bool all = cl->full;
                int t = t0 + turn, ug = t / npb, pb = t - ug * npb;
                const int dug = stride / npb, dpb = stride - dug * npb;
                turn -= t1 - t0;
#pragma unroll 1
                for (; t < t1; t += stride, turn += stride) {
                    const int li = ug * lpg + ln, gi = ge.G == 1 ? (li >= nlines) : li / nlines, line = li - gi * nlines;
                    const bool act = ln < lpg && gi < imgs;
                    const int gt = tbuf + pair * PB + (act ? gi : 0) * ge.img_bytes;         // first output of the image
                    // the block's first position in the direction of the walk, and in the image
                    const int q0 = pb * bl;
                    const bool mir = mirrored(id, MERGED);
                    const int p0 = mir ? plen - 1 - q0 : q0;
                    // Output pixel.  Where a block's outputs lie is worked out from a few numbers, anew behind the body:
                    // kept over it the addresses and strides cost registers (56x56x96 bf16, batch 128: 194 us, now 169).
                    auto out = [&](int gi, int h, int w) {
                        return y + (((size_t)(n0 + gi) * p.H + h0 + h) * p.W + w0 + w) * p.C + c0 + 2 * pair;
                    };
                    auto task = [&](f32x2 (&Wt)[kMaxTaps], f32x2 bias) {
                    if (kind == KIND_SLANT) {
                        f32x2 O[kSR * kST];
                        const int l0 = line * kSR, sgn = sgn_of(id, MERGED);
                        const bool hf = fr == FR_H;
                        const int lstep = hf ? row_bytes : px, pstep = hf ? px : row_bytes;
                        const int plo = hf ? ge.plo_w : ge.plo_h, phi = hf ? ge.phi_w : ge.phi_h;
                        const int cut = hf ? ge.halo_h : ge.halo_w;
                        const int llo = (hf ? ge.plo_h : ge.plo_w) + 1 - cut, lhi = (hf ? ge.phi_h : ge.phi_w) - 1 + cut;
                        const int lzero = cut ? 0 : hf ? ge.plo_h : ge.phi_w;
                        // line r of the block, `left` positions of it
                        auto each_line = [&](int id, int l0, int gi, int q0, auto &&f) {
                            const bool hf = frame_of(id) == FR_H, mir = mirrored(id, MERGED);
                            const int plen = hf ? lenw : lenh, llen = hf ? lenh : lenw, p0 = mir ? plen - 1 - q0 : q0, sgn = sgn_of(id, MERGED);
                            const ptrdiff_t ps = hf ? p.C : (ptrdiff_t)p.W * p.C;
#pragma unroll
                            for (int r = 0; r < kSR; r++) {
                                const int l = sgn > 0 ? l0 + r : l0 + kSR - 1 - r;
                                f(r, out(gi, hf ? l : p0, hf ? p0 : l), mir ? -ps : ps, act && l < llen ? plen - q0 : 0);
                            }
                        };
                        if constexpr (WG) each_line(id, l0, gi, q0, [&](int r, T *q, ptrdiff_t ps, int left) { load_line<T, kST>(q, ps, &O[r * kST], left); });
                        else {
#pragma unroll
                            for (int o = 0; o < kSR * kST; o++) O[o] = bias;
                        }
                        slant_body<T, R, WG, MERGED>(gt + p0 * pstep, lstep, mir ? -pstep : pstep, l0, sgn, llo, lhi, lzero,
                                                     mir ? p0 - phi : plo - p0, mir ? p0 - plo : phi - p0, O, Wt);
                        if constexpr (WG) {
#pragma unroll
                            for (int o = 0; o < kSR * kST; o++) add2(dbias, O[o]);
                        } else
                            each_line(anew(id), anew(l0), anew(gi), anew(q0), [&](int r, T *q, ptrdiff_t ps, int left) { store_line<T, kST>(q, ps, &O[r * kST], left, all, mask); });
                    } else if (kind == KIND_AXIS) {
                        f32x2 O[LT];
                        const bool hf = fr == FR_H;
                        const int step = hf ? px : row_bytes, base = gt + line * (hf ? row_bytes : px);
                        const int plo = hf ? ge.plo_w : ge.plo_h, phi = hf ? ge.phi_w : ge.phi_h;
                        const bool cut = hf ? ge.halo_w : ge.halo_h;
                        auto place = [&](int id, int line, int gi, int q0, auto &&f) {
                            const bool hf = frame_of(id) == FR_H, mir = mirrored(id, MERGED);
                            const int plen = hf ? lenw : lenh, p0 = mir ? plen - 1 - q0 : q0;
                            const ptrdiff_t ps = hf ? p.C : (ptrdiff_t)p.W * p.C;
                            f(out(gi, hf ? line : p0, hf ? p0 : line), mir ? -ps : ps, act ? plen - q0 : 0);
                        };
                        if constexpr (WG) place(id, line, gi, q0, [&](T *q, ptrdiff_t ps, int left) { load_line<T, LT>(q, ps, O, left); });
                        else {
#pragma unroll
                            for (int o = 0; o < LT; o++) O[o] = bias;
                        }
                        line_body<T, KIND_AXIS, R, LT, WG, MERGED>(base + p0 * step, mir ? -step : step, mir ? p0 - phi : plo - p0,
                                                                   mir ? p0 - plo : phi - p0, q0 > 0 || cut, q0 + LT < plen || cut, O, Wt);
                        if constexpr (WG) {
#pragma unroll
                            for (int o = 0; o < LT; o++) add2(dbias, O[o]);
                        } else
                            place(anew(id), anew(line), anew(gi), anew(q0), [&](T *q, ptrdiff_t ps, int left) { store_line<T, LT>(q, ps, O, left, all, mask); });
                    } else {
                        f32x2 O[kTD];
                        // per position: a row up, dw pixels to the right
                        const int dw = id == 2 ? 1 : -1, w = dw > 0 ? line - (kTD - 1) : line;
                        auto outputs = [&](int id, int line, int gi, int q0, auto &&f) {
                            const int dw = id == 2 ? 1 : -1, w = dw > 0 ? line - (kTD - 1) : line;
                            T *q = out(gi, lenh - 1 - q0, w);
                            const ptrdiff_t ps = ((ptrdiff_t)dw - p.W) * p.C;
#pragma unroll
                            for (int o = 0; o < kTD; o++) {
                                f(o, q, act && q0 + o < lenh && (unsigned)(w + o * dw) < (unsigned)lenw);
                                q += ps;
                            }
                        };
                        if constexpr (WG) {
                            outputs(id, line, gi, q0, [&](int o, const T *q, bool in) { O[o] = Pair<T>::ldg_if(in, q); });
                        } else {
#pragma unroll
                            for (int o = 0; o < kTD; o++) O[o] = bias;
                        }
                        // where the diagonal enters and leaves the tile (at the zeros around a whole map), from the block's first position
                        const int f = max(dw > 0 ? ge.plo_w - w : w - ge.phi_w, p0 - ge.phi_h);
                        const int l = min(dw > 0 ? ge.phi_w - w : w - ge.plo_w, p0 - ge.plo_h);
                        // (a diagonal that misses the tile reads its first row, zeros around a whole map)
                        const bool miss = f > l;
                        line_body<T, KIND_DIAG, R, kTD, WG, MERGED>(miss ? gt + ge.plo_h * row_bytes : gt + p0 * row_bytes + w * px,
                                                                    dw * px - row_bytes, miss ? 0 : f, miss ? 0 : l,
                                                                    q0 > 0 || ge.halo_h, q0 + kTD < plen || ge.halo_h, O, Wt);
                        if constexpr (WG) {
#pragma unroll
                            for (int o = 0; o < kTD; o++) add2(dbias, O[o]);
                        } else {
                            outputs(anew(id), anew(line), anew(gi), anew(q0), [&](int o, T *q, bool in) {
                                if (in) {
                                    if (all) Pair<T>::st(q, O[o]); else store_pair(q, O[o], mask);
                                }
                            });
                        }
                    }
                    };
                    if constexpr (WG) task(Wg, 0);
                    else {
                        f32x2 Wt[kMaxTaps];
#pragma unroll
                        for (int i = 0; i < kMaxTaps; i++) Wt[i] = tab->w[i][pair];
                        task(Wt, tab->bias[pair]);
                    }
                    ug += dug;
                    pb += dpb;
                    if (pb >= npb) { pb -= npb; ug++; }
                }
            }
            __syncwarp();
            if (lane == 0 && last_warp(&cnt[buf]) && s + ge.nbuf < nitems) issue(g, s + ge.nbuf, buf);
            if (++buf == ge.nbuf) buf = 0;
        }
        if constexpr (WG) {
            // lanes of a pair, then the warps of a class, each in a fixed order
            const int np = tab->cls[my_class].n, ln = lane / np;
            __syncthreads();
            f32x2 *red = reinterpret_cast<f32x2 *>(sm + p.off_tile);         // [warp][32][kMaxPairs]
#pragma unroll 1
            for (int n = 32 / np; n > 1;) {
                const int half = (n + 1) / 2;
                const bool take = ln + half < n;
                static_for<0, kMaxTaps + 1>([&](auto i_) {
                    constexpr int i = decltype(i_)::value;
                    f32x2 &v = i < kMaxTaps ? Wg[i < kMaxTaps ? i : 0] : dbias;
                    const f32x2 u = __shfl_down_sync(~0u, v, half * np);
                    if (take) add2(v, u);
                });
                n = half;
            }
            if (lane < np)
                static_for<0, kMaxTaps + 1>([&](auto i_) {
                    constexpr int i = decltype(i_)::value;
                    red[(warp * 32 + i) * kMaxPairs + lane] = i < kMaxTaps ? Wg[i < kMaxTaps ? i : 0] : dbias;
                });
            __syncthreads();
            const int slot = p.per_chunk ? (int)blockIdx.x : (int)blockIdx.x + p.run[g.run].chunk0 + g.chunk;
#pragma unroll 1
            for (int ci = 0; ci < tab->ncls; ci++) {
                const Class &cl = tab->cls[ci];
#pragma unroll 1
                for (int i = tid; i < cl.n * 64; i += kThreads) {
                    const int e = i >> 6, half = i >> 5 & 1, t = i & 31, entry = cl.entry[e];
                    if (!(entry >> 4 >> half & 1)) continue;
                    float sum = 0.f;
#pragma unroll 1
                    for (int w = cl.warp0; w < cl.warp0 + cl.warps; w++)
                        sum += reinterpret_cast<const float *>(&red[(w * 32 + t) * kMaxPairs + e])[half];
                    partial[((size_t)slot * p.CC + 2 * (entry & 15) + half) * 32 + t] = sum;
                }
            }
        }
    }
}

// Adds the shares of a chunk (one CTA each) in the order of the CTAs and writes the weight and bias gradients.
static __global__ void __launch_bounds__(256)
seg_wgrad_final_kernel(const float *__restrict__ partial, const int8_t *__restrict__ chan, void *__restrict__ dw, void *__restrict__ db,
                       int out_bf16, int ctas, const __grid_constant__ SegParams p) {
    __shared__ int slots[256], nslots;
    const int chunk = blockIdx.x, tid = threadIdx.x;
    bool has = false;                            // does CTA `tid` have a segment of this chunk?
    int slot = tid;
    if (tid < ctas) {
        Segment g;
        Spot at{0, 0, 0}, end{0, 0, 0};
        if (!p.per_chunk) {
            at = spot_of(p, p.total_cost * tid / ctas);
            end = spot_of(p, p.total_cost * (tid + 1) / ctas);
            slot = tid + chunk;
        }
        bool more = first_segment(p, g, at, end, tid);
#pragma unroll 1
        while (more && !has) {
            has = p.run[g.run].chunk0 + g.chunk == chunk;
            more = !p.per_chunk && first_segment(p, g, at, end, tid);
        }
    }
    slots[tid] = has ? slot : -1;
    __syncthreads();
    if (tid == 0) {
        int n = 0;
#pragma unroll 1
        for (int i = 0; i < ctas; i++)
            if (slots[i] >= 0) slots[n++] = slots[i];
        nslots = n;
    }
    __syncthreads();
#pragma unroll 1
    for (int i = blockIdx.y * 256 + tid; i < p.CC * 32; i += gridDim.y * 256) {
        const int cc = i >> 5, c = chunk * p.CC + cc, k = i & 31;      // k: tap of the kernel, 31: the bias
        if (c >= p.C || (k < 31 ? k >= p.K : db == nullptr)) continue;
        int at = 31;
        if (k < 31) {
            const int id = chan[c], kind = kind_of(id), j = k - p.K / 2 + kHalf, t = backwards(id, true) ? kMaxTaps - 1 - j : j;
            at = kind == KIND_SLANT ? (t == 14 || t == 16 ? 15 : t) : kind == KIND_DIAG ? g_diag_at[t] : t;
        }
        float sum = 0.f;
#pragma unroll 8
        for (int n = 0; n < nslots; n++) sum += partial[((size_t)slots[n] * p.CC + cc) * 32 + at];
        const size_t o = k < 31 ? (size_t)c * p.K + k : c;
        void *out = k < 31 ? dw : db;
        if (out_bf16) ((__nv_bfloat16 *)out)[o] = __float2bfloat16_rn(sum); else ((float *)out)[o] = sum;
    }
}

}  // namespace seg
}  // namespace o1d
