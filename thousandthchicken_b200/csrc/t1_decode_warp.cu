// t1_decode_warp.cu -- Tier-1 EBCOT/MQ code-block decoder for sm_100a, one
// warp per code-block (the default; t1_decode.cu keeps the decoder of several
// blocks per warp).
//
// A block's decisions are one serial chain, so the warp's instructions per
// decision bound it: their latency when blocks are few, issue slots and the
// integer ALU when they fill the GPU.  Hence:
//   * what the next decision is, and its context, is prepared by the lanes in
//     parallel before a stripe's serial part: bitmaps of the samples to code,
//     in scan order, and a context label for each.  A decision is then find
//     first bit, label, context word, interval arithmetic; no neighbourhood is
//     looked at, no column or row loop is walked.  A sample that becomes
//     significant makes five lanes recompute the labels that it changes, and a
//     table lookup adds the samples that it makes candidates.  A run-length
//     column is its first row alone, under its own label.
//   * the serial part runs on all lanes alike (see BlockState for what keeps
//     them apart from one another's context words); the next label and context word are loaded while the
//     current decision is decoded, and both successor states as soon as its
//     context word is known.
//   * magnitudes are bit-planes in shared memory (512 B each), gathered by the
//     epilogue with the inverse quantiser (ISO E.1); with the significance,
//     sign, visited and refined bitmaps a block of 8 bit-planes takes 7 KB.
//     Blocks of any depth share one launch: when room for its deepest block
//     would cost the others their places, deep blocks move their bits on to
//     their output words (see kFewPlanes).
// Against the decoder of per-column flag words that was here before (one warp
// per block too), Tier-1 of one 64x64 block of 8 bit-planes 6.39 -> 3.03 ms,
// of 14 bit-planes 10.4 -> 4.7 ms; 4096x4096x3 lossy 14.4 -> 12.6 ms (issue
// 74% -> 87% of cycles, ALU pipe 76% busy), 2048x2048x3 12-bit lossless
// 16.4 -> 9.0 ms.
//
// Code-blocks with a coding style (bypass, context reset, termination on every
// pass, vertically causal contexts, segmentation symbols; ISO D.4-D.7) run in
// a launch of their own, an instantiation of the same decoder that switches
// codeword segments at pass boundaries; the reference decodes style 0 only.
#include <cuda_runtime.h>

#include <algorithm>

#include "t1_common.cuh"
#include "tc_internal.cuh"

namespace tc {
namespace {

constexpr int kRow = 9;          // words per stripe of a sample bitmap: 64 columns and a zero guard
constexpr int kLabRun = 72, kLabUni = 68;   // context labels are kept as byte offsets (4 x label)
constexpr int kMaxSlots = 12;    // code-blocks per CTA at most
constexpr int kStyledSlots = 8;  // the same for styled blocks, which take up to 128 registers
// Launches of fewer blocks per SM than this decode Deep: the label of the
// sample after the next is loaded too and one branch leaves the straight line,
// more instructions but shorter waits.  Against the other kernel: 1024x1024x3
// lossy (5 blocks per SM) 1.86 and 2.12 ms, 2048x2048 16-bit lossless (7) 5.66
// and 6.64; 1792x1792x3 lossy (16) 3.40 and 3.29, 4096x4096x3 13.8 and 12.6.
// From 9 to 13 it depends on the blocks: where a few are much longer than the
// rest Deep is faster (1472x1472x3 8-bit lossless 3.49 and 3.84, sparse lossy
// 0.39 and 0.47), where all are alike the other one is (lossy 2.56 and 2.51,
// 1536x1536x3 2.76 and 2.42).
constexpr int kDeepBlocks = 13;

// Label and probability tables of a CTA.
struct WarpTables {
    uint8_t zc[4][512];   // zero-coding label x 4 per orientation and 3x3 neighbourhood
    uint8_t sc[1280];     // sign label x 4 | XOR bit << 7, by sign index (see build_warp_tables)
    uint2 next[94];       // context words after an MPS and after an LPS, by 2 x state + MPS
    uint2 adds[2][32];    // by pass (propagation, cleanup) and place: see build_warp_tables
};

// A context word: Qe << 16 | (2 x state + MPS) << 3.
__device__ __forceinline__ uint32_t ctx_word(int state, int mps)
{
    return ((uint32_t)c_qe[state] << 16) | (uint32_t)((2 * state + mps) << 3);
}

// A code-block's state.  Bitmaps of samples have eight words a stripe, each
// of eight columns of four rows, in scan order from the top bit down (column
// c, row k: bit 31 - 4 (c & 7) - k, so that bit & 3 is 3 - k); a zero word
// ends every stripe, and S and G have a zero stripe above and below.  The
// magnitude bits follow as bit-planes of kPlaneWords words.
//
// All lanes run the serial part, but nothing keeps them in step there: a lane
// must not store a context word that another has yet to read.  Deep: each lane
// has context words of its own (21 words apart, so in different banks), and
// between two new samples no lane waits for another.  Otherwise all share one
// set, which keeps the state small, and a warp barrier stands before every
// store; own sets, or contexts in registers and shuffles, cost such launches
// more (4096x4096x3 lossy 12.7 ms with the barrier, 13.9 with sets for eight
// lanes; shuffles take 10% longer than the barrier.  2048x2048 16-bit lossless,
// Deep, 5.2 ms with own words and 5.5 with the barrier).
template <bool Deep>
struct BlockState {
    static constexpr int kSets = Deep ? 32 : 1;
    static constexpr int kSetWords = Deep ? 21 : 20;
    uint32_t S[1 + 18 * kRow];   // significance (from S + 1: the guard before the first word)
    uint32_t G[1 + 18 * kRow];   // signs of the significant samples
    uint32_t P[16 * 8];          // coded in this plane's significance propagation pass
    uint32_t R[16 * 8];          // refined at least once
    uint32_t F[66];              // flag words of the current stripe's columns
    uint8_t lab[9 * 32];         // context label of every sample of the current stripe, in scan order
    uint32_t ctx[kSets * kSetWords];   // context words

    // The contexts' first states (ISO Table D.7).
    __device__ void reset_contexts(int lane)
    {
        for (int i = lane; i < kSets * 19; i += 32) {
            const int k = i / kSets;
            ctx[i % kSets * kSetWords + k] = ctx_word(k == 0 ? 4 : (k == 17 ? 46 : (k == 18 ? 3 : 0)), 0);
        }
    }
};
constexpr int kPlaneWords = 128;
// A launch that does not fit the GPU at once with room for all bit-planes of
// its deepest block, and that would fit more blocks with room for this many, has
// room for no more than these places allow (12 with 24 places per SM); a deeper
// block moves its bits to its output words as it goes.  So one deep block, or a
// caller's bound of 31, costs the others no places: 4096x4096x3 lossy, most blocks
// of 4 bit-planes, takes 12.6 ms alone, with one block of 20 and under a bound of
// 31 (13.6, 16.4 and 16.4 before, with 24, 16 and 12 places; the first is the
// code's difference), 2048x2048x3 16-bit lossless 12.0 (13.4).  A launch that fits
// anyway moves nothing.
constexpr int kFewPlanes = 8;

// Flag word of a stripe column: bits 3j + i (j = 0..5: rows 4..-1, i = 0
// right, 1 this, 2 left column) significance; bits 18..23 the signs of the
// column's rows 4..-1; bits 24..27 and 28..31 the signs of rows 3..0 of the
// columns to the left and to the right.  The 3x3 neighbourhood of row k is
// (F >> 3 (3 - k)) & 0x1FF.
constexpr int kOwnSign = 18, kLeftSign = 24, kRightSign = 28;

__device__ void build_warp_tables(WarpTables &t)
{
    for (int i = threadIdx.x; i < 94; i += blockDim.x) {
        const int st = i >> 1, mps = i & 1, sw = st == 0 || st == 6 || st == 14;
        t.next[i] = make_uint2(ctx_word(c_nmps[st], mps), ctx_word(c_nlps[st], mps ^ sw));
    }
    for (int i = threadIdx.x; i < 4 * 512; i += blockDim.x) {
        const int o = i >> 9, p = i & 511;
        const int h = ((p >> 3) & 1) + ((p >> 5) & 1);
        const int v = ((p >> 1) & 1) + ((p >> 7) & 1);
        const int d = (p & 1) + ((p >> 2) & 1) + ((p >> 6) & 1) + ((p >> 8) & 1);
        t.zc[o][p] = (uint8_t)(4 * zc_label(o, h, v, d));
    }
    // Sign index: significance of down, right, left, up in bits 1, 3, 5, 7
    // (their places in the 3x3 neighbourhood), their signs in bits 0, 10, 6
    // and 2 (their places in the flag word from bit kOwnSign + 3 - row on).
    // ISO Tables D.2/D.3.
    for (int i = threadIdx.x; i < 1280; i += blockDim.x) {
        auto ctb = [&](int sig, int neg) { return (i >> sig) & 1 ? ((i >> neg) & 1 ? -1 : 1) : 0; };
        int vc = ctb(7, 2) + ctb(1, 0), hc = ctb(5, 6) + ctb(3, 10);
        hc = hc > 1 ? 1 : (hc < -1 ? -1 : hc);
        vc = vc > 1 ? 1 : (vc < -1 ? -1 : vc);
        const int cx = hc == 0 ? (vc == 0 ? 9 : 10) : 12 + hc * vc;
        const int xr = hc == 0 ? vc < 0 : hc < 0;
        t.sc[i] = (uint8_t)((4 * cx) | (xr << 7));
    }
    // The candidates that a newly significant sample at bit `at` can add, in
    // its own word (x) and the next (y).  Propagation: the next row and the
    // next column's rows k - 1 .. k + 1; cleanup: the next column's rows
    // (it may have been a run-length column).
    for (int i = threadIdx.x; i < 64; i += blockDim.x) {
        const int at = i & 31, r = at & 3, col = at & ~3;   // r = 3 - row
        unsigned long long m = 0;                            // bit 32 + b: bit b of this word
        for (int q = 0; q < 4; q++)
            if (i >= 32 || (q >= r - 1 && q <= r + 1)) m |= 1ull << (32 + col - 4 + q);
        if (i < 32 && r > 0) m |= 1ull << (32 + at - 1);
        t.adds[i >> 5][at] = make_uint2((uint32_t)(m >> 32), (uint32_t)m);
    }
}

// Index of the highest set bit (-1 for 0), and the count of leading zeros of
// a nonzero word: one instruction each.
__device__ __forceinline__ int top_bit(uint32_t x)
{
    int r;
    asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}
__device__ __forceinline__ int lead_zeros(uint32_t x)
{
    int r;
    asm("bfind.shiftamt.u32 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}

// MQ decoder (ISO C.3), the interval register A scaled by 2^16.
struct WarpMQ {
    const uint8_t *p;
    int len, bp, ct;
    uint32_t a, c, cur, nxt;

    __device__ __forceinline__ uint32_t byte_at(int i) const { return i < len ? (uint32_t)__ldg(p + i) : 0xFFu; }
    __device__ __forceinline__ void bytein()
    {
        if (cur == 0xFF) {
            if (nxt > 0x8F) {
                c += 0xFF00;  // marker (or past the end): feed 1-bits, do not advance
                ct = 8;
                return;
            }
            c += nxt << 9;
            ct = 7;
        } else {
            c += nxt << 8;
            ct = 8;
        }
        bp++;
        cur = nxt;
        nxt = byte_at(bp + 1);
    }
    __device__ __forceinline__ void init(const uint8_t *d, int n)
    {
        p = d;
        len = n;
        bp = 0;
        cur = byte_at(0);
        nxt = byte_at(1);
        c = cur << 16;
        bytein();
        c <<= 7;
        ct -= 7;
        a = 0x80000000u;
    }
    // One decision of the context whose word is w; out: its word afterwards.
    // Both successors are loaded as soon as w is known, and the shift is
    // taken without a branch (0 when no renormalisation is due), so the
    // chain from one decision to the next is arithmetic alone.
    __device__ __forceinline__ bool decide(const WarpTables &T, uint32_t w, uint32_t &out)
    {
        const uint2 nx = *reinterpret_cast<const uint2 *>(reinterpret_cast<const char *>(T.next) + (w & 0x3F8u));
        const uint32_t q = w & 0xFFFF0000u;
        const uint32_t a1 = a - q;
        const bool lower = c < q;    // the code value lies in the Qe sub-interval
        const bool lps = lower != (a1 < q);
        c = lower ? c : c - q;
        a = lower ? q : a1;
        int sh = lead_zeros(a);
        out = sh ? (lps ? nx.y : nx.x) : w;
        while (sh > ct) {
            a <<= ct;
            c <<= ct;
            sh -= ct;
            bytein();
        }
        a <<= sh;
        c <<= sh;
        ct -= sh;
        return lps != ((w & 8u) != 0u);
    }
    // The same without a branch: the shift is taken whether it is 0 or not and
    // may leave ct negative, for the caller to refill; due: the state moves on,
    // to nx.
    __device__ __forceinline__ bool decide_ahead(const WarpTables &T, uint32_t w, uint32_t &nx, bool &due)
    {
        const uint2 succ = *reinterpret_cast<const uint2 *>(reinterpret_cast<const char *>(T.next) + (w & 0x3F8u));
        const uint32_t q = w & 0xFFFF0000u;
        const uint32_t a1 = a - q;
        const bool lower = c < q;
        const bool lps = lower != (a1 < q);
        c = lower ? c : c - q;
        a = lower ? q : a1;
        due = (int)a >= 0;
        nx = lps ? succ.y : succ.x;
        const int sh = lead_zeros(a);
        a <<= sh;
        c <<= sh;
        ct -= sh;
        return lps != ((w & 8u) != 0u);
    }
    // The bytes that are due (ct < 0: bits taken by the last shift that the
    // register did not hold).  Adding a byte after the shift, shifted up by
    // the bits that were missing, equals adding it before.
    __device__ __forceinline__ void refill()
    {
        while (ct < 0) {
            uint32_t add = 0xFF00u;
            int n = 8;
            if (cur != 0xFF || nxt <= 0x8F) {
                n = cur == 0xFF ? 7 : 8;
                add = nxt << (16 - n);
                bp++;
                cur = nxt;
                nxt = byte_at(bp + 1);
            }
            c += add << -ct;
            ct += n;
        }
    }
};

// Raw (bypass) bits of ISO D.6.
struct WarpRaw {
    const uint8_t *p;
    int len, bp, ct;
    uint32_t b;

    __device__ __forceinline__ void init(const uint8_t *d, int n)
    {
        p = d;
        len = n;
        bp = 0;
        ct = 0;
        b = 0;
    }
    __device__ __forceinline__ bool bit()
    {
        if (ct == 0) {
            const uint32_t nb = bp < len ? (uint32_t)__ldg(p + bp) : 0xFFu;
            if (b == 0xFF && nb > 0x8F) {
                ct = 8;
            } else {
                ct = b == 0xFF ? 7 : 8;
                b = nb;
                bp++;
            }
        }
        --ct;
        return (b >> ct) & 1u;
    }
};

constexpr unsigned kFull = 0xffffffffu;

// The magnitude bits of column x in stripe s, from n bit-planes after those in m.
__device__ __forceinline__ void gather_planes(uint32_t (&m)[4], const uint32_t *planes, int n, int s, int x)
{
    const uint32_t *word = planes + s * 8 + (x >> 3);
    const int sh = 28 - 4 * (x & 7);
    for (int q = 0; q < n; q++) {
        const uint32_t b = word[q * kPlaneWords] >> sh;
#pragma unroll
        for (int k = 0; k < 4; k++) m[k] = 2 * m[k] + ((b >> (3 - k)) & 1u);
    }
}

// A state without room for another bit-plane: the np planes that it holds move
// to the block's output words (more: below those that moved before).  A lane has
// the same columns as in the epilogue, so no lane reads what another wrote.  Not
// inlined: a block moves planes three times at most, and the serial part keeps
// its registers.
__device__ __noinline__ void move_planes(const uint32_t *planes, int np, uint32_t *ob, uint32_t pitch, int w, int h,
                                         bool more, int lane)
{
    for (int s = 0; 4 * s < h; s++)
        for (int x = lane; x < w; x += 32) {
            uint32_t m[4] = {0u, 0u, 0u, 0u};
            gather_planes(m, planes, np, s, x);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (4 * s + k >= h) break;
                uint32_t *o = ob + (uint64_t)(4 * s + k) * pitch + x;
                *o = more ? (*o << np) | m[k] : m[k];
            }
        }
}

// Decode one code-block, all lanes alike.  Returns the last pass type
// (0 cleanup, 1 significance propagation, 2 refinement) and its plane.
// Modes: the code-block style `style` applies; lens, when not null, holds the
// lengths of the codeword's terminated segments (BYPASS / TERMALL), which
// follow one another from seg.  Raw: the block has raw (bypass) passes.
template <bool Modes, bool Raw, bool Deep>
__device__ int decode_block_warp(BlockState<Deep> &B, uint32_t *planes, int np, const WarpTables &T, const uint8_t *seg,
                                 int len, int w, int h, int orient, int numbps, int passes, int *last_plane, int lane, int style,
                                 const uint32_t *lens, uint32_t *ob, uint32_t pitch)
{
    WarpMQ mq;
    WarpRaw rw;
    bool raw = false;      // the current segment is raw-coded
    int segi = 0;          // current segment
    uint32_t segoff = 0;   // its first byte
    const bool vsc = Modes && (style & TC_CBLK_STYLE_VSC);
    if (!Modes || !lens) mq.init(seg, len);
    char *ctxb = reinterpret_cast<char *>(B.ctx + (Deep ? lane * B.kSetWords : 0));
    auto ctx_at = [&](int lab) -> uint32_t & { return *reinterpret_cast<uint32_t *>(ctxb + lab); };
    const uint8_t *zc = T.zc[orient];
    const int nstripes = (h + 3) >> 2;

    // The columns of this lane's word that lie in the block.
    const int ncol = lane < 8 ? min(8, max(0, w - 8 * lane)) : 0;
    const uint32_t colmask = ncol ? 0xffffffffu << (32 - 4 * ncol) : 0u;
    // Where the window of three columns around this lane's column starts (its
    // second column, 32 further on, four words later).
    const int win = ((lane + 7) >> 3) - 1, winsh = 4 * ((lane + 7) & 7);
    // When a sample becomes significant, lanes 0..3 compute the labels of the
    // next column's rows, the other lanes that of the next sample in scan
    // order: bit (at & lab_col) - lab_next.
    const int lab_col = lane < 4 ? ~3 : ~0, lab_next = lane < 4 ? lane + 1 : 1;

    // Before a context word is stored that all lanes share.  No lane is then
    // more than a decision ahead, which the labels and flag words need as well.
    auto before_store = [&]() {
        if constexpr (!Deep) __syncwarp();
    };
    auto begin_pass = [&](int t) {
        if constexpr (Modes) {
            if (!lens || (t > 0 && !style_pass_terminates(style, t - 1))) return;
            if (t > 0) segoff += lens[segi++];
            if constexpr (Raw) {
                raw = style_pass_raw(style, t);
                if (raw) {
                    rw.init(seg + segoff, (int)lens[segi]);
                    return;
                }
            }
            mq.init(seg + segoff, (int)lens[segi]);
        }
    };
    // One decision of context word cw, out: the word afterwards, due: whether
    // it changed.  Deep: the caller refills.
    auto decide = [&](uint32_t cw, uint32_t &out, bool &due) -> bool {
        if constexpr (Raw) {
            if (raw) {
                out = cw;
                due = false;
                return rw.bit();
            }
        }
        if constexpr (Deep) return mq.decide_ahead(T, cw, out, due);
        due = true;
        return mq.decide(T, cw, out);
    };
    // A decision outside the pipelined loops, its context updated.
    auto decide_now = [&](int lab) -> bool {
        uint32_t out;
        const bool d = mq.decide(T, ctx_at(lab), out);
        before_store();
        ctx_at(lab) = out;
        return d;
    };

    int type = 0, p = numbps - 1;
    uint32_t *plane = planes - kPlaneWords;   // the bits of plane p
    for (int t = 0;;) {
        begin_pass(t);
        if (type == 1 || t == 0) {   // a new plane
            plane += kPlaneWords;
            if (plane == planes + np * kPlaneWords) {
                __syncwarp();
                move_planes(planes, np, ob, pitch, w, h, p + 1 + np < numbps, lane);
                __syncwarp();
                plane = planes;
            }
            for (int i = lane; i < nstripes * 8; i += 32) plane[i] = 0u;
        }

        for (int s = 0; s < nstripes; s++) {
            const int rows = min(4, h - 4 * s);
            const uint32_t valid = colmask & ((0xF0u >> rows) & 0xFu) * 0x11111111u;
            __syncwarp();
            // ---- candidates: lane j < 8 holds word j of the stripe ----
            const uint32_t *Srow = B.S + 1 + (s + 1) * kRow;
            uint32_t S0 = 0, V = 0, E = 0, A = 0, N = 0;
            if (lane < 8) {
                S0 = Srow[lane];
                const uint32_t up = Srow[lane - kRow], dn = vsc ? 0u : Srow[lane + kRow];
                V = ((S0 >> 1) & 0x77777777u) | ((S0 << 1) & 0xEEEEEEEEu) | ((up & 0x11111111u) << 3) |
                    ((dn >> 3) & 0x11111111u);
            }
            const uint32_t VS = V | S0;
            const uint32_t prev = __shfl_sync(kFull, VS, (lane + 31) & 31), next = __shfl_sync(kFull, VS, (lane + 1) & 31);
            // samples with a significant neighbour
            const uint32_t nb = V | __funnelshift_r(VS, prev, 4) | __funnelshift_l(next, VS, 4);
            if (type == 2) {
                if (lane < 8) E = S0 & ~B.P[s * 8 + lane];
            } else {
                A = ~S0 & valid;   // samples that may still become candidates
                if (type == 1) {
                    E = nb & A;
                    if (lane < 8) B.P[s * 8 + lane] = 0u;
                } else {
                    if (lane < 8) E = A & ~B.P[s * 8 + lane];
                    // run-length columns (four rows, nothing significant in
                    // or around them) have their first row as their only
                    // candidate
                    const uint32_t any = nb | S0;
                    const uint32_t some = (any | (any >> 1) | (any >> 2) | (any >> 3)) & 0x11111111u;
                    A = rows == 4 ? (valid & 0x11111111u & ~some) * 7u : 0u;
                    E &= ~A;
                }
            }
            uint32_t wm = __ballot_sync(kFull, E != 0u);
            if (wm == 0u) continue;

            // ---- flag words and labels: each lane its columns ----
#pragma unroll
            for (int half = 0; half < 2; half++) {
                const int c = lane + 32 * half;
                if (32 * half >= w || (Raw && raw && type == 2)) break;
                uint32_t l4;
                if (type == 2) {
                    // 16 after the first refinement, else 15 with a
                    // significant neighbour, else 14
                    const int sh = 28 - 4 * (c & 7);
                    const uint32_t rn = (B.R[s * 8 + (c >> 3)] >> sh) & 15u;
                    const uint32_t nn = (__shfl_sync(kFull, nb, c >> 3) >> sh) & ~rn & 15u;
                    auto bytes = [](uint32_t n) { return ((n >> 3) | (n << 6) | (n << 15) | (n << 24)) & 0x01010101u; };
                    l4 = 0x38383838u + 4u * bytes(nn) + 8u * bytes(rn);
                } else {
                    // three columns of this stripe (four rows each), of the
                    // row above and of the row below: left, this, right
                    auto window = [&](const uint32_t *row) {
                        const uint32_t *q = row + win + 4 * half;
                        return __funnelshift_l(q[1], q[0], winsh) >> 20;
                    };
                    auto spread = [](uint32_t n) {   // bit i -> bit 3i
                        return (n & 1u) | ((n & 2u) << 2) | ((n & 4u) << 4) | ((n & 8u) << 6);
                    };
                    auto three = [](uint32_t x) { return (x | (x >> 3) | (x >> 6)) & 7u; };   // bits 8, 4, 0 -> 2, 1, 0
                    const uint32_t *Grow = B.G + 1 + (s + 1) * kRow;
                    const uint32_t x = window(Srow), g = window(Grow);
                    const uint32_t xu = window(Srow - kRow) & 0x111u, gu = window(Grow - kRow);
                    const uint32_t xd = vsc ? 0u : (window(Srow + kRow) >> 3) & 0x111u;
                    const uint32_t gd = vsc ? 0u : window(Grow + kRow) >> 3;
                    const uint32_t sig = ((spread(x & 15u) | (spread((x >> 4) & 15u) << 1) | (spread(x >> 8) << 2)) << 3) |
                                         three(xd) | (three(xu) << 15);
                    B.F[c] = sig | (((gd >> 4) & 1u) << kOwnSign) | (((g >> 4) & 15u) << (kOwnSign + 1)) |
                             (((gu >> 4) & 1u) << (kOwnSign + 5)) | ((g >> 8) << kLeftSign) | ((g & 15u) << kRightSign);
                    l4 = (uint32_t)zc[sig >> 9] | ((uint32_t)zc[(sig >> 6) & 0x1FFu] << 8) |
                         ((uint32_t)zc[(sig >> 3) & 0x1FFu] << 16) | ((uint32_t)zc[sig & 0x1FFu] << 24);
                    if (type == 0 && rows == 4 && sig == 0u) l4 = kLabRun;
                }
                *reinterpret_cast<uint32_t *>(B.lab + 4 * c) = l4;
            }
            __syncwarp();

            uint32_t vis = 0;   // lane j: the samples of word j coded in this pass
            if (type == 2) {
                // ---- magnitude refinement (ISO D.3.3) ----
                if (Raw && raw) {
                    // raw bits, one a sample in scan order: no labels, no
                    // contexts (1536x1100x3 lossless with bypass: 3.77 ms, 0.55 less)
                    do {
                        const int j = __ffs(wm) - 1;
                        wm &= wm - 1;
                        uint32_t e = __shfl_sync(kFull, E, j), bits = 0;
                        while (e) {
                            const uint32_t bit = 1u << top_bit(e);
                            e ^= bit;
                            if (rw.bit()) bits |= bit;
                        }
                        if (lane == j) N = bits;
                    } while (wm);
                } else {
                do {
                    const int j = __ffs(wm) - 1;
                    wm &= wm - 1;
                    uint32_t e = __shfl_sync(kFull, E, j), bits = 0;
                    const uint8_t *labp = B.lab + 32 * j + 31;
                    int at = top_bit(e);
                    int lab = labp[-at];
                    uint32_t cw = ctx_at(lab);
                    if constexpr (Deep) {
                        e ^= 1u << at;
                        int an = top_bit(e);
                        int ln = labp[-an];
                        // the sample at a0, a1 next; the one after that takes
                        // a0's place (two steps by turns: no register moves)
                        auto step = [&](int &a0, int &l0, const int a1, const int l1) -> bool {
                            const bool last = e == 0u;
                            const uint32_t bit = 1u << a0;
                            e &= ~(1u << (a1 & 31));
                            const int a2 = top_bit(e);
                            const int l2 = labp[-a2];
                            const uint32_t cn = ctx_at(l1);
                            uint32_t nx;
                            bool due;
                            const bool d = decide(cw, nx, due);
                            if (due) ctx_at(l0) = nx;
                            if (d) bits |= bit;
                            cw = due && l1 == l0 ? nx : cn;
                            if (mq.ct < 0) mq.refill();
                            a0 = a2;
                            l0 = l2;
                            return last;
                        };
                        for (;;) {
                            if (step(at, lab, an, ln)) break;
                            if (step(an, ln, at, lab)) break;
                        }
                    } else {
                        for (;;) {
                            const uint32_t bit = 1u << at;
                            e ^= bit;
                            const int an = top_bit(e);
                            const int ln = labp[-an];
                            const uint32_t cn = ctx_at(ln);
                            uint32_t nx;
                            bool due;
                            if (decide(cw, nx, due)) bits |= bit;
                            before_store();
                            ctx_at(lab) = nx;
                            if (!e) break;
                            cw = ln == lab ? nx : cn;
                            at = an;
                            lab = ln;
                        }
                    }
                    if (lane == j) N = bits;
                } while (wm);
                }
                if (lane < 8) {
                    B.R[s * 8 + lane] |= E;
                    plane[s * 8 + lane] |= N;
                }
                continue;
            }

            // ---- significance propagation (ISO D.3.1) and cleanup (D.3.4) ----
            uint32_t gn = 0;   // lane j: the signs of word j's new samples
            const uint2 *adds = T.adds[type == 1 ? 0 : 1];
            do {
                const int j = __ffs(wm) - 1;
                wm &= wm - 1;
                uint32_t e = __shfl_sync(kFull, E, j), seen = e, sig = 0, sgn = 0;
                const uint32_t avail = __shfl_sync(kFull, A, j), avail1 = __shfl_sync(kFull, A, j + 1);
                uint8_t *labp = B.lab + 32 * j + 31;
                char *fp = reinterpret_cast<char *>(B.F + 8 * j + 7);   // the word's last column
                int at = top_bit(e);
                int lab = labp[-at];
                uint32_t cw = ctx_at(lab);
                int an = 0, ln = 0;
                if constexpr (Deep) {
                    e ^= 1u << at;
                    an = top_bit(e);
                    ln = labp[-an];
                }
                for (;;) {
                    // at, lab, cw: the current sample; an, ln: the next one;
                    // e: the samples after the current one; Deep: a2, l2, e2
                    // the same one sample on
                    uint32_t e2 = 0;
                    int a2 = 0, l2 = 0;
                    if constexpr (Deep) {
                        e2 = e & ~(1u << (an & 31));
                        a2 = top_bit(e2);
                        l2 = labp[-a2];
                    } else {
                        e ^= 1u << at;
                        an = top_bit(e);
                        ln = labp[-an];
                    }
                    const uint32_t cn = ctx_at(ln);
                    uint32_t nx;
                    bool due;
                    const bool d = decide(cw, nx, due);
                    before_store();
                    if (due) ctx_at(lab) = nx;
                    cw = due && ln == lab ? nx : cn;
                    // Deep: one branch leaves the straight line
                    if (!Deep || d || mq.ct < 0 || !e) {
                        if (Deep && mq.ct < 0) mq.refill();
                        if (d) {
                            if (lab == kLabRun) {
                                // a run-length column with a significant
                                // sample: its row, then the rows below it
                                const int top = at;
                                const int r1 = decide_now(kLabUni), r0 = decide_now(kLabUni);
                                at -= 2 * r1 + r0;
                                e |= (1u << at) - (1u << (top - 3));
                            }
                            const uint32_t bit = 1u << at;
                            sig |= bit;
                            const int r = at & 3;
                            // The lane's sample: its flag word with this
                            // sample in it, and its label.  Stored before the
                            // sign is decoded, so that the next context is
                            // loaded meanwhile.
                            const int to = (at & lab_col) - lab_next;
                            uint32_t *fw = reinterpret_cast<uint32_t *>(fp - (to & ~3));
                            const bool other = ((to ^ at) & ~3) != 0;   // the next column
                            if constexpr (Deep) __syncwarp();   // else: the barrier before the store above
                            const uint32_t f = *reinterpret_cast<const uint32_t *>(fp - (at & ~3));
                            uint32_t v = *fw | ((other ? 32u : 16u) << (3 * r));
                            const uint2 add = adds[at];
                            labp[-to] = zc[(v >> (3 * (to & 3))) & 0x1FFu];
                            const uint32_t sv = T.sc[((f >> (3 * r)) & 0xAAu) | ((f >> (kOwnSign + r)) & 0x445u)];
                            e |= add.x & avail;
                            seen |= add.x & avail;
                            an = top_bit(e);
                            __syncwarp();
                            const int sl = (int)(sv & 0x7Fu);
                            const uint32_t sw = ctx_at(sl);
                            ln = labp[-an];
                            cw = ctx_at(ln);   // not a sign context
                            if constexpr (Deep) {
                                e2 = e & ~(1u << (an & 31));
                                a2 = top_bit(e2);
                                l2 = labp[-a2];
                            }
                            uint32_t snx;
                            bool sdue;
                            const bool neg = decide(sw, snx, sdue) != ((Raw && raw) ? false : (sv >> 7) != 0u);
                            before_store();
                            if (sdue) ctx_at(sl) = snx;
                            if (neg) {
                                v |= (other ? 1u << kLeftSign : 2u << kOwnSign) << r;
                                sgn |= bit;
                            }
                            *fw = v;
                            if (add.y & avail1) {
                                if (lane == j + 1) E |= add.y & avail1;
                                wm |= 2u << j;
                            }
                            if (Deep && mq.ct < 0) mq.refill();
                        }
                        if (!e) break;
                    }
                    at = an;
                    lab = ln;
                    if constexpr (Deep) {
                        an = a2;
                        ln = l2;
                        e = e2;
                    }
                }
                if (lane == j) {
                    N = sig;
                    gn = sgn;
                    vis = seen;
                }
            } while (wm);
            if (lane < 8) {
                const int i = 1 + (s + 1) * kRow + lane;
                B.S[i] = S0 | N;
                B.G[i] |= gn;
                plane[s * 8 + lane] |= N;
                if (type == 1) B.P[s * 8 + lane] = vis;
            }
        }

        if constexpr (Modes) {
            if (type == 0 && (style & TC_CBLK_STYLE_SEGSYM)) {   // segmentation symbol 1010 (ISO D.5)
                for (int i = 0; i < 4; i++) decide_now(kLabUni);
            }
            if (style & TC_CBLK_STYLE_RESET) {
                __syncwarp();
                B.reset_contexts(lane);
            }
        }
        if (++t >= passes) break;
        if (type == 0) {
            --p;
            type = 1;
        } else {
            type = type == 1 ? 2 : 0;
        }
    }
    *last_plane = p;
    return type;
}

// Decode code-block `bi` with the state B and write it out.  np: the
// bit-planes that the state has room for; limit: the most that a block may have.
template <bool Modes, bool Deep>
__device__ __forceinline__ void process_block_warp(BlockState<Deep> &B, uint32_t *planes, int np, int limit, const WarpTables &T,
                                                   const tc_cblk_desc *__restrict__ desc, uint32_t bi, int ndesc,
                                                   const uint8_t *__restrict__ pool, uint64_t pool_len,
                                                   char *__restrict__ out, uint64_t out_elems, int out_mode, float recon_r,
                                                   uint32_t *__restrict__ err, int lane)
{
    if (bi >= (uint32_t)ndesc) {
        if (lane == 0) atomicOr(err, TC_DERR_DESC);
        return;
    }
    const tc_cblk_desc d = desc[bi];
    const int w = d.w, h = d.h;
    const bool geom_ok = w >= 1 && w <= 64 && h >= 1 && h <= 64;
    const int numbps = (int)d.mb - (int)d.zero_bitplanes;
    bool ok = geom_ok && d.mb >= 1 && d.mb <= 31 && d.orient <= 3 && numbps >= 0 &&
              (numbps == 0 || d.passes <= 3 * numbps - 2) && numbps <= limit;
    const bool pool_ok = d.seg_off <= pool_len && (uint64_t)d.seg_len <= pool_len - d.seg_off;
    if (!geom_ok) {
        if (lane == 0) atomicOr(err, TC_DERR_DESC);
        return;
    }
    // the block's last sample, out_off + (h-1) * out_pitch + w - 1, must lie
    // inside the output; a block that does not is skipped before any write
    if (d.out_off > out_elems || (uint64_t)(h - 1) * d.out_pitch + (uint64_t)w > out_elems - d.out_off) {
        if (lane == 0) atomicOr(err, TC_DERR_OUT);
        return;
    }
    if (!ok || !pool_ok) {
        if (lane == 0) atomicOr(err, ok ? TC_DERR_POOL : TC_DERR_DESC);
        ok = false;
    }
    // Styled blocks: only the Modes launch decodes them.  A segment table
    // (BYPASS / TERMALL) sits 4-byte aligned at seg_off, the codeword after
    // it, and its lengths add up to seg_len.
    const int style = d.style & kStyleDecodeBits;
    const uint32_t *lens = nullptr;
    uint64_t cw_off = d.seg_off;
    if (!Modes && style) {
        if (lane == 0) atomicOr(err, TC_DERR_STYLE);
        ok = false;
    }
    if (Modes && ok && (style & (TC_CBLK_STYLE_BYPASS | TC_CBLK_STYLE_TERMALL)) && numbps > 0 && d.passes > 0) {
        const int nseg = style_segments(style, d.passes);
        const uint64_t tab = 4ull * (uint64_t)nseg;
        bool tab_ok = (d.seg_off & 3u) == 0 && d.seg_off + tab <= pool_len &&
                      (uint64_t)d.seg_len <= pool_len - d.seg_off - tab;
        if (tab_ok) {
            lens = reinterpret_cast<const uint32_t *>(pool + d.seg_off);
            uint64_t sum = 0;
            for (int i = 0; i < nseg; i++) sum += __ldg(lens + i);
            tab_ok = sum == d.seg_len;
            cw_off += tab;
        }
        if (!tab_ok) {
            if (lane == 0) atomicOr(err, TC_DERR_STYLE);
            ok = false;
        }
    }
    const bool coded = ok && numbps > 0 && d.passes > 0;
    const int nstripes = (h + 3) >> 2;

    // clear the state
    for (int i = lane; i < 1 + (nstripes + 2) * kRow; i += 32) B.S[i] = B.G[i] = 0u;
    for (int i = lane; i < nstripes * 8; i += 32) B.P[i] = B.R[i] = 0u;
    for (int i = lane; i < 9 * 8; i += 32) reinterpret_cast<uint32_t *>(B.lab)[i] = 0u;
    B.reset_contexts(lane);
    __syncwarp();

    int type = 0, last_plane = 0;
    uint32_t *ob = reinterpret_cast<uint32_t *>(out) + d.out_off;   // the block's output words
    if (coded) {
        if (Modes && (style & TC_CBLK_STYLE_BYPASS) && d.passes > 10)
            type = decode_block_warp<Modes, Modes, Deep>(B, planes, np, T, pool + cw_off, (int)d.seg_len, w, h, d.orient,
                                                          numbps, d.passes, &last_plane, lane, style, lens, ob, d.out_pitch);
        else
            type = decode_block_warp<Modes, false, Deep>(B, planes, np, T, pool + cw_off, (int)d.seg_len, w, h, d.orient,
                                                          numbps, d.passes, &last_plane, lane, style, lens, ob, d.out_pitch);
    }
    __syncwarp();

    // epilogue: magnitudes gathered from the bit-planes, reconstruction and
    // inverse quantisation, coalesced rows; an ROI magnitude (>= 2^roi) is
    // shifted down by roi (ISO H.1), and so is its count of undecoded planes
    const bool irrev = (d.flags & TC_CBLK_IRREVERSIBLE) != 0;
    const int roi = d.roi_shift < d.mb ? d.roi_shift : 0;
    const int mb_out = d.mb - roi;  // magnitude bits after the ROI shift
    // the decoded bit-planes that are still in the state, after those that moved
    const int nplanes = coded ? numbps - last_plane : 0;
    int held = nplanes;
    while (held > np) held -= np;
    for (int s = 0; s < nstripes; s++) {
        const int rows = min(4, h - 4 * s);
        for (int x = lane; x < w; x += 32) {
            const int word = s * 8 + (x >> 3), sh = 28 - 4 * (x & 7);
            uint32_t gn = 0, sn = 0, pn = 0, m[4] = {0u, 0u, 0u, 0u};
            if (coded) {
                sn = B.S[1 + (s + 1) * kRow + (x >> 3)] >> sh;
                gn = B.G[1 + (s + 1) * kRow + (x >> 3)] >> sh;
                pn = B.P[word] >> sh;
                if (nplanes > held) {
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if (k < rows) m[k] = ob[(uint64_t)(4 * s + k) * d.out_pitch + x];
                }
                gather_planes(m, planes, held, s, x);
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (k >= rows) break;
                char *row = out + 4 * (d.out_off + (uint64_t)(4 * s + k) * d.out_pitch);
                const bool sg = ((sn >> (3 - k)) & 1u) != 0u;
                uint32_t mg = 0, neg = 0, u = 0;
                if (sg) {
                    mg = m[k] << last_plane;
                    neg = (gn >> (3 - k)) & 1u;
                    u = (uint32_t)last_plane;
                    if (type == 1 && !((pn >> (3 - k)) & 1u)) u++;
                    if (roi && (mg >> roi)) {
                        mg >>= roi;
                        u = u > (uint32_t)roi ? u - roi : 0u;
                    }
                }
                if (out_mode == TC_T1_OUT_RAW) {
                    reinterpret_cast<uint32_t *>(row)[x] = sg ? ((mg << (31 - mb_out)) | (neg << 31)) : 0u;
                } else if (irrev) {
                    float v = 0.0f;
                    if (sg) v = ((float)mg + recon_r * (float)(1u << u)) * d.step;
                    reinterpret_cast<float *>(row)[x] = neg ? -v : v;
                } else {
                    int32_t v = 0;
                    if (sg) v = (int32_t)mg + (u ? (int32_t)floorf(recon_r * (float)(1u << u)) : 0);
                    reinterpret_cast<int32_t *>(row)[x] = neg ? -v : v;
                }
            }
        }
    }
    __syncwarp();
}

// The blocks of a launch: up to three slices of the order array, taken one
// after the other (deepest class first).
struct BlockQueue {
    const uint32_t *o0, *o1, *o2;   // nullptr: the blocks 0, 1, ... in order
    int n0, n1, n2;
};

template <bool Modes, bool Deep>
__global__ void __launch_bounds__(32 * (Modes ? kStyledSlots : kMaxSlots), 2)
t1_decode_warp_kernel(const tc_cblk_desc *__restrict__ desc, BlockQueue queue, int ndesc, int slots, int np, int limit,
                      const uint8_t *__restrict__ pool, uint64_t pool_len, char *__restrict__ out, uint64_t out_elems,
                      int out_mode, float recon_r, uint32_t *__restrict__ counter, uint32_t *__restrict__ err)
{
    extern __shared__ __align__(16) unsigned char smem[];
    WarpTables &T = *reinterpret_cast<WarpTables *>(smem);
    build_warp_tables(T);
    __syncthreads();
    // A warp's slot, alternately up and down the SM's four schedulers, so that
    // the first (longest) blocks share theirs with the shortest or with none.
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, slot = (warp & 4) ? warp ^ 3 : warp;
    if (slot >= slots) return;
    const size_t stride = sizeof(BlockState<Deep>) + (size_t)np * kPlaneWords * 4;
    BlockState<Deep> &B = *reinterpret_cast<BlockState<Deep> *>(smem + sizeof(WarpTables) + slot * stride);
    uint32_t *planes = reinterpret_cast<uint32_t *>(&B + 1);
    // The first block of every warp is dealt out over the CTAs, longest first,
    // so that an SM does not start with twelve of the longest (mixed batch of
    // 12 images 6.30 -> 5.49 ms, 3001x2047x3 12-bit lossless 12.98 -> 12.06);
    // then the queue.
    for (bool dealt = true;; dealt = false) {
        int idx = slot * (int)gridDim.x + (int)blockIdx.x;
        if (!dealt) {
            if (lane == 0) idx = slots * (int)gridDim.x + (int)atomicAdd(counter, 1u);
            idx = __shfl_sync(kFull, idx, 0);
        }
        const uint32_t *order = queue.o0;
        if (idx >= queue.n0) {
            idx -= queue.n0;
            order = queue.o1;
            if (idx >= queue.n1) {
                idx -= queue.n1;
                order = queue.o2;
                if (idx >= queue.n2) break;
            }
        }
        const uint32_t bi = order ? order[idx] : (uint32_t)idx;
        process_block_warp<Modes, Deep>(B, planes, np, limit, T, desc, bi, ndesc, pool, pool_len, out, out_elems, out_mode,
                                        recon_r, err, lane);
    }
}

static_assert(sizeof(WarpTables) % 16 == 0 && sizeof(BlockState<false>) % 16 == 0 && sizeof(BlockState<true>) % 16 == 0,
              "state alignment");

struct WarpLaunch {
    int regs = 0;
    int smem_sm = 0;    // shared memory per SM
    int smem_cta = 0;   // the most one CTA can take
};

template <bool Modes, bool Deep>
cudaError_t warp_launch_info(tc_ctx *ctx, WarpLaunch **out)
{
    static WarpLaunch info[64];
    static DeviceFlags ready;
    WarpLaunch &I = info[ctx->device & 63];
    const cudaError_t e = once_per_device(ready, ctx->device, [&] {
        cudaError_t r = cudaDeviceGetAttribute(&I.smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, ctx->device);
        if (r == cudaSuccess)
            r = cudaDeviceGetAttribute(&I.smem_cta, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device);
        if (r == cudaSuccess)
            r = cudaFuncSetAttribute(t1_decode_warp_kernel<Modes, Deep>, cudaFuncAttributeMaxDynamicSharedMemorySize, I.smem_cta);
        cudaFuncAttributes a{};
        if (r == cudaSuccess) r = cudaFuncGetAttributes(&a, t1_decode_warp_kernel<Modes, Deep>);
        I.regs = a.numRegs;
        return r;
    });
    *out = &I;
    return e;
}

}  // namespace

bool t1_warp_deep(const tc_ctx *ctx, int n) { return n < kDeepBlocks * num_sms(ctx->device); }

cudaError_t launch_t1_warp(tc_ctx *ctx, bool styled, const tc_cblk_desc *d_desc, const uint32_t *const order[3],
                           const int n[3], int ndesc, int max_planes,
                           const uint8_t *d_pool, uint64_t pool_len, void *d_out, uint64_t out_elems, int out_mode,
                           float recon_r, int word)
{
    const int total = n[0] + n[1] + n[2], sms = num_sms(ctx->device);
    const bool deep = t1_warp_deep(ctx, total);
    WarpLaunch *I = nullptr;
    cudaError_t e = styled ? warp_launch_info<true, true>(ctx, &I)
                           : (deep ? warp_launch_info<false, true>(ctx, &I) : warp_launch_info<false, false>(ctx, &I));
    if (e != cudaSuccess) return e;
    const BlockQueue q{order[0], order[1], order[2], n[0], n[1], n[2]};
    const size_t state = styled || deep ? sizeof(BlockState<true>) : sizeof(BlockState<false>);
    const size_t plane = kPlaneWords * 4;
    auto smem_of = [&](int slots, int np) { return sizeof(WarpTables) + slots * (state + np * plane); };
    // CTA shape: the most code-blocks resident on an SM (24 for up to 8 bit-planes)
    struct Shape {
        int slots = 1, per_sm = 1, places = 0;
    };
    auto shape_of = [&](int np) {
        Shape best;
        for (int s = 1; s <= (styled ? kStyledSlots : kMaxSlots); s++) {
            const size_t sm = smem_of(s, np);
            if (sm > (size_t)I->smem_cta) break;
            const int threads = 128 * ((s + 3) / 4);
            const int ctas = std::min((int)(I->smem_sm / (sm + 1024)), 65536 / (threads * ((I->regs + 7) & ~7)));
            if (ctas >= 1 && ctas * s >= best.places) best = Shape{s, ctas, ctas * s};
        }
        return best;
    };
    const int each = std::max(1, (total + sms - 1) / sms);
    int np = max_planes;
    Shape shape = shape_of(np);
    if (np > kFewPlanes && shape.places < each) {
        const Shape few = shape_of(kFewPlanes);
        if (few.places > shape.places) {
            shape = few;
            while (smem_of(few.slots, np) > (size_t)I->smem_cta ||
                   (int)(I->smem_sm / (smem_of(few.slots, np) + 1024)) < few.per_sm)
                np--;
        }
    }
    // Blocks that all fit at once are spread evenly over the SMs: with 16 per
    // SM as two CTAs of 8 (1792x1792x3 lossy: 3.3 ms), not as 12 on every SM
    // and a second CTA on some of them (0.6 ms more).
    int slots = shape.slots, per_sm = shape.per_sm;
    if (each < shape.places) {
        per_sm = (each + slots - 1) / slots;
        slots = (each + per_sm - 1) / per_sm;
    }
    const int grid = std::max(1, std::min((total + slots - 1) / slots, per_sm * sms));
    const int threads = 128 * ((slots + 3) / 4);
    uint32_t *words = ctx->d_words;
    auto kernel = styled ? t1_decode_warp_kernel<true, true>
                         : (deep ? t1_decode_warp_kernel<false, true> : t1_decode_warp_kernel<false, false>);
    kernel<<<grid, threads, smem_of(slots, np), ctx->stream>>>(d_desc, q, ndesc, slots, np, max_planes, d_pool, pool_len,
                                                               static_cast<char *>(d_out), out_elems, out_mode, recon_r,
                                                               words + word, words);
    ctx->launches++;
    return cudaGetLastError();
}

}  // namespace tc
