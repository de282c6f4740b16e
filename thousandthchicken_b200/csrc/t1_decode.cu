// t1_decode.cu -- Tier-1 EBCOT/MQ code-block decoder with several blocks per
// warp (tc_ctx_set_t1_group 8 or 16), the class launches of either decoder,
// and the standalone inverse quantiser.
//
// The default, one warp per block (t1_decode_warp.cu), is the faster one
// wherever it was measured; this one stays for callers that ask for lane
// groups.  Replaces the reference g_decode kernel (coefficient_coder.cl:778-819)
// and the dequantiser kernels (quantizer_*_inverse.cl) with persistent launches:
//   * groups of G lanes pull block indices from a device work queue (an atomic
//     counter over a longest-first order);
//   * blocks are split by coded bit-planes (<= 8, <= 16, <= 31) into classes:
//     8-bit magnitudes in shared memory, deeper ones in the block's output
//     words; the classes run as concurrent launches, heaviest first;
//   * the code-block state is one 32-bit flag word per stripe column: the
//     significance of its 3x6 neighbourhood interleaved so that row k's 3x3
//     neighbourhood is (F >> 3k) & 0x1FF, the visited (pi) and refined
//     (sigma') bits of its four rows, and the signs of its six rows (-1..4).
//     (The reference rebuilds a 3x3 window of packed words from global memory
//     at every step, coefficient_coder.cl:271-298.)
//   * a group's lanes run the decoder alike; at every stripe they find
//     the candidate columns of the pass with __ballot_sync and the serial loop
//     visits only those;
//   * the pass loop honours the coding-pass count (defect D3 fixed) and
//     updates the state it reads (defects D1/D2 fixed); every codeword byte is
//     consumed (defect D22 fixed) and one-column blocks stay in bounds (D23);
//   * the epilogue writes the block out coalesced with the inverse quantiser
//     fused in (ISO E.1, reconstruction point r).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "t1_common.cuh"
#include "tc_internal.cuh"

namespace tc {
namespace {

#ifndef TC_T1_BLOCKS8
#define TC_T1_BLOCKS8 12
#endif
constexpr int kBlocks8 = TC_T1_BLOCKS8;  // code-blocks per CTA of the 8-bit class

// Blocks of more than 8 coded bit-planes keep their magnitude bits in their
// own output words instead of shared memory, which keeps their state as small
// as an 8-bit block's.
template <typename MagT>
constexpr bool kOutMag = sizeof(MagT) > 1;

template <typename MagT>
struct WarpState {
    uint32_t F[kMaxStripes * 64];          // flag word per stripe column (with signs, bits 26-31)
    uint32_t ctx[20];                      // packed probability state per context
    uint8_t mrow[64];                      // refinement pass: rows of the stripe to refine
    uint8_t mctx[64];                      // refinement pass: 2-bit context code per row
    MagT mag[kOutMag<MagT> ? 4 : 64 * 64]; // magnitude bits decoded so far
};

// Signs in the decoder's flag word: bit 26 + j holds the sign of row j - 1 of
// the stripe column (j = 0..5, rows -1..4), set when that row becomes
// significant; rows -1 and 4 belong to the stripes above and below.
constexpr int kSignShift = 26;

// Sign-coding index (ISO Table D.3 neighbourhood) of row k of the column at
// F[i], whose flag word is f and 3x3 neighbourhood n9: the signs of the rows
// above and below come from f, those of the left and right neighbours from
// their own words.  Bits: up sign 0, up 1, left sign 2, left 3, right sign 4,
// right 5, down sign 6, down 7.
__device__ __forceinline__ uint32_t dec_sign_index(const uint32_t *F, uint32_t f, uint32_t n9, int i, int k, int c,
                                                   int w)
{
    const uint32_t lf = c > 0 ? F[i - 1] : 0u, rt = c + 1 < w ? F[i + 1] : 0u;
    const int own = kSignShift + 1 + k;  // this row's sign bit in a word of its stripe
    return (n9 & 0xAAu) | ((f >> (own - 1)) & 1u) | (((lf >> own) & 1u) << 2) | (((rt >> own) & 1u) << 4) |
           (((f >> (own + 1)) & 1u) << 6);
}

// Row k of stripe s in column c became significant with sign neg: the flag
// words of the neighbouring columns see its significance, and those of the
// stripes above and below also its sign.  The caller sets the column's own
// significance and sign bits.
__device__ __forceinline__ void dec_mark_significant(uint32_t *F, int s, int k, int c, int w, int nstripes,
                                                     uint32_t neg)
{
    const int i = s * 64 + c;
    if (c > 0) F[i - 1] |= 1u << (3 * k + 5);
    if (c + 1 < w) F[i + 1] |= 1u << (3 * k + 3);
    if (k == 0 && s > 0) {
        const int u = i - 64;
        F[u] |= (1u << 16) | (neg << (kSignShift + 5));
        if (c > 0) F[u - 1] |= 1u << 17;
        if (c + 1 < w) F[u + 1] |= 1u << 15;
    }
    if (k == 3 && s + 1 < nstripes) {
        const int d = i + 64;
        F[d] |= (1u << 1) | (neg << kSignShift);
        if (c > 0) F[d - 1] |= 1u << 2;
        if (c + 1 < w) F[d + 1] |= 1u << 0;
    }
}

// MQ decoder (ISO C.3; bytein/renormd/mqDecode, coefficient_coder.cl:121-252).
// The interval register A is kept scaled by 2^16 so that it lives in the same
// bit positions as C's upper half: the Qe comparison against C, the
// "A < 0x8000" test (sign bit of the scaled A) and the renormalisation shift
// (count of leading zeros) need no extra shifts.  Each context word is an
// entry of Tables::mqd: Qe << 16, the entries of its two successor states
// (after an MPS, after an LPS with the MPS switched where ISO Table C.2 says
// so) and the MPS in bit 0.  The byte after the current one is loaded ahead
// of use.
struct MQ {
    const uint8_t *p;
    int len, bp, ct;
    uint32_t a, c, cur, nxt;
    unsigned group;   // the lanes that decode this block

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
        nxt = byte_at(bp + 1);   // used about nine decisions later: no prefetch needed
    }
    __device__ __forceinline__ void init(const uint8_t *d, int n, unsigned lanes)
    {
        p = d;
        len = n;
        group = lanes;
        bp = 0;
        cur = byte_at(0);
        nxt = byte_at(1);
        c = cur << 16;
        bytein();
        c <<= 7;
        ct -= 7;
        a = 0x80000000u;
    }
    __device__ __forceinline__ void renorm()
    {
        int sh = __clz(a);
        while (sh > ct) {
            a <<= ct;
            c <<= ct;
            sh -= ct;
            bytein();
        }
        a <<= sh;
        c <<= sh;
        ct -= sh;
    }
    // One decision.  The interval arithmetic of ISO C.3.2 (both the MPS and
    // the LPS sub-interval, with the conditional exchange) is done with
    // selects; the one branch left is the renormalisation, which is also
    // where the context's state moves on.  The barrier keeps the group's lanes
    // within a decision of one another: none stores a context or a flag word
    // that another has yet to read as it was.
    __device__ __forceinline__ uint32_t decode(uint32_t *ctx, const uint32_t *tbl, int cx)
    {
        const uint32_t w = ctx[cx];
        __syncwarp(group);
        const uint32_t qs = w & 0xFFFF0000u, mps = w & 1u;
        const uint32_t a1 = a - qs;
        const bool lower = c < qs;   // the code value lies in the Qe sub-interval
        const bool exch = a1 < qs;   // the conditional exchange swaps the symbols
        const uint32_t d = mps ^ (uint32_t)(lower != exch);
        c = lower ? c : c - qs;
        a = lower ? qs : a1;
        if (lower || (int)a1 >= 0) {
            ctx[cx] = tbl[d != mps ? (w >> 7) & 127u : w & 127u];
            renorm();
        }
        return d;
    }
};

// Decode one code-block.  Every lane of the group runs this function alike;
// the lanes split the per-stripe candidate searches between them (lane l owns
// columns l, l + G, ...) and the serial loop visits only candidate
// columns, in scan order.  Returns the last pass type (0 cleanup,
// 1 significance propagation, 2 refinement) and its plane.
template <typename MagT, int G>
__device__ int decode_block(WarpState<MagT> &S, const Tables &T, const uint8_t *seg, int len, int w,
                            int h, int orient, int numbps, int passes, int *last_plane, int lane, unsigned gmask,
                            int gshift, uint32_t *ob, uint32_t pitch)
{
    // magnitude bits: in shared memory, or (deep blocks) in the block's own
    // output words ob (row pitch `pitch`), where lane 0 of the group stores a
    // sample's first bit and ORs refinement bits in with fire-and-forget
    // atomics; the epilogue reads them back
    auto mag_set = [&](int y, int c, uint32_t v) {
        if constexpr (kOutMag<MagT>) {
            if (lane == 0) ob[(size_t)y * pitch + c] = v;
        } else {
            S.mag[y * 64 + c] = (MagT)v;
        }
    };
    auto mag_or = [&](int y, int c, uint32_t v) {
        if constexpr (kOutMag<MagT>) {
            if (lane == 0) atomicOr(ob + (size_t)y * pitch + c, v);
        } else {
            S.mag[y * 64 + c] |= (MagT)v;
        }
    };
    MQ mq;
    mq.init(seg, len, gmask);
    uint32_t *ctx = S.ctx;
    const uint32_t *tbl = T.mqd;
    const uint8_t *zc = T.zc[orient];
    uint32_t *F = S.F;
    const int nstripes = (h + 3) >> 2;
    constexpr int CPL = 64 / G;  // columns per lane
    int type = 0, pass = 0;
    *last_plane = numbps - 1;

    for (int p = numbps - 1; p >= 0; --p) {
        const uint32_t pbit = 1u << p;
        if (p != numbps - 1) {
            // ---- significance propagation pass (ISO D.3.1; SigPropPassFunctor) ----
            for (int s = 0; s < nstripes; s++) {
                const int rows = min(4, h - 4 * s);
                __syncwarp(gmask);
                bool any[CPL];
#pragma unroll
                for (int j = 0; j < CPL; j++) {
                    const int c = lane + G * j;
                    bool a = false;
                    if (c < w) {
                        // bit 3j of g: a significant sample in row j - 1 of
                        // the three columns; bit 3k of the test: row k is not
                        // significant and has a significant neighbour
                        const uint32_t f = F[s * 64 + c];
                        const uint32_t g = (f | (f >> 1) | (f >> 2)) & 0x9249u;
                        a = ((g | (g >> 3) | (g >> 6)) & ~(f >> 4) & (0x249u >> (3 * (4 - rows)))) != 0u;
                    }
                    any[j] = a;
                }
                const unsigned long long cand64 = group_ballot<G>(any, gmask, gshift);
                uint32_t chi = (uint32_t)(cand64 >> 32);  // columns 32-63
#pragma unroll 1
                for (int half = 0; half < 2; half++) {
                    uint32_t cand = half ? chi : (uint32_t)cand64;
                    while (cand) {
                        const int c = 32 * half + __ffs(cand) - 1;
                        cand &= cand - 1;
                        uint32_t f = F[s * 64 + c];
                        for (int k = 0; k < rows; k++) {
                            const uint32_t fk = f >> (3 * k);   // row k's window at bit 0, self at bit 4
                            if (fk & 0x10u) continue;
                            const uint32_t n9 = fk & 0x1FFu;
                            if (!(n9 & 0x1EFu)) continue;
                            f |= pi_bit(k);
                            if (mq.decode(ctx, tbl, zc[n9])) {
                                const uint32_t si = T.sc[dec_sign_index(F, f, n9, s * 64 + c, k, c, w)];
                                const uint32_t neg = (uint32_t)mq.decode(ctx, tbl, si & 15) ^ (si >> 4);
                                f |= self_bit(k) | (neg << (kSignShift + 1 + k));
                                dec_mark_significant(F, s, k, c, w, nstripes, neg);
                                mag_set(4 * s + k, c, pbit);
                                if (c + 1 < w) {  // the next column gained a neighbour
                                    cand |= 2u << (c & 31);
                                    chi |= (uint32_t)(c == 31);
                                }
                            }
                        }
                        // stored unconditionally: a visited column nearly
                        // always had a row coded (its pi bit set)
                        F[s * 64 + c] = f;
                    }
                }
            }
            type = 1;
            *last_plane = p;
            if (++pass >= passes) break;

            // ---- magnitude refinement pass (ISO D.3.3; MagRefPassFunctor) ----
            // Rows to refine and their contexts do not change during the pass:
            // the lanes precompute them for their columns.
            for (int s = 0; s < nstripes; s++) {
                const int rows = min(4, h - 4 * s);
                __syncwarp(gmask);
                bool any[CPL];
#pragma unroll
                for (int j = 0; j < CPL; j++) {
                    const int c = lane + G * j;
                    uint32_t rr = 0, codes = 0;
                    if (c < w) {
                        const uint32_t f = F[s * 64 + c];
                        for (int k = 0; k < rows; k++) {
                            if ((f & self_bit(k)) && !(f & pi_bit(k))) {
                                rr |= 1u << k;
                                const uint32_t code = (f & ref_bit(k)) ? 2u : (((f >> (3 * k)) & 0x1EFu) ? 1u : 0u);
                                codes |= code << (2 * k);
                            }
                        }
                        S.mrow[c] = (uint8_t)rr;
                        S.mctx[c] = (uint8_t)codes;
                        if (rr) F[s * 64 + c] = f | (rr << 22);
                    }
                    any[j] = rr != 0;
                }
                const unsigned long long cand64 = group_ballot<G>(any, gmask, gshift);
                __syncwarp(gmask);
#pragma unroll 1
                for (int half = 0; half < 2; half++) {
                    uint32_t cand = half ? (uint32_t)(cand64 >> 32) : (uint32_t)cand64;
                    while (cand) {
                        const int c = 32 * half + __ffs(cand) - 1;
                        cand &= cand - 1;
                        uint32_t rr = S.mrow[c];
                        const uint32_t codes = S.mctx[c];
                        while (rr) {
                            const int k = __ffs(rr) - 1;
                            rr &= rr - 1;
                            if (mq.decode(ctx, tbl, 14 + ((codes >> (2 * k)) & 3u))) mag_or(4 * s + k, c, pbit);
                        }
                    }
                }
            }
            type = 2;
            if (++pass >= passes) break;
        }

        // ---- cleanup pass (ISO D.3.4; CleanUpPassFunctor) ----
        for (int s = 0; s < nstripes; s++) {
            const int rows = min(4, h - 4 * s);
            const uint32_t rmask = (1u << rows) - 1u;
            __syncwarp(gmask);
            bool any[CPL];
#pragma unroll
            for (int j = 0; j < CPL; j++) {
                const int c = lane + G * j;
                bool a = false;
                if (c < w) {
                    const uint32_t f = F[s * 64 + c];
                    uint32_t done = (f >> 18) & 0xFu;  // pi
#pragma unroll
                    for (int k = 0; k < 4; k++) done |= ((f >> (3 * k + 4)) & 1u) << k;
                    a = (~done & rmask) != 0u;
                }
                any[j] = a;
            }
            const unsigned long long cand64 = group_ballot<G>(any, gmask, gshift);
#pragma unroll 1
            for (int half = 0; half < 2; half++) {
                uint32_t cand = half ? (uint32_t)(cand64 >> 32) : (uint32_t)cand64;
                while (cand) {
                    const int c = 32 * half + __ffs(cand) - 1;
                    cand &= cand - 1;
                    uint32_t f = F[s * 64 + c];
                    const uint32_t f0 = f;
                    int k = 0;
                    if (rows == 4 && (f & kSigMask) == 0u) {
                        // run-length mode: four rows with an all-zero neighbourhood
                        if (!mq.decode(ctx, tbl, 18)) continue;
                        int r = mq.decode(ctx, tbl, 17) << 1;
                        r |= mq.decode(ctx, tbl, 17);
                        const uint32_t si = T.sc[dec_sign_index(F, f, (f >> (3 * r)) & 0x1FFu, s * 64 + c, r, c, w)];
                        const uint32_t neg = (uint32_t)mq.decode(ctx, tbl, si & 15) ^ (si >> 4);
                        f |= self_bit(r) | (neg << (kSignShift + 1 + r));
                        dec_mark_significant(F, s, r, c, w, nstripes, neg);
                        mag_set(4 * s + r, c, pbit);
                        k = r + 1;
                    }
                    for (; k < rows; k++) {
                        if (f & (self_bit(k) | pi_bit(k))) continue;
                        const uint32_t n9 = (f >> (3 * k)) & 0x1FFu;
                        if (mq.decode(ctx, tbl, zc[n9])) {
                            const uint32_t si = T.sc[dec_sign_index(F, f, n9, s * 64 + c, k, c, w)];
                            const uint32_t neg = (uint32_t)mq.decode(ctx, tbl, si & 15) ^ (si >> 4);
                            f |= self_bit(k) | (neg << (kSignShift + 1 + k));
                            dec_mark_significant(F, s, k, c, w, nstripes, neg);
                            mag_set(4 * s + k, c, pbit);
                        }
                    }
                    if (f != f0) F[s * 64 + c] = f;
                }
            }
        }
        type = 0;
        *last_plane = p;
        if (++pass >= passes) break;
        __syncwarp(gmask);
        for (int i = lane; i < nstripes * 64; i += G) F[i] &= ~0x3C0000u;  // clear pi
        __syncwarp(gmask);
    }
    return type;
}

// Lanes per code-block G (16 or 8): a warp splits into 32 / G groups that
// decode different code-blocks (each group runs the serial
// decoder redundantly across its lanes and splits the candidate searches
// between them), so one warp instruction can advance several code-blocks.
// Code-blocks per CTA: the per-CTA label tables are shared by more blocks
// when the block state is small.
template <typename MagT, int G>
struct GroupCfg {
    static constexpr int blocks = sizeof(MagT) == 1 ? kBlocks8 : 4;
    static constexpr int warps = blocks * G / 32 > 0 ? blocks * G / 32 : 1;
};

// Decode code-block `bi` with the state S and write it out (the group's
// lanes, all alike).  MagT bounds the coded bit-planes it accepts.
template <typename MagT, int G>
__device__ __forceinline__ void process_block(WarpState<MagT> &S, const Tables &T, const tc_cblk_desc *__restrict__ desc,
                                              uint32_t bi, int ndesc, const uint8_t *__restrict__ pool,
                                              uint64_t pool_len, char *__restrict__ out, uint64_t out_elems, int out_mode,
                                              float recon_r, uint32_t *__restrict__ err, int gl, unsigned gmask,
                                              int gshift)
{
    if (bi >= (uint32_t)ndesc) {
        if (gl == 0) atomicOr(err, TC_DERR_DESC);
        return;
    }
    const tc_cblk_desc d = desc[bi];
    const int w = d.w, h = d.h;
    const bool geom_ok = w >= 1 && w <= 64 && h >= 1 && h <= 64;
    const int numbps = (int)d.mb - (int)d.zero_bitplanes;
    bool ok = geom_ok && d.mb >= 1 && d.mb <= 31 && d.orient <= 3 && numbps >= 0 &&
              (numbps == 0 || d.passes <= 3 * numbps - 2) && numbps <= (int)(8 * sizeof(MagT));
    const bool pool_ok = d.seg_off <= pool_len && (uint64_t)d.seg_len <= pool_len - d.seg_off;
    if (!geom_ok) {
        if (gl == 0) atomicOr(err, TC_DERR_DESC);
        return;
    }
    // the block's last sample, out_off + (h-1) * out_pitch + w - 1, must lie
    // inside the output; a block that does not is skipped before any write
    if (d.out_off > out_elems || (uint64_t)(h - 1) * d.out_pitch + (uint64_t)w > out_elems - d.out_off) {
        if (gl == 0) atomicOr(err, TC_DERR_OUT);
        return;
    }
    if (!ok || !pool_ok) {
        if (gl == 0) atomicOr(err, ok ? TC_DERR_POOL : TC_DERR_DESC);
        ok = false;
    }
    // styled blocks run in t1_decode_warp.cu's styled launch
    if (d.style & kStyleDecodeBits) {
        if (gl == 0) atomicOr(err, TC_DERR_STYLE);
        ok = false;
    }
    const bool coded = ok && numbps > 0 && d.passes > 0;
    const int nstripes = (h + 3) >> 2;

    // clear the state (the group's lanes)
    for (int i = gl; i < nstripes * 64; i += G) S.F[i] = 0u;
    for (int i = gl; i < 19; i += G) {
        const int st = i == 0 ? 4 : (i == 17 ? 46 : (i == 18 ? 3 : 0));
        S.ctx[i] = T.mqd[2 * st];   // MPS 0
    }
    __syncwarp(gmask);

    int type = 0, last_plane = 0;
    uint32_t *ob = reinterpret_cast<uint32_t *>(out) + d.out_off;   // the block's output words
    if (coded)
        type = decode_block<MagT, G>(S, T, pool + d.seg_off, (int)d.seg_len, w, h, d.orient, numbps, d.passes, &last_plane,
                                     gl, gmask, gshift, ob, d.out_pitch);
    if constexpr (kOutMag<MagT>) __threadfence();   // lane 0's magnitude writes, before the group reads them
    __syncwarp(gmask);

    // epilogue: reconstruction + inverse quantisation, coalesced rows; an
    // ROI magnitude (>= 2^roi) is shifted down by roi (ISO H.1), and so is
    // its count of undecoded planes
    const bool irrev = (d.flags & TC_CBLK_IRREVERSIBLE) != 0;
    const int roi = d.roi_shift < d.mb ? d.roi_shift : 0;
    const int mb_out = d.mb - roi;  // magnitude bits after the ROI shift
    for (int y = 0; y < h; y++) {
        char *row = out + 4 * (d.out_off + (uint64_t)y * d.out_pitch);
        const int s = y >> 2, k = y & 3;
        for (int x = gl; x < w; x += G) {
            const uint32_t f = coded ? S.F[s * 64 + x] : 0u;
            const bool sg = (f & self_bit(k)) != 0u;
            uint32_t mg = 0, neg = 0, u = 0;
            if (sg) {
                if constexpr (kOutMag<MagT>)
                    mg = __ldcg(reinterpret_cast<const uint32_t *>(row) + x);
                else
                    mg = (uint32_t)S.mag[y * 64 + x];
                neg = (f >> (kSignShift + 1 + k)) & 1u;
                u = (uint32_t)last_plane;
                if (type == 1 && !(f & pi_bit(k))) u++;
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
    __syncwarp(gmask);
}

// Persistent Tier-1 launch over one magnitude class.
template <typename MagT, int G>
__global__ void __launch_bounds__(32 * GroupCfg<MagT, G>::warps, 1)
t1_decode_kernel(const tc_cblk_desc *__restrict__ desc, const uint32_t *__restrict__ order, int n, int ndesc,
                 const uint8_t *__restrict__ pool, uint64_t pool_len, char *__restrict__ out, uint64_t out_elems,
                 int out_mode, float recon_r, uint32_t *__restrict__ counter, uint32_t *__restrict__ err)
{
    extern __shared__ __align__(16) unsigned char smem[];
    Tables &T = *reinterpret_cast<Tables *>(smem);
    WarpState<MagT> *states = reinterpret_cast<WarpState<MagT> *>(smem + ((sizeof(Tables) + 15) & ~size_t(15)));
    build_tables(T);
    __syncthreads();

    const int wl = threadIdx.x & 31;             // lane in the warp
    const int gidx = wl / G, gl = wl % G;         // group in the warp, lane in the group
    const int gshift = gidx * G;
    const unsigned gmask = ((1u << G) - 1u) << gshift;
    const int slot = (threadIdx.x >> 5) * (32 / G) + gidx;
    WarpState<MagT> &S = states[slot];
    for (;;) {
        int idx = 0;
        if (gl == 0) idx = (int)atomicAdd(counter, 1u);
        idx = __shfl_sync(gmask, idx, gshift);
        if (idx >= n) break;
        const uint32_t bi = order ? order[idx] : (uint32_t)idx;
        process_block<MagT, G>(S, T, desc, bi, ndesc, pool, pool_len, out, out_elems, out_mode, recon_r, err, gl, gmask,
                               gshift);
    }
}

// Standalone inverse quantiser over raw sign-magnitude words.
__global__ void dequant_raw_kernel(const tc_cblk_desc *__restrict__ desc, int n,
                                   const uint32_t *__restrict__ raw, char *__restrict__ out, uint64_t elems,
                                   float recon_r, uint32_t *words, bool base16)
{
    const int b = blockIdx.x;
    if (b >= n) return;
    const tc_cblk_desc d = desc[b];
    if (d.w < 1 || d.w > 64 || d.h < 1 || d.h > 64 || d.mb < 1 || d.mb > 31) {
        if (threadIdx.x == 0) atomicOr(&words[0], TC_DERR_DESC);
        return;
    }
    // raw words and output share the block's place: both hold `elems`
    if (d.out_off > elems || (uint64_t)(d.h - 1) * d.out_pitch + (uint64_t)d.w > elems - d.out_off) {
        if (threadIdx.x == 0) atomicOr(&words[0], TC_DERR_OUT);
        return;
    }
    const int numbps = (int)d.mb - (int)d.zero_bitplanes;
    const int roi = d.roi_shift < d.mb ? d.roi_shift : 0;
    const int mb = d.mb - roi;  // magnitude bits of the raw words
    // Decoded planes from the pass count: the last pass ran on plane p_last
    // (counted in the ROI-shifted domain for an ROI block).
    int u = 0;
    if (numbps > 0 && d.passes > 0) {
        const int p_last = numbps - 1 - (d.passes + 1) / 3 - roi;
        u = p_last < 0 ? 0 : p_last;
    }
    const bool irrev = (d.flags & TC_CBLK_IRREVERSIBLE) != 0;
    const float fr = recon_r * (float)(1u << u);
    const int32_t ir = u ? (int32_t)floorf(fr) : 0;
    // 16 threads per row, four consecutive coefficients each (one 16-byte
    // load and store when the block's rows are aligned): whole rows, no
    // index division
    auto one = [&](uint32_t r) -> uint32_t {
        const uint32_t mg = (r & 0x7FFFFFFFu) >> (31 - mb);
        const bool neg = (r >> 31) != 0;
        if (irrev) {
            const float v = mg ? ((float)mg + fr) * d.step : 0.0f;
            return __float_as_uint(neg ? -v : v);
        }
        const int32_t v = mg ? (int32_t)mg + ir : 0;
        return (uint32_t)(neg ? -v : v);
    };
    const int x = 4 * (threadIdx.x & 15);
    if (x >= d.w) return;
    const bool vec = base16 && ((d.out_off | (uint64_t)d.out_pitch) & 3u) == 0 && x + 4 <= d.w;
    uint32_t *dst = reinterpret_cast<uint32_t *>(out);
    for (int y = threadIdx.x >> 4; y < d.h; y += blockDim.x >> 4) {
        const uint64_t o = d.out_off + (uint64_t)y * d.out_pitch + x;
        if (vec) {
            const uint4 r = *reinterpret_cast<const uint4 *>(raw + o);
            *reinterpret_cast<uint4 *>(dst + o) = make_uint4(one(r.x), one(r.y), one(r.z), one(r.w));
        } else {
            for (int j = 0; j < 4 && x + j < d.w; j++) dst[o + j] = one(raw[o + j]);
        }
    }
}

struct LaunchCfg {
    int per_sm = 1;    // resident CTAs per SM
    int per_cta = 4;   // code-blocks in flight per CTA
    size_t smem = 0;   // dynamic shared memory per CTA
};

// One class launch: a persistent grid pulling the class's blocks from its
// work counter d_words[slot] (zeroed beforehand).
template <typename MagT, int G>
cudaError_t launch_class(tc_ctx *ctx, cudaStream_t stream, const tc_cblk_desc *d_desc, const uint32_t *d_order, int n,
                         int ndesc, const uint8_t *d_pool, uint64_t pool_len, void *d_out, uint64_t out_elems,
                         int out_mode, float recon_r, int slot)
{
    constexpr int kWarps = GroupCfg<MagT, G>::warps;
    static LaunchCfg cfg[64];
    static DeviceFlags ready;
    LaunchCfg &C = cfg[ctx->device & 63];
    const cudaError_t e = once_per_device(ready, ctx->device, [&] {
        C.smem = ((sizeof(Tables) + 15) & ~size_t(15)) + kWarps * (32 / G) * sizeof(WarpState<MagT>);
        C.per_cta = kWarps * (32 / G);
        cudaError_t r = cudaFuncSetAttribute(t1_decode_kernel<MagT, G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)C.smem);
        if (r == cudaSuccess)
            r = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&C.per_sm, t1_decode_kernel<MagT, G>, 32 * kWarps, C.smem);
        if (C.per_sm < 1) C.per_sm = 1;
        return r;
    });
    if (e != cudaSuccess) return e;
    const int grid = std::max(1, std::min((n + C.per_cta - 1) / C.per_cta, C.per_sm * num_sms(ctx->device)));
    t1_decode_kernel<MagT, G><<<grid, 32 * kWarps, C.smem, stream>>>(d_desc, d_order, n, ndesc, d_pool, pool_len,
                                                                     static_cast<char *>(d_out), out_elems, out_mode,
                                                                     recon_r, ctx->d_words + slot, ctx->d_words);
    ctx->launches++;
    return cudaGetLastError();
}

template <typename MagT>
cudaError_t launch_class_g(tc_ctx *ctx, cudaStream_t stream, const tc_cblk_desc *d_desc, const uint32_t *d_order,
                           int n, int ndesc, const uint8_t *d_pool, uint64_t pool_len, void *d_out, uint64_t out_elems, int out_mode,
                           float recon_r, int slot)
{
    if (ctx->t1_group == 8)
        return launch_class<MagT, 8>(ctx, stream, d_desc, d_order, n, ndesc, d_pool, pool_len, d_out, out_elems, out_mode,
                                     recon_r, slot);
    return launch_class<MagT, 16>(ctx, stream, d_desc, d_order, n, ndesc, d_pool, pool_len, d_out, out_elems, out_mode,
                                  recon_r, slot);
}

}  // namespace

cudaError_t launch_t1_decode(tc_ctx *ctx, const tc_cblk_desc *d_desc, const uint32_t *d_order, int n,
                             const uint8_t *d_pool, uint64_t pool_len, void *d_out, uint64_t out_elems, int out_mode, float recon_r,
                             int max_bitplanes)
{
    if (out_mode & TC_T1_STYLED) {
        const int s[3] = {max_bitplanes <= 8 ? n : 0, max_bitplanes > 8 && max_bitplanes <= 16 ? n : 0,
                          max_bitplanes > 16 ? n : 0};
        return launch_t1_classes(ctx, d_desc, d_order, n, 0, 0, 0, d_pool, pool_len, d_out, out_elems, out_mode & ~TC_T1_STYLED,
                                 recon_r, s);
    }
    return launch_t1_classes(ctx, d_desc, d_order, n, max_bitplanes <= 8 ? n : 0,
                             max_bitplanes > 8 && max_bitplanes <= 16 ? n : 0, max_bitplanes > 16 ? n : 0, d_pool,
                             pool_len, d_out, out_elems, out_mode, recon_r);
}

// Classes: blocks of <= 8, <= 16 and <= 31 coded bit-planes, in that order in
// d_order (each slice longest first), then styled blocks in the same three.
// One warp per block takes the three classes in one launch, the deepest (the
// longest chains) first, whose state has room for the deepest block (planes, or
// the class's bound) or less, and the styled ones in a launch of their own
// before it.
// With lane groups the plain classes run as concurrent launches, the 32- and
// 16-bit ones on side streams; an 8-bit class at most half the size of the
// 16-bit class joins its launch (a wider state decodes any narrower block).
cudaError_t launch_t1_classes(tc_ctx *ctx, const tc_cblk_desc *d_desc, const uint32_t *d_order, int ndesc,
                              int n8, int n16, int n32, const uint8_t *d_pool, uint64_t pool_len, void *d_out,
                              uint64_t out_elems, int out_mode, float recon_r, const int *nstyled, const int *planes)
{
    const int ns8 = nstyled ? nstyled[0] : 0, ns16 = nstyled ? nstyled[1] : 0, ns32 = nstyled ? nstyled[2] : 0;
    if (n8 + n16 + n32 + ns8 + ns16 + ns32 == 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(ctx->d_words + 1, 0, 6 * sizeof(uint32_t), ctx->stream);
    if (e != cudaSuccess) return e;
    auto warp_launch = [&](bool styled, const uint32_t *o, int a8, int a16, int a32, int word) {
        const uint32_t *orders[3] = {o ? o + a8 + a16 : nullptr, o ? o + a8 : nullptr, o};
        const int counts[3] = {a32, a16, a8};
        const int np = planes ? planes[styled] : (a32 > 0 ? 31 : (a16 > 0 ? 16 : 8));
        return launch_t1_warp(ctx, styled, d_desc, orders, counts, ndesc, np, d_pool, pool_len, d_out, out_elems, out_mode,
                              recon_r, word);
    };
    if (ns8 + ns16 + ns32 > 0) {
        e = warp_launch(true, d_order ? d_order + n8 + n16 + n32 : nullptr, ns8, ns16, ns32, 4);
        if (e != cudaSuccess || n8 + n16 + n32 == 0) return e;
    }
    if (ctx->t1_group == 32) return warp_launch(false, d_order, n8, n16, n32, 1);

    const uint32_t *o16 = d_order ? d_order + n8 : nullptr;
    const uint32_t *o32 = d_order ? d_order + n8 + n16 : nullptr;
    if (n8 > 0 && n16 > 0 && 2 * n8 <= n16 && d_order) {
        o16 = d_order;  // the 8-bit slice directly precedes the 16-bit one
        n16 += n8;
        n8 = 0;
    }
    const int nlaunch = (n8 > 0) + (n16 > 0) + (n32 > 0);
    cudaStream_t s8 = ctx->stream, s16 = ctx->stream, s32 = ctx->stream;
    if (nlaunch > 1) {
        // Fork: the heavier classes run on side streams, concurrently with
        // the 8-bit class on the context's stream, and are joined after it.
        if ((e = ensure_side_streams(ctx)) != cudaSuccess) return e;
        if ((e = cudaEventRecord(ctx->ev_fork, ctx->stream)) != cudaSuccess) return e;
        for (int i = 0; i < 2; i++)
            if ((e = cudaStreamWaitEvent(ctx->side[i], ctx->ev_fork, 0)) != cudaSuccess) return e;
        s32 = ctx->side[0];
        s16 = ctx->side[1];
    }
    if (n32 > 0)
        e = launch_class_g<uint32_t>(ctx, s32, d_desc, o32, n32, ndesc, d_pool, pool_len, d_out, out_elems, out_mode,
                                     recon_r, 3);
    if (e == cudaSuccess && n16 > 0)
        e = launch_class_g<uint16_t>(ctx, s16, d_desc, o16, n16, ndesc, d_pool, pool_len, d_out, out_elems, out_mode,
                                     recon_r, 2);
    if (e == cudaSuccess && n8 > 0)
        e = launch_class_g<uint8_t>(ctx, s8, d_desc, d_order, n8, ndesc, d_pool, pool_len, d_out, out_elems, out_mode,
                                    recon_r, 1);
    if (nlaunch > 1) {
        for (int i = 0; i < 2; i++) {
            cudaError_t e2 = cudaEventRecord(ctx->ev_join[i], ctx->side[i]);
            if (e2 == cudaSuccess) e2 = cudaStreamWaitEvent(ctx->stream, ctx->ev_join[i], 0);
            if (e == cudaSuccess) e = e2;
        }
    }
    return e;
}

cudaError_t launch_dequant_raw(tc_ctx *ctx, const tc_cblk_desc *d_desc, int n, const uint32_t *d_raw,
                               void *d_out, uint64_t elems, float recon_r)
{
    if (n <= 0) return cudaSuccess;
    const bool base16 = ((reinterpret_cast<uintptr_t>(d_raw) | reinterpret_cast<uintptr_t>(d_out)) & 15) == 0;
    dequant_raw_kernel<<<n, 256, 0, ctx->stream>>>(d_desc, n, d_raw, static_cast<char *>(d_out), elems, recon_r,
                                                   ctx->d_words, base16);
    ctx->launches++;
    return cudaGetLastError();
}

}  // namespace tc
