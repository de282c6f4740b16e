// t1_encode.cu -- Tier-1 EBCOT/MQ code-block encoder for sm_100a.
//
// The reference has no Tier-1 encoder; this is the GPU half of the forward
// pipeline (forward colour transform and DWT in color.cu / dwt.cu).  It
// produces, block for block, the same codeword as the project's host encoder
// (t1_encode_block in j2k_host.cpp): all coding passes, or the first
// max_passes of them, MQ termination by the FLUSH procedure of ISO C.2.9.
//
// One warp per code-block.  The samples are known, so only the MQ coder is
// serial: for every stripe of a pass the lanes work out in parallel which
// samples the pass codes, their contexts and signs, and put the decisions
// (context label, bit) into a list in scan order; the warp then runs the list
// through the MQ coder, all lanes alike.
//   * a lane holds two columns of the block (c and c + 32) as 64-bit masks in
//     registers: significance, signs, the plane's bits, visited, refined; its
//     neighbours' rows come by shuffles;
//   * in the significance propagation pass a sample that becomes significant
//     makes its later neighbours candidates: the lanes iterate this to its
//     fixed point, columns to the left first seen as they will be by then;
//   * a sample's context sees the column to the left and the row above it as
//     this pass leaves them, the rest as it found them.
// The coder is bound by the decisions' chain when blocks are few and by issue
// slots when they fill the GPU; the list takes the context search that ran
// between decisions off both (64x64 blocks of 9 bit-planes: 48 of them 8.4 ->
// 3.39 ms, 3,072 11.8 -> 7.4 ms, 12,288 42.2 -> 23.1 ms).  80 registers, six
// CTAs (24 warps) per SM: at 96 and five, 768 CTAs left a second wave of 28
// (8.1 ms); at 64 registers every block took 37% longer.
#include <cuda_runtime.h>

#include <cmath>

#include "t1_common.cuh"
#include "tc_internal.cuh"

namespace tc {
namespace {

constexpr int kEncWarps = 4;   // code-blocks per CTA
constexpr int kSymRun = 72, kSymUni = 68;   // labels are kept as byte offsets (4 x label)

// Label and probability tables of a CTA.
struct EncTables {
    uint8_t zc[4][256];   // zero-coding label x 4: left rows k-1..k+1 in bits 0-2, right 3-5, up 6, down 7
    uint8_t sc[256];      // sign label x 4 | XOR bit: significance of left, right, up, down in bits 0-3, signs 4-7
    uint2 next[94];       // context words after an MPS and after an LPS, by 2 x state + MPS
};

// A block's decisions of one stripe and pass (at most ten a column) and its
// context words (Qe << 16 | (2 x state + MPS) << 3).
struct EncState {
    uint8_t sym[64 * 10 + 16];   // label x 4 | decision
    uint32_t ctx[20];
};

__device__ __forceinline__ uint32_t enc_word(int state, int mps)
{
    return ((uint32_t)c_qe[state] << 16) | (uint32_t)((2 * state + mps) << 3);
}

__device__ void build_enc_tables(EncTables &t)
{
    for (int i = threadIdx.x; i < 94; i += blockDim.x) {
        const int st = i >> 1, mps = i & 1, sw = st == 0 || st == 6 || st == 14;
        t.next[i] = make_uint2(enc_word(c_nmps[st], mps), enc_word(c_nlps[st], mps ^ sw));
    }
    for (int i = threadIdx.x; i < 4 * 256; i += blockDim.x) {
        const int b = i & 255;
        auto bit = [&](int k) { return (b >> k) & 1; };
        t.zc[i >> 8][b] = (uint8_t)(4 * zc_label(i >> 8, bit(1) + bit(4), bit(6) + bit(7),
                                                 bit(0) + bit(2) + bit(3) + bit(5)));
    }
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {   // ISO Tables D.2/D.3
        auto ctb = [&](int k) { return (i >> k) & 1 ? ((i >> (4 + k)) & 1 ? -1 : 1) : 0; };
        int hc = ctb(0) + ctb(1), vc = ctb(2) + ctb(3);
        hc = hc > 1 ? 1 : (hc < -1 ? -1 : hc);
        vc = vc > 1 ? 1 : (vc < -1 ? -1 : vc);
        const int cx = hc == 0 ? (vc == 0 ? 9 : 10) : 12 + hc * vc;
        const int xr = hc == 0 ? vc < 0 : hc < 0;
        t.sc[i] = (uint8_t)((4 * cx) | xr);
    }
}

// A sample's bits as they lie in the input, and their magnitude: the int32
// input, or the float input quantised floor(|v| / step) (ISO E.2 deadzone).
__device__ __forceinline__ uint32_t sample(const tc_t1_enc_desc &d, const void *in, int x, int y)
{
    return __ldg(static_cast<const uint32_t *>(in) + (d.in_off + (size_t)y * d.in_pitch + x));
}
__device__ __forceinline__ uint32_t magnitude(const tc_t1_enc_desc &d, uint32_t bits)
{
    if (d.flags & TC_CBLK_IRREVERSIBLE) return (uint32_t)floorf(fabsf(__uint_as_float(bits)) * d.inv_step);
    const int32_t v = (int32_t)bits;
    return (uint32_t)(v < 0 ? -(int64_t)v : v);
}

// MQ encoder (ISO C.2.1-C.2.9).  A is 16 bits wide as in the standard.  The last byte emitted (B of the
// standard) stays in a register until the next one is emitted, since a
// carry can still increment it; bytes before it are final.
struct MQEnc {
    uint8_t *out;
    uint32_t cap, n;   // n: bytes emitted so far (B is byte n - 1; n == 0: B is the byte before the codeword)
    uint32_t a, c, b;
    int ct;
    bool writer, overflow;

    __device__ __forceinline__ void init(uint8_t *o, uint32_t capacity, bool w)
    {
        out = o;
        cap = capacity;
        n = 0;
        a = 0x8000u;
        c = 0;
        b = 0;
        ct = 12;
        writer = w;
        overflow = false;
    }
    __device__ __forceinline__ void put(uint32_t v)
    {
        if (n >= 1) {
            if (n - 1 < cap) {
                if (writer) out[n - 1] = (uint8_t)b;
            } else {
                overflow = true;
            }
        }
        n++;
        b = v & 0xFFu;
    }
    __device__ __forceinline__ void byteout()
    {
        if (b == 0xFFu) {
            put(c >> 20);
            c &= 0xFFFFFu;
            ct = 7;
        } else if (c < 0x8000000u) {
            put(c >> 19);
            c &= 0x7FFFFu;
            ct = 8;
        } else {
            b++;
            if (b == 0xFFu) {
                c &= 0x7FFFFFFu;
                put(c >> 20);
                c &= 0xFFFFFu;
                ct = 7;
            } else {
                put(c >> 19);
                c &= 0x7FFFFu;
                ct = 8;
            }
        }
    }
    // One decision of the context whose word is w; returns its word afterwards.
    __device__ __forceinline__ uint32_t encode(const EncTables &T, uint32_t w, uint32_t d)
    {
        const uint2 succ = *reinterpret_cast<const uint2 *>(reinterpret_cast<const char *>(T.next) + (w & 0x3F8u));
        const uint32_t qe = w >> 16, a1 = a - qe;
        const bool lps = d != ((w >> 3) & 1u);
        const bool upper = lps == (a1 < qe);   // the upper sub-interval (conditional exchange included)
        a = upper ? a1 : qe;
        c = upper ? c + qe : c;
        int sh = __clz(a) - 16;
        const uint32_t nx = sh ? (lps ? succ.y : succ.x) : w;
        a <<= sh;
        while (sh >= ct) {
            c <<= ct;
            sh -= ct;
            byteout();
        }
        c <<= sh;
        ct -= sh;
        return nx;
    }
    // FLUSH (ISO C.2.9); returns the codeword length (a final 0xFF dropped).
    __device__ __forceinline__ uint32_t flush()
    {
        const uint32_t tempc = c + a;
        c |= 0xFFFFu;
        if (c >= tempc) c -= 0x8000u;
        c <<= ct;
        byteout();
        c <<= ct;
        byteout();
        const uint32_t len = b == 0xFFu ? n - 1 : n;
        if (n >= 1 && n - 1 < len) {  // the last byte is part of the codeword
            if (n - 1 < cap) {
                if (writer) out[n - 1] = (uint8_t)b;
            } else {
                overflow = true;
            }
        }
        return len;
    }
};

constexpr unsigned kAll = 0xffffffffu;

// The first `limit` coding passes of a block.  neg: the lane's columns' signs.
__device__ void encode_block(EncState &S, const EncTables &T, MQEnc &mq, const tc_t1_enc_desc &d, const void *in,
                             const unsigned long long (&neg)[2], int numbps, int limit, int lane)
{
    const int w = d.w, h = d.h, nstripes = (h + 3) >> 2;
    const uint8_t *zc = T.zc[d.orient];
    char *ctxb = reinterpret_cast<char *>(S.ctx);
    auto ctx_at = [&](uint32_t sym) -> uint32_t { return *reinterpret_cast<const uint32_t *>(ctxb + (sym & 0x7Cu)); };
    // all lanes run the list; none stores a word that another has yet to read
    auto store_ctx = [&](uint32_t sym, uint32_t word) {
        __syncwarp();
        *reinterpret_cast<uint32_t *>(ctxb + (sym & 0x7Cu)) = word;
    };
    unsigned long long sig[2] = {0ull, 0ull}, pi[2] = {0ull, 0ull}, ref[2] = {0ull, 0ull}, bits[2] = {0ull, 0ull};
    // six rows, -1..4, of stripe s of a column
    auto window = [](unsigned long long m, int s) -> uint32_t {
        return (uint32_t)(s ? m >> (4 * s - 1) : m << 1) & 63u;
    };
    auto spread3 = [](uint32_t x) -> uint32_t { return (x | (x >> 1) | (x >> 2)) & 15u; };   // rows k-1..k+1 of a window

    // the list through the MQ coder
    auto run_list = [&](int n) {
        if (n == 0) return;
        __syncwarp();
        uint32_t s0 = S.sym[0];
        uint32_t cw = ctx_at(s0);
        for (int i = 1;; i++) {
            const uint32_t s1 = S.sym[i];   // one past the end for the last
            const uint32_t cn = ctx_at(s1);
            const uint32_t nx = mq.encode(T, cw, s0 & 1u);
            store_ctx(s0, nx);
            if (i >= n) break;
            cw = ((s0 ^ s1) & 0x7Cu) ? cn : nx;
            s0 = s1;
        }
        __syncwarp();
    };

    int p = numbps - 1, type = 0;   // 0 cleanup, 1 significance propagation, 2 refinement
    for (int done = 0; done < limit; done++) {
        if (type == 1 || done == 0) {
            // this bit-plane's bits
#pragma unroll
            for (int j = 0; j < 2; j++) {
                unsigned long long m = 0;
                if (lane + 32 * j < w) {
#pragma unroll 8
                    for (int y = 0; y < h; y++)
                        m |= (unsigned long long)((magnitude(d, sample(d, in, lane + 32 * j, y)) >> p) & 1u) << y;
                }
                bits[j] = m;
                pi[j] = 0ull;
            }
        }
        for (int s = 0; s < nstripes; s++) {
            const int rows = min(4, h - 4 * s);
            const uint32_t rowmask = (1u << rows) - 1u;
            // windows of the lane's columns: significance in bits 0-5, signs in 6-11
            const uint32_t v0 = window(sig[0], s) | (window(neg[0], s) << 6);
            const uint32_t v1 = window(sig[1], s) | (window(neg[1], s) << 6);
            int n = 0;                 // decisions in the list
            uint32_t carry = 0;        // column 31's new samples, for column 32
#pragma unroll
            for (int j = 0; j < 2; j++) {
                if (32 * j >= w) break;
                const uint32_t v = j ? v1 : v0;
                uint32_t lv = __shfl_up_sync(kAll, v, 1), rv = __shfl_down_sync(kAll, v, 1);
                const uint32_t edge = j ? __shfl_sync(kAll, v0, 31) : __shfl_sync(kAll, v1, 0);
                if (lane == 0) lv = j ? edge : 0u;
                if (lane == 31) rv = j ? 0u : edge;
                const uint32_t own = v & 63u, right = rv & 63u;
                const uint32_t here = (own >> 1) & 15u;                       // the stripe's significant samples
                const uint32_t b = (uint32_t)(bits[j] >> (4 * s)) & 15u;
                const uint32_t mask = lane + 32 * j < w ? rowmask : 0u;
                const uint32_t near = spread3(lv & 63u) | spread3(right) | ((own | (own >> 2)) & 15u);

                if (type == 2) {
                    // ---- magnitude refinement (ISO D.3.3) ----
                    const uint32_t m = here & ~(uint32_t)(pi[j] >> (4 * s)) & mask;
                    const uint32_t r = (uint32_t)(ref[j] >> (4 * s)) & 15u;
                    int at = __popc(m), sum = at;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int u = __shfl_up_sync(kAll, sum, o);
                        if (lane >= o) sum += u;
                    }
                    at = n + sum - at;
                    n += __shfl_sync(kAll, sum, 31);
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if ((m >> k) & 1u)
                            S.sym[at++] = (uint8_t)(((r >> k) & 1u ? 64u : ((near >> k) & 1u ? 60u : 56u)) | ((b >> k) & 1u));
                    ref[j] |= (unsigned long long)m << (4 * s);
                    continue;
                }

                const uint32_t avail = ~here & mask;
                uint32_t m, left_new;   // samples coded; the left column's new ones
                if (type == 1) {
                    // ---- significance propagation (ISO D.3.1) ----
                    m = avail & near;
                    left_new = lane == 0 ? carry : 0u;
                    for (;;) {
                        m |= avail & (left_new | (left_new << 1) | (left_new >> 1));
                        m |= avail & ((m & b) << 1);
                        m |= avail & ((m & b) << 1);
                        m |= avail & ((m & b) << 1);
                        const uint32_t l = __shfl_up_sync(kAll, m & b, 1);
                        const uint32_t now = lane == 0 ? carry : l;
                        const bool changed = now != left_new;
                        left_new = now;
                        if (!__any_sync(kAll, changed)) break;
                    }
                    pi[j] |= (unsigned long long)m << (4 * s);
                } else {
                    // ---- cleanup (ISO D.3.4) ----
                    m = avail & ~(uint32_t)(pi[j] >> (4 * s));
                    const uint32_t l = __shfl_up_sync(kAll, m & b, 1);
                    left_new = lane == 0 ? carry : l;
                }
                const uint32_t fresh = m & b;
                carry = __shfl_sync(kAll, fresh, 31);
                if (type == 1 && !__any_sync(kAll, m != 0u)) continue;
                const uint32_t left = (lv & 63u) | (left_new << 1), up = own | (fresh << 1);
                // run-length column: four rows, nothing significant around
                const bool run = type == 0 && rows == 4 && mask && (own | left | right) == 0u;
                const int first = run ? (b ? __ffs((int)b) - 1 : 4) : -1;   // its first significant row
                int at = run ? (b ? 4 + 3 - first + __popc(b >> (first + 1)) : 1) : __popc(m) + __popc(fresh), sum = at;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(kAll, sum, o);
                    if (lane >= o) sum += u;
                }
                at = n + sum - at;
                n += __shfl_sync(kAll, sum, 31);
                if (run) {
                    S.sym[at++] = (uint8_t)(kSymRun | (b != 0u));
                    if (b) {
                        S.sym[at++] = (uint8_t)(kSymUni | (first >> 1));
                        S.sym[at++] = (uint8_t)(kSymUni | (first & 1));
                    }
                }
                const uint32_t ln = lv >> 6, rn = rv >> 6, on = v >> 6;   // signs
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (((m >> k) & 1u) && k > first)
                        S.sym[at++] = (uint8_t)(zc[((left >> k) & 7u) | (((right >> k) & 7u) << 3) | (((up >> k) & 1u) << 6) |
                                                   (((own >> (k + 2)) & 1u) << 7)] |
                                                ((b >> k) & 1u));
                    if (((fresh >> k) & 1u) && k >= first) {
                        const uint32_t i = ((left >> (k + 1)) & 1u) | (((right >> (k + 1)) & 1u) << 1) |
                                           (((up >> k) & 1u) << 2) | (((own >> (k + 2)) & 1u) << 3) |
                                           (((ln >> (k + 1)) & 1u) << 4) | (((rn >> (k + 1)) & 1u) << 5) |
                                           (((on >> k) & 1u) << 6) | (((on >> (k + 2)) & 1u) << 7);
                        S.sym[at++] = (uint8_t)(T.sc[i] ^ ((on >> (k + 1)) & 1u));
                    }
                }
                sig[j] |= (unsigned long long)fresh << (4 * s);
            }
            run_list(n);
        }
        if (type == 0) --p;
        type = type == 0 ? 1 : (type == 1 ? 2 : 0);
    }
}

// One code-block per warp; blocks b = blockIdx.x * kEncWarps + warp.
__global__ void __launch_bounds__(32 * kEncWarps, 6)
    t1_encode_kernel(const tc_t1_enc_desc *__restrict__ desc, int n, const void *__restrict__ in,
                     uint8_t *__restrict__ out, uint32_t cap, tc_t1_enc_result *__restrict__ res)
{
    __shared__ EncTables T;
    __shared__ EncState states[kEncWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    EncState &S = states[warp];
    build_enc_tables(T);
    __syncthreads();
    const int bi = blockIdx.x * kEncWarps + warp;
    if (bi >= n) return;
    const tc_t1_enc_desc d = desc[bi];
    const int w = d.w, h = d.h;
    tc_t1_enc_result r{0u, 0u, 0u, 0u};
    if (w < 1 || w > 64 || h < 1 || h > 64 || d.orient > 3 || d.mb < 1 || d.mb > 31) {
        r.status = 1;
        if (lane == 0) res[bi] = r;
        return;
    }
    // largest magnitude and the signs, rows coalesced across the lanes
    uint32_t mx = 0;
    unsigned long long neg[2] = {0ull, 0ull};  // columns lane and lane + 32
    // Eight rows' loads in flight at once: a block with nothing to code is no more
    // than this scan (12,000 empty 64x64 blocks, with the calls around the launch,
    // 520 us row by row, 325 so; 3,000 of 9 bit-planes 6.74 -> 6.43 ms).
    for (int y0 = 0; y0 < h; y0 += 8) {
        uint32_t v[8][2];
#pragma unroll
        for (int k = 0; k < 8; k++)
#pragma unroll
            for (int j = 0; j < 2; j++) v[k][j] = y0 + k < h && lane + 32 * j < w ? sample(d, in, lane + 32 * j, y0 + k) : 0u;
#pragma unroll
        for (int k = 0; k < 8; k++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const uint32_t m = magnitude(d, v[k][j]);
                mx = max(mx, m);
                if (m && (v[k][j] >> 31)) neg[j] |= 1ull << (y0 + k);
            }
    }
    if (lane < 19) S.ctx[lane] = enc_word(lane == 0 ? 4 : (lane == 17 ? 46 : (lane == 18 ? 3 : 0)), 0);
    for (int i = lane; i < (int)sizeof S.sym; i += 32) S.sym[i] = 0;   // one past a list is read, too
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    __syncwarp();
    const int numbps = 32 - __clz(mx);
    if (numbps > d.mb) {
        r.status = 2;  // the magnitudes need more bit-planes than the band has
    } else if (numbps > 0) {
        // passes kept: d.max_passes (0 or more than the block has: all)
        const int total = 3 * numbps - 2;
        const int limit = d.max_passes && d.max_passes < total ? (int)d.max_passes : total;
        MQEnc mq;
        mq.init(out + (size_t)bi * cap, cap, lane == 0);
        encode_block(S, T, mq, d, in, neg, numbps, limit, lane);
        r.len = mq.flush();
        r.passes = (uint32_t)limit;
        if (mq.overflow || r.len > cap) {
            r.status = 3;
            r.len = 0;
        }
    }
    r.zero_bitplanes = (uint32_t)(d.mb - min(numbps, (int)d.mb));
    if (lane == 0) res[bi] = r;
}

}  // namespace

cudaError_t launch_t1_encode(tc_ctx *ctx, const tc_t1_enc_desc *d_desc, int n, const void *d_in, uint8_t *d_out,
                             uint32_t cap, tc_t1_enc_result *d_res)
{
    if (n <= 0) return cudaSuccess;
    t1_encode_kernel<<<(n + kEncWarps - 1) / kEncWarps, 32 * kEncWarps, 0, ctx->stream>>>(d_desc, n, d_in, d_out, cap, d_res);
    ctx->launches++;
    return cudaGetLastError();
}

}  // namespace tc

namespace tc {
namespace {

// Packs the codewords: block k's len[k] bytes from src + k * cap to
// dst + off[k] (one CTA per block).
__global__ void gather_codewords_kernel(const uint8_t *__restrict__ src, uint32_t cap,
                                        const tc_t1_enc_result *__restrict__ res, const uint64_t *__restrict__ off,
                                        int n, uint8_t *__restrict__ dst)
{
    const int k = blockIdx.x;
    if (k >= n) return;
    const uint32_t len = res[k].len;
    const uint8_t *s = src + (size_t)k * cap;
    uint8_t *d = dst + off[k];
    for (uint32_t i = threadIdx.x; i < len && i < cap; i += blockDim.x) d[i] = s[i];
}

}  // namespace

cudaError_t launch_gather_codewords(tc_ctx *ctx, const uint8_t *src, uint32_t cap, const tc_t1_enc_result *res,
                                    const uint64_t *off, int n, uint8_t *dst)
{
    if (n <= 0) return cudaSuccess;
    gather_codewords_kernel<<<n, 128, 0, ctx->stream>>>(src, cap, res, off, n, dst);
    ctx->launches++;
    return cudaGetLastError();
}

}  // namespace tc
