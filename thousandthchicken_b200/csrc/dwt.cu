// dwt.cu -- forward 5/3 (int32) and 9/7 (fp32) lifting DWT levels for
// sm_100a (the encoder's and the tc_dwt_forward* entry points; the reverse
// levels are in dwt_rev.cu).
//
// Replaces the reference's forward kernels (dwt_f53.cl, dwt_f97.cl over
// dwt_transform_buffer.cl / dwt_io.cl).  One 256-thread CTA transforms a tile
// of 120 output columns by 56 (9/7) or 60 (5/3) output rows of one level:
//   * it stages the extended tile (halo of H = 4 or 2 samples on every side)
//     in shared memory with 4-byte asynchronous copies, whole-sample
//     symmetric extension at the image edges (ISO F.3.7; the reference's
//     single reflection, dwt_io.cl:7-38, is defect D14);
//   * vertical lifting first (ISO 2D_SD: columns, then rows): two threads
//     per column each lift an overlapping half of it in registers;
//   * horizontal lifting: one thread per 30-output row segment, in
//     registers, whose low- and high-pass results go back to shared memory
//     de-interleaved;
//   * the store writes each row's low and high halves to the level's LL and
//     HL (even rows) or LH and HH (odd rows) bands, coalesced.
// The odd row stride keeps the row walk of the horizontal pass free of bank
// conflicts, a lane's (mirrored) columns are worked out once, a thread's store
// stays in one band, and the levels are chained with programmatic dependent
// launch (not the first: its early CTAs would crowd out the previous
// transform's last levels, 2048x2048 81 against 56 us).  Five levels of
// 2999x2001 5/3 68 -> 33 us, six of 4096x4096 9/7 130 -> 69 us (1.9 TB/s of
// level traffic); the rest is the levels of 512x512 and less, 4 to 5 us each.
// 5/3 uses floor (ISO) or truncating (reference, defect D13) rounding; 9/7
// uses fp32 with the scaling factors applied as floats (defects D10-D12
// fixed).  The lifting steps and their order follow ISO F.4.8.
#include <cuda_runtime.h>

#include <type_traits>

#include "dwt_common.cuh"
#include "tc_internal.cuh"

namespace tc {
namespace {

using namespace dwt;

constexpr int kThreads = 256;

template <int WAVELET>
struct FwdGeo {
    static constexpr int H = WAVELET ? 4 : 2;     // halo
    static constexpr int NR = 64;                 // extended rows per tile
    static constexpr int TY = NR - 2 * H;         // output rows per tile
    static constexpr int TX = 120;                // output columns per tile (even)
    static constexpr int NC = TX + 2 * H;         // extended columns
    static constexpr int S = NC + 1;              // row stride, odd: threads on consecutive rows hit different banks
    static constexpr int SEG = 30;                // outputs per row segment (even)
    static constexpr int SEGN = SEG + 2 * H;      // inputs per row segment
    static constexpr int VN = 32 + H;             // rows lifted by one thread of a column pair
    static constexpr int OUTV = 32 - H;           // rows it keeps
};

// In-place 1-D forward lifting of a signal held in registers (v[0] at an
// even position).  Only samples at least H away from both ends are exact.
template <typename T, int WAVELET, int RND, int N>
__device__ __forceinline__ void lift_forward(T (&v)[N])
{
    if constexpr (WAVELET == 0) {
#pragma unroll
        for (int k = 1; k <= N - 2; k += 2) v[k] -= div2r<RND>(v[k - 1] + v[k + 1]);
#pragma unroll
        for (int k = 2; k <= N - 2; k += 2) v[k] += div4r<RND>(v[k - 1] + v[k + 1] + 2);
    } else {
#pragma unroll
        for (int k = 1; k <= N - 2; k += 2) v[k] = fmaf(kA, v[k - 1] + v[k + 1], v[k]);
#pragma unroll
        for (int k = 2; k <= N - 2; k += 2) v[k] = fmaf(kB, v[k - 1] + v[k + 1], v[k]);
#pragma unroll
        for (int k = 1; k <= N - 2; k += 2) v[k] = fmaf(kG, v[k - 1] + v[k + 1], v[k]);
#pragma unroll
        for (int k = 2; k <= N - 2; k += 2) v[k] = fmaf(kD, v[k - 1] + v[k + 1], v[k]);
#pragma unroll
        for (int k = 0; k + 1 < N; k += 2) {
            v[k] *= kInvK;
            v[k + 1] *= kK;
        }
    }
}

__device__ __forceinline__ void cp_async4(void *smem, const void *gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Forward level, one component per blockIdx.z: io.ll[c] is the spatial input
// (pitch ll_pitch), io.out[c] receives LL (out_pitch), io.bands[c] the Mallat
// plane holding HL/LH/HH (bands_pitch).
template <typename T, int WAVELET, int RND>
__global__ void __launch_bounds__(kThreads) fdwt_level_kernel(LevelIO io)
{
    using G = FwdGeo<WAVELET>;
    constexpr int H = G::H, NR = G::NR, TY = G::TY, TX = G::TX, NC = G::NC, S = G::S;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *t = reinterpret_cast<T *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c = blockIdx.z;
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
    const int w = io.w, h = io.h;
    const T *in = static_cast<const T *>(io.ll[c]);
    pdl_allow_next();
    pdl_wait_prev();

    // 1. stage the extended tile; a lane's columns are the same in every row
    constexpr int kCols = (NC + 31) / 32;
    int xo[kCols];
#pragma unroll
    for (int j = 0; j < kCols; j++) xo[j] = lane + 32 * j < NC ? mirror(x0 - H + lane + 32 * j, w) : -1;
#pragma unroll 2
    for (int r = warp; r < NR; r += kThreads / 32) {
        const T *row = in + (size_t)mirror(y0 - H + r, h) * io.ll_pitch;
#pragma unroll
        for (int j = 0; j < kCols; j++)
            if (xo[j] >= 0) cp_async4(t + r * S + lane + 32 * j, row + xo[j]);
    }
    cp_async_wait_all();
    __syncthreads();

    // 2. vertical lifting: column pairs of threads, rows [0, VN) and
    //    [NR - VN, NR); the results go back in place once all have read
    {
        const int col = tid % 128, half = tid / 128;
        const int vbase = half ? NR - G::VN : 0;
        T v[G::VN];
        if (col < NC) {
#pragma unroll
            for (int k = 0; k < G::VN; k++) v[k] = t[(vbase + k) * S + col];
        }
        __syncthreads();
        if (col < NC) {
            if (h > 1) lift_forward<T, WAVELET, RND, G::VN>(v);
#pragma unroll
            for (int k = 0; k < G::OUTV; k++) t[(vbase + H + k) * S + col] = v[H + k];
        }
        __syncthreads();
    }

    // 3. horizontal lifting of the TY output rows, one 30-output segment per
    //    thread; low outputs go to row words [0, TX/2), high to [64, 64 + TX/2)
    {
        constexpr int NSEG = TX / G::SEG;
        const bool active = tid < TY * NSEG;
        const int seg = tid / TY, r = H + tid % TY;  // a warp walks consecutive rows
        T v[G::SEGN];
        if (active) {
#pragma unroll
            for (int k = 0; k < G::SEGN; k++) v[k] = t[r * S + seg * G::SEG + k];
        }
        __syncthreads();  // segments overlap, and the outputs overwrite the inputs
        if (active) {
            if (w > 1) lift_forward<T, WAVELET, RND, G::SEGN>(v);
#pragma unroll
            for (int i = 0; i < G::SEG / 2; i++) {
                t[r * S + seg * (G::SEG / 2) + i] = v[H + 2 * i];
                t[r * S + 64 + seg * (G::SEG / 2) + i] = v[H + 2 * i + 1];
            }
        }
        __syncthreads();
    }

    // 4. store: row by row, the low half to LL / LH, the high half to HL / HH;
    //    a thread keeps one of the 120 output slots of a row (60 low, 60 high)
    //    and walks every other row, so it stays in one band
    const int wl = (w + 1) >> 1, hl = (h + 1) >> 1;
    constexpr int HALF = TX / 2;
    const int j = tid % 128, odd = tid / 128;
    if (j < TX) {
        const bool hi = j >= HALF;
        const int i = hi ? j - HALF : j;
        const int x = x0 + 2 * i + (hi ? 1 : 0);
        if (x < w) {
            const int xb = (x0 >> 1) + i, yb = y0 >> 1;
            const bool ll = !odd && !hi;
            const size_t pitch = ll ? (size_t)io.out_pitch : (size_t)io.bands_pitch;
            T *dst = static_cast<T *>(ll ? io.out[c] : io.bands[c]) + (size_t)(odd ? hl + yb : yb) * pitch + xb + (hi ? wl : 0);
            const T *src = t + (H + odd) * S + (hi ? 64 : 0) + i;
            const int n = (min(TY, h - y0) - odd + 1) >> 1;
#pragma unroll 4
            for (int k = 0; k < n; k++, dst += pitch, src += 2 * S) *dst = *src;
        }
    }
}

template <typename T, int WAVELET, int RND>
cudaError_t run_fdwt(tc_ctx *ctx, const LevelIO &io, bool chained)
{
    using G = FwdGeo<WAVELET>;
    constexpr size_t smem = (size_t)G::NR * G::S * sizeof(T);
    static DeviceFlags attr;
    if (cudaError_t e = set_smem_once(attr, ctx->device, fdwt_level_kernel<T, WAVELET, RND>, smem)) return e;
    dim3 grid((io.w + G::TX - 1) / G::TX, (io.h + G::TY - 1) / G::TY, io.ncomp);
    if (chained) {
        if (cudaError_t e = launch_pdl(fdwt_level_kernel<T, WAVELET, RND>, grid, dim3(kThreads), smem, ctx->stream, io))
            return e;
    } else {
        fdwt_level_kernel<T, WAVELET, RND><<<grid, kThreads, smem, ctx->stream>>>(io);
    }
    ctx->launches++;
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_fdwt_level(tc_ctx *ctx, const LevelIO &io, int wavelet, int rounding, bool chained)
{
    if (io.w <= 0 || io.h <= 0) return cudaSuccess;
    if (wavelet) return run_fdwt<float, 1, 0>(ctx, io, chained);
    if (rounding == TC_ROUND_TRUNC) return run_fdwt<int32_t, 0, TC_ROUND_TRUNC>(ctx, io, chained);
    return run_fdwt<int32_t, 0, TC_ROUND_FLOOR>(ctx, io, chained);
}

}  // namespace tc
