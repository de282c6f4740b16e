/*
 * drivers.cc -- runs the Tier-1 device functions on the emulated warp (see
 * cuda_runtime.h here).  TEST INFRASTRUCTURE ONLY.  EMU_SOURCE is a kernel
 * file's device part, which ends inside namespace tc's anonymous namespace.
 */
#include EMU_SOURCE

}  // namespace
}  // namespace tc

// The order in which the lanes take their turns.
struct Order {
    int lane[32];
    explicit Order(uint32_t seed)   // 0 ascending, 1 descending, else shuffled
    {
        for (int l = 0; l < 32; l++) lane[l] = seed == 1 ? 31 - l : l;
        for (int l = 31; seed > 1 && l > 0; l--) {
            seed = seed * 1664525u + 1013904223u;
            std::swap(lane[l], lane[(seed >> 8) % (uint32_t)(l + 1)]);
        }
    }
};

// A buffer of exactly `bytes` between two guard zones, filled with junk.
struct Guarded {
    static constexpr size_t kZone = 4096;
    std::vector<unsigned char> mem;
    size_t bytes;
    explicit Guarded(size_t n) : mem(n + 2 * kZone, 0xA5), bytes(n) {}
    unsigned char *data() { return mem.data() + kZone; }
    bool intact() const
    {
        for (size_t i = 0; i < kZone; i++)
            if (mem[i] != 0xA5 || mem[kZone + bytes + i] != 0xA5) return false;
        return true;
    }
};

enum { kOk = 0, kStuck = 1, kOutOfBounds = 2 };

#if defined(EMU_WARP)
template <bool Modes, bool Deep>
static int decode(const tc_cblk_desc *desc, int n, const uint8_t *pool, uint64_t pool_len, uint32_t *out, uint64_t elems,
                  int mode, float r, int planes, int limit, uint32_t seed, uint32_t *err)
{
    using namespace tc;
    const Order order(seed);
    Guarded tables(sizeof(WarpTables)), state(sizeof(BlockState<Deep>) + (size_t)planes * kPlaneWords * 4);
    WarpTables &T = *reinterpret_cast<WarpTables *>(tables.data());
    BlockState<Deep> &B = *reinterpret_cast<BlockState<Deep> *>(state.data());
    const bool ok = emu::run(order.lane, [&](int lane) {
        build_warp_tables(T);
        __syncthreads();
        for (int i = 0; i < n; i++)
            process_block_warp<Modes, Deep>(B, reinterpret_cast<uint32_t *>(&B + 1), planes, limit, T, desc, (uint32_t)i, n, pool,
                                            pool_len, reinterpret_cast<char *>(out), elems, mode, r, err, lane);
    });
    return !tables.intact() || !state.intact() ? kOutOfBounds : (ok ? kOk : kStuck);
}

extern "C" int emu_decode(int modes, int deep, const tc_cblk_desc *desc, int n, const uint8_t *pool, uint64_t pool_len,
                          uint32_t *out, uint64_t elems, int mode, float r, int planes, int limit, uint32_t seed,
                          uint32_t *err)
{
    if (modes) return decode<true, true>(desc, n, pool, pool_len, out, elems, mode, r, planes, limit, seed, err);
    if (deep) return decode<false, true>(desc, n, pool, pool_len, out, elems, mode, r, planes, limit, seed, err);
    return decode<false, false>(desc, n, pool, pool_len, out, elems, mode, r, planes, limit, seed, err);
}
#elif defined(EMU_GROUPS)
template <typename MagT, int G>
static int decode(const tc_cblk_desc *desc, int n, const uint8_t *pool, uint64_t pool_len, uint32_t *out, uint64_t elems,
                  int mode, float r, uint32_t seed, uint32_t *err)
{
    using namespace tc;
    constexpr int kGroups = 32 / G;
    const Order order(seed);
    Guarded tables(sizeof(Tables)), states(kGroups * sizeof(WarpState<MagT>));
    Tables &T = *reinterpret_cast<Tables *>(tables.data());
    WarpState<MagT> *S = reinterpret_cast<WarpState<MagT> *>(states.data());
    const bool ok = emu::run(order.lane, [&](int lane) {
        build_tables(T);
        __syncthreads();
        const int g = lane / G, shift = g * G;
        for (int i = g; i < n; i += kGroups)
            process_block<MagT, G>(S[g], T, desc, (uint32_t)i, n, pool, pool_len, reinterpret_cast<char *>(out), elems, mode, r,
                                   err, lane % G, ((1u << G) - 1u) << shift, shift);
    });
    return !tables.intact() || !states.intact() ? kOutOfBounds : (ok ? kOk : kStuck);
}

extern "C" int emu_decode_groups(int lanes, int wide, const tc_cblk_desc *desc, int n, const uint8_t *pool,
                                 uint64_t pool_len, uint32_t *out, uint64_t elems, int mode, float r, uint32_t seed,
                                 uint32_t *err)
{
    if (lanes == 8)
        return wide ? decode<uint16_t, 8>(desc, n, pool, pool_len, out, elems, mode, r, seed, err)
                    : decode<uint8_t, 8>(desc, n, pool, pool_len, out, elems, mode, r, seed, err);
    return wide ? decode<uint16_t, 16>(desc, n, pool, pool_len, out, elems, mode, r, seed, err)
                : decode<uint8_t, 16>(desc, n, pool, pool_len, out, elems, mode, r, seed, err);
}
#elif defined(EMU_ENCODE)
// Block i is the descriptor i * kEncWarps, the first warp of its CTA.
extern "C" int emu_encode(const tc_t1_enc_desc *desc, int n, const void *in, uint8_t *out, uint32_t cap,
                          tc_t1_enc_result *res, uint32_t seed)
{
    const Order order(seed);
    for (int i = 0; i < n; i += tc::kEncWarps) {
        emu::block_idx.x = (unsigned)(i / tc::kEncWarps);
        if (!emu::run(order.lane, [&](int) { tc::t1_encode_kernel(desc, n, in, out, cap, res); })) return kStuck;
    }
    return kOk;
}
#endif
