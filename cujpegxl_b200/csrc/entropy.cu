// Device entropy coding and assembly (see entropy.cuh for the data model).
//
// Token and context semantics follow the reference encoder exactly: AC
// tokens as src/entropy.cu:649-681 with the contexts of src/ac_context.h and
// the fixed 32-cluster map; DC residuals with the modular Gradient predictor
// inside each DC group (src/entropy.cu:114-124); AcMetadata samples YtoX,
// YtoB, strategy row, quant-field row and EPF zeros under the Zero predictor
// (src/entropy.cu:252-274); hybrid-uint (4,2,0) tokens; prefix codes from
// prefix_code.cuh; section layout and headers as src/frame_encoder.cu:88-292
// and src/bitstream/{frame_assembly,codestream,container}.cc.
//
// AC block-channels of the frontend's planes are tokenised one lane per token:
// a bitmap of the non-zeros in scan order gives every position the reference's
// sequential state (non-zeros left, previous-coefficient flag) by population
// counts. Planes given by a caller go one warp per item, a lane per position of
// a 32-position chunk, with ballots for that state. Every other item (header
// blobs, DC residuals, AcMetadata samples) takes one thread.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstring>

#include "chained_launch.cuh"
#include "entropy.cuh"
#include "jxl_constants.cuh"
#include "prefix_code.cuh"

namespace jxb {
namespace {

constexpr unsigned kFull = 0xffffffffu;

// Token channel order Y, X, B over planes stored X, Y, B.
__device__ __forceinline__ int phys_channel(int p) { return p == 0 ? 1 : (p == 1 ? 0 : 2); }

// Section holding `item`, which lies in section s or a little later.
__device__ __forceinline__ Section section_from(const EntropyDev& e, int& s, std::uint32_t item) {
    Section sec{e.sections[s]};
    while (item >= sec.first + sec.count) sec = e.sections[++s];
    return sec;
}

struct GroupGeom {
    int bx0, by0, gw, gh;
};

__device__ __forceinline__ GroupGeom ac_group_geom(const EntropyDev& e, int g) {
    GroupGeom r;
    r.bx0 = (g % e.xg) * kAcGroupBlocks;
    r.by0 = (g / e.xg) * kAcGroupBlocks;
    r.gw = min(kAcGroupBlocks, e.bw - r.bx0);
    r.gh = min(kAcGroupBlocks, e.bh - r.by0);
    return r;
}

__device__ __forceinline__ GroupGeom dc_group_geom(const EntropyDev& e, int g) {
    GroupGeom r;
    const int gy{e.xdg == 1 ? g : g / e.xdg};
    r.bx0 = (g - gy * e.xdg) * kDcGroupBlocks;
    r.by0 = gy * kDcGroupBlocks;
    r.gw = min(kDcGroupBlocks, e.bw - r.bx0);
    r.gh = min(kDcGroupBlocks, e.bh - r.by0);
    return r;
}

enum TokTable : int { kTabDc = 1, kTabAm = 2 };

// ---- items other than AC block-channels -------------------------------------------

// a / b for a < 2^23 and b < 2^16: the float quotient is within one of it.
__device__ __forceinline__ std::uint32_t div_small(std::uint32_t a, std::uint32_t b) {
    std::uint32_t q{static_cast<std::uint32_t>(__fdividef(static_cast<float>(a), static_cast<float>(b)))};
    if (q * b > a) --q;
    if (a - q * b >= b) ++q;
    return q;
}

// Visits the bits of non-AC item j of section `sec` in stream order:
// blob(bytes, nbits), varlen(v), count_field(group, nbits), epf(group), first_block(group),
// token(table, group, symbol, extra_bits, extra_value).
template <class V>
__device__ void visit_misc(const EntropyDev& e, const Section& sec, std::uint32_t j, V& v) {
    if (sec.kind == kSecDcGlobal) {
        v.blob(e.dc_global, e.dc_global_bits);
        return;
    }
    if (sec.kind == kSecAcGlobal) {
        if (j == 0) {
            v.blob(e.ac_prefix, e.ac_prefix_bits);
        } else if (j <= 32) {
            v.varlen(e.ac_alpha[j - 1] - 1);
        } else {
            v.blob(e.desc + (j - 33) * kDescBytes, e.desc_bits[j - 33]);
        }
        return;
    }
    const int g{sec.group};
    const GroupGeom gg{dc_group_geom(e, g)};
    const std::uint32_t n{static_cast<std::uint32_t>(gg.gw * gg.gh)};
    // Row and column of block b of the group.
    auto locate = [&](std::uint32_t b, int& x, int& y) {
        y = static_cast<int>(div_small(b, static_cast<std::uint32_t>(gg.gw)));
        x = static_cast<int>(b) - y * gg.gw;
    };
    if (j == 0) {
        v.blob(e.pre_const, e.pre_const_bits);
        return;
    }
    if (j == 1) {
        v.blob(e.desc + (32 + g) * kDescBytes, e.desc_bits[32 + g]);
        return;
    }
    if (j < 2 + 3 * n) {
        const std::uint32_t sidx{j - 2};
        const int p{(sidx >= n ? 1 : 0) + (sidx >= 2 * n ? 1 : 0)};
        const int c{phys_channel(p)};
        int bx, by;
        locate(sidx - p * n, bx, by);
        bx += gg.bx0;
        by += gg.by0;
        const std::int32_t* plane{e.dc + static_cast<std::size_t>(c) * e.nblocks};
        const std::size_t blk{static_cast<std::size_t>(by) * e.bw + bx};
        const bool hl{bx > gg.bx0};
        const bool ht{by > gg.by0};
        const std::int32_t w{hl ? plane[blk - 1] : 0};
        const std::int32_t nn{ht ? plane[blk - e.bw] : 0};
        const std::int32_t nw{(hl && ht) ? plane[blk - e.bw - 1] : 0};
        const std::int32_t pred{gradient_predict(hl, ht, w, nn, nw)};
        std::uint32_t tok, nb, bits;
        hybrid_uint(pack_signed(plane[blk] - pred), tok, nb, bits);
        v.token(kTabDc, g, tok, nb, bits);
        return;
    }
    if (j == 2 + 3 * n) {
        v.count_field(g, ceil_log2_u(n));
        return;
    }
    if (j == 3 + 3 * n) {
        v.blob(e.mid_const, e.mid_const_bits);
        return;
    }
    if (j == 4 + 3 * n) {
        v.blob(e.desc + (32 + e.ndc + g) * kDescBytes, e.desc_bits[32 + e.ndc + g]);
        return;
    }
    const std::uint32_t m{j - (5 + 3 * n)};
    const int cw{(gg.gw + 7) / 8};
    const int ch{(gg.gh + 7) / 8};
    const std::uint32_t cwch{static_cast<std::uint32_t>(cw * ch)};
    std::int32_t val{0};
    if (m < 2 * cwch) {
        const std::uint32_t t{m < cwch ? m : m - cwch};
        const std::size_t tile{static_cast<std::size_t>(gg.by0 / 8 + static_cast<int>(t) / cw) * e.cmw +
                               gg.bx0 / 8 + static_cast<int>(t) % cw};
        val = m < cwch ? e.ytox[tile] : e.ytob[tile];
    } else if (m < 2 * cwch + 2 * n) {
        const std::uint32_t r{m - 2 * cwch};
        int bx, by;
        locate(r < n ? r : r - n, bx, by);
        const std::size_t blk{static_cast<std::size_t>(gg.by0 + by) * e.bw + gg.bx0 + bx};
        const int side{e.acs[blk]};
        if (side == 0) return;
        if (r < n) {
            val = raw_strategy(side);
            v.first_block(g);
        } else {
            val = e.qf[blk] - 1;
        }
    } else {
        v.epf(g);
        return;
    }
    std::uint32_t tok, nb, bits;
    hybrid_uint(pack_signed(val), tok, nb, bits);
    v.token(kTabAm, g, tok, nb, bits);
}

// ---- AC block-channels: one CTA per stripe staged in shared memory -------------------

constexpr int kAcThreads = 256;
constexpr int kAcWarps = kAcThreads / 32;
constexpr int kStripeItems = 3 * kStripeRows * kAcGroupBlocks;  // 384
constexpr int kRowSlots = kAcGroupBlocks * kCoeffsPerBlock;      // 2048
// AC token symbols are hybrid-uint (4, 2, 0) tokens of values below 2^16
// (packed int16 coefficients, counts up to 1008): at most 63.
constexpr int kAcSymbols = 64;
constexpr int kWindowWords = 4096;  // 16 KB of output bits assembled per CTA

// Bits before section s (s == nsec: all of them).
__device__ __forceinline__ unsigned long long section_start(const EntropyDev& e, int s) {
    if (s >= e.nsec) return e.unit_off[e.misc_units + static_cast<std::uint32_t>(e.nstripes)];
    const Section sec{e.sections[s]};
    const unsigned long long off{e.unit_off[sec.unit]};
    return sec.kind == kSecAcGroup ? off : off + e.item_pre[sec.first];
}

// ORs `n` (<= 32) bits of `v` at bit position `pos` of a zeroed word array in
// shared or global memory.
__device__ __forceinline__ void put_bits_at(unsigned int* words, unsigned long long pos, std::uint32_t n,
                                            std::uint32_t v) {
    while (n > 0) {
        const unsigned long long wi{pos >> 5};
        const std::uint32_t off{static_cast<std::uint32_t>(pos & 31)};
        const std::uint32_t take{n < 32 - off ? n : 32 - off};
        const std::uint32_t chunk{take == 32 ? v : (v & ((1u << take) - 1u))};
        if (chunk != 0) atomicOr(&words[wi], chunk << off);
        v = take == 32 ? 0 : v >> take;
        n -= take;
        pos += take;
    }
}

// A stripe's inputs in shared memory: the three coefficient planes of its
// block rows (row stride kRowSlots), the natural orders, strategies and
// non-zero counts (nzn row 0 is the block row above the stripe).
// Rows of the zero-density cluster table, padded to 16 bytes.
constexpr int kZdRow = (kZeroDensityCount + 15) & ~15;
constexpr int kCoeffCtxBytes = 64 + 64 + 2 * kZdRow;
// The context tables every stripe CTA stages (layout of StripeStage's
// nz_ctx .. zd_cluster), filled on each device by entropy_kernels_init.
__device__ __align__(16) std::uint8_t g_coeff_ctx[kCoeffCtxBytes];

struct StripeStage {
    std::int16_t coef[3][kStripeRows][kRowSlots];
    std::uint16_t order[64 + 256 + 1024];
    std::uint16_t nzc[3][kStripeRows][kAcGroupBlocks];
    std::uint8_t nzn[3][kStripeRows + 1][kAcGroupBlocks];
    std::int8_t acs[kStripeRows][kAcGroupBlocks];
    std::uint16_t active[kStripeItems];  // items with coefficient tokens
    std::uint32_t aux[kStripeItems];     // per-item bits (bits pass) or bit offset (emit pass)
    // The coefficient-token context as table lookups (a copy of
    // g_coeff_ctx): coeff_nz_ctx and coeff_freq_ctx of 1..63, and the
    // cluster of zero-density context z for luma (row 0) and chroma (row 1)
    // block contexts.
    alignas(16) std::uint8_t nz_ctx[64];
    std::uint8_t freq_ctx[64];
    std::uint8_t zd_cluster[2][kZdRow];
    int nactive;
};

// Asynchronous global -> shared copies (cp.async, sm_80 and later): a thread
// issues all of its copies before waiting once for them (cp_async_wait_all).
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
    const unsigned dst{static_cast<unsigned>(__cvta_generic_to_shared(smem_dst))};
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gmem_src) {
    const unsigned dst{static_cast<unsigned>(__cvta_generic_to_shared(smem_dst))};
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The caller's barrier after this publishes the stage to the whole CTA.
__device__ void stage_stripe(const EntropyDev& e, const Stripe& st, const GroupGeom& gg, StripeStage& s) {
    const int tid{static_cast<int>(threadIdx.x)};
    const int vpr{gg.gw * (kCoeffsPerBlock * 2 / 16)};  // 16-byte vectors per block row
    for (int c{0}; c < 3; ++c) {
        const std::int16_t* plane{e.ac + static_cast<std::size_t>(c) * e.nblocks * kCoeffsPerBlock};
        for (int r{0}; r < st.rows; ++r) {
            const std::size_t blk0{static_cast<std::size_t>(gg.by0 + st.r0 + r) * e.bw + gg.bx0};
            const uint4* src{reinterpret_cast<const uint4*>(plane + blk0 * kCoeffsPerBlock)};
            uint4* dst{reinterpret_cast<uint4*>(&s.coef[c][r][0])};
            for (int v{tid}; v < vpr; v += kAcThreads) cp_async16(&dst[v], &src[v]);
        }
    }
    for (int i{tid}; i < (64 + 256 + 1024) / 2; i += kAcThreads) {
        cp_async4(&reinterpret_cast<std::uint32_t*>(s.order)[i], &reinterpret_cast<const std::uint32_t*>(e.order)[i]);
    }
    const int cells{st.rows * gg.gw};
    for (int i{tid}; i < cells; i += kAcThreads) {
        const int r{i / gg.gw};
        const int x{i - r * gg.gw};
        const std::size_t blk{static_cast<std::size_t>(gg.by0 + st.r0 + r) * e.bw + gg.bx0 + x};
        s.acs[r][x] = e.acs[blk];
        for (int c{0}; c < 3; ++c) {
            const std::size_t cb{static_cast<std::size_t>(c) * e.nblocks + blk};
            s.nzc[c][r][x] = e.nzc[cb];
            s.nzn[c][r + 1][x] = e.nzn[cb];
            if (r == 0) s.nzn[c][0][x] = st.r0 > 0 ? e.nzn[cb - e.bw] : 0;
        }
    }
    static_assert(kCoeffCtxBytes % 16 == 0 && offsetof(StripeStage, zd_cluster) + 2 * kZdRow ==
                                                   offsetof(StripeStage, nz_ctx) + kCoeffCtxBytes,
                  "context tables: one contiguous 16-byte-aligned copy");
    for (int i{tid}; i < kCoeffCtxBytes / 16; i += kAcThreads) {
        cp_async16(reinterpret_cast<uint4*>(s.nz_ctx) + i, reinterpret_cast<const uint4*>(g_coeff_ctx) + i);
    }
    if (tid == 0) s.nactive = 0;
    cp_async_wait_all();
}

// Stripe-local item j: block (bx, by) of the stripe, plane c.
struct StripeItem {
    int c, bx, by, n;
    std::uint32_t nz;
};

__device__ __forceinline__ StripeItem stripe_item(const StripeStage& s, int gw, int j) {
    StripeItem it;
    const int bidx{j / 3};
    it.c = phys_channel(j - 3 * bidx);
    it.by = bidx / gw;
    it.bx = bidx - it.by * gw;
    it.n = s.acs[it.by][it.bx];
    it.nz = it.n != 0 ? s.nzc[it.c][it.by][it.bx] : 0u;
    return it;
}

// Count token of a non-covered item: cluster from the non-zero prediction of
// the group-local top and left neighbours (src/entropy.cu:649-652).
__device__ __forceinline__ void count_token(const StripeStage& s, const Stripe& st, const StripeItem& it, int& cl,
                                            std::uint32_t& tok, std::uint32_t& nb, std::uint32_t& bits) {
    const bool hl{it.bx > 0};
    const bool ht{st.r0 + it.by > 0};
    const std::uint32_t top{ht ? s.nzn[it.c][it.by][it.bx] : 0u};
    const std::uint32_t left{hl ? s.nzn[it.c][it.by + 1][it.bx - 1] : 0u};
    cl = context_cluster(nonzero_context(predict_nonzeros(hl, ht, top, left), block_ctx(it.c, it.n)));
    hybrid_uint(it.nz, tok, nb, bits);
}

// Calls f(has, cluster, symbol, extra_bits, extra_value) with all 32 lanes
// once per 32-position chunk of the item's scan, one coefficient token per
// lane in stream order. Ballots give each lane the reference's sequential
// state at its position (src/entropy.cu:653-680): a position is coded while
// non-zeros remain before it, and its context uses that count and whether the
// previous coefficient was non-zero.
template <class F>
__device__ void coeff_tokens(const StripeStage& s, const StripeItem& it, int lane, F&& f) {
    const int n{it.n};
    const int side{n >> 3};
    const int lside{side == 1 ? 0 : (side == 2 ? 1 : 2)};
    const std::uint32_t covered{static_cast<std::uint32_t>(side * side)};
    const std::uint32_t size{static_cast<std::uint32_t>(n * n)};
    const std::uint32_t l2{static_cast<std::uint32_t>(2 * lside)};
    const int bctx{block_ctx(it.c, n)};
    const std::uint16_t* ord{s.order + (n == 8 ? 0 : (n == 16 ? 64 : 320))};
    const std::int16_t* plane{&s.coef[it.c][it.by][it.bx * kCoeffsPerBlock]};
    std::uint32_t remaining{it.nz};
    std::uint32_t prev{it.nz > size / 16 ? 0u : 1u};
    const unsigned below{(1u << lane) - 1u};
    for (std::uint32_t k0{covered}; k0 < size && remaining > 0; k0 += 32) {
        const std::uint32_t k{k0 + static_cast<std::uint32_t>(lane)};
        std::int32_t val{0};
        if (k < size) {
            const int raw{ord[k]};
            const int q{raw >> 6};
            const int qy{q >> lside};
            const int qx{q & (side - 1)};
            // Transforms start at multiples of their size inside the group, so
            // the covered blocks lie in the stripe; planes that break this
            // layout read zeros instead of leaving the staged area.
            if (it.by + qy < kStripeRows && it.bx + qx < kAcGroupBlocks) {
                val = plane[qy * kRowSlots + qx * kCoeffsPerBlock + (raw & 63)];
            }
        }
        const unsigned nzmask{__ballot_sync(kFull, val != 0)};
        const std::uint32_t left{remaining - static_cast<std::uint32_t>(__popc(nzmask & below))};
        const std::uint32_t p{lane == 0 ? prev : ((nzmask >> (lane - 1)) & 1u)};
        const bool has{k < size && left > 0};
        std::uint32_t tok{0}, nb{0}, bits{0};
        int cl{0};
        if (has) {
            // context_cluster(coeff_context(bctx, left, k, covered, l2, p)):
            // the context is the block context's zero-density base plus z,
            // and its cluster depends only on z and luma/chroma. coeff_nz_ctx
            // is constant from 33 on, so the clamp to 63 changes nothing; z
            // stays below kZeroDensityCount whenever the item's count is its
            // non-zeros, and the clamp keeps the lookup in the table otherwise.
            const std::uint32_t nzi{min((left + covered - 1) >> l2, 63u)};
            const std::uint32_t z{min((static_cast<std::uint32_t>(s.nz_ctx[nzi]) + s.freq_ctx[k >> l2]) * 2 + p,
                                      static_cast<std::uint32_t>(kZeroDensityCount - 1))};
            cl = s.zd_cluster[bctx < 7 ? 0 : 1][z];
            hybrid_uint(pack_signed(val), tok, nb, bits);
        }
        f(has, cl, tok, nb, bits);
        remaining -= static_cast<std::uint32_t>(__popc(nzmask));
        prev = (nzmask >> 31) & 1u;
    }
}

__device__ __forceinline__ std::uint32_t warp_sum(std::uint32_t v) {
#pragma unroll
    for (int off{16}; off > 0; off >>= 1) v += __shfl_xor_sync(kFull, v, off);
    return v;
}

__device__ __forceinline__ std::uint32_t warp_incl_scan(std::uint32_t v, int lane) {
#pragma unroll
    for (int off{1}; off < 32; off <<= 1) {
        const std::uint32_t t{__shfl_up_sync(kFull, v, off)};
        if (lane >= off) v += t;
    }
    return v;
}

// An AC token in 32 bits: symbol (6 bits), cluster (5), extra-bit count (4)
// and extra bits (at most 13: packed coefficients stay below 2^16).
__device__ __forceinline__ std::uint32_t pack_ac_token(int cl, std::uint32_t sym, std::uint32_t nb,
                                                       std::uint32_t bits) {
    return (bits << 15) | (nb << 11) | (static_cast<std::uint32_t>(cl) << 6) | sym;
}
// Its entry in EntropyDev::code.
__device__ __forceinline__ std::uint32_t token_code_index(std::uint32_t t) { return t & 2047u; }
__device__ __forceinline__ std::uint32_t token_extra_count(std::uint32_t t) { return (t >> 11) & 15u; }
__device__ __forceinline__ std::uint32_t token_extra_bits(std::uint32_t t) { return t >> 15; }

// Where a stripe's tokens are: tokens below `split` at near[t], the others at
// far[t]; near is null when they did not fit the pool. Direct stripes have
// kTokensPerBlock places a block of their own, and what exceeds those runs of
// the output buffer's end (dense_tokens). Otherwise the stripe's run of the
// pool holds all of them. `split` is a multiple of 32.
struct StripeTokens {
    const std::uint32_t* near;
    const std::uint32_t* far;
    std::uint32_t split;
    __device__ __forceinline__ const std::uint32_t* at(std::uint32_t t) const { return (t < split ? near : far) + t; }
};

__device__ __forceinline__ std::uint32_t stripe_blocks(const EntropyDev& e, const Stripe& st) {
    return (st.item0 - e.ac_first) / 3;  // blocks of the stripes before it
}

// Place of a direct stripe's tokens from `split` on, given its offset (in
// tokens, counted back from the end of the output buffer) there.
//
// The file cannot reach them. A token is at most 13 extra bits and a code; a
// cluster's code is optimal for its counts raised to a floor that adds less
// than 15% to their sum (a depth above 15 needs a total of a thousand times
// the floor), so no worse than 6 bits a token on that sum, the length of a
// fixed code for 64 symbols. With at most 192 tokens a block that is 2.5 x 192
// bytes of tokens and, for the other items, less than 48, against the
// buffer's 1200 bytes a block (worst_case_output) and 4 x (192 - 32) of
// tokens kept here. The layout checks it all the same.
__device__ __forceinline__ std::uint32_t* dense_tokens(const EntropyDev& e, std::uint32_t back) {
    return reinterpret_cast<std::uint32_t*>(e.out + e.out_capacity) - back;
}

__device__ __forceinline__ StripeTokens stripe_tokens(const EntropyDev& e, const Stripe& st, unsigned blk, int cells) {
    const std::uint32_t place{e.stripe_tok[2 * blk]};
    if (!e.direct) {
        return {place != kNoTokens ? e.tok_pool + place : nullptr, nullptr, 0xffffffe0u};
    }
    const std::uint32_t split{static_cast<std::uint32_t>(cells) * kTokensPerBlock};
    return {e.tok_pool + static_cast<std::size_t>(stripe_blocks(e, st)) * kTokensPerBlock,
            dense_tokens(e, place) - split, split};
}

// Number of coefficient tokens of an item: the scan positions from `covered`
// through its last non-zero coefficient, exactly those on which
// coeff_tokens reports `has` (all positions to the end of the transform when
// the staged coefficients hold fewer non-zeros than the item's count).
__device__ std::uint32_t coeff_extent(const StripeStage& s, const StripeItem& it, int lane) {
    const int n{it.n};
    const int side{n >> 3};
    const int lside{side == 1 ? 0 : (side == 2 ? 1 : 2)};
    const std::uint32_t covered{static_cast<std::uint32_t>(side * side)};
    const std::uint32_t size{static_cast<std::uint32_t>(n * n)};
    const std::uint16_t* ord{s.order + (n == 8 ? 0 : (n == 16 ? 64 : 320))};
    const std::int16_t* plane{&s.coef[it.c][it.by][it.bx * kCoeffsPerBlock]};
    std::uint32_t remaining{it.nz};
    if (remaining == 0) return 0;
    const unsigned upto{(2u << lane) - 1u};  // lanes 0..lane
    for (std::uint32_t k0{covered}; k0 < size; k0 += 32) {
        const std::uint32_t k{k0 + static_cast<std::uint32_t>(lane)};
        std::int32_t val{0};
        if (k < size) {
            const int raw{ord[k]};
            const int q{raw >> 6};
            const int qy{q >> lside};
            const int qx{q & (side - 1)};
            if (it.by + qy < kStripeRows && it.bx + qx < kAcGroupBlocks) {
                val = plane[qy * kRowSlots + qx * kCoeffsPerBlock + (raw & 63)];
            }
        }
        const unsigned m{__ballot_sync(kFull, val != 0)};
        const std::uint32_t pc{static_cast<std::uint32_t>(__popc(m))};
        if (pc >= remaining) {
            // The lane holding the remaining-th non-zero of this chunk.
            const bool last{val != 0 && static_cast<std::uint32_t>(__popc(m & upto)) == remaining};
            const unsigned who{__ballot_sync(kFull, last)};
            return k0 + static_cast<std::uint32_t>(__ffs(who) - 1) - covered + 1;
        }
        remaining -= pc;
    }
    return size - covered;
}

// Exclusive scan over a CTA of kAcThreads threads; `warp_sums` holds
// kAcWarps + 1 words and receives the total in its last entry.
__device__ std::uint32_t cta_exclusive_scan(std::uint32_t v, std::uint32_t* warp_sums, std::uint32_t& total) {
    const int lane{static_cast<int>(threadIdx.x) & 31};
    const int warp{static_cast<int>(threadIdx.x) >> 5};
    const std::uint32_t incl{warp_incl_scan(v, lane)};
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const std::uint32_t ws{lane < kAcWarps ? warp_sums[lane] : 0u};
        const std::uint32_t wi{warp_incl_scan(ws, lane)};
        if (lane < kAcWarps) warp_sums[lane] = wi - ws;
        if (lane == kAcWarps - 1) warp_sums[kAcWarps] = wi;
    }
    __syncthreads();
    const std::uint32_t off{warp_sums[warp] + incl - v};
    total = warp_sums[kAcWarps];
    __syncthreads();
    return off;
}

// ---- pass 1: histograms ---------------------------------------------------------

// One CTA per stripe: the stripe's coefficient planes are read once, its
// tokens counted into the 32-cluster histogram and written, in stream order,
// to a run of the token pool that the stripe reserves once it knows their
// number (count tokens first sized, then the coefficient extents).
__device__ __forceinline__ void ac_tok_body(const EntropyDev& e, const unsigned blk) {
    extern __shared__ __align__(16) unsigned char ac_smem[];
    StripeStage& s{*reinterpret_cast<StripeStage*>(ac_smem)};
    std::uint32_t* hist{reinterpret_cast<std::uint32_t*>(ac_smem + sizeof(StripeStage))};  // [32][64]
    __shared__ std::uint32_t sh_scan[kAcWarps + 1];
    __shared__ std::uint32_t sh_base;
    __shared__ int sh_stored;
    const int tid{static_cast<int>(threadIdx.x)};
    const int lane{tid & 31};
    const Stripe st{e.stripes[blk]};
    const GroupGeom gg{ac_group_geom(e, st.group)};
    for (int i{tid}; i < kNumClusters * kAcSymbols; i += kAcThreads) hist[i] = 0;
    stage_stripe(e, st, gg, s);
    __syncthreads();
    const int nitems{3 * st.rows * gg.gw};
    for (int j{tid}; j < nitems; j += kAcThreads) {
        const StripeItem it{stripe_item(s, gg.gw, j)};
        if (it.n == 0) {
            s.aux[j] = 0;
            continue;
        }
        int cl;
        std::uint32_t tok, nb, bits;
        count_token(s, st, it, cl, tok, nb, bits);
        atomicAdd(&hist[cl * kAcSymbols + tok], 1u);
        s.aux[j] = 1;
        if (it.nz != 0) s.active[atomicAdd(&s.nactive, 1)] = static_cast<std::uint16_t>(j);
    }
    __syncthreads();
    for (int a{tid >> 5}; a < s.nactive; a += kAcWarps) {
        const int j{s.active[a]};
        const std::uint32_t ext{coeff_extent(s, stripe_item(s, gg.gw, j), lane)};
        if (lane == 0) s.aux[j] += ext;
    }
    __syncthreads();
    // Token offsets of the items: each thread scans two adjacent items.
    const int j0{2 * tid};
    const std::uint32_t c0{j0 < nitems ? s.aux[j0] : 0u};
    const std::uint32_t c1{j0 + 1 < nitems ? s.aux[j0 + 1] : 0u};
    std::uint32_t total{0};
    const std::uint32_t off{cta_exclusive_scan(c0 + c1, sh_scan, total)};
    if (j0 < nitems) s.aux[j0] = off;
    if (j0 + 1 < nitems) s.aux[j0 + 1] = off + c0;
    if (tid == 0) {
        std::uint32_t base{0};
        bool stored{true};
        if (total != 0) {
            base = atomicAdd(e.tok_count, total);
            stored = base <= e.tok_capacity && total <= e.tok_capacity - base;
        }
        sh_base = base;
        sh_stored = stored ? 1 : 0;
        e.stripe_tok[2 * blk] = stored ? base : kNoTokens;
        e.stripe_tok[2 * blk + 1] = total;
    }
    __syncthreads();
    const bool stored{sh_stored != 0};
    std::uint32_t* pool{e.tok_pool + sh_base};
    if (stored) {
        for (int j{tid}; j < nitems; j += kAcThreads) {
            const StripeItem it{stripe_item(s, gg.gw, j)};
            if (it.n == 0) continue;
            int cl;
            std::uint32_t tok, nb, bits;
            count_token(s, st, it, cl, tok, nb, bits);
            pool[s.aux[j]] = pack_ac_token(cl, tok, nb, bits);
        }
    }
    for (int a{tid >> 5}; a < s.nactive; a += kAcWarps) {
        const int j{s.active[a]};
        const StripeItem it{stripe_item(s, gg.gw, j)};
        std::uint32_t* dst{pool + s.aux[j] + 1 + static_cast<std::uint32_t>(lane)};
        coeff_tokens(s, it, lane, [&](bool has, int cl, std::uint32_t sym, std::uint32_t nb, std::uint32_t bits) {
            const unsigned key{has ? static_cast<unsigned>(cl * kAcSymbols + sym) : 0xffffffffu};
            const unsigned peers{__match_any_sync(kFull, key)};
            if (has && (__ffs(peers) - 1) == lane) atomicAdd(&hist[key], static_cast<unsigned>(__popc(peers)));
            if (has && stored) *dst = pack_ac_token(cl, sym, nb, bits);
            dst += 32;
        });
    }
    __syncthreads();
    for (int i{tid}; i < kNumClusters * kAcSymbols; i += kAcThreads) {
        if (hist[i]) atomicAdd(&e.ac_hist[(i / kAcSymbols) * 256 + i % kAcSymbols], hist[i]);
    }
}

// ---- pass 1 for the frontend's own planes: one lane per token -------------------------

constexpr int kStripeRegions = kAcGroupBlocks / 4;  // 32x32-pixel regions of a stripe

// What the direct token pass keeps in shared memory (the coefficients
// themselves stay in global memory).
struct DirectStage {
    std::uint32_t hist[kNumClusters * kAcSymbols];
    // Non-zero coefficients in scan order, two words per block. The 16 blocks
    // of a region lie in Z order, in which the blocks of an aligned DCT16 or
    // DCT32 are adjacent, so an item's words are contiguous.
    std::uint32_t bitmap[3][kStripeRegions][32];
    std::uint16_t before[3][kStripeRegions][32];     // the item's non-zeros in its earlier words
    alignas(16) std::uint8_t flag[kAcWarps][32 * 32];  // a warp's non-zeros of one region and plane, a byte each
    std::uint16_t count[kStripeItems];               // tokens of each item
    std::uint32_t info[kStripeItems];                // what a token needs to know of each item (pack_direct_item)
    std::uint32_t item_off[kStripeItems + 33];       // first token of each item that has any, then a sentinel
    std::uint32_t item_info[kStripeItems];           // and its info
    alignas(16) std::uint16_t order[64 + 256 + 1024];  // raw index of each scan position
    std::uint16_t rank[64 + 256 + 1024];               // scan position of each raw index
    alignas(16) std::uint8_t nz_ctx[64];               // copy of g_coeff_ctx, as in StripeStage
    std::uint8_t freq_ctx[64];
    std::uint8_t zd_cluster[2][kZdRow];
    std::uint8_t nzn[3][kStripeRows + 1][kAcGroupBlocks];  // row 0: the block row above the stripe
    // Of each block: its transform's log2 side in blocks (bits 9-10), the
    // block's ordinal in it (bits 5-8) and its first bitmap word (bits 0-4).
    std::uint16_t owner[kStripeRows][kAcGroupBlocks];
    std::uint32_t scan[kAcWarps + 1];
    std::uint32_t far;  // offset of the tokens past the stripe's own places (dense_tokens)
};
static_assert(offsetof(DirectStage, zd_cluster) + 2 * kZdRow == offsetof(DirectStage, nz_ctx) + kCoeffCtxBytes &&
                  offsetof(DirectStage, nz_ctx) % 16 == 0 && offsetof(DirectStage, order) % 16 == 0 &&
                  offsetof(DirectStage, rank) % 16 == 0,
              "context and order tables: aligned contiguous copies");
constexpr unsigned kNoOwner = 0xffffu;

// First entry of a transform of 2^lside blocks a side in the concatenated orders.
__device__ __forceinline__ int order_base(int lside) { return lside == 0 ? 0 : (lside == 1 ? 64 : 320); }

// First bitmap word of stripe block (r, x) in its region: twice its Z-order index.
__device__ __forceinline__ int bitmap_word(int r, int x) {
    return 2 * ((x & 1) | ((r & 1) << 1) | ((x & 2) << 1) | ((r & 2) << 2));
}

// Non-zeros (11 bits), log2 side (2), block column (5) and row (2), plane (2).
__device__ __forceinline__ std::uint32_t pack_direct_item(std::uint32_t nz, int lside, int x, int r, int c) {
    return nz | (static_cast<std::uint32_t>(lside) << 11) | (static_cast<std::uint32_t>(x) << 13) |
           (static_cast<std::uint32_t>(r) << 18) | (static_cast<std::uint32_t>(c) << 20);
}

// One CTA per stripe of planes the frontend wrote (every block covered by
// exactly one transform, transforms at multiples of their size, non-zero
// counts exact; anything else would give other tokens but stays inside the
// stripe's arrays and pool run). A first pass reads the coefficients in
// storage order, eight per load, and sets one bit per non-zero at its scan
// position; an item's token count, and for every position the non-zeros left
// and the previous coefficient, then follow from population counts, so the
// tokens are independent of each other and are written one per lane, whatever
// the mix of item sizes. The stripe's tokens have a fixed place in the pool;
// only a stripe of more than kTokensPerBlock a block reserves room for the
// rest, so everything is stored and stored once.
__device__ __forceinline__ void ac_tok_direct_body(const EntropyDev& e, const unsigned blk) {
    extern __shared__ __align__(16) unsigned char ac_smem[];
    DirectStage& s{*reinterpret_cast<DirectStage*>(ac_smem)};
    const int tid{static_cast<int>(threadIdx.x)};
    const int lane{tid & 31};
    const int warp{tid >> 5};
    const Stripe st{e.stripes[blk]};
    const GroupGeom gg{ac_group_geom(e, st.group)};
    const std::size_t blk0{static_cast<std::size_t>(gg.by0 + st.r0) * e.bw + gg.bx0};
    const int cells{st.rows * gg.gw};

    // The stripe's coefficients, 16 bytes (eight of one block) per load, all
    // loads issued before anything waits.
    static_assert(kAcGroupBlocks * (kCoeffsPerBlock / 8) <= kAcThreads, "one vector of each block row per thread");
    const bool loads{tid < gg.gw * (kCoeffsPerBlock / 8)};
    uint4 v[3][kStripeRows];
#pragma unroll
    for (int c{0}; c < 3; ++c) {
        const uint4* src{reinterpret_cast<const uint4*>(
                             e.ac + (static_cast<std::size_t>(c) * e.nblocks + blk0) * kCoeffsPerBlock) + tid};
#pragma unroll
        for (int r{0}; r < kStripeRows; ++r) {
            v[c][r] = loads && r < st.rows ? src[static_cast<std::size_t>(r) * e.bw * (kCoeffsPerBlock / 8)]
                                           : make_uint4(0, 0, 0, 0);
        }
    }
    // Tables, strategies and count predictions; cleared bitmap and histogram.
    constexpr int kOrderVecs{(64 + 256 + 1024) * 2 / 16};
    for (int i{tid}; i < kOrderVecs; i += kAcThreads) {
        cp_async16(reinterpret_cast<uint4*>(s.order) + i, reinterpret_cast<const uint4*>(e.order) + i);
        cp_async16(reinterpret_cast<uint4*>(s.rank) + i, reinterpret_cast<const uint4*>(e.rank) + i);
    }
    for (int i{tid}; i < kCoeffCtxBytes / 16; i += kAcThreads) {
        cp_async16(reinterpret_cast<uint4*>(s.nz_ctx) + i, reinterpret_cast<const uint4*>(g_coeff_ctx) + i);
    }
    // One block per thread, so a block's default owner is written by the
    // thread that may then claim it for its own transform.
    static_assert(kStripeRows * kAcGroupBlocks <= kAcThreads, "one block per thread");
    const int cr{tid / gg.gw};
    const int cx{tid - cr * gg.gw};
    int side{0};
    if (tid < cells) {
        const std::size_t b{blk0 + static_cast<std::size_t>(cr) * e.bw + cx};
        const int n{e.acs[b]};
        std::uint8_t pn[3], pt[3];
#pragma unroll
        for (int c{0}; c < 3; ++c) {
            const std::size_t cb{static_cast<std::size_t>(c) * e.nblocks + b};
            pn[c] = e.nzn[cb];
            pt[c] = cr == 0 && st.r0 > 0 ? e.nzn[cb - e.bw] : 0;
        }
        s.owner[cr][cx] = kNoOwner;
        side = n == 8 ? 1 : (n == 16 ? 2 : (n == 32 ? 4 : 0));
        if (cr + side > st.rows || cx + side > gg.gw || ((cr | cx) & (side - 1)) != 0) side = 0;
#pragma unroll
        for (int c{0}; c < 3; ++c) {
            s.nzn[c][cr + 1][cx] = pn[c];
            if (cr == 0) s.nzn[c][0][cx] = pt[c];
        }
    }
    for (int i{tid}; i < kNumClusters * kAcSymbols; i += kAcThreads) s.hist[i] = 0;
    __syncthreads();
    if (side != 0) {
        const int lside{side >> 1};
        const int own{(lside << 9) | bitmap_word(cr, cx)};
        for (int q{0}; q < side * side; ++q) {
            s.owner[cr + (q >> lside)][cx + (q & (side - 1))] = static_cast<std::uint16_t>(own | (q << 5));
        }
    }
    cp_async_wait_all();
    __syncthreads();

    // A warp holds one region's four block rows (a lane an eighth of a block
    // of each), so it makes that region's bitmaps by itself: plane by plane,
    // each non-zero stores a byte at its scan position, and lane w gathers
    // word w from 32 bytes. (ORing the bits in place with shared-memory atomics
    // took up to 20K cycles for a dense stripe: low frequencies of one
    // transform share a few words.) The tokens of each item follow: its count
    // token, then every scan position through its last non-zero; sums over an
    // item's words are segmented warp scans.
    static_assert(kStripeRegions == kAcWarps && kAcGroupBlocks / kStripeRegions * (kCoeffsPerBlock / 8) == 32,
                  "a warp per region");
    uint4 ranks[kStripeRows];    // scan positions of the lane's eight coefficients of each row
    std::uint32_t rowinfo[kStripeRows];  // 32 * first bitmap word
#pragma unroll
    for (int r{0}; r < kStripeRows; ++r) {
        const unsigned own{loads && r < st.rows ? s.owner[r][tid >> 3] : kNoOwner};
        const int lside{own != kNoOwner ? static_cast<int>(own >> 9) : 0};
        const std::uint16_t* rank{s.rank + order_base(lside) + (own != kNoOwner ? (own >> 5) & 15u : 0u) * kCoeffsPerBlock +
                                  (tid & 7) * 8};
        ranks[r] = *reinterpret_cast<const uint4*>(rank);
        rowinfo[r] = own != kNoOwner ? 32 * (own & 31u) : 0u;
    }
    std::uint8_t* flag{s.flag[warp]};
#pragma unroll
    for (int c{0}; c < 3; ++c) {
        reinterpret_cast<uint4*>(flag)[lane] = make_uint4(0, 0, 0, 0);
        reinterpret_cast<uint4*>(flag)[lane + 32] = make_uint4(0, 0, 0, 0);
        __syncwarp();
#pragma unroll
        for (int r{0}; r < kStripeRows; ++r) {
            const std::uint32_t word[4]{v[c][r].x, v[c][r].y, v[c][r].z, v[c][r].w};
            if ((word[0] | word[1] | word[2] | word[3]) == 0) continue;
            const std::uint32_t pos[4]{ranks[r].x, ranks[r].y, ranks[r].z, ranks[r].w};
            std::uint8_t* at{flag + rowinfo[r]};
#pragma unroll
            for (int i{0}; i < 8; ++i) {
                const std::uint32_t k{(pos[i >> 1] >> (16 * (i & 1))) & 0xffffu};
                // (The low frequencies, which are not coded here, are zero in
                // the frontend's planes.)
                if (((word[i >> 1] >> (16 * (i & 1))) & 0xffffu) != 0) at[k] = 1;
            }
        }
        __syncwarp();
        std::uint32_t m{0};
#pragma unroll
        for (int q{0}; q < 2; ++q) {
            const uint4 b{reinterpret_cast<const uint4*>(flag)[2 * lane + q]};
            // Four 0/1 bytes to four bits: byte i's product lands in bit 24 + i.
            const std::uint32_t n[4]{b.x * 0x01020408u >> 24, b.y * 0x01020408u >> 24, b.z * 0x01020408u >> 24,
                                     b.w * 0x01020408u >> 24};
#pragma unroll
            for (int i{0}; i < 4; ++i) m |= n[i] << (16 * q + 4 * i);
        }
        __syncwarp();
        const int region{warp};
        const int z{lane >> 1};
        const int r{((z >> 1) & 1) | ((z >> 2) & 2)};
        const int x{4 * region + ((z & 1) | ((z >> 1) & 2))};
        const unsigned own{r < st.rows && x < gg.gw ? s.owner[r][x] : kNoOwner};
        s.bitmap[c][region][lane] = m;
        const int lside{own != kNoOwner ? static_cast<int>(own >> 9) : 0};
        const int words{2 << (2 * lside)};
        const int seg{lane & ~(words - 1)};
        const std::uint32_t pc{static_cast<std::uint32_t>(__popc(m))};
        std::uint32_t sum{pc};
#pragma unroll
        for (int off{1}; off < 32; off <<= 1) {
            const std::uint32_t t{__shfl_up_sync(kFull, sum, off)};
            if (lane - seg >= off) sum += t;
        }
        s.before[c][region][lane] = static_cast<std::uint16_t>(sum - pc);
        const std::uint32_t nz{__shfl_sync(kFull, sum, seg + words - 1)};
        const unsigned filled{__ballot_sync(kFull, m != 0) & (kFull >> (32 - words) << seg)};
        const int last{filled != 0 ? 31 - __clz(static_cast<int>(filled)) : seg};
        const std::uint32_t lm{__shfl_sync(kFull, m, last)};
        const std::uint32_t covered{1u << (2 * lside)};
        const std::uint32_t end{max(covered, 32u * static_cast<std::uint32_t>(last - seg + 1) -
                                                 static_cast<std::uint32_t>(__clz(static_cast<int>(lm))))};
        if ((lane & 1) == 0 && r < st.rows && x < gg.gw) {
            const int j{3 * (r * gg.gw + x) + (c == 1 ? 0 : (c == 0 ? 1 : 2))};
            const bool first{own != kNoOwner && lane == seg};
            s.count[j] = first ? static_cast<std::uint16_t>(1 + end - covered) : static_cast<std::uint16_t>(0);
            s.info[j] = pack_direct_item(nz, lside, x, r, c);
        }
    }
    __syncthreads();
    // Offsets: tokens in the low half of the scanned word, items with tokens
    // in the high half. Each thread takes two adjacent items.
    const int nitems{3 * cells};
    std::uint32_t count[2];
#pragma unroll
    for (int h{0}; h < 2; ++h) count[h] = 2 * tid + h < nitems ? s.count[2 * tid + h] : 0u;
    const std::uint32_t mine{count[0] + count[1] + ((count[0] != 0 ? 0x10000u : 0u) + (count[1] != 0 ? 0x10000u : 0u))};
    std::uint32_t both{0};
    std::uint32_t off{cta_exclusive_scan(mine, s.scan, both)};
#pragma unroll
    for (int h{0}; h < 2; ++h) {
        if (count[h] == 0) continue;
        s.item_off[off >> 16] = off & 0xffffu;
        s.item_info[off >> 16] = s.info[2 * tid + h];
        off += 0x10000u + count[h];
    }
    const int nactive{static_cast<int>(both >> 16)};
    if (tid < 33) s.item_off[nactive + tid] = 0xffffffffu;
    const std::uint32_t total{min(both & 0xffffu, static_cast<std::uint32_t>(cells) * kMaxTokensPerBlock)};
    const std::uint32_t own{static_cast<std::uint32_t>(cells) * kTokensPerBlock};
    if (tid == 0) {
        std::uint32_t far{0};
        if (total > own) {
            const std::uint32_t more{(total - own + 31u) & ~31u};
            far = atomicAdd(e.tok_count, more) + more;
        }
        s.far = far;
        e.stripe_tok[2 * blk] = far;
        e.stripe_tok[2 * blk + 1] = total;
    }
    __syncthreads();

    // Each warp takes a contiguous run of tokens, 32 at a time: the items that
    // start among them come from one load and one reduction, so a lane knows
    // its item without a search. kAhead groups are prepared together, so that
    // their coefficient loads overlap.
    constexpr int kAhead{4};
    std::uint32_t* near{e.tok_pool + static_cast<std::size_t>(stripe_blocks(e, st)) * kTokensPerBlock};
    std::uint32_t* far{dense_tokens(e, s.far) - own};
    const std::uint32_t groups{(total + 31) / 32};
    const std::uint32_t per_warp{(groups + kAcWarps - 1) / kAcWarps};
    const std::uint32_t t_first{32 * per_warp * static_cast<std::uint32_t>(warp)};
    const std::uint32_t t_end{min(total, t_first + 32 * per_warp)};
    int base{0};  // the item of token t0
    if (t_first < t_end) {
        int hi{nactive - 1};
        while (base < hi) {
            const int mid{(base + hi + 1) >> 1};
            if (s.item_off[mid] <= t_first) {
                base = mid;
            } else {
                hi = mid - 1;
            }
        }
    }
    for (std::uint32_t t0{t_first}; t0 < t_end; t0 += 32 * kAhead) {
        std::uint32_t info[kAhead];
        std::uint32_t at[kAhead];      // token index inside its item
        std::uint32_t state[kAhead];   // non-zeros left << 1 | previous coefficient non-zero
        std::int32_t val[kAhead];
#pragma unroll
        for (int g{0}; g < kAhead; ++g) {
            const std::uint32_t tg{t0 + 32 * g};
            if (tg >= t_end) break;
            const std::uint32_t rel{s.item_off[min(base + 1 + lane, nactive)] - tg};
            const unsigned starts{__reduce_or_sync(kFull, rel < 32 ? 1u << rel : 0u)};
            const int item{min(base + __popc(starts & ((2u << lane) - 1u)), nactive - 1)};
            base += __popc(starts) + (__ballot_sync(kFull, rel == 32) != 0 ? 1 : 0);
            info[g] = s.item_info[item];
            at[g] = tg + lane - s.item_off[item];
            val[g] = 0;
            state[g] = 0;
            if (tg + lane >= t_end || at[g] == 0) continue;
            // Scan position k: the non-zeros left from the bits before it, the
            // previous coefficient's bit (or the rule for the first position).
            const int lside{static_cast<int>((info[g] >> 11) & 3u)};
            const int x{static_cast<int>((info[g] >> 13) & 31u)};
            const int r{static_cast<int>((info[g] >> 18) & 3u)};
            const int c{static_cast<int>((info[g] >> 20) & 3u)};
            const std::uint32_t nz{info[g] & 2047u};
            const std::uint32_t covered{1u << (2 * lside)};
            const std::uint32_t k{covered + at[g] - 1};
            const int w{min(bitmap_word(r, x) + static_cast<int>(k >> 5), 31)};
            const std::uint32_t m{s.bitmap[c][x >> 2][w]};
            const std::uint32_t bit{k & 31u};
            const std::uint32_t left{nz - s.before[c][x >> 2][w] -
                                     static_cast<std::uint32_t>(__popc(m & ((1u << bit) - 1u)))};
            const std::uint32_t earlier{bit != 0 ? m << (32 - bit) : s.bitmap[c][x >> 2][max(w - 1, 0)]};
            const std::uint32_t prev{at[g] == 1 ? (nz > (covered * kCoeffsPerBlock) / 16 ? 0u : 1u) : earlier >> 31};
            state[g] = (left << 1) | prev;
            if ((m >> bit) & 1u) {
                const int raw{s.order[order_base(lside) + static_cast<int>(k)]};
                const int q{raw >> 6};
                const std::size_t b{blk0 + static_cast<std::size_t>(r + (q >> lside)) * e.bw + x +
                                    (q & ((1 << lside) - 1))};
                val[g] = e.ac[(static_cast<std::size_t>(c) * e.nblocks + b) * kCoeffsPerBlock + (raw & 63)];
            }
        }
#pragma unroll
        for (int g{0}; g < kAhead; ++g) {
            const std::uint32_t t{t0 + 32 * g + lane};
            if (t0 + 32 * g >= t_end) break;
            const int lside{static_cast<int>((info[g] >> 11) & 3u)};
            const int c{static_cast<int>((info[g] >> 20) & 3u)};
            std::uint32_t value;
            int cl;
            if (at[g] == 0) {
                const int x{static_cast<int>((info[g] >> 13) & 31u)};
                const int r{static_cast<int>((info[g] >> 18) & 3u)};
                const bool hl{x > 0};
                const bool ht{st.r0 + r > 0};
                const std::uint32_t top{ht ? s.nzn[c][r][x] : 0u};
                const std::uint32_t left{hl ? s.nzn[c][r + 1][x - 1] : 0u};
                cl = context_cluster(nonzero_context(predict_nonzeros(hl, ht, top, left), block_ctx(c, 8 << lside)));
                value = info[g] & 2047u;
            } else {
                // The context tables and clamps of coeff_tokens.
                const std::uint32_t l2{static_cast<std::uint32_t>(2 * lside)};
                const std::uint32_t covered{1u << l2};
                const std::uint32_t k{covered + at[g] - 1};
                const std::uint32_t nzi{min(((state[g] >> 1) + covered - 1) >> l2, 63u)};
                const std::uint32_t z{min((static_cast<std::uint32_t>(s.nz_ctx[nzi]) + s.freq_ctx[min(k >> l2, 63u)]) * 2 +
                                              (state[g] & 1u),
                                          static_cast<std::uint32_t>(kZeroDensityCount - 1))};
                cl = s.zd_cluster[c == 1 ? 0 : 1][z];
                value = pack_signed(val[g]);
            }
            std::uint32_t tok, nb, bits;
            hybrid_uint(value, tok, nb, bits);
            // Lanes of equal tokens count once: shared-memory atomics on one
            // address serialise.
            const unsigned key{t < t_end ? static_cast<unsigned>(cl * kAcSymbols) + tok : 0xffffffffu};
            const unsigned peers{__match_any_sync(kFull, key)};
            if (t < t_end) {
                if (__ffs(static_cast<int>(peers)) - 1 == lane) {
                    atomicAdd(&s.hist[key], static_cast<unsigned>(__popc(peers)));
                }
                (t < own ? near : far)[t] = pack_ac_token(cl, tok, nb, bits);
            }
        }
    }
    __syncthreads();
    for (int i{tid}; i < kNumClusters * kAcSymbols; i += kAcThreads) {
        if (s.hist[i]) atomicAdd(&e.ac_hist[(i / kAcSymbols) * 256 + i % kAcSymbols], s.hist[i]);
    }
}

// The token of an item other than an AC block-channel, kept from the token
// pass for the later passes: symbol (7 bits; hybrid-uint (4, 2, 0) symbols of
// 32-bit values are below 128), extra-bit count (5), extra bits (18), table.
// kMiscVisit: blobs, counts and wider tokens, which the later passes visit
// again; kMiscNone: nothing is written for the item.
constexpr std::uint32_t kMiscVisit = 0x80000000u;
constexpr std::uint32_t kMiscNone = 0x80000001u;
constexpr std::uint32_t kMiscExtraBits = 18;
constexpr int kMiscSymbols = 128;
__device__ __forceinline__ std::uint32_t pack_misc_token(int tab, std::uint32_t sym, std::uint32_t nb, std::uint32_t bits) {
    if (nb > kMiscExtraBits) return kMiscVisit;
    return (tab == kTabAm ? 0x40000000u : 0u) | (bits << 12) | (nb << 7) | sym;
}
// Entry of EntropyDev::code where a DC group's DC or AcMetadata symbols start.
__device__ __forceinline__ int misc_code_base(const EntropyDev& e, bool am, int g) {
    return kNumClusters * kAcSymbols + ((am ? e.ndc : 0) + g) * kMiscSymbols;
}
// Its depth << 16 | code bits, in DC group g.
__device__ __forceinline__ std::uint32_t misc_code(const EntropyDev& e, int g, std::uint32_t t) {
    return e.code[misc_code_base(e, (t & 0x40000000u) != 0, g) + (t & 127u)];
}
__device__ __forceinline__ std::uint32_t misc_extra_count(std::uint32_t t) { return (t >> 7) & 31u; }
__device__ __forceinline__ std::uint32_t misc_extra_bits(std::uint32_t t) { return (t >> 12) & 0x3ffffu; }

struct HistVisitor {
    std::uint32_t* sh_g;      // [2 slots][2 tables][256]
    std::uint32_t* sh_fb;     // [2 slots]
    int g0, g1;
    const EntropyDev* e;
    std::uint32_t kept{kMiscNone};  // what item_tok gets
    __device__ void blob(const std::uint8_t*, std::uint32_t) { kept = kMiscVisit; }
    __device__ void varlen(std::uint32_t) { kept = kMiscVisit; }
    __device__ void count_field(int, unsigned) { kept = kMiscVisit; }
    __device__ void epf(int) { kept = pack_misc_token(kTabAm, 0, 0, 0); }  // counted by the code pass
    __device__ void first_block(int g) {
        if (g == g0) {
            atomicAdd(&sh_fb[0], 1u);
        } else if (g == g1) {
            atomicAdd(&sh_fb[1], 1u);
        } else {
            atomicAdd(&e->fb_count[g], 1u);
        }
    }
    __device__ void token(int tab, int g, std::uint32_t sym, std::uint32_t nb, std::uint32_t bits) {
        kept = pack_misc_token(tab, sym, nb, bits);
        const int t{tab == kTabDc ? 0 : 1};
        if (g == g0) {
            atomicAdd(&sh_g[t * 256 + sym], 1u);
        } else if (g == g1) {
            atomicAdd(&sh_g[(2 + t) * 256 + sym], 1u);
        } else {
            atomicAdd(&(t == 0 ? e->dc_hist : e->am_hist)[g * 256 + sym], 1u);
        }
    }
};

// Other items per thread of the item passes.
constexpr int kMiscPerThread = 2;
static_assert(kMiscItemsPerUnit == kMiscPerThread * kAcThreads, "a unit of other items is one CTA's");

__device__ __forceinline__ void misc_hist_body(const EntropyDev& e, const unsigned blk) {
    extern __shared__ __align__(16) unsigned char misc_smem[];
    std::uint32_t* sh_g{reinterpret_cast<std::uint32_t*>(misc_smem)};  // [4 * 256]
    std::uint32_t* sh_fb{sh_g + 4 * 256};                              // [2]
    if (threadIdx.x < 2) sh_fb[threadIdx.x] = 0;
    for (int i{static_cast<int>(threadIdx.x)}; i < 4 * 256; i += blockDim.x) sh_g[i] = 0;
    const std::uint32_t first{blk * kMiscItemsPerUnit};
    const std::uint32_t last{min(first + kMiscItemsPerUnit, e.ac_first) - 1};
    const int sfirst{static_cast<int>(e.unit_section[blk])};
    const Section s0{e.sections[sfirst]};
    int slast{sfirst};
    const Section s1{section_from(e, slast, last)};
    HistVisitor v{sh_g, sh_fb, s0.kind == kSecDcGroup ? s0.group : -1,
                  s1.kind == kSecDcGroup && s1.group != s0.group ? s1.group : -2, &e};
    __syncthreads();
#pragma unroll
    for (int k{0}; k < kMiscPerThread; ++k) {
        const std::uint32_t item{first + threadIdx.x + k * blockDim.x};
        if (item < e.ac_first) {
            int sat{sfirst};
            const Section sec{section_from(e, sat, item)};
            v.kept = kMiscNone;
            visit_misc(e, sec, item - sec.first, v);
            e.item_tok[item] = v.kept;
        }
    }
    __syncthreads();
    for (int i{static_cast<int>(threadIdx.x)}; i < 4 * 256; i += blockDim.x) {
        const int slot{i >> 9};
        const int t{(i >> 8) & 1};
        const int g{slot == 0 ? v.g0 : v.g1};
        if (sh_g[i] && g >= 0) atomicAdd(&(t == 0 ? e.dc_hist : e.am_hist)[g * 256 + (i & 255)], sh_g[i]);
    }
    if (threadIdx.x < 2) {
        const int g{threadIdx.x == 0 ? v.g0 : v.g1};
        if (g >= 0 && sh_fb[threadIdx.x]) atomicAdd(&e.fb_count[g], sh_fb[threadIdx.x]);
    }
}

// ---- pass 2: prefix codes ---------------------------------------------------------

struct WarpCodeSmem {
    std::uint32_t hist[256];
    std::uint32_t cnt[256];            // leaf counts in rank order (count floor 1)
    std::uint16_t leaf_sym[256];       // symbol of the leaf of each rank
    std::uint16_t floor_sym[256];      // symbols of the clamped leaves in descending order
    std::uint8_t depth[256];
    std::uint16_t bits[256];
    std::uint16_t used[256];           // compacted list of used symbols
    alignas(16) std::uint32_t used_cnt[256 + 4];  // their counts, padded to a multiple of four
    std::uint32_t len_count[18];       // depths per code length (canonical codes, header)
    std::uint32_t len_next[18];
    alignas(4) std::uint8_t desc[kDescBytes];
    CodeLengthScratch cl;
    // One tree per lane, lane-interleaved: internal node counts, heights and
    // every node's parent, for the count floor 2^lane.
    std::uint32_t icnt[256 * 32];
    std::uint8_t height[256 * 32];
    std::int16_t parent[512 * 32];
};

// Depths for a histogram with at least two used symbols, equal to the
// reference's serial construction (src/bitstream/prefix_code.cc:65-125):
// leaves ranked by (count ascending, symbol descending), two-queue merge (a
// leaf wins ties), the whole construction repeated with the count floor
// doubled until no depth exceeds `limit`.
//
// Warp-cooperative: the used symbols are compacted and ranked once. Raising
// the floor to F only clamps the smallest counts to F - 1, so the leaves of
// floor F are the same ranks with counts max(count, F - 1), the clamped ones
// (count <= F - 1, a prefix of the ranks) re-ordered by descending symbol.
// Every lane runs the merge for its own floor 2^lane at once, without
// branches, recording parents and internal heights; the smallest floor whose
// tree is no higher than `limit` is the one the serial loop stops at, and its
// leaves are walked to the root.
//
// hist[0..length) is read, depth[] of the used symbols written (the caller
// zeroes the rest); the rest of `s` other than hist and depth is scratch. A
// single used symbol gets depth 1, as the serial builder gives it.
__device__ void warp_create_tree(WarpCodeSmem& s, const std::uint32_t* hist, int length, int limit,
                                 std::uint8_t* depth, int lane) {
    int n{0};
    for (int base{0}; base < length; base += 32) {
        const int sym{base + lane};
        const bool used{sym < length && hist[sym] != 0};
        const unsigned m{__ballot_sync(kFull, used)};
        if (used) {
            const int at{n + __popc(m & ((1u << lane) - 1u))};
            s.used[at] = static_cast<std::uint16_t>(sym);
            s.used_cnt[at] = hist[sym];
        }
        n += __popc(m);
    }
    constexpr std::uint32_t kInf{0xffffffffu};
    if (lane < 4) s.used_cnt[n + lane] = kInf;
    __syncwarp();
    if (n < 2) {
        if (n == 1 && lane == 0) depth[s.used[0]] = 1;
        __syncwarp();
        return;
    }
    // Rank of used symbol i: those with a smaller count, or the same count and
    // a larger symbol (a later place in the list), come before it.
    for (int i{lane}; i < n; i += 32) {
        const std::uint32_t c{s.used_cnt[i]};
        int rank{0};
        for (int t{0}; t < n; t += 4) {
            const uint4 q{*reinterpret_cast<const uint4*>(&s.used_cnt[t])};
            rank += (q.x < c || (q.x == c && t > i)) ? 1 : 0;
            rank += (q.y < c || (q.y == c && t + 1 > i)) ? 1 : 0;
            rank += (q.z < c || (q.z == c && t + 2 > i)) ? 1 : 0;
            rank += (q.w < c || (q.w == c && t + 3 > i)) ? 1 : 0;
        }
        // The padding counts as equal to a symbol of the largest count.
        if (c == kInf) rank -= -n & 3;
        s.cnt[rank] = c;
        s.leaf_sym[rank] = s.used[i];
    }
    __syncwarp();
    // Lane L: floor 2^L, leaf r has count max(cnt[r], 2^L - 1). The heads of
    // both queues and the entries behind them are held in registers, so one
    // step (two picks) waits for one round of loads.
    const std::uint32_t fm1{lane == 31 ? 0x7fffffffu : (1u << lane) - 1u};
    std::uint32_t* icnt{s.icnt + lane};
    std::uint8_t* height{s.height + lane};
    std::int16_t* parent{s.parent + lane};
    int i{0};
    int j{0};
    std::uint32_t a0{max(s.cnt[0], fm1)};  // leaves i and i + 1 (n is at least 2)
    std::uint32_t a1{max(s.cnt[1], fm1)};
    std::uint32_t b0{kInf};                // internal nodes j and j + 1
    std::uint32_t b1{kInf};
    int h0{0};
    int h1{0};
    for (int t{0}; t < n - 1; ++t) {
        const bool leaf0{a0 <= b0};
        const std::uint32_t a{leaf0 ? a1 : a0};
        const std::uint32_t b{leaf0 ? b0 : b1};
        const bool leaf1{a <= b};
        const std::uint32_t v0{leaf0 ? a0 : b0};
        const std::uint32_t v1{leaf1 ? a : b};
        // Saturating: only floors far above any that can fit reach it.
        const std::uint32_t sum{v0 > kInf - 1u - v1 ? kInf - 1u : v0 + v1};
        const int h{max(leaf0 ? 0 : h0, leaf1 ? 0 : (leaf0 ? h0 : h1))};
        parent[32 * (leaf0 ? i : n + j)] = static_cast<std::int16_t>(n + t);
        i += leaf0 ? 1 : 0;
        j += leaf0 ? 0 : 1;
        parent[32 * (leaf1 ? i : n + j)] = static_cast<std::int16_t>(n + t);
        i += leaf1 ? 1 : 0;
        j += leaf1 ? 0 : 1;
        icnt[32 * t] = sum;
        height[32 * t] = static_cast<std::uint8_t>(h + 1);
        // The next heads; nodes up to t exist (entries of leaves past the
        // last, and of nodes past t, never win a pick).
        a0 = i < n ? max(s.cnt[min(i, n - 1)], fm1) : kInf;
        a1 = i + 1 < n ? max(s.cnt[min(i + 1, n - 1)], fm1) : kInf;
        b0 = j <= t ? icnt[32 * min(j, t)] : kInf;
        b1 = j + 1 <= t ? icnt[32 * min(j + 1, t)] : kInf;
        h0 = height[32 * min(j, t)];
        h1 = height[32 * min(j + 1, t)];
    }
    const int root_h{static_cast<int>(height[32 * (n - 2)])};
    const unsigned fit{__ballot_sync(kFull, root_h <= limit)};
    __syncwarp();
    const int best{__ffs(fit) - 1};  // a floor of 2^31 leaves every count equal: always fits
    // Leaves clamped at the chosen floor, in descending symbol order.
    const std::uint32_t bm1{best == 31 ? 0x7fffffffu : (1u << best) - 1u};
    int m{0};
    for (int base{0}; base < n; base += 32) {
        const int r{base + lane};
        m += __popc(__ballot_sync(kFull, r < n && s.cnt[r] <= bm1));
    }
    for (int q{lane}; q < m; q += 32) {
        const int sym{s.leaf_sym[q]};
        int rank{0};
        for (int t{0}; t < m; ++t) rank += s.leaf_sym[t] > sym ? 1 : 0;
        s.floor_sym[rank] = static_cast<std::uint16_t>(sym);
    }
    __syncwarp();
    const std::int16_t* bp{s.parent + best};
    const int root{2 * n - 2};
    for (int r{lane}; r < n; r += 32) {
        int d{0};
        for (int v{r}; v != root; v = bp[32 * v]) ++d;
        depth[r < m ? s.floor_sym[r] : s.leaf_sym[r]] = static_cast<std::uint8_t>(d);
    }
    __syncwarp();
}

// Canonical codes of depth[0..len) (canonical_codes in prefix_code.cuh),
// warp-cooperative: codes of equal length are handed out in symbol order.
__device__ void warp_canonical_codes(WarpCodeSmem& s, const std::uint8_t* depth, int len, std::uint16_t* bits,
                                     int lane) {
    if (lane < 18) s.len_count[lane] = 0;
    __syncwarp();
    for (int base{0}; base < len; base += 32) {
        const int sym{base + lane};
        const int d{sym < len ? depth[sym] : 0};
        const unsigned peers{__match_any_sync(kFull, d)};
        if (d != 0 && (__ffs(peers) - 1) == lane) s.len_count[d] += static_cast<std::uint32_t>(__popc(peers));
        __syncwarp();
    }
    // First code of each length, next[l] = (next[l - 1] + count[l - 1]) << 1,
    // as a sum of the shorter lengths' counts in units of 2^-15.
    {
        const std::uint32_t share{lane > 0 && lane < 16 ? s.len_count[lane] << (15 - lane) : 0u};
        const std::uint32_t before{warp_incl_scan(share, lane) - share};
        if (lane < 16) s.len_next[lane] = before >> (15 - lane);
    }
    __syncwarp();
    const unsigned below{(1u << lane) - 1u};
    for (int base{0}; base < len; base += 32) {
        const int sym{base + lane};
        const int d{sym < len ? depth[sym] : 0};
        const unsigned peers{__match_any_sync(kFull, d)};
        const std::uint32_t code{d != 0 ? s.len_next[d] + static_cast<std::uint32_t>(__popc(peers & below)) : 0u};
        __syncwarp();
        if (d != 0 && (__ffs(peers) - 1) == lane) s.len_next[d] += static_cast<std::uint32_t>(__popc(peers));
        if (sym < len) bits[sym] = d != 0 ? static_cast<std::uint16_t>(__brev(code) >> (32 - d)) : 0;
        __syncwarp();
    }
}

// ORs `n` (<= 32) bits of `v` at bit `pos` of a zeroed little-endian byte
// buffer held as 32-bit words; bits at or past `cap` are dropped.
__device__ __forceinline__ void or_bits(std::uint8_t* buf, std::uint32_t pos, std::uint32_t n, std::uint32_t v,
                                        std::uint32_t cap) {
    if (n == 0) return;
    if (n < 32) v &= (1u << n) - 1u;
    unsigned int* words{reinterpret_cast<unsigned int*>(buf)};
    const std::uint32_t off{pos & 31u};
    if (pos < cap) atomicOr(&words[pos >> 5], v << off);
    if (off + n > 32 && pos + (32 - off) < cap) atomicOr(&words[(pos >> 5) + 1], v >> (32 - off));
}

// store_complex (prefix_code.cuh) with the per-symbol depth codes written by
// the whole warp: lane 0 builds the code-length code and writes its part of
// the header, then every lane places its symbols' codes at offsets from a
// warp scan.
__device__ void warp_store_complex(WarpCodeSmem& s, int num, BitSink& w, int lane) {
    int new_len{0};
    for (int i{lane}; i < num; i += 32) {
        if (s.depth[i] != 0) new_len = i + 1;
    }
#pragma unroll
    for (int off{16}; off > 0; off >>= 1) new_len = max(new_len, __shfl_xor_sync(kFull, new_len, off));
    CodeLengthScratch& scr{s.cl};
    if (lane < 18) scr.hist[lane] = 0;
    __syncwarp();
    for (int base{0}; base < new_len; base += 32) {
        const int i{base + lane};
        const int d{i < new_len ? s.depth[i] : -1};
        const unsigned peers{__match_any_sync(kFull, d)};
        if (d >= 0 && (__ffs(peers) - 1) == lane) scr.hist[d] += static_cast<std::uint32_t>(__popc(peers));
        __syncwarp();
    }
    // The code-length code: the same construction (limit 5) and canonical
    // codes, across the warp.
    if (lane < 18) {
        scr.cl_depth[lane] = 0;
        scr.cl_bits[lane] = 0;
    }
    __syncwarp();
    warp_create_tree(s, scr.hist, 18, 5, scr.cl_depth, lane);
    warp_canonical_codes(s, scr.cl_depth, 18, scr.cl_bits, lane);
    // Code-length-code header: lane i takes entry i of the transmission order
    // {1, 2, 3, 4, 0, 5, 17, 6, 16, 7, ..., 15} (six bits each below), whose
    // depth 0..5 is sent as {length, code} {2,0} {4,7} {3,3} {2,2} {2,1} {4,15}
    // (four bits each).
    const unsigned used{__ballot_sync(kFull, lane < 18 && scr.hist[lane] != 0)};
    const int num_codes{__popc(used)};
    const std::uint64_t lo10{1ull | 2ull << 6 | 3ull << 12 | 4ull << 18 | 0ull << 24 | 5ull << 30 | 17ull << 36 |
                             6ull << 42 | 16ull << 48 | 7ull << 54};
    const std::uint64_t hi8{8ull | 9ull << 6 | 10ull << 12 | 11ull << 18 | 12ull << 24 | 13ull << 30 | 14ull << 36 |
                            15ull << 42};
    const int entry{lane < 10 ? static_cast<int>((lo10 >> (6 * lane)) & 63u)
                              : (lane < 18 ? static_cast<int>((hi8 >> (6 * (lane - 10))) & 63u) : 0)};
    const int l{lane < 18 ? scr.cl_depth[entry] : 0};
    const unsigned sent{__ballot_sync(kFull, l != 0)};
    const int to_store{num_codes > 1 ? 32 - __clz(static_cast<int>(sent)) : 18};
    const int skip{(sent & 3u) != 0 ? 0 : ((sent & 4u) != 0 ? 2 : 3)};
    const std::uint32_t ln{lane >= skip && lane < to_store ? (0x422342u >> (4 * l)) & 15u : 0u};
    const std::uint32_t lincl{warp_incl_scan(ln, lane)};
    std::uint32_t pos{__shfl_sync(kFull, w.pos, 0)};
    if (lane == 0) or_bits(w.buf, pos, 2, static_cast<std::uint32_t>(skip), w.cap);
    or_bits(w.buf, pos + 2 + lincl - ln, ln, (0xf12370u >> (4 * l)) & 15u, w.cap);
    pos += 2 + __shfl_sync(kFull, lincl, 31);
    __syncwarp();
    if (num_codes == 1 && lane == 0) scr.cl_depth[__ffs(used) - 1] = 0;
    __syncwarp();
    const std::uint32_t cap{w.cap};
    for (int base{0}; base < new_len; base += 32) {
        const int i{base + lane};
        const int d{i < new_len ? s.depth[i] : 0};
        const std::uint32_t n{i < new_len ? scr.cl_depth[d] : 0u};
        const std::uint32_t incl{warp_incl_scan(n, lane)};
        or_bits(w.buf, pos + incl - n, n, scr.cl_bits[d], cap);
        pos += __shfl_sync(kFull, incl, 31);
    }
    __syncwarp();
    if (lane == 0) {
        if (pos > cap) w.overflow = true;
        w.pos = pos;
    }
}

// build_and_store for s.hist[0..length) (src/bitstream/prefix_code.cc:387-426);
// the header goes to w (lane 0's copy holds the final position).
__device__ void warp_build_and_store(WarpCodeSmem& s, int length, BitSink& w, int lane) {
    int s4[4]{0, 0, 0, 0};
    int count{0};
    for (int base{0}; base < length && count <= 4; base += 32) {
        const int sym{base + lane};
        unsigned m{__ballot_sync(kFull, sym < length && s.hist[sym] != 0)};
        while (m != 0 && count <= 4) {
            if (count < 4) s4[count] = base + __ffs(m) - 1;
            ++count;
            m &= m - 1;
        }
    }
    if (count <= 1) {
        if (lane == 0) {
            w.put(4, 1);
            w.put(alphabet_bits(length), static_cast<std::uint32_t>(s4[0]));
        }
        __syncwarp();
        return;
    }
    warp_create_tree(s, s.hist, length, 15, s.depth, lane);
    warp_canonical_codes(s, s.depth, length, s.bits, lane);
    if (count <= 4) {
        if (lane == 0) store_code_header(count, s4, length, s.depth, w, s.cl);
        __syncwarp();
        return;
    }
    warp_store_complex(s, length, w, lane);
}

// One single-warp CTA per histogram (the 32 AC clusters, then the DC and the
// AcMetadata histogram of every DC group): the merges, a tree per lane, are
// serial chains of up to 255 steps, so each warp gets an SM to itself.
__device__ __forceinline__ void codes_body(const EntropyDev& e, const unsigned blk) {
    extern __shared__ __align__(16) unsigned char code_smem[];
    const int lane{static_cast<int>(threadIdx.x) & 31};
    WarpCodeSmem& s{*reinterpret_cast<WarpCodeSmem*>(code_smem)};
    int idx;
    std::uint32_t* src;
    std::uint8_t* dst_depth;
    std::uint16_t* dst_bits;
    bool clustered;
    std::uint32_t extra0{0};
    if (blk < kNumClusters) {
        const int c{static_cast<int>(blk)};
        idx = c;
        src = e.ac_hist + c * 256;
        dst_depth = e.ac_depth + c * 256;
        dst_bits = e.ac_bits + c * 256;
        clustered = true;
    } else {
        const int g{(static_cast<int>(blk) - kNumClusters) >> 1};
        const int warp{(static_cast<int>(blk) - kNumClusters) & 1};
        if (warp == 0) {
            idx = 32 + g;
            src = e.dc_hist + g * 256;
            dst_depth = e.dc_depth + g * 256;
            dst_bits = e.dc_bits + g * 256;
        } else {
            idx = 32 + e.ndc + g;
            src = e.am_hist + g * 256;
            dst_depth = e.am_depth + g * 256;
            dst_bits = e.am_bits + g * 256;
            const GroupGeom gg{dc_group_geom(e, g)};
            extra0 = static_cast<std::uint32_t>(gg.gw * gg.gh);  // EPF zeros
        }
        clustered = false;
    }
    std::uint32_t hv[8];
#pragma unroll
    for (int k{0}; k < 8; ++k) hv[k] = src[lane + 32 * k];  // all eight loads in flight at once
    // Leave the histograms and counters zeroed for the next frame; the passes
    // after this one read the counters' frozen copies.
#pragma unroll
    for (int k{0}; k < 8; ++k) src[lane + 32 * k] = 0;
    if (lane == 0 && blk == 0) {
        e.frozen[0] = *e.tok_count;
        *e.tok_count = 0;
    }
    if (lane == 0 && idx >= 32 + e.ndc) {
        const int g{idx - 32 - e.ndc};
        e.frozen[1 + g] = e.fb_count[g];
        e.fb_count[g] = 0;
    }
#pragma unroll
    for (int k{0}; k < 8; ++k) {
        const int i{lane + 32 * k};
        s.hist[i] = hv[k] + (i == 0 ? extra0 : 0u);
        s.depth[i] = 0;
        s.bits[i] = 0;
    }
    for (int i{lane}; i < kDescBytes / 4; i += 32) reinterpret_cast<std::uint32_t*>(s.desc)[i] = 0;
    __syncwarp();
    int alpha{1};
    for (int i{lane}; i < 256; i += 32) {
        if (s.hist[i]) alpha = i + 1;
    }
#pragma unroll
    for (int off{16}; off > 0; off >>= 1) alpha = max(alpha, __shfl_xor_sync(kFull, alpha, off));
    BitSink w{s.desc, 0, kDescBytes * 8, false};
    if (!clustered && lane == 0) {
        // Single-context prefix histogram header (src/bitstream/histogram_writer.cc:59-83).
        w.put(1, 0);
        w.put(1, 1);
        put_uint_config(w, 4, 2, 0);
        put_var_len_u16(w, static_cast<std::uint32_t>(alpha - 1));
    }
    if (clustered && lane == 0) e.ac_alpha[idx] = static_cast<std::uint32_t>(alpha);
    if (alpha > 1) warp_build_and_store(s, alpha, w, lane);
    __syncwarp();
    std::uint32_t nbits{w.overflow ? 0u : w.pos};
    nbits = __shfl_sync(kFull, nbits, 0);
    if (lane == 0) e.desc_bits[idx] = nbits;
    std::uint8_t* d{e.desc + idx * kDescBytes};
    for (int i{lane}; i < kDescBytes; i += 32) d[i] = s.desc[i];
    for (int i{lane}; i < 256; i += 32) {
        dst_depth[i] = s.depth[i];
        dst_bits[i] = s.bits[i];
    }
    std::uint32_t* code{e.code + (clustered ? idx * kAcSymbols : kNumClusters * kAcSymbols + (idx - 32) * kMiscSymbols)};
    for (int i{lane}; i < (clustered ? kAcSymbols : kMiscSymbols); i += 32) {
        code[i] = (static_cast<std::uint32_t>(s.depth[i]) << 16) | s.bits[i];
    }
}

// One histogram through the device builder (test hook): `length` symbols,
// depths, codes and the header (simple or code-length-code form) out.
__global__ void __launch_bounds__(32) prefix_code_test_kernel(const std::uint32_t* hist, int length,
                                                              std::uint8_t* depth, std::uint16_t* bits,
                                                              std::uint8_t* header, std::uint32_t* nbits) {
    extern __shared__ __align__(16) unsigned char code_smem[];
    const int lane{static_cast<int>(threadIdx.x) & 31};
    WarpCodeSmem& s{*reinterpret_cast<WarpCodeSmem*>(code_smem)};
    for (int i{lane}; i < 256; i += 32) {
        s.hist[i] = i < length ? hist[i] : 0u;
        s.depth[i] = 0;
        s.bits[i] = 0;
    }
    for (int i{lane}; i < kDescBytes; i += 32) s.desc[i] = 0;
    __syncwarp();
    BitSink w{s.desc, 0, kDescBytes * 8, false};
    warp_build_and_store(s, length, w, lane);
    __syncwarp();
    for (int i{lane}; i < length; i += 32) {
        depth[i] = s.depth[i];
        bits[i] = s.bits[i];
    }
    for (int i{lane}; i < kDescBytes; i += 32) header[i] = s.desc[i];
    if (lane == 0) *nbits = w.overflow ? 0xffffffffu : w.pos;
}

// ---- pass 3: bit lengths, scan and layout ----------------------------------------------------

// Bits of a stripe whose tokens are stored: the sum over its tokens. (Only
// the start of a stripe is ever looked up, so its items get no prefixes.)
__device__ __forceinline__ void ac_bits_stored_body(const EntropyDev& e, const unsigned blk) {
    __shared__ std::uint32_t sh_sum[kAcWarps];
    const int tid{static_cast<int>(threadIdx.x)};
    const Stripe st{e.stripes[blk]};
    const StripeTokens pool{stripe_tokens(e, st, blk, st.rows * st.cols)};
    if (pool.near == nullptr) return;  // summed by the pass over unstored stripes
    const std::uint32_t ntok{e.stripe_tok[2 * blk + 1]};
    std::uint32_t sum{0};
#pragma unroll 4
    for (std::uint32_t t{static_cast<std::uint32_t>(tid)}; t < ntok; t += kAcThreads) {
        const std::uint32_t tk{*pool.at(t)};
        sum += (e.code[token_code_index(tk)] >> 16) + token_extra_count(tk);
    }
    sum = warp_sum(sum);
    if ((tid & 31) == 0) sh_sum[tid >> 5] = sum;
    __syncthreads();
    if (tid == 0) {
        std::uint32_t total{0};
        for (int w{0}; w < kAcWarps; ++w) total += sh_sum[w];
        e.unit_sum[e.misc_units + blk] = total;
    }
}

// Bits of a stripe whose tokens are not stored, and each item's prefix.
__device__ __forceinline__ void ac_bits_unstored_body(const EntropyDev& e, const unsigned blk) {
    extern __shared__ __align__(16) unsigned char ac_smem[];
    StripeStage& s{*reinterpret_cast<StripeStage*>(ac_smem)};
    __shared__ std::uint32_t sh_scan[kAcWarps + 1];
    const int tid{static_cast<int>(threadIdx.x)};
    const int lane{tid & 31};
    const Stripe st{e.stripes[blk]};
    const GroupGeom gg{ac_group_geom(e, st.group)};
    stage_stripe(e, st, gg, s);
    __syncthreads();
    const int nitems{3 * st.rows * gg.gw};
    for (int j{tid}; j < nitems; j += kAcThreads) {
        const StripeItem it{stripe_item(s, gg.gw, j)};
        std::uint32_t b{0};
        if (it.n != 0) {
            int cl;
            std::uint32_t tok, nb, bits;
            count_token(s, st, it, cl, tok, nb, bits);
            b = e.ac_depth[cl * 256 + tok] + nb;
            if (it.nz != 0) s.active[atomicAdd(&s.nactive, 1)] = static_cast<std::uint16_t>(j);
        }
        s.aux[j] = b;
    }
    __syncthreads();
    for (int a{tid >> 5}; a < s.nactive; a += kAcWarps) {
        const int j{s.active[a]};
        const StripeItem it{stripe_item(s, gg.gw, j)};
        std::uint32_t total{0};
        coeff_tokens(s, it, lane, [&](bool has, int cl, std::uint32_t sym, std::uint32_t nb, std::uint32_t) {
            if (has) total += e.ac_depth[cl * 256 + sym] + nb;
        });
        total = warp_sum(total);
        if (lane == 0) s.aux[j] += total;
    }
    __syncthreads();
    const int j0{2 * tid};
    const std::uint32_t b0{j0 < nitems ? s.aux[j0] : 0u};
    const std::uint32_t b1{j0 + 1 < nitems ? s.aux[j0 + 1] : 0u};
    std::uint32_t total{0};
    const std::uint32_t off{cta_exclusive_scan(b0 + b1, sh_scan, total)};
    if (j0 < nitems) e.item_pre[st.item0 + j0] = off;
    if (j0 + 1 < nitems) e.item_pre[st.item0 + j0 + 1] = off + b0;
    if (tid == 0) e.unit_sum[e.misc_units + blk] = total;
}

struct BitsVisitor {
    const EntropyDev* e;
    std::uint32_t total;
    __device__ void blob(const std::uint8_t*, std::uint32_t nbits) { total += nbits; }
    __device__ void varlen(std::uint32_t v) {
        if (v == 0) {
            total += 1;
        } else {
            unsigned nb{0};
            for (std::uint32_t x{v}; x > 1; x >>= 1) ++nb;
            total += 5 + nb;
        }
    }
    __device__ void count_field(int, unsigned nbits) { total += nbits; }
    __device__ void epf(int) {}  // kept as tokens, not visited again
    __device__ void first_block(int) {}
    __device__ void token(int tab, int g, std::uint32_t sym, std::uint32_t nb, std::uint32_t) {
        total += (tab == kTabDc ? e->dc_depth : e->am_depth)[g * 256 + sym] + nb;
    }
};

// Bits of a unit of other items, and each item's prefix in it; thread t takes
// items 2t and 2t + 1.
__device__ __forceinline__ void misc_bits_body(const EntropyDev& e, const unsigned blk) {
    __shared__ std::uint32_t sh_scan[kAcWarps + 1];
    const std::uint32_t item0{blk * kMiscItemsPerUnit + kMiscPerThread * threadIdx.x};
    std::uint32_t bits[kMiscPerThread]{};
    std::uint32_t tok[kMiscPerThread];
#pragma unroll
    for (int k{0}; k < kMiscPerThread; ++k) tok[k] = item0 + k < e.ac_first ? e.item_tok[item0 + k] : kMiscNone;
    int sat{static_cast<int>(e.unit_section[blk])};
#pragma unroll
    for (int k{0}; k < kMiscPerThread; ++k) {
        if (tok[k] == kMiscNone) continue;
        const Section sec{section_from(e, sat, item0 + k)};
        if (tok[k] == kMiscVisit) {
            BitsVisitor v{&e, 0};
            visit_misc(e, sec, item0 + k - sec.first, v);
            bits[k] = v.total;
        } else {
            bits[k] = (misc_code(e, sec.group, tok[k]) >> 16) + misc_extra_count(tok[k]);
        }
    }
    std::uint32_t total{0};
    const std::uint32_t off{cta_exclusive_scan(bits[0] + bits[1], sh_scan, total)};
    if (item0 < e.ac_first) e.item_pre[item0] = off;
    if (item0 + 1 < e.ac_first) e.item_pre[item0 + 1] = off + bits[0];
    if (threadIdx.x == 0) e.unit_sum[blk] = total;
}

// ---- pass 4: layout ---------------------------------------------------------------

// TOC entry of a section of `bytes` bytes: U32 with selectors 0 + 10 bits,
// 1024 + 14, 17408 + 22, 4211712 + 30 (src/bitstream/codestream.cc:16-18, 91-98);
// the smallest selector that holds the value, as one LSB-first field.
__device__ __forceinline__ void toc_entry(std::uint32_t bytes, std::uint32_t& nbits, std::uint32_t& field) {
    std::uint32_t sel;
    std::uint32_t base;
    std::uint32_t extra;
    if (bytes < 1024u) {
        sel = 0; base = 0; extra = 10;
    } else if (bytes < 17408u) {
        sel = 1; base = 1024; extra = 14;
    } else if (bytes < 4211712u) {
        sel = 2; base = 17408; extra = 22;
    } else {
        sel = 3; base = 4211712; extra = 30;
    }
    nbits = 2 + extra;
    field = sel | ((bytes - base) << 2);
}

constexpr int kLayoutThreads = 1024;
constexpr int kLayoutWarps = kLayoutThreads / 32;

// Block-wide exclusive scan of one 64-bit value per thread of the layout CTA;
// returns the thread's offset and sets `total`.
__device__ unsigned long long block_scan(unsigned long long v, unsigned long long* warp_sums,
                                         unsigned long long& total) {
    const int lane{static_cast<int>(threadIdx.x) & 31};
    const int warp{static_cast<int>(threadIdx.x) >> 5};
    unsigned long long incl{v};
#pragma unroll
    for (int off{1}; off < 32; off <<= 1) {
        const unsigned long long t{__shfl_up_sync(kFull, incl, off)};
        if (lane >= off) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    // Every warp scans the warps' sums itself.
    const unsigned long long x{warp_sums[lane]};
    unsigned long long sums{x};
#pragma unroll
    for (int off{1}; off < 32; off <<= 1) {
        const unsigned long long t{__shfl_up_sync(kFull, sums, off)};
        if (lane >= off) sums += t;
    }
    const unsigned long long before{__shfl_sync(kFull, sums - x, warp)};
    total = __shfl_sync(kFull, sums, 31);
    __syncthreads();
    return before + incl - v;
}

// Zeroes word w of the output, or those of its bytes that lie in the file.
__device__ __forceinline__ void zero_out_word(const EntropyDev& e, unsigned long long w, unsigned long long file_bytes) {
    if (4 * w + 4 <= file_bytes) {
        reinterpret_cast<std::uint32_t*>(e.out)[w] = 0;
    } else {
        for (unsigned long long b{4 * w}; b < file_bytes; ++b) e.out[b] = 0;
    }
}

// Scans the units, sizes the sections, places sections and units, and writes
// the container framing, the codestream headers and the TOC
// (src/bitstream/codestream.cc:57-135, src/bitstream/container.cc:35-62). The
// emission ORs its bits into the words that units or sections share, so those
// are zeroed here; a unit stores the words it has to itself.
//
// One CTA per frame. Its time is that of its chains of dependent loads, so
// sections and units are looked up two levels deep and loads go ahead of
// stores.
__device__ __forceinline__ void layout_body(const EntropyDev& e) {
    __shared__ unsigned long long scan_sums[kLayoutWarps];
    const int tid{static_cast<int>(threadIdx.x)};
    const std::uint32_t units{e.misc_units + static_cast<std::uint32_t>(e.nstripes)};
    // This thread's sections (a contiguous run of TOC entries): what their
    // starts depend on, loaded while the units are scanned. With one AC group
    // the four sections are one combined TOC entry: their bits follow each
    // other with no padding between them (tools/bitstream/vardct_frame.cc:414-449).
    const bool single{e.nac == 1};
    const int ntoc{single ? 1 : e.nsec};
    const int per{(ntoc + kLayoutThreads - 1) / kLayoutThreads};
    const int lo{min(ntoc, tid * per)};
    const int hi{min(ntoc, lo + per)};
    // Unit offsets, four units per thread and round (unit_sum and unit_off
    // have room for whole vectors of four).
    unsigned long long carry{0};
    for (std::uint32_t u0{0}; u0 < units; u0 += kLayoutThreads * 4) {
        const std::uint32_t at{u0 + static_cast<std::uint32_t>(tid) * 4};
        uint4 x{at < units ? *reinterpret_cast<const uint4*>(e.unit_sum + at) : make_uint4(0, 0, 0, 0)};
        if (at + 1 >= units) x.y = 0;
        if (at + 2 >= units) x.z = 0;
        if (at + 3 >= units) x.w = 0;
        unsigned long long total{0};
        const unsigned long long off{
            carry + block_scan(static_cast<unsigned long long>(x.x) + x.y + x.z + x.w, scan_sums, total)};
        if (at < units) {
            auto* dst{reinterpret_cast<ulonglong2*>(e.unit_off + at)};
            dst[0] = make_ulonglong2(off, off + x.x);
            dst[1] = make_ulonglong2(off + x.x + x.y, off + x.x + x.y + x.z);
        }
        carry += total;
    }
    __syncthreads();
    if (tid == 0) e.unit_off[units] = carry;
    __syncthreads();

    std::uint32_t nb{0};  // of the last entry: of the only one in all but the largest frames
    std::uint32_t field{0};
    unsigned long long my_bits{0};
    unsigned long long my_bytes{0};
    unsigned long long start{lo < hi ? section_start(e, lo) : 0ull};
    for (int s{lo}; s < hi; ++s) {
        const unsigned long long next{section_start(e, single ? e.nsec : s + 1)};
        const std::uint32_t bytes{static_cast<std::uint32_t>((next - start + 7) / 8)};
        start = next;
        toc_entry(bytes, nb, field);
        my_bits += nb;
        my_bytes += bytes;
        e.sec_shift[s] = bytes;
    }
    unsigned long long toc_bits{0};
    unsigned long long body{0};
    const unsigned long long toc_off{block_scan(my_bits, scan_sums, toc_bits)};
    const unsigned long long byte_off{block_scan(my_bytes, scan_sums, body)};
    const unsigned long long head{e.head_bytes + (toc_bits + 7) / 8};
    const unsigned long long cs{head + body};
    const bool large{cs >= 0x100000000ull - 8};
    const unsigned long long framing{32ull + (large ? 16 : 8)};
    const unsigned long long file{framing + cs};
    // 2: the file would reach the tokens kept at the buffer's end (never:
    // dense_tokens).
    const unsigned long long dense{e.direct ? 4ull * e.frozen[0] : 0ull};
    const unsigned long long status{
        file > e.out_capacity ? 1ull : (dense != 0 && file + dense > e.out_capacity ? 2ull : 0ull)};
    if (tid == 0) {
        e.result[0] = file;
        e.result[1] = framing + head;
        e.result[2] = status;
    }
    if (status != 0) return;

    // Each section's shift from its bits' place in the scan to their place in
    // the file (sections are padded to whole bytes, but not the combined ones).
    if (single) {
        for (int s{tid}; s < e.nsec; s += kLayoutThreads) e.sec_shift[s] = 8 * (framing + head);
    } else {
        unsigned long long pos{framing + head + byte_off};
        start = lo < hi ? section_start(e, lo) : 0ull;
        for (int s{lo}; s < hi; ++s) {
            const unsigned long long bytes{e.sec_shift[s]};
            e.sec_shift[s] = 8 * pos - start;
            pos += bytes;
            if (s + 1 < hi) start = section_start(e, s + 1);
        }
    }
    __syncthreads();
    // Unit positions; the words that hold a unit's first or last bit. Four
    // units' loads at a time, ahead of their stores.
    for (std::uint32_t u0{static_cast<std::uint32_t>(tid)}; u0 < units; u0 += 4 * kLayoutThreads) {
        unsigned long long pos[4];
        std::uint32_t bits[4];
        std::uint32_t sec[4];
#pragma unroll
        for (int k{0}; k < 4; ++k) {
            const std::uint32_t u{min(u0 + k * kLayoutThreads, units - 1)};
            sec[k] = e.unit_section[u];
            pos[k] = e.unit_off[u];
            bits[k] = e.unit_sum[u];
        }
#pragma unroll
        for (int k{0}; k < 4; ++k) pos[k] += e.sec_shift[sec[k]];
#pragma unroll
        for (int k{0}; k < 4; ++k) {
            const std::uint32_t u{u0 + k * kLayoutThreads};
            if (u >= units) break;
            e.unit_pos[u] = pos[k];
            // A unit of several sections has its last bit elsewhere, in words
            // zeroed below; the one found here is then some other word of the body.
            const unsigned long long last{(pos[k] + (bits[k] != 0 ? bits[k] - 1 : 0)) >> 5};
            zero_out_word(e, pos[k] >> 5, file);
            zero_out_word(e, last, file);
        }
    }
    // Sections that start inside a unit: the emission ORs that unit's part of
    // them bit by bit, and the section before them ends there. A warp each.
    for (int s{1 + (tid >> 5)}; s < e.ndc + 2; s += kLayoutWarps) {
        const Section sec{e.sections[s]};
        if (sec.first % kMiscItemsPerUnit == 0) continue;
        const std::uint32_t end{min(sec.first + sec.count, (sec.unit + 1) * kMiscItemsPerUnit)};
        const unsigned long long from{section_start(e, s)};
        const unsigned long long to{end < sec.first + sec.count ? e.unit_off[sec.unit + 1] : section_start(e, s + 1)};
        const unsigned long long shift{e.sec_shift[s]};
        for (unsigned long long w{((shift + from) >> 5) + (tid & 31)}; w < (shift + to + 31) >> 5; w += 32) {
            zero_out_word(e, w, file);
        }
        if ((tid & 31) == 0) zero_out_word(e, (e.sec_shift[s - 1] + from - 1) >> 5, file);
    }
    const unsigned long long head_w0{framing / 4};
    for (unsigned long long w{head_w0 + tid}; 4 * w < framing + head; w += kLayoutThreads) zero_out_word(e, w, file);
    __syncthreads();

    // Container framing in bytes, headers and TOC ORed in.
    if (tid < 48) {
        constexpr std::uint8_t kHead[32]{0, 0, 0, 0x0c, 'J', 'X', 'L', ' ', 0x0d, 0x0a, 0x87, 0x0a, 0, 0, 0, 0x14,
                                         'f', 't', 'y', 'p', 'j', 'x', 'l', ' ', 0, 0, 0, 0, 'j', 'x', 'l', ' '};
        constexpr std::uint8_t kBox[4]{'j', 'x', 'l', 'c'};
        const unsigned long long box{cs + (large ? 16 : 8)};
        const std::uint32_t sf{large ? 1u : static_cast<std::uint32_t>(box)};
        if (tid < 32) {
            e.out[tid] = kHead[tid];
        } else if (tid < 36) {
            e.out[tid] = static_cast<std::uint8_t>(sf >> (8 * (35 - tid)));
        } else if (tid < 40) {
            e.out[tid] = kBox[tid - 36];
        } else if (large) {
            e.out[tid] = static_cast<std::uint8_t>(box >> (8 * (47 - tid)));
        }
    }
    auto* words{reinterpret_cast<unsigned int*>(e.out)};
    if (tid < 4 && e.head_words[tid] != 0) atomicOr(&words[head_w0 + tid], e.head_words[tid]);
    unsigned long long p{8 * (framing + e.head_bytes) + toc_off};
    for (int s{lo}; s < hi; ++s) {
        if (hi - lo > 1) {
            const unsigned long long from{section_start(e, s)};
            toc_entry(static_cast<std::uint32_t>((section_start(e, s + 1) - from + 7) / 8), nb, field);
        }
        const std::uint32_t off{static_cast<std::uint32_t>(p & 31)};
        atomicOr(&words[p >> 5], field << off);
        if (off + nb > 32) atomicOr(&words[(p >> 5) + 1], field >> (32 - off));
        p += nb;
    }
}

__device__ __forceinline__ void lengths_body(const EntropyDev& e, const unsigned blk) {
    if (blk < static_cast<unsigned>(e.nstripes)) {
        ac_bits_stored_body(e, blk);
    } else {
        misc_bits_body(e, blk - static_cast<unsigned>(e.nstripes));
    }
}

// ---- pass 5: emission ------------------------------------------------------------

// Copies a window of `nwords` assembled words to global word w0 onward. The
// first and last words can share bits with neighbouring items and are ORed
// in; every word between lies wholly inside the window's bit range and is
// stored.
__device__ void flush_window(const unsigned int* win, int nwords, unsigned int* gwords, unsigned long long w0) {
    for (int i{static_cast<int>(threadIdx.x)}; i < nwords; i += blockDim.x) {
        const unsigned int v{win[i]};
        if (i == 0 || i == nwords - 1) {
            if (v != 0) atomicOr(&gwords[w0 + i], v);
        } else {
            gwords[w0 + i] = v;
        }
    }
}

// Where a unit's bits go: a shared-memory window of the words they touch, or,
// when those exceed the window, the output itself, whose words between the
// unit's first and last (zeroed by the layout) the CTA zeroes here. `base` is
// the unit's first bit in `words`.
struct EmitTarget {
    unsigned int* words;
    unsigned long long base;
    unsigned long long w0;  // first word of the unit in the output
    int window;             // words of the window, -1 without one
};

__device__ __forceinline__ EmitTarget emit_target(const EntropyDev& e, unsigned long long pos, std::uint32_t bits,
                                                  unsigned int* win, int capacity) {
    auto* out{reinterpret_cast<unsigned int*>(e.out)};
    const unsigned long long w0{pos >> 5};
    const unsigned long long nw{bits == 0 ? 0ull : ((pos + bits + 31) >> 5) - w0};
    if (nw <= static_cast<unsigned long long>(capacity)) {
        for (int i{static_cast<int>(threadIdx.x)}; i < static_cast<int>(nw); i += blockDim.x) win[i] = 0;
        return {win, pos & 31, w0, static_cast<int>(nw)};
    }
    for (unsigned long long w{w0 + 1 + threadIdx.x}; w + 1 < w0 + nw; w += blockDim.x) out[w] = 0;
    return {out, pos, w0, -1};
}

// Writes a stored stripe's tokens, in stream order: their lengths, a CTA scan
// for their offsets, and their bits, eight consecutive tokens per thread and
// round gathered into whole words on the way to the window.
//
// Latency-bound: one round (2048 tokens; a stripe of a 4K frame at distance 1
// has some 1400) is a pool load, the scan and the stores, where rounds of four
// tokens with two or three ORs each into shared memory took several: 9-12K
// cycles a stripe, now 3-5K. The code table is copied to shared memory while
// the first tokens load.
__device__ __forceinline__ void ac_emit_stored_body(const EntropyDev& e, const unsigned blk) {
    extern __shared__ __align__(16) unsigned char ac_smem[];
    unsigned int* win{reinterpret_cast<unsigned int*>(ac_smem)};                     // [kWindowWords]
    auto* code{reinterpret_cast<std::uint32_t*>(ac_smem + kWindowWords * 4)};        // [32][64]
    __shared__ std::uint32_t sh_scan[kAcWarps + 1];
    constexpr int kPer{8};
    const std::uint32_t tid{threadIdx.x};
    const Stripe st{e.stripes[blk]};
    const StripeTokens pool{stripe_tokens(e, st, blk, st.rows * st.cols)};
    if (pool.near == nullptr || e.result[2] != 0) return;
    const std::uint32_t ntok{e.stripe_tok[2 * blk + 1]};
    const unsigned long long pos{e.unit_pos[e.misc_units + blk]};
    const std::uint32_t bits{e.unit_sum[e.misc_units + blk]};
    for (int i{static_cast<int>(tid)}; i < kNumClusters * kAcSymbols / 4; i += kAcThreads) {
        reinterpret_cast<uint4*>(code)[i] = reinterpret_cast<const uint4*>(e.code)[i];
    }
    const EmitTarget to{emit_target(e, pos, bits, win, kWindowWords)};
    __syncthreads();
    unsigned long long run{to.base};
    for (std::uint32_t t0{0}; t0 < ntok; t0 += kAcThreads * kPer) {
        const std::uint32_t t{t0 + tid * kPer};
        std::uint32_t tk[kPer];
        std::uint32_t cd[kPer];
        std::uint32_t local{0};
        // A thread's eight tokens lie on one side of the split. Direct places
        // are 16-byte aligned, reserved runs may not be.
        const std::uint32_t* src{pool.at(t)};
        if (t + kPer <= ntok && (reinterpret_cast<std::uintptr_t>(src) & 15u) == 0) {
            const uint4 a{reinterpret_cast<const uint4*>(src)[0]};
            const uint4 b{reinterpret_cast<const uint4*>(src)[1]};
            tk[0] = a.x; tk[1] = a.y; tk[2] = a.z; tk[3] = a.w;
            tk[4] = b.x; tk[5] = b.y; tk[6] = b.z; tk[7] = b.w;
        } else {
#pragma unroll
            for (int i{0}; i < kPer; ++i) tk[i] = t + i < ntok ? src[i] : 0u;
        }
#pragma unroll
        for (int i{0}; i < kPer; ++i) {
            cd[i] = t + i < ntok ? code[token_code_index(tk[i])] : 0u;
            local += (cd[i] >> 16) + (t + i < ntok ? token_extra_count(tk[i]) : 0u);
        }
        std::uint32_t total{0};
        const unsigned long long at{run + cta_exclusive_scan(local, sh_scan, total)};
        unsigned int* w{to.words + (at >> 5)};
        unsigned long long acc{0};
        std::uint32_t fill{static_cast<std::uint32_t>(at & 31)};
#pragma unroll
        for (int i{0}; i < kPer; ++i) {
            if (t + i >= ntok) break;
            const std::uint32_t depth{cd[i] >> 16};
            const std::uint32_t v{(cd[i] & 0xffffu) | (token_extra_bits(tk[i]) << depth)};
            acc |= static_cast<unsigned long long>(v) << fill;  // at most 15 + 13 bits on at most 31
            fill += depth + token_extra_count(tk[i]);
            if (fill >= 32) {
                atomicOr(w++, static_cast<unsigned int>(acc));
                acc >>= 32;
                fill -= 32;
            }
        }
        if (acc != 0) atomicOr(w, static_cast<unsigned int>(acc));
        run += total;
    }
    __syncthreads();
    if (to.window > 0) flush_window(win, to.window, reinterpret_cast<unsigned int*>(e.out), to.w0);
}

// Tokenises an unstored stripe again and writes its tokens.
__device__ __forceinline__ void ac_emit_unstored_body(const EntropyDev& e, const unsigned blk) {
    extern __shared__ __align__(16) unsigned char ac_smem[];
    StripeStage& s{*reinterpret_cast<StripeStage*>(ac_smem)};
    unsigned int* win{reinterpret_cast<unsigned int*>(ac_smem + sizeof(StripeStage))};
    const int tid{static_cast<int>(threadIdx.x)};
    const int lane{tid & 31};
    const Stripe st{e.stripes[blk]};
    const GroupGeom gg{ac_group_geom(e, st.group)};
    const int nitems{3 * st.rows * gg.gw};
    stage_stripe(e, st, gg, s);
    const EmitTarget to{
        emit_target(e, e.unit_pos[e.misc_units + blk], e.unit_sum[e.misc_units + blk], win, kWindowWords)};
    __syncthreads();
    for (int j{tid}; j < nitems; j += kAcThreads) s.aux[j] = e.item_pre[st.item0 + j];
    __syncthreads();
    for (int j{tid}; j < nitems; j += kAcThreads) {
        const StripeItem it{stripe_item(s, gg.gw, j)};
        if (it.n == 0) continue;
        int cl;
        std::uint32_t tok, nb, bits;
        count_token(s, st, it, cl, tok, nb, bits);
        const std::uint32_t d{e.ac_depth[cl * 256 + tok]};
        const unsigned long long at{to.base + s.aux[j]};
        put_bits_at(to.words, at, d, e.ac_bits[cl * 256 + tok]);
        if (nb) put_bits_at(to.words, at + d, nb, bits);
        if (it.nz != 0) {
            s.active[atomicAdd(&s.nactive, 1)] = static_cast<std::uint16_t>(j);
            s.aux[j] += d + nb;  // coefficient tokens start after the count token
        }
    }
    __syncthreads();
    for (int a{tid >> 5}; a < s.nactive; a += kAcWarps) {
        const int j{s.active[a]};
        const StripeItem it{stripe_item(s, gg.gw, j)};
        unsigned long long pos{to.base + s.aux[j]};
        coeff_tokens(s, it, lane, [&](bool has, int cl, std::uint32_t sym, std::uint32_t nb, std::uint32_t bits) {
            const std::uint32_t d{has ? e.ac_depth[cl * 256 + sym] : 0u};
            const std::uint32_t tb{has ? d + nb : 0u};
            const std::uint32_t incl{warp_incl_scan(tb, lane)};
            if (has) {
                const unsigned long long at{pos + incl - tb};
                put_bits_at(to.words, at, d, e.ac_bits[cl * 256 + sym]);
                if (nb) put_bits_at(to.words, at + d, nb, bits);
            }
            pos += __shfl_sync(kFull, incl, 31);
        });
    }
    __syncthreads();
    if (to.window > 0) flush_window(win, to.window, reinterpret_cast<unsigned int*>(e.out), to.w0);
}

// A header blob long enough to be written by the whole CTA (the AcGlobal
// prefix with its context map runs to tens of thousands of bits).
struct DeferredBlob {
    unsigned int* words;
    unsigned long long pos;
    const std::uint8_t* src;  // 4-byte aligned, readable in whole words
    std::uint32_t nbits;
};
constexpr int kMaxDeferred = 32;
constexpr std::uint32_t kDeferBits = 256;

struct EmitVisitor {
    const EntropyDev* e;
    unsigned int* words;
    unsigned long long pos;
    DeferredBlob* deferred{nullptr};
    int* ndeferred{nullptr};
    __device__ void put(std::uint32_t n, std::uint32_t v) {
        if (n == 0) return;
        if (n < 32) v &= (1u << n) - 1u;
        put_bits_at(words, pos, n, v);
        pos += n;
    }
    __device__ void blob(const std::uint8_t* b, std::uint32_t nbits) {
        if (deferred != nullptr && nbits > kDeferBits) {
            const int k{atomicAdd(ndeferred, 1)};
            if (k < kMaxDeferred) {
                deferred[k] = DeferredBlob{words, pos, b, nbits};
                pos += nbits;
                return;
            }
        }
        std::uint32_t i{0};
        for (; i + 32 <= nbits; i += 32) {
            put(32, static_cast<std::uint32_t>(b[i >> 3]) | (static_cast<std::uint32_t>(b[(i >> 3) + 1]) << 8) |
                        (static_cast<std::uint32_t>(b[(i >> 3) + 2]) << 16) |
                        (static_cast<std::uint32_t>(b[(i >> 3) + 3]) << 24));
        }
        for (; i + 8 <= nbits; i += 8) put(8, b[i >> 3]);
        if (i < nbits) put(nbits - i, b[i >> 3]);
    }
    __device__ void varlen(std::uint32_t v) {
        if (v == 0) {
            put(1, 0);
            return;
        }
        put(1, 1);
        unsigned nb{0};
        for (std::uint32_t x{v}; x > 1; x >>= 1) ++nb;
        put(4, nb);
        put(nb, v - (1u << nb));
    }
    __device__ void count_field(int g, unsigned nbits) { put(nbits, e->frozen[1 + g] - 1); }
    __device__ void epf(int) {}  // kept as tokens, not visited again
    __device__ void first_block(int) {}
    __device__ void token(int tab, int g, std::uint32_t sym, std::uint32_t nb, std::uint32_t bits) {
        const std::uint8_t* d{tab == kTabDc ? e->dc_depth : e->am_depth};
        const std::uint16_t* c{tab == kTabDc ? e->dc_bits : e->am_bits};
        put(d[g * 256 + sym], c[g * 256 + sym]);
        if (nb) put(nb, bits);
    }
};

constexpr int kMiscWindowWords = 2048;

// One unit of other items, two per thread; the bits of the items that share the
// first item's section go through a shared-memory window.
__device__ __forceinline__ void misc_emit_body(const EntropyDev& e, const unsigned blk) {
    extern __shared__ __align__(16) unsigned char misc_smem[];
    unsigned int* win{reinterpret_cast<unsigned int*>(misc_smem)};                              // [kMiscWindowWords]
    DeferredBlob* deferred{reinterpret_cast<DeferredBlob*>(misc_smem + kMiscWindowWords * 4)};  // [kMaxDeferred]
    __shared__ int sh_ndeferred;
    if (e.result[2] != 0) return;
    const std::uint32_t first{blk * kMiscItemsPerUnit};
    const int sfirst{static_cast<int>(e.unit_section[blk])};
    const Section sec0{e.sections[sfirst]};
    const unsigned long long pos0{e.unit_pos[blk]};
    if (threadIdx.x == 0) sh_ndeferred = 0;
    const bool whole{sec0.first + sec0.count >= min(first + kMiscItemsPerUnit, e.ac_first)};
    const std::uint32_t bits{whole ? e.unit_sum[blk]
                                   : static_cast<std::uint32_t>(section_start(e, sfirst + 1) - e.unit_off[blk])};
    const EmitTarget to{emit_target(e, pos0, bits, win, kMiscWindowWords)};
    __syncthreads();
    std::uint32_t tok[kMiscPerThread];
    std::uint32_t pre[kMiscPerThread];
#pragma unroll
    for (int k{0}; k < kMiscPerThread; ++k) {
        const std::uint32_t item{first + threadIdx.x + k * kAcThreads};
        tok[k] = item < e.ac_first ? e.item_tok[item] : kMiscNone;
        pre[k] = item < e.ac_first ? e.item_pre[item] : 0u;
    }
#pragma unroll
    for (int k{0}; k < kMiscPerThread; ++k) {
        if (tok[k] == kMiscNone) continue;
        const std::uint32_t item{first + threadIdx.x + k * kAcThreads};
        int sat{sfirst};
        const Section sec{section_from(e, sat, item)};
        unsigned int* words{to.words};
        unsigned long long pos{to.base + pre[k]};
        if (sat != sfirst) {
            words = reinterpret_cast<unsigned int*>(e.out);
            pos = e.sec_shift[sat] + e.unit_off[blk] + pre[k];
        }
        if (tok[k] == kMiscVisit) {
            EmitVisitor v{&e, words, pos, deferred, &sh_ndeferred};
            visit_misc(e, sec, item - sec.first, v);
        } else {
            // At most 15 + 18 bits on at most 31: two words.
            const std::uint32_t cd{misc_code(e, sec.group, tok[k])};
            const unsigned long long v{((cd & 0xffffu) |
                                        (static_cast<unsigned long long>(misc_extra_bits(tok[k])) << (cd >> 16)))
                                       << (pos & 31)};
            if (static_cast<unsigned int>(v) != 0) atomicOr(&words[pos >> 5], static_cast<unsigned int>(v));
            if ((v >> 32) != 0) atomicOr(&words[(pos >> 5) + 1], static_cast<unsigned int>(v >> 32));
        }
    }
    __syncthreads();
    // Long blobs, one 32-bit word of each per thread.
    const int nd{min(sh_ndeferred, kMaxDeferred)};
    for (int k{0}; k < nd; ++k) {
        const DeferredBlob d{deferred[k]};
        const auto* src{reinterpret_cast<const std::uint32_t*>(d.src)};
        for (std::uint32_t w{threadIdx.x}; 32 * w < d.nbits; w += blockDim.x) {
            const std::uint32_t n{min(32u, d.nbits - 32 * w)};
            std::uint32_t v{src[w]};
            if (n < 32) v &= (1u << n) - 1u;
            put_bits_at(d.words, d.pos + 32ull * w, n, v);
        }
    }
    __syncthreads();
    if (to.window > 0) flush_window(win, to.window, reinterpret_cast<unsigned int*>(e.out), to.w0);
}

// Zeroes a frame's histograms, first-block counts and token-pool fill; block
// blk of nblk takes every nblk-th 256-word stretch.
__device__ __forceinline__ void clear_body(const EntropyDev& e, unsigned blk, unsigned nblk) {
    const unsigned stride{nblk * blockDim.x};
    const unsigned t0{blk * blockDim.x + threadIdx.x};
    for (unsigned i{t0}; i < static_cast<unsigned>(kNumClusters * 256); i += stride) e.ac_hist[i] = 0;
    for (unsigned i{t0}; i < static_cast<unsigned>(e.ndc) * 256u; i += stride) {
        e.dc_hist[i] = 0;
        e.am_hist[i] = 0;
    }
    for (unsigned i{t0}; i < static_cast<unsigned>(e.ndc); i += stride) e.fb_count[i] = 0;
    if (t0 == 0) *e.tok_count = 0;
}

// Blocks of a frame's clear: one per 32 DC groups (8192 histogram words each).
__host__ __device__ constexpr unsigned clear_blocks(int ndc) { return 1u + static_cast<unsigned>(ndc) / 32u; }

// ---- kernels: one frame per launch, and every frame of a batch per launch -----------

#define JXB_ENTROPY_KERNELS(NAME, BOUNDS, PHASE)                                                           \
    __global__ void BOUNDS NAME##_kernel(const __grid_constant__ EntropyDev e) {                              \
        wait_for_previous_grid();                                                                             \
        NAME##_body(e, blockIdx.x);                                                                           \
    }                                                                                                         \
    __global__ void BOUNDS NAME##_batch_kernel(const __grid_constant__ EntropyBatch b) {                      \
        const int f{batch_frame(b, PHASE, blockIdx.x)};                                                      \
        NAME##_body(b.frames[f], blockIdx.x - b.begin[PHASE][f]);                                             \
    }

// Frame of block `blk` of a batched launch of `phase` (binary search over the
// frames' first blocks).
__device__ __forceinline__ int batch_frame(const EntropyBatch& b, int phase, unsigned blk) {
    int lo{0};
    int hi{b.nframes - 1};
    while (lo < hi) {
        const int mid{(lo + hi + 1) >> 1};
        if (b.begin[phase][mid] <= blk) {
            lo = mid;
        } else {
            hi = mid - 1;
        }
    }
    return lo;
}

// The three item passes run the AC stripes (blocks 0 .. nstripes - 1, the
// long ones, scheduled first) and the other items (the blocks after them) as
// one launch: the two kinds are independent within a pass.
__device__ __forceinline__ void tokens_body(const EntropyDev& e, const unsigned blk) {
    if (blk < static_cast<unsigned>(e.nstripes)) {
        ac_tok_direct_body(e, blk);
    } else {
        misc_hist_body(e, blk - static_cast<unsigned>(e.nstripes));
    }
}
__device__ __forceinline__ void emit_body(const EntropyDev& e, const unsigned blk) {
    if (blk < static_cast<unsigned>(e.nstripes)) {
        ac_emit_stored_body(e, blk);
    } else {
        misc_emit_body(e, blk - static_cast<unsigned>(e.nstripes));
    }
}

JXB_ENTROPY_KERNELS(tokens, __launch_bounds__(kAcThreads, 3), kPhaseItems)
JXB_ENTROPY_KERNELS(codes, __launch_bounds__(32), kPhaseCodes)
JXB_ENTROPY_KERNELS(lengths, __launch_bounds__(kAcThreads, 8), kPhaseItems)
__global__ void __launch_bounds__(kLayoutThreads) layout_kernel(const __grid_constant__ EntropyDev e) {
    wait_for_previous_grid();
    layout_body(e);
}
__global__ void __launch_bounds__(kLayoutThreads) layout_batch_kernel(const __grid_constant__ EntropyBatch b) {
    layout_body(b.frames[blockIdx.x]);
}
// Five CTAs per SM (latency-bound: the window and code table fill the rest).
JXB_ENTROPY_KERNELS(emit, __launch_bounds__(kAcThreads, 5), kPhaseItems)
// Stripes whose tokens did not fit the pool are rare, so their passes run on
// a few resident CTAs that skip the stored stripes with one load each.
constexpr unsigned kUnstoredCtas = 148;

// Every stripe adds its token count to the pool fill whether or not it fits,
// so a frame has an unstored stripe exactly when its final fill exceeds the
// capacity; a frame without one is passed over after one load.
__device__ __forceinline__ bool frame_all_stored(const EntropyDev& e) { return e.frozen[0] <= e.tok_capacity; }

__global__ void __launch_bounds__(kAcThreads) lengths_unstored_kernel(const __grid_constant__ EntropyDev e) {
    if (frame_all_stored(e)) return;
    for (unsigned s{blockIdx.x}; s < static_cast<unsigned>(e.nstripes); s += gridDim.x) {
        if (e.stripe_tok[2 * s] != kNoTokens) continue;
        ac_bits_unstored_body(e, s);
        __syncthreads();
    }
}
__global__ void __launch_bounds__(kAcThreads) emit_unstored_kernel(const __grid_constant__ EntropyDev e) {
    if (frame_all_stored(e) || e.result[2] != 0) return;
    for (unsigned s{blockIdx.x}; s < static_cast<unsigned>(e.nstripes); s += gridDim.x) {
        if (e.stripe_tok[2 * s] != kNoTokens) continue;
        ac_emit_unstored_body(e, s);
        __syncthreads();
    }
}
#undef JXB_ENTROPY_KERNELS

__global__ void __launch_bounds__(256) clear_kernel(const __grid_constant__ EntropyDev e) {
    clear_body(e, blockIdx.x, gridDim.x);
}

// The token pass of planes given by the caller.
__global__ void __launch_bounds__(kAcThreads) tokens_staged_kernel(const __grid_constant__ EntropyDev e) {
    if (blockIdx.x < static_cast<unsigned>(e.nstripes)) {
        ac_tok_body(e, blockIdx.x);
    } else {
        misc_hist_body(e, blockIdx.x - static_cast<unsigned>(e.nstripes));
    }
}

constexpr std::size_t kHistSmem{sizeof(StripeStage) + kNumClusters * kAcSymbols * sizeof(std::uint32_t)};
constexpr std::size_t kBitsSmem{sizeof(StripeStage)};
constexpr std::size_t kEmitSmem{sizeof(StripeStage) + kWindowWords * sizeof(unsigned int)};
// Emission of stored stripes (window and code table) and of other items.
constexpr std::size_t kEmitStoredSmem{(kWindowWords + kNumClusters * kAcSymbols) * sizeof(unsigned int)};
static_assert(kEmitStoredSmem >= kMiscWindowWords * sizeof(unsigned int) + kMaxDeferred * sizeof(DeferredBlob),
              "emission shared memory");
// The other items' passes share these launches and their shared memory.
constexpr std::size_t kDirectSmem{sizeof(DirectStage)};
static_assert(kHistSmem >= (4 * 256 + 2) * sizeof(std::uint32_t) && kDirectSmem >= (4 * 256 + 2) * sizeof(std::uint32_t) &&
                  kDirectSmem <= 48 * 1024,
              "token pass shared memory");


}  // namespace

static_assert(sizeof(EntropyBatch) <= 32000, "a batched entropy launch's parameters exceed the kernel parameter limit");

bool entropy_launch(const EntropyDev& e, void* stream) {
    if (e.nsec > kMaxSections) return false;
    cudaStream_t st{static_cast<cudaStream_t>(stream)};
    const unsigned units{e.misc_units + static_cast<unsigned>(e.nstripes)};
    if (e.clear_first && !launch_plain(clear_kernel, clear_blocks(e.ndc), 256, 0, st, e)) return false;
    const auto codes{static_cast<unsigned>(kNumClusters + 2 * e.ndc)};
    if (e.direct) {
        return launch_chained(tokens_kernel, units, kAcThreads, kDirectSmem, st, e) &&
               launch_chained(codes_kernel, codes, 32, sizeof(WarpCodeSmem), st, e) &&
               launch_chained(lengths_kernel, units, kAcThreads, 0, st, e) &&
               launch_chained(layout_kernel, 1, kLayoutThreads, 0, st, e) &&
               launch_chained(emit_kernel, units, kAcThreads, kEmitStoredSmem, st, e);
    }
    return launch_plain(tokens_staged_kernel, units, kAcThreads, kHistSmem, st, e) &&
           launch_plain(codes_kernel, codes, 32, sizeof(WarpCodeSmem), st, e) &&
           launch_plain(lengths_unstored_kernel, kUnstoredCtas, kAcThreads, kBitsSmem, st, e) &&
           launch_plain(lengths_kernel, units, kAcThreads, 0, st, e) &&
           launch_plain(layout_kernel, 1, kLayoutThreads, 0, st, e) &&
           launch_plain(emit_kernel, units, kAcThreads, kEmitStoredSmem, st, e) &&
           launch_plain(emit_unstored_kernel, kUnstoredCtas, kAcThreads, kEmitSmem, st, e);
}

void entropy_batch_plan(EntropyBatch& b) {
    for (int p{0}; p < kEntropyPhases; ++p) b.begin[p][0] = 0;
    for (int f{0}; f < b.nframes; ++f) {
        const EntropyDev& e{b.frames[f]};
        const std::uint32_t per[kEntropyPhases]{e.misc_units + static_cast<std::uint32_t>(e.nstripes),
                                                 static_cast<std::uint32_t>(kNumClusters + 2 * e.ndc)};
        for (int p{0}; p < kEntropyPhases; ++p) b.begin[p][f + 1] = b.begin[p][f] + per[p];
    }
}

bool entropy_batch_launch(const EntropyBatch& b, void* stream) {
    if (b.nframes <= 0 || b.nframes > kEntropyBatchFrames) return false;
    for (int f{0}; f < b.nframes; ++f) {
        if (b.frames[f].nsec > kMaxSections) return false;
    }
    cudaStream_t st{static_cast<cudaStream_t>(stream)};
    const int nf{b.nframes};
    const unsigned items{b.begin[kPhaseItems][nf]};
    tokens_batch_kernel<<<items, kAcThreads, kDirectSmem, st>>>(b);
    codes_batch_kernel<<<b.begin[kPhaseCodes][nf], 32, sizeof(WarpCodeSmem), st>>>(b);
    lengths_batch_kernel<<<items, kAcThreads, 0, st>>>(b);
    layout_batch_kernel<<<static_cast<unsigned>(nf), kLayoutThreads, 0, st>>>(b);
    emit_batch_kernel<<<items, kAcThreads, kEmitStoredSmem, st>>>(b);
    return cudaGetLastError() == cudaSuccess;
}

bool prefix_code_test(const std::uint32_t* hist, int length, std::uint8_t* depth, std::uint16_t* bits,
                      std::uint8_t* header, std::size_t header_cap, std::uint32_t* nbits) {
    if (length < 1 || length > 256 || header_cap < static_cast<std::size_t>(kDescBytes)) return false;
    unsigned char* dev{nullptr};
    const std::size_t bytes{256 * 4 + 256 + 256 * 2 + kDescBytes + 4};
    if (cudaMalloc(&dev, bytes) != cudaSuccess) return false;
    auto* dh{reinterpret_cast<std::uint32_t*>(dev)};
    auto* dd{dev + 1024};
    auto* db{reinterpret_cast<std::uint16_t*>(dev + 1280)};
    auto* dhead{dev + 1792};
    auto* dn{reinterpret_cast<std::uint32_t*>(dev + 1792 + kDescBytes)};
    bool ok{cudaFuncSetAttribute(prefix_code_test_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(sizeof(WarpCodeSmem))) == cudaSuccess &&
            cudaMemcpy(dh, hist, static_cast<std::size_t>(length) * 4, cudaMemcpyHostToDevice) == cudaSuccess};
    if (ok) {
        prefix_code_test_kernel<<<1, 32, sizeof(WarpCodeSmem)>>>(dh, length, dd, db, dhead, dn);
        ok = cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess &&
             cudaMemcpy(depth, dd, static_cast<std::size_t>(length), cudaMemcpyDeviceToHost) == cudaSuccess &&
             cudaMemcpy(bits, db, static_cast<std::size_t>(length) * 2, cudaMemcpyDeviceToHost) == cudaSuccess &&
             cudaMemcpy(header, dhead, kDescBytes, cudaMemcpyDeviceToHost) == cudaSuccess &&
             cudaMemcpy(nbits, dn, 4, cudaMemcpyDeviceToHost) == cudaSuccess;
    }
    cudaFree(dev);
    return ok;
}

bool entropy_kernels_init() {
    std::uint8_t ctx[kCoeffCtxBytes]{};
    for (int i{1}; i < 64; ++i) {
        ctx[i] = static_cast<std::uint8_t>(coeff_nz_ctx(static_cast<std::uint32_t>(i)));
        ctx[64 + i] = static_cast<std::uint8_t>(coeff_freq_ctx(static_cast<std::uint32_t>(i)));
    }
    for (int g{0}; g < 2; ++g) {
        for (int z{0}; z < kZeroDensityCount; ++z) {
            // Block context 0 stands for every luma context, 7 for every chroma one.
            ctx[128 + g * kZdRow + z] = static_cast<std::uint8_t>(context_cluster(
                static_cast<std::uint32_t>(kNumBlockCtx * kNonZeroBuckets + kZeroDensityCount * (7 * g) + z)));
        }
    }
    if (cudaMemcpyToSymbol(g_coeff_ctx, ctx, sizeof(ctx)) != cudaSuccess) return false;
    return cudaFuncSetAttribute(codes_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(sizeof(WarpCodeSmem))) == cudaSuccess &&
           cudaFuncSetAttribute(tokens_staged_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(kHistSmem)) == cudaSuccess &&
           cudaFuncSetAttribute(lengths_unstored_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(kBitsSmem)) == cudaSuccess &&
           cudaFuncSetAttribute(emit_unstored_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(kEmitSmem)) == cudaSuccess &&
           cudaFuncSetAttribute(codes_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(sizeof(WarpCodeSmem))) == cudaSuccess;
}

}  // namespace jxb
