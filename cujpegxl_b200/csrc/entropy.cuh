// Device entropy coding and frame assembly: quantised planes -> .jxl bytes in
// device memory, with no host round trip.
//
// The codestream is modelled as a list of sections (DcGlobal, the DcGroups,
// AcGlobal, the AcGroups, in TOC order), each a list of "items" whose bit
// lengths are data dependent but whose number is fixed by the frame geometry:
// a header blob, one AC block-channel, one DC sample, one AcMetadata sample.
// Per frame:
//   1. token pass over all items: the AC stripes' tokens are counted into
//      the 32 cluster histograms and stored once in a token pool; the other
//      items fill the per-DC-group DC and AcMetadata histograms;
//   2. prefix codes built on the device, one warp per histogram;
//   3. bit-length pass over all items: each unit (an AC stripe or 512 other
//      items, the work of one CTA) sums and scans its own;
//   4. a layout CTA scans the units, sizes every section, writes the
//      container, headers and TOC, and places sections and units;
//   5. an emit pass writes every item's bits at its final position.
// Passes 1, 3 and 5 are one launch each: a CTA per AC stripe (one lane per
// token), then a CTA per 512 other items (two per thread). Planes given by
// the caller are tokenised a warp per block-channel instead, and stripes whose
// tokens did not fit the pool go through passes 3 and 5 in one more launch
// each, with their coefficients staged again. The code pass leaves the
// histograms and counters zeroed for the next frame.
#pragma once

#include <cstddef>
#include <cstdint>
#include <vector>

namespace jxb {

enum SectionKind : int { kSecDcGlobal = 0, kSecDcGroup = 1, kSecAcGlobal = 2, kSecAcGroup = 3 };

struct Section {
    std::uint32_t first;   // first global item index
    std::uint32_t count;   // items in the section
    int kind;
    int group;             // DC or AC group index
    std::uint32_t unit;    // unit that holds the first item
};

// Up to kStripeRows block rows of one AC group: the unit one CTA stages in
// shared memory for the AC passes. Rows start at multiples of 4 inside the
// group, so every DCT16/DCT32 transform lies inside one stripe.
constexpr int kStripeRows = 4;
struct alignas(16) Stripe {
    std::uint32_t item0;   // global index of the stripe's first item
    std::int32_t section;  // section index of the AC group
    std::uint16_t group;   // AC group index
    std::uint8_t r0;       // first block row inside the group
    std::uint8_t rows;     // block rows, 1..kStripeRows
    std::uint32_t cols;    // blocks per row
};

// Geometry and per-frame device state of the entropy stage. All pointers are
// device memory owned by the encoder.
struct EntropyDev {
    // geometry
    int width, height, bw, bh, nblocks, xg, nac, xdg, ndc, cmw, nsec;
    std::uint32_t total_items;
    std::uint32_t ac_first;          // first item of the first AcGroup; AC block-channels follow
    std::uint32_t misc_units;        // units of the items before ac_first; the stripes' units follow
    const Section* sections;
    const Stripe* stripes;
    int nstripes;
    const std::uint32_t* unit_section;  // [misc_units + nstripes] section that holds each unit's first item

    // inputs (frontend outputs)
    const std::int16_t* ac;
    const std::int32_t* dc;
    const std::int8_t* acs;
    const std::int32_t* qf;
    const std::int8_t* ytox;
    const std::int8_t* ytob;
    const std::uint8_t* nzn;
    const std::uint16_t* nzc;

    // constant tables
    const std::uint16_t* order;      // natural orders: 64 (DCT8) | 256 (DCT16) | 1024 (DCT32)
    const std::uint16_t* rank;       // their inverses: scan position of each raw index (direct passes only)
    const std::uint8_t* pre_const;   // DcGroup header bits before the DC code description
    std::uint32_t pre_const_bits;
    const std::uint8_t* mid_const;   // AcMetadata header bits after the count field
    std::uint32_t mid_const_bits;
    const std::uint8_t* ac_prefix;   // AcGlobal bits before the per-cluster sizes
    std::uint32_t ac_prefix_bits;
    const std::uint8_t* dc_global;   // DcGlobal section bits (per distance)
    std::uint32_t dc_global_bits;
    std::uint32_t head_words[4];     // codestream header up to the TOC: signature, sizes, frame header
    std::uint32_t head_bytes;

    // Per-frame scratch. The histograms and counters (ac_hist to tok_count)
    // are zero between encodes: the passes that read them last clear them (with
    // clear_first, for scratch without that history, a kernel clears them
    // before the first pass).
    bool clear_first;
    std::uint32_t* ac_hist;          // [32][256]
    std::uint32_t* dc_hist;          // [ndc][256]
    std::uint32_t* am_hist;          // [ndc][256]
    std::uint32_t* fb_count;         // [ndc] first blocks counted by the token pass
    std::uint32_t* tok_count;        // [1] pool fill, or tokens at the output's end (direct)
    std::uint32_t* frozen;           // [1 + ndc] tok_count and fb_count as the code pass found them
    std::uint8_t* ac_depth;          // [32][256]
    std::uint16_t* ac_bits;
    // Depth << 16 | code bits of each symbol: [32][64] AC, then [ndc][128] DC
    // and [ndc][128] AcMetadata.
    std::uint32_t* code;
    std::uint8_t* dc_depth;          // [ndc][256]
    std::uint16_t* dc_bits;
    std::uint8_t* am_depth;          // [ndc][256]
    std::uint16_t* am_bits;
    std::uint32_t* ac_alpha;         // [32]
    std::uint8_t* desc;              // [32 + 2*ndc][kDescBytes] code descriptions
    std::uint32_t* desc_bits;        // [32 + 2*ndc]
    std::uint32_t* item_pre;         // [total_items] exclusive prefix of the bits within the item's unit
    std::uint32_t* item_tok;         // [ac_first] tokens of the items before the AC groups (pack_misc_token)
    std::uint32_t* unit_sum;         // [unit_words] bits of each unit
    unsigned long long* unit_off;    // [unit_words] bits before each unit, then their total
    unsigned long long* unit_pos;    // [misc_units + nstripes] absolute bit offset of each unit in `out`
    unsigned long long* sec_shift;   // [nsec] from a bit's place in the scan to its place in `out`
    unsigned long long* result;      // [4]: total bytes, body start, status, 0

    // AC tokens, written once by the token pass in stream order and read by
    // the bit-length and emission passes. `direct`: the planes come from the
    // frontend, and each stripe has kTokensPerBlock places a block in the
    // pool; the tokens of a stripe that has more go to the end of the output
    // buffer, which the file does not reach. Otherwise (planes given by the
    // caller, which may break the block layout, and a buffer of any size) each
    // stripe reserves a contiguous run of the pool; one that finds it full
    // keeps its tokens unstored and the later passes tokenise its
    // coefficients again.
    bool direct;
    std::uint32_t* tok_pool;         // [tok_capacity] packed tokens (pack_ac_token)
    std::uint32_t tok_capacity;
    std::uint32_t* stripe_tok;       // [2 * nstripes]: place (pool offset or kNoTokens, or dense_tokens offset), token count
    std::uint8_t* out;               // output buffer (container + codestream)
    std::size_t out_capacity;
};

constexpr int kDescBytes = 256;
// Items of a unit that is not an AC stripe.
constexpr std::uint32_t kMiscItemsPerUnit = 512;
// Token pool capacity per 8x8 block: 4K frames at distance 0.5 use about 27,
// at distance 1 about 11.
constexpr std::uint32_t kTokensPerBlock = 32;
// A block's tokens at most: three channels of one count and 63 coefficients
// (DCT8; larger transforms have fewer a block).
constexpr std::uint32_t kMaxTokensPerBlock = 192;
constexpr std::uint32_t kNoTokens = 0xffffffffu;

// Sections of a frame at most (25,000: 1.6 gigapixels).
constexpr int kMaxSections = 25584;

// Builds the constant header blobs and section table for a geometry. Fills the
// host-side vectors; the caller uploads them.
struct EntropyHostPlan {
    std::vector<Section> sections;
    std::vector<Stripe> stripes;
    std::uint32_t misc_units{0};
    std::vector<std::uint32_t> unit_section;
    std::uint32_t head_words[4]{};
    std::uint32_t head_bytes{0};
    std::uint32_t total_items{0};
    std::uint32_t ac_first{0};
    std::vector<std::uint8_t> pre_const;
    std::uint32_t pre_const_bits{0};
    std::vector<std::uint8_t> mid_const;
    std::uint32_t mid_const_bits{0};
    std::vector<std::uint8_t> ac_prefix;
    std::uint32_t ac_prefix_bits{0};
    std::vector<std::uint16_t> order;
    std::vector<std::uint16_t> rank;  // inverse of each order, concatenated likewise
};
EntropyHostPlan entropy_plan(int width, int height);

// DcGlobal section bits for the quantiser state.
std::vector<std::uint8_t> dc_global_bits(std::uint32_t global_scale, std::uint32_t quant_dc,
                                         std::uint32_t* nbits);

// Worst-case output size (same bound as the reference's cujpegxl.cc:50-59).
std::size_t worst_case_output(std::uint32_t width, std::uint32_t height);

// Enqueues the whole entropy + assembly stage on `stream`. After completion
// result[0] holds the file size and result[2] a status (0 = ok, 1 = output
// capacity exceeded).
bool entropy_launch(const EntropyDev& e, void* stream);

// Several frames' entropy stages as one launch per pass: each pass runs the
// blocks of every frame, frame f owning blocks begin[phase][f] ..
// begin[phase][f + 1] - 1. The frames live in the launch's parameter block.
constexpr int kEntropyBatchFrames = 64;
enum EntropyPhase : int {
    kPhaseItems = 0,  // item passes: one block per AC stripe, then one per 512 other items
    kPhaseCodes = 1,  // prefix codes: one block per histogram
    kEntropyPhases = 2
};
struct EntropyBatch {
    int nframes;
    std::uint32_t begin[kEntropyPhases][kEntropyBatchFrames + 1];
    EntropyDev frames[kEntropyBatchFrames];
};

// Fills b.begin from b.frames[0 .. b.nframes).
void entropy_batch_plan(EntropyBatch& b);

// Enqueues every frame's entropy stage on `stream` (b planned).
bool entropy_batch_launch(const EntropyBatch& b, void* stream);

// Entries of unit_sum and unit_off: the units and one more, in whole vectors of four.
inline std::size_t unit_words(const EntropyHostPlan& p) { return (p.unit_section.size() + 4) & ~std::size_t{3}; }

// The device prefix-code builder on one histogram of `length` (1..256)
// symbols, synchronously on the current device (test hook): depths, codes and
// the header (header_cap >= kDescBytes), its length in bits.
bool prefix_code_test(const std::uint32_t* hist, int length, std::uint8_t* depth, std::uint16_t* bits,
                      std::uint8_t* header, std::size_t header_cap, std::uint32_t* nbits);

}  // namespace jxb
