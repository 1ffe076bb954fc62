// Decode attention over an FP8 latent KV cache on sm_100a tensor cores.
//
// A cluster pair of thread blocks (two SMs) works through a list of work items.  An item is (query-token row n,
// group of 128 heads, a range of 64-entry tiles of that row).  The list is either the single item the pair's grid
// position names (one launch = rows x head groups x splits pairs) or this pair's slice of a schedule a planner kernel
// wrote (sched.cuh): the pair then stays resident, keeps its tensor memory and barriers, and overlaps the set-up of
// the next item with the tail of the current one.
//
// The pair computes a tile with paired MMAs (cta_group::2, M = 128): each block owns 64 of the 128
// heads (its rows of Q, S, P and O) and supplies half of the B operand of every MMA:
//   S[128 heads x 64 entries] = Q . K^T     each block brings the K rows of ITS 32 entries (all 576 columns)
//   O[128 heads x 512]       += P . V       each block brings ITS 256 value columns of all 64 entries
// so an entry is dequantised once for S and half of it a second time for V, O (64 heads x 512) takes half of a
// block's tensor memory, and S is computed once per pair.  The roles of a block's 26 warps:
//   resolve warps  (2) walk the items and work out where the entries live (index list -> block table -> record number), tiles
//                  ahead: one for the block's own 32 entries of a tile, one for the other block's;
//   fetch warps    (2) have TMA fetch the raw records into a ring in shared memory: one the own entries,
//                  one this block's half of the others;
//   K, V warps     (8 + 8) dequantise FP8 * scale -> FP16 (BF16 for the reference layouts) from the ring into the K and V
//                  tiles, in the 128-byte-swizzled operand layout;
//   S, O warps     (of the even block) issue the MMAs of the pair;
//   softmax warps  (4) read S from tensor memory (half a row per thread), run the online softmax with a lazily updated
//                  reference maximum, write P to shared memory, rescale O in tensor memory when the maximum
//                  moved, and finally normalise and store.
//
// What bounds it, in SM cycles per tile: tensor pipe 24 x 18 + 12 x 25 (S) + 8 x 64 (O) = 1244 (counted: 1445); shared-memory port
// (128 B/clk) about 2000 (counted: bank reads 1172 + writes 845 = 2017): raw records in and out 520, operand writes 610, operand reads 860;
// TMA gather of 656-byte records 1200 alone, up to 1900 with every SM gathering from DRAM.  A tile takes 2380 with few SMs at work, 2570 with
// all of them and the inputs in L2, 2630 from DRAM: the port is busy for 77 to 85 % of it.  Loads through the load/store unit (4 records
// x 128 bytes per instruction, straight into registers) took 3300: records at a pitch of 656 bytes cost eight tag look-ups per
// instruction.  Measured, B200, 128 heads, inputs from DRAM: CSA, 64 requests x top-k 2048 60 us (one block per SM with its own copy of
// S: 92), HCA, 64 requests x 910 entries 32 us (45): 1.34 us a tile (2.0-2.9) and some 12 us a launch.
//
// All waits are bounded; a wait that gives up records where in `status` and the pair leaves through the common
// exit, where it stays until its copies and MMAs in flight have landed, and frees its tensor memory.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <math_constants.h>
#include <stdint.h>
#include <type_traits>

#include "ptx.cuh"

namespace dsv4 {

constexpr int kTileN = 64;             // entries per tile (MMA N of S, K of P.V)
constexpr int kRowsPerBlock = 32;      // K rows a block supplies per tile
constexpr int kHeadsPerCta = 128;      // heads of an item (MMA M over the pair)
constexpr int kHeadsPerBlock = 64;     // of which one block owns half
constexpr int kQChunkBytes = 64 * 128;    // 64 heads x 64 16-bit values, swizzled: a chunk of Q, and P
constexpr int kKChunkBytes = 32 * 128;    // 32 entries x 64 16-bit values
constexpr int kVChunkBytes = 64 * 128;    // 64 entries x 64 value columns
// Warp roles, four warpgroups of four warps (tensor-memory lane quarter = warp % 4).
constexpr int kNumSoftmaxWarps = 4;    // warps 0-3: softmax + epilogue
constexpr int kNumKWarps = 8;          // warps 4-11: K tile, four rows each
constexpr int kNumVWarps = 8;          // warps 12-19: V tile, 16 rows of one 128-column span each; and Q's set-up
constexpr int kFirstKWarp = 4;
constexpr int kFirstVWarp = 12;
constexpr int kSWarp = 20;             // Q load, tensor-memory allocation and (even block) issue of the S MMAs
constexpr int kOWarp = 21;             // (even block) issue of the O MMAs: a warp of its own, so that a ready P never waits behind S MMAs
constexpr int kFetchWarp = 22;         // 22: own entries; 23: this block's half of the other block's
constexpr int kResolveWarp = 24;       // 24, 25: the record numbers for warps 22, 23 (a warp that did both spent half of its time on either)
constexpr int kNumWarps = 26;
constexpr int kNumThreads = kNumWarps * 32;  // 832
constexpr int kTmemCols = 512;
constexpr int kTmemS = 0;              // two S buffers of 32 columns (lanes 0-63: entries of the even block, 64-127: of the odd one)
constexpr int kTmemO = 64;             // O: 256 columns (lanes 0-63: value columns 0-255, lanes 64-127: 256-511)
constexpr int kTmemQ = 320;            // Q chunks 0-5 as packed 16-bit values, 32 columns each, rows in both lane halves
constexpr int kQTmemChunks = 6;        // as the A operand from here they take neither room nor bandwidth of shared memory
constexpr int kQStageChunks = 3;       // chunks on their way to tensor memory staged at a time
constexpr unsigned long long kDefaultWaitNs = 2000000000ull;  // 2 s
constexpr float kRescaleThreshold = 8.0f;  // log2 units; O is rescaled only when the max grows by more
constexpr int kItemWords = 8;          // int32 words per work item of a schedule
constexpr int kStages = 3;             // raw tiles in the ring (with two, and a second K buffer in the room of the third: 71 us against 63 at 32 tiles)
constexpr int kIdRing = 4;             // tiles the resolve warps may be ahead of the fetch warps
constexpr int kTagRing = 8;            // tags and validity masks kept: the softmax of a tile is done before the tile eight later is fetched

enum SourceKind : int {
    kSrcCsa = 0,   // index list + block table, packed 656-byte entries
    kSrcHca = 1,   // dense [0, kv_len) through the block table, then the window buffer
    kSrcRef = 2,   // reference layout: separate planes, 448 e4m3 + 7 UE8M0 + 64 bf16
    kSrcRefPaged = 3,   // the same bytes in packed pages: per page, page_size tokens of [448 e4m3 | 64 bf16]
                        // followed by page_size x 8 scale bytes (7 UE8M0 + 1 pad), behind block tables
};

// both kinds with the reference's quantisation (448 latent elements, one UE8M0 byte per 64)
__host__ __device__ constexpr bool is_ref_layout(int src) { return src == kSrcRef || src == kSrcRefPaged; }

// Operand format of the MMAs.  The packed 656-byte layout goes through FP16: FP8 -> FP16 is one
// exact conversion instruction per two elements and one packed multiply by the scale (the BF16
// route costs five integer/FP instructions per two elements), and FP16 keeps three more mantissa bits of fp8 x scale
// than BF16.  Q and P are converted to FP16 as well (exact for Q inside FP16's normal range; P <= 2^8).
// Limits: |q| below 65504; block scales above 146 (entries beyond +-65408) are clamped to 146 (the
// BF16 route's own limit on scales is 128).
// The reference layouts keep BF16: their power-of-two scales span BF16's exponent range.
__host__ __device__ constexpr bool use_f16(int src) { return !is_ref_layout(src); }

enum StatusCode : int {
    kStatusOk = 0,
    kStatusWaitKvFull = 1,
    kStatusWaitKvFree = 2,
    kStatusWaitSFull = 3,
    kStatusWaitPFull = 4,
    kStatusWaitOFull = 5,
    kStatusWaitQ = 6,
    kStatusBadIndex = 7,       // an index, length or block-table value pointed outside the cache: entry left out, not read
    kStatusWaitRaw = 9,
};

struct DecodeArgs {
    // TMA descriptor of Q viewed as [rows = B*s_q*H, cols = 64*NCHUNK] bf16, box 64 x 64, 128-byte swizzle
    alignas(64) CUtensorMap q_map;
    // Record fetch, per pool (0 cache, 1 window), 32-bit elements.  tile::gather4, one row high:
    //   packed 656-byte records: whole record | 256 bytes of latent | 16 bytes of scales
    //   reference planes: latent row (448) | 256 bytes of it | 192 bytes of it;  RoPE row (128) in rope_map
    // tiled, four tokens of a page:
    //   packed reference pages: token (576) | 256 bytes of it | 320 bytes of it
    alignas(64) CUtensorMap rec_map[2][3];
    alignas(64) CUtensorMap rope_map[2];
    int B, s_q, H;
    int topk;            // CSA
    int max_pages;
    int win_cap;         // HCA
    int num_splits;
    float scale_log2;    // sm_scale * log2(e)
    long long num_pages; // pages in kv_pool: block-table values outside [0, num_pages) are not followed
    const __nv_bfloat16* q;
    const uint8_t* kv_pool;
    const int32_t* block_table;
    const int32_t* indices;
    const int32_t* kv_len;
    const int32_t* topk_len;
    const uint8_t* win_pool;
    const int32_t* win_len;
    const float* attn_sink;
    __nv_bfloat16* out;
    float* lse;
    float* partial_o;            // split partials, stored as BF16 (the area is sized for FP32)
    float* partial_lse;
    int32_t* status;
    // schedule (sched.cuh): null = one item per pair, named by the grid position
    const int32_t* sched_pair_begin;   // [pairs + 1]: first item of every pair
    const int32_t* sched_items;        // [items][kItemWords]
#ifdef DSV4_TRACE
    unsigned long long* trace;         // development builds only: block 0 stores cycle counts here, 1024 slots per role
#endif
    uint32_t wait_ns;                  // limit of every bounded wait (below four seconds)
    int dbg_drop_tile;                 // test aid (-1 = off): the loaders withhold the hand-over of the pair's tile with this
                                       // running number, so that a bounded wait runs out and the error path can be checked
    // reference layout planes (kSrcRef)
    const uint8_t* ref_kc;  const uint8_t* ref_kc_s;  const __nv_bfloat16* ref_kc_rope;
    const uint8_t* ref_ks;  const uint8_t* ref_ks_s;  const __nv_bfloat16* ref_ks_rope;
    int ref_m_cur, ref_swa_len;
    // packed pages (kSrcRefPaged): two pools (compressed cache, sliding window) with their block tables;
    // per-request lengths come through kv_len / win_len
    const uint8_t* pg_kv;  const uint8_t* pg_swa;
    const int32_t* pg_swa_table;
    int pg_swa_max_pages;
    int pg_page_shift;           // log2(page_size), page_size <= 64
    int64_t pg_page_bytes;       // page_size * 584
    int64_t pg_num_pages, pg_swa_num_pages;
};

// One unit of work of a pair: tiles [tile0, tile0 + ntiles) of row n for head group hg.
struct Item {
    int n, hg;
    int tile0, ntiles;
    int n_tok;        // entries of the row that take part (index-list slots in use, or kv_len + win_len)
    int kv_len_n;     // CSA: causal bound on index values; HCA: entries read through the block table
    int slot;         // < 0: the item is the whole row, write out / lse; else the partial slot to write

    // entries of the item's tile `it` (1 .. 64)
    __device__ __forceinline__ int tile_entries(int it) const { return min(n_tok - (tile0 + it) * kTileN, kTileN); }
};

// Entries are dealt to the two blocks four at a time: slot s of a tile is K row 4 (s / 8) + s % 4 of block (s / 4) % 2,
// so that a tile that is not full fills the leading rows of both blocks evenly.  Groups of four rows of each block
// that a tile of n entries uses; its P.V reads the leading 16 or 32 rows of each block.
__device__ __forceinline__ int tile_groups(int n) { return (n + 7) >> 3; }
__device__ __forceinline__ int tile_ksteps(int n) { return n > 32 ? 2 : 1; }

// A raw tile in the ring.  Rows come in groups of four (one gather); a gather's destination starts at a multiple of 128 bytes.
// Own rows hold whole entries; half rows the other block's entries' latent of this block's value columns.
template <int SRC>
struct RawLayout {
    static constexpr bool kPacked = !is_ref_layout(SRC);
    static constexpr int kOwnRow = kPacked ? 656 : (SRC == kSrcRefPaged ? 576 : 448);
    static constexpr int kOwnGroup = (4 * kOwnRow + 127) / 128 * 128;
    static constexpr int kOwnRope = 0;      // planes only: RoPE rows of the own entries, 128 bytes each
    // half rows: packed 256 bytes; planes 256 (even block) or 192 (odd block) bytes; pages 256 or, with the RoPE tail, 320 bytes
    __host__ __device__ static constexpr int half_row(int rank) { return kPacked || rank == 0 ? 256 : (SRC == kSrcRefPaged ? 320 : 192); }
    static constexpr int kHalfGroup = SRC == kSrcRefPaged ? 1280 : 1024;
    static constexpr int kRopeOff = 8 * kOwnGroup;                                         // planes: own RoPE
    static constexpr int kHalfOff = kRopeOff + (SRC == kSrcRef ? 8 * 512 : 0);
    static constexpr int kHalfRopeOff = kHalfOff + 8 * kHalfGroup;                         // planes: RoPE of the half rows
    static constexpr int kScaleOff = kHalfRopeOff + (SRC == kSrcRef ? 8 * 512 : 0);
    // packed: the four FP32 scales of the half rows, 128 bytes a group; reference layouts: 8 bytes of UE8M0 scales per entry,
    // [block][row], written by the producers
    static constexpr int kBytes = kScaleOff + (kPacked ? 8 * 128 : 512);
    static_assert(kBytes % 128 == 0, "stages start at multiples of 128 bytes");
    __device__ static uint32_t own(uint32_t row) { return (row >> 2) * kOwnGroup + (row & 3u) * kOwnRow; }
    __device__ static uint32_t own_rope(uint32_t row) {
        return kPacked ? own(row) + 528u : (SRC == kSrcRefPaged ? own(row) + 448u : kRopeOff + row * 128u);
    }
    __device__ static uint32_t half(uint32_t row, int rank) { return kHalfOff + (row >> 2) * kHalfGroup + (row & 3u) * half_row(rank); }
    __device__ static uint32_t half_rope(uint32_t row) {     // odd block only
        return SRC == kSrcRefPaged ? half(row, 1) + 192u : kHalfRopeOff + row * 128u;
    }
};

template <int NCHUNK, int SRC>
struct SmemLayout {
    static constexpr int kQChunks = NCHUNK - kQTmemChunks;          // Q chunks that stay in shared memory
    static constexpr int kQOff = 0;
    static constexpr int kQStageOff = kQOff + kQChunks * kQChunkBytes;
    static constexpr int kKOff = kQStageOff + kQStageChunks * kQChunkBytes;
    static constexpr int kKBytes = NCHUNK * kKChunkBytes;
    static constexpr int kVOff = kKOff + kKBytes;                   // four chunks: this block's value columns
    static constexpr int kPOff = kVOff + 4 * kVChunkBytes;          // two buffers
    static constexpr int kRawOff = kPOff + 2 * kQChunkBytes;
    static constexpr int kMiscOff = kRawOff + kStages * RawLayout<SRC>::kBytes;
    static constexpr int kMiscBytes = 5120;
    static constexpr int kTotal = kMiscOff + kMiscBytes;            // no slack: dynamic shared memory starts 1 KB-aligned (checked)
    static_assert(kTotal <= 232448, "shared memory of a block");
    static_assert(kKOff % 1024 == 0 && kVOff % 1024 == 0 && kPOff % 1024 == 0, "swizzled operands");
    static_assert(kQStageChunks * kQChunkBytes <= 4 * kVChunkBytes, "the first item's second staging round uses the V tile");
};

// What a resolve warp hands its fetch warp for one tile.
struct IdSlot {
    int32_t num[kRowsPerBlock];      // record number per K row, 0 where none
    uint2 scales[kRowsPerBlock];     // reference layouts: the row's UE8M0 bytes
    uint32_t valid, second;          // bit r: row r takes part / comes from the second pool
    uint32_t meta, pad;
};

struct SmemMisc {
    IdSlot id_ring[2][kIdRing];
    uint64_t bar_id_full[2][kIdRing], bar_id_free[2][kIdRing];
    float exch[2 * kHeadsPerBlock];  // softmax: values the two threads of a head row exchange
    uint64_t bar_raw_full[kStages];  // raw tile fetched (both producers, TMA transaction count)
    uint64_t bar_raw_free[kStages];  // raw tile read by all K and V warps
    uint64_t bar_q_full[2];          // per item: staging round landed in shared memory (TMA transaction count)
    uint64_t bar_q_copied[2];        // per item: round copied out by every V warp
    uint64_t bar_tmem;               // tensor memory allocated
    // signalled in both blocks by the commits of the MMA warps
    uint64_t bar_s_full[2];          // S of a tile complete: S buffer full, K tile free
    uint64_t bar_v_free;             // P.V of a tile complete for the first value-column span: its V chunks free
    uint64_t bar_o_full[2];          // P.V of a tile complete, by P buffer: that buffer and the V chunks of the second span free, O up to date
    // in the even block only, signalled by the warps of both
    uint64_t bar_q_ready;            // per item: Q in place
    uint64_t bar_k_full[2];          // K chunks 0-3 / the others written
    uint64_t bar_v_full[2];          // V span j written
    uint64_t bar_p_full[2];          // P of a tile written (and its S buffer read, O rescaled), by buffer
    uint32_t mask[kTagRing][2];      // per tile and block: bit r = K row r takes part in the softmax
    uint32_t meta[kTagRing];
    uint32_t tmem_base;
};
static_assert(sizeof(SmemMisc) <= 5120 - 16, "misc area; the last word of the block's shared memory is failed_flag()");

// (out of line: it is called from many places and hardly ever runs)
__device__ __noinline__ void report_status(int32_t* status, int code, int role, int tile) {
    if (status != nullptr) {
        if (atomicCAS(status, 0, code) == 0) {
            status[1] = int(blockIdx.x) | (int(blockIdx.y) << 8) | (int(blockIdx.z) << 20);
            status[2] = role;
            status[3] = tile;
        }
    }
}

// Set when a wait of the pair has run out: the last word of a block's dynamic shared memory (found without an argument, which would
// take a register at every wait: HCA, 64 requests, 32.0 us instead of 32.3).
__device__ __forceinline__ uint32_t failed_flag() {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint32_t bytes;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(bytes));
    return ptx::smem_u32(smem_raw) + bytes - 4u;
}

// A wait that ran out: reported, and marked in both blocks of the pair.
__device__ __noinline__ void wait_ran_out(int32_t* status, int code, int role, int tile) {
    ptx::sts_cluster_u32(ptx::mapa(failed_flag(), 0), 1u);
    ptx::sts_cluster_u32(ptx::mapa(failed_flag(), 1), 1u);
    report_status(status, code, role, tile);
}

// Copies and MMAs must not outlive the blocks they work for.  After an ordinary run every one has been waited for by the role that uses its result; where
// a wait ran out that role is gone, so the block stays for a time that any copy needs less than (a few microseconds), counted from when all
// roles have ended and none can be added.  (Waiting for their barriers instead, in the fetch and MMA warps, cost every launch 4 to 6 %.)
constexpr uint32_t kHoldNs = 1000000u;
__device__ __noinline__ void hold_block() {
    const uint32_t t0 = ptx::globaltimer_lo();
    while (ptx::globaltimer_lo() - t0 < kHoldNs) __nanosleep(1000);
}

// Development builds (-DDSV4_TRACE): block 0 records when its roles pass their pipeline points
// (role 0 softmax, 1 S issue, 2 loader warp 0, 3 O issue).  Compiled out of the product.
#ifdef DSV4_TRACE
__device__ __forceinline__ void trace_mark(const DecodeArgs& a, int role, int slot) {
    if (a.trace != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && slot < 1024) a.trace[role * 1024 + slot] = clock64();
}
#else
__device__ __forceinline__ void trace_mark(const DecodeArgs&, int, int) {}
#endif

// Two FP8 e4m3 bytes sitting in bits [15:8] and [31:24] of `r` -> two BF16 bit
// patterns whose values are the FP8 values times 2^-120 (the e4m3 exponent and
// mantissa bits dropped into the BF16 exponent/mantissa fields; e4m3
// subnormals become BF16 subnormals, so one multiply fixes both).
__device__ __forceinline__ uint32_t e4m3x2_to_bf16x2_bits(uint32_t r) {
    return (r & 0x80008000u) | ((r >> 4) & 0x07F007F0u);
}

// Four FP8 e4m3 (one 32-bit word) times the block scale -> 4 BF16 (two packed
// words).  `scale2` holds scale * 2^120 in both halves; integer ALU plus one
// packed BF16 multiply per pair (no slow-rate conversion instructions).
__device__ __forceinline__ void dequant4(uint32_t w, __nv_bfloat162 scale2, uint32_t& lo, uint32_t& hi) {
    uint32_t r01 = e4m3x2_to_bf16x2_bits(__byte_perm(w, 0u, 0x1404u));
    uint32_t r23 = e4m3x2_to_bf16x2_bits(__byte_perm(w, 0u, 0x3424u));
    __nv_bfloat162 a = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&r01), scale2);
    __nv_bfloat162 b = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&r23), scale2);
    lo = *reinterpret_cast<uint32_t*>(&a);
    hi = *reinterpret_cast<uint32_t*>(&b);
}

// Four FP8 e4m3 (one 32-bit word) times the block scale -> 4 FP16 (two packed words).
__device__ __forceinline__ void dequant4_f16(uint32_t w, __half2 scale2, uint32_t& lo, uint32_t& hi) {
    uint32_t a, b;
    ptx::e4m3x4_to_f16x4(w, a, b);
    const __half2 x = __hmul2(*reinterpret_cast<const __half2*>(&a), scale2);
    const __half2 y = __hmul2(*reinterpret_cast<const __half2*>(&b), scale2);
    lo = *reinterpret_cast<const uint32_t*>(&x);
    hi = *reinterpret_cast<const uint32_t*>(&y);
}

// Where an entry lives, as a 32-bit record number with bit 31 = "takes part" and bit 30 = "second pool"
// (the window buffer / the sliding-window planes or pages): for the packed layout the number of its
// 656-byte record in the pool (page * 64 + slot) or in the window buffer (request * win_cap + row); for
// packed reference pages page << 6 | slot; for the reference planes the row number in the plane.  The
// resolver warp works these out several tiles ahead of the data loads, in stages, so that no stage uses
// the result of a load issued in the same step: the index -> block table -> record chain is off the
// critical path.
constexpr uint32_t kIdValid = 1u << 31, kIdSecond = 1u << 30, kIdNumber = (1u << 30) - 1u;

// What a tile's position in its row needs to be resolved (the same in all lanes of a warp).
struct TileCtx {
    int n, b, hg;
    int n_tok, kv_len_n;
    int v0;              // first entry of the tile in its row
    uint32_t meta;
};
// a tile's tag: first tile of its item, its entries, bit 31: a tile at all
constexpr uint32_t kMetaFirst = 1u << 24, kMetaTile = 1u << 31;
__device__ __forceinline__ int meta_entries(uint32_t meta) { return int(meta & 0xFFu); }

// A resolution in flight: the block-table value requested (not yet looked at) and what is known already.
struct PendingId {
    int page;          // block-table value on its way; kNoPage: `id` is final
    uint32_t id;       // paged: kIdValid | second pool | slot in the page;  otherwise the final record number
};
constexpr int kNoPage = -2;

// Stage 1 (CSA only): the index-list value of entry `ent` of the tile, -1 where there is none.
__device__ __forceinline__ int resolve_index(const DecodeArgs& a, const TileCtx& c, int ent) {
    const int v = c.v0 + ent;
    if ((c.meta & kMetaTile) && v < c.n_tok) return ptx::ld(a.indices + int64_t(c.n) * a.topk + v);
    return -1;
}

// Stage 2: issue the block-table load (where there is one).  `e` is the index-list value (CSA).  An entry
// whose page slot lies outside the block table, or whose window row lies outside the window buffer, is
// reported and left out; nothing is read through it.
template <int SRC>
__device__ __forceinline__ PendingId resolve_issue(const DecodeArgs& a, const TileCtx& c, int e, int ent) {
    PendingId p{kNoPage, 0u};
    const int v = c.v0 + ent;
    const bool in_row = (c.meta & kMetaTile) && v < c.n_tok;
    if constexpr (SRC == kSrcCsa) {
        if (e >= 0 && e < c.kv_len_n) {
            if ((e >> 6) < a.max_pages) {
                p.page = ptx::ld(a.block_table + int64_t(c.b) * a.max_pages + (e >> 6));
                p.id = kIdValid | uint32_t(e & 63);
            } else {
                report_status(a.status, kStatusBadIndex, 4, e);
            }
        }
    } else if constexpr (SRC == kSrcHca) {
        if (in_row) {
            if (v < c.kv_len_n) {
                if ((v >> 6) < a.max_pages) {
                    p.page = ptx::ld(a.block_table + int64_t(c.b) * a.max_pages + (v >> 6));
                    p.id = kIdValid | uint32_t(v & 63);
                } else {
                    report_status(a.status, kStatusBadIndex, 4, v);
                }
            } else if (v - c.kv_len_n < a.win_cap) {
                p.id = kIdValid | kIdSecond | uint32_t(c.b * a.win_cap + (v - c.kv_len_n));
            } else {
                report_status(a.status, kStatusBadIndex, 4, v);
            }
        }
    } else if constexpr (SRC == kSrcRefPaged) {
        // a token outside its block table, or a table value outside the pool, is left out of the
        // softmax instead of being read
        if (in_row) {
            const int slot_mask = (1 << a.pg_page_shift) - 1;
            const bool swa = v >= c.kv_len_n;
            const int w = swa ? v - c.kv_len_n : v;
            const uint8_t* pool = swa ? a.pg_swa : a.pg_kv;
            const int32_t* table = swa ? a.pg_swa_table : a.block_table;
            const int cols = swa ? a.pg_swa_max_pages : a.max_pages;
            if (pool != nullptr && (w >> a.pg_page_shift) < cols) {
                p.page = ptx::ld(table + int64_t(c.b) * cols + (w >> a.pg_page_shift));
                p.id = kIdValid | (swa ? kIdSecond : 0u) | uint32_t(w & slot_mask);
            }
        }
    } else {
        if (in_row)
            p.id = kIdValid | ((v < a.ref_m_cur) ? uint32_t(c.b * a.ref_m_cur + v)
                                                 : (uint32_t(c.b * a.ref_swa_len + (v - a.ref_m_cur)) | kIdSecond));
    }
    return p;
}

// Stage 3 (a step later, when the block-table value has arrived): the record number.  A table value
// outside the pool is reported and the entry left out.
template <int SRC>
__device__ __forceinline__ uint32_t resolve_finish(const DecodeArgs& a, const PendingId& p) {
    if (p.page == kNoPage || !(p.id & kIdValid)) return p.id;
    if constexpr (SRC == kSrcRefPaged) {
        const int64_t pages = (p.id & kIdSecond) ? a.pg_swa_num_pages : a.pg_num_pages;
        if (p.page < 0 || p.page >= pages) return 0u;
        return (p.id & (kIdValid | kIdSecond)) | (uint32_t(p.page) << 6) | (p.id & 63u);
    } else {
        if (p.page < 0 || (long long)p.page >= a.num_pages) {
            report_status(a.status, kStatusBadIndex, 4, p.page);
            return 0u;
        }
        return kIdValid | (uint32_t(p.page) * 64u + (p.id & 63u));
    }
}

// This block's Q rows of an item pulled into L2 ahead of their use: 64 rows x NCHUNK x 128 bytes, by one warp.
template <int NCHUNK>
__device__ __forceinline__ void prefetch_q_l2(const DecodeArgs& a, int n, int hg, int rank, int lane) {
    const int h0 = hg * kHeadsPerCta + rank * kHeadsPerBlock;
    const uint8_t* base = reinterpret_cast<const uint8_t*>(a.q + (int64_t(n) * a.H + h0) * (64 * NCHUNK));
    const int lines = min(kHeadsPerBlock, a.H - h0) * NCHUNK;
#pragma unroll 1
    for (int l = lane; l < lines; l += 32) ptx::prefetch_l2(base + int64_t(l) * 128);
}

// What the chain from a row's lengths to its first records runs through (lengths, index list, block table), and its Q, pulled
// into L2 at the very start of a launch on the static grid, where the row is known from the grid position: the chain then
// waits for DRAM once instead of three times (with Q set up meanwhile: CSA, 64 x 2048 62.5 -> 60.3 us, one request 15.0 -> 13.7).
// Nothing is read, so the kernel before may still be writing these.
template <int NCHUNK, int SRC>
__device__ __forceinline__ void prefetch_start(const DecodeArgs& a, int n, int hg, int rank, int warp, int lane) {
    constexpr int kMostLines = 128;
    auto row = [&](const void* p, int64_t bytes) {
        const int lines = int(min(bytes, int64_t(kMostLines) * 128));
#pragma unroll 1
        for (int at = lane * 128; at < lines; at += 32 * 128) ptx::prefetch_l2(static_cast<const uint8_t*>(p) + at);
    };
    const int b = n / a.s_q;
    if (warp == 0) {
        if (lane == 0 && a.kv_len != nullptr) ptx::prefetch_l2(a.kv_len + n);
        if (lane == 1 && a.topk_len != nullptr) ptx::prefetch_l2(a.topk_len + n);
        if (lane == 2 && a.win_len != nullptr) ptx::prefetch_l2(a.win_len + n);
    } else if (warp == 1) {
        if (SRC == kSrcCsa && rank == 0) row(a.indices + int64_t(n) * a.topk, int64_t(a.topk) * 4);
    } else if (warp == 2) {
        if (rank == 1) row(a.block_table + int64_t(b) * a.max_pages, int64_t(a.max_pages) * 4);
    } else {
        const int h0 = hg * kHeadsPerCta + rank * kHeadsPerBlock;
        const uint8_t* base = reinterpret_cast<const uint8_t*>(a.q + (int64_t(n) * a.H + h0) * (64 * NCHUNK));
        const int lines = min(kHeadsPerBlock, a.H - h0) * NCHUNK;
#pragma unroll 1
        for (int l = (warp - 3) * 32 + lane; l < lines; l += (kNumVWarps - 3) * 32) ptx::prefetch_l2(base + int64_t(l) * 128);
    }
}

// The row lengths of an item, from the per-row length arrays.
template <int SRC>
__device__ __forceinline__ void row_lengths(const DecodeArgs& a, int n, int& n_tok, int& kv_len_n) {
    if constexpr (SRC == kSrcCsa) {
        const int raw = (a.topk_len != nullptr) ? ptx::ld(a.topk_len + n) : a.topk;
        n_tok = min(max(raw, 0), a.topk);
        kv_len_n = (a.kv_len != nullptr) ? ptx::ld(a.kv_len + n) : 0x7FFFFFFF;
    } else if constexpr (SRC == kSrcHca || SRC == kSrcRefPaged) {
        kv_len_n = max(ptx::ld(a.kv_len + n), 0);
        n_tok = kv_len_n + max(ptx::ld(a.win_len + n), 0);
    } else {
        kv_len_n = a.ref_m_cur;
        n_tok = a.ref_m_cur + a.ref_swa_len;
    }
}

// ── producers ──
template <int SRC>
struct RecordPtr {
    const uint8_t* lat;
    const uint8_t* scale;
    const uint8_t* rope;
    __device__ __forceinline__ RecordPtr(const DecodeArgs& a, uint32_t id) {
        const uint32_t num = id & kIdNumber;
        const bool second = (id & kIdSecond) != 0u;
        if constexpr (!is_ref_layout(SRC)) {
            lat = (second ? a.win_pool : a.kv_pool) + int64_t(num) * 656;
            scale = lat + 512;
            rope = lat + 528;
        } else if constexpr (SRC == kSrcRefPaged) {
            const int slot = int(num & 63u);
            lat = (second ? a.pg_swa : a.pg_kv) + int64_t(num >> 6) * a.pg_page_bytes + slot * 576;
            // the page's scale area starts after its page_size tokens: 8 bytes per token
            scale = lat + int64_t((1 << a.pg_page_shift) - slot) * 576 + slot * 8;
            rope = lat + 448;
        } else {
            lat = (second ? a.ref_ks : a.ref_kc) + int64_t(num) * 448;
            scale = (second ? a.ref_ks_s : a.ref_kc_s) + int64_t(num) * 7;
            rope = reinterpret_cast<const uint8_t*>(second ? a.ref_ks_rope : a.ref_kc_rope) + int64_t(num) * 128;
        }
    }
};

// The reference layouts' seven UE8M0 bytes of an entry (planes: 7 bytes at any alignment; pages: 8 aligned bytes).
template <int SRC>
__device__ __forceinline__ uint2 load_ref_scales(const DecodeArgs& a, uint32_t id) {
    uint2 w = make_uint2(0u, 0u);
    if (id & kIdValid) {
        const RecordPtr<SRC> p(a, id);
        if constexpr (SRC == kSrcRefPaged) {
            w = ptx::ld(reinterpret_cast<const uint2*>(p.scale));
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) w.x |= uint32_t(ptx::ld(p.scale + i)) << (8 * i);
#pragma unroll
            for (int i = 0; i < 3; ++i) w.y |= uint32_t(ptx::ld(p.scale + 4 + i)) << (8 * i);
        }
    }
    return w;
}

// Sends for the raw data of one tile that fetch warp `p` of block `rank` owns: record numbers in ids[0..31] (0 where
// none), validity and second-pool bits by row.  Groups of four rows without a valid entry are left out; in the others
// an entry that takes no part is fetched as record 0 of the pool and never used.  Called by all lanes.
template <int SRC>
__device__ __forceinline__ void fetch_raw(const DecodeArgs& a, const int32_t* ids, uint32_t valid, uint32_t second, int p, int rank,
                                          uint32_t stage, uint32_t bar, int lane) {
    using R = RawLayout<SRC>;
    if constexpr (SRC == kSrcRefPaged) {
        // A group of four rows is one box where its tokens follow one another in one page; at the end of a row, and where a row of
        // window tokens crosses a page, it is one bulk copy per token.  (32 of those occupy a warp for 2000 cycles.)
        const uint32_t bytes = p == 0 ? 576u : (rank ? 320u : 256u);
        const int id = ids[lane], id0 = __shfl_sync(0xFFFFFFFFu, id, lane & ~3);
        const uint32_t swa = (second >> lane) & 1u, swa0 = (second >> (lane & ~3)) & 1u;
        // (the first test: record numbers follow one another across pages of 64 that do)
        const uint32_t odd = __ballot_sync(0xFFFFFFFFu, (id0 & 63) > 60 || !((valid >> lane) & 1u) || id != id0 + (lane & 3) || swa != swa0);
        const uint32_t boxes = ~(odd | (odd >> 1) | (odd >> 2) | (odd >> 3)) & 0x11111111u, single = valid & ~(boxes * 15u);
        if (lane == 0) ptx::mbar_arrive_expect_tx(bar, uint32_t(4 * __popc(boxes) + __popc(single)) * bytes);
        __syncwarp();
        if (ptx::elect_one()) {
            int first[8];
#pragma unroll
            for (int g = 0; g < 8; ++g) first[g] = ids[4 * g];
#pragma unroll
            for (int g = 0; g < 8; ++g)
                if ((boxes >> (4 * g)) & 1u)
                    ptx::tma_load_3d(stage + (p == 0 ? R::own(4 * g) : R::half(4 * g, rank)), &a.rec_map[(second >> (4 * g)) & 1u][p == 0 ? 0 : 1 + rank],
                                     p == 0 ? 0 : 64 * rank, first[g] & 63, first[g] >> 6, bar);
        }
        __syncwarp();
        if ((single >> lane) & 1u) {
            const RecordPtr<SRC> r(a, uint32_t(id) | (swa ? kIdSecond : 0u));
            ptx::bulk_load(stage + (p == 0 ? R::own(lane) : R::half(lane, rank)), r.lat + (p == 0 ? 0 : 256 * rank), bytes, bar);
        }
        __syncwarp();
        return;
    }
    const uint32_t any = (valid | (valid >> 1) | (valid >> 2) | (valid >> 3)) & 0x11111111u;       // bit 4 g: group g has a valid entry
    const uint32_t group_bytes = p == 0 ? (R::kPacked ? 4u * 656u : 4u * (448u + 128u)) : (R::kPacked ? 4u * (256u + 16u) : (rank ? 4u * (192u + 128u) : 4u * 256u));
    // groups with entries of both pools (at most one in a dense row: where the cache ends and the window begins)
    const uint32_t s4 = (second | (second >> 1) | (second >> 2) | (second >> 3)) & 0x11111111u;
    const uint32_t f = valid & ~second, f4 = (f | (f >> 1) | (f >> 2) | (f >> 3)) & 0x11111111u;
    const uint32_t mixed = s4 & f4;
    if (ptx::elect_one()) {
        ptx::mbar_arrive_expect_tx(bar, uint32_t(__popc(any)) * group_bytes);
        // Unrolled, with the record numbers read ahead: a gather goes out every 50 cycles (290 in a rolled loop).
        const uint32_t todo = any & ~mixed;
        int4 r[8];
#pragma unroll
        for (int g = 0; g < 8; ++g) r[g] = *reinterpret_cast<const int4*>(ids + 4 * g);
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            if (!((todo >> (4 * g)) & 1u)) continue;
            const int pool = SRC == kSrcCsa ? 0 : int((s4 >> (4 * g)) & 1u);
            const CUtensorMap* m = a.rec_map[pool];
            if constexpr (R::kPacked) {
                ptx::tma_gather4(p == 0 ? stage + R::own(4 * g) : stage + R::half(4 * g, 0), p == 0 ? &m[0] : &m[1], p == 0 ? 0 : 64 * rank, r[g], bar);
                if (p != 0) ptx::tma_gather4(stage + R::kScaleOff + uint32_t(g) * 128u, &m[2], 128, r[g], bar);
            } else {
                ptx::tma_gather4(p == 0 ? stage + R::own(4 * g) : stage + R::half(4 * g, rank), p == 0 ? &m[0] : &m[1 + rank], p == 0 ? 0 : 64 * rank, r[g], bar);
                if (p == 0 || rank) ptx::tma_gather4(p == 0 ? stage + R::own_rope(4 * g) : stage + R::half_rope(4 * g), &a.rope_map[pool], 0, r[g], bar);
            }
        }
        if (SRC != kSrcCsa && mixed) {
            // row by row
#pragma unroll 1
            for (int row = 0; row < 32; ++row) {
                if (!((mixed >> (row & ~3)) & 1u)) continue;
                const RecordPtr<SRC> q(a, uint32_t(ids[row]) | (((second >> row) & 1u) ? kIdSecond : 0u));
                if (p == 0) {
                    ptx::bulk_load(stage + R::own(row), q.lat, R::kOwnRow, bar);
                    if constexpr (!R::kPacked) ptx::bulk_load(stage + R::own_rope(row), q.rope, 128, bar);
                } else {
                    ptx::bulk_load(stage + R::half(row, rank), q.lat + 256 * rank, uint32_t(R::half_row(rank)), bar);
                    if constexpr (R::kPacked) ptx::bulk_load(stage + R::kScaleOff + uint32_t(row >> 2) * 128u + uint32_t(row & 3) * 16u, q.scale, 16, bar);
                    else if (rank) ptx::bulk_load(stage + R::half_rope(row), q.rope, 128, bar);
                }
            }
        }
    }
    __syncwarp();
}

// ── K and V warps ──
// One load or store instruction covers four rows; eight lanes take the eight 16-byte pieces of a row's 128-byte span (two
// 64-element latent chunks, or the RoPE tail).  Shared memory serves a quarter-warp (8 lanes) at a time, and both ways
// its lanes have to cover all eight 16-byte bank groups:
//  * stores: piece p becomes columns 2 (p % 4) and + 1 of chunk p / 4 of its row, swizzled by the row number.  A quarter-warp takes
//    four pieces (no two with the same p % 4) of each of two neighbouring rows, whose swizzles differ in the lowest bit:
//    even columns of the one, odd ones of the other.
//  * loads: raw rows lie `pitch` bytes apart, pitch / 16 = s (mod 8) bank groups, so the odd row's pieces are rotated by s:
//    lanes 4-7 of a quarter take pieces 4 - s .. 7 - s (mod 8).  (Without it every load took twice its time.)
__device__ __forceinline__ int loader_row(int lane) { return (lane >> 3) ^ ((lane >> 2) & 1); }
__device__ __forceinline__ int loader_piece(int lane, int pitch) { return ((lane & 7) - (loader_row(lane) & 1) * (pitch / 16)) & 7; }

// Dequantise 16 latent bytes and store them as two 16-byte columns at `at` and `at` ^ 16.
template <int SRC>
__device__ __forceinline__ void store_latent(uint32_t at, const uint4& x, uint32_t w) {
    uint4 w0, w1;
    if constexpr (use_f16(SRC)) {
        // scales above 146 would take 448 x scale past FP16's largest finite value: such blocks saturate
        const __half2 scale2 = __float2half2_rn(fminf(__uint_as_float(w), 146.f));
        dequant4_f16(x.x, scale2, w0.x, w0.y);
        dequant4_f16(x.y, scale2, w0.z, w0.w);
        dequant4_f16(x.z, scale2, w1.x, w1.y);
        dequant4_f16(x.w, scale2, w1.z, w1.w);
    } else {
        // one UE8M0 byte per 64 elements: 2^(byte-127) * 2^120; a zero byte means a zero
        // scale, as in the reference's dequantiser
        const float s120 = w ? __uint_as_float((w + 120u) << 23) : 0.f;
        const __nv_bfloat162 scale2 = __float2bfloat162_rn(s120);
        dequant4(x.x, scale2, w0.x, w0.y);
        dequant4(x.y, scale2, w0.z, w0.w);
        dequant4(x.z, scale2, w1.x, w1.y);
        dequant4(x.w, scale2, w1.z, w1.w);
    }
    ptx::sts_v4(at, w0);
    ptx::sts_v4(at ^ 16u, w1);
}

// Where a lane's stores go.  Row t of a chunk is 128 bytes; 16-byte column c16 of row t lives at (c16 ^ (t % 8)) << 4.
// Its 16 latent bytes of a span (piece p) become columns 2 (p % 4) and + 1 of the span's chunk `flip` = p / 4.
struct LoaderAddr {
    uint32_t row;        // row of this lane's first entry
    uint32_t flip;
    uint32_t lat;        // byte offset of the first of those columns of that row inside a chunk
    uint32_t rope;       // byte offset of RoPE column p
    // row0: first row of the warp (a multiple of 8).  Its entries are rows row + 4 i; at odd i the swizzle of a row differs in
    // bit 2, that is, in bit 6 of the offset.
    __device__ __forceinline__ LoaderAddr(int row0, uint32_t piece, int lane) {
        row = uint32_t(row0 + loader_row(lane));
        flip = piece >> 2;
        lat = row * 128u + (((2u * (piece & 3u)) ^ (row & 7u)) << 4);
        rope = row * 128u + ((piece ^ (row & 7u)) << 4);
    }
    static __device__ __forceinline__ uint32_t at(uint32_t off, int i) { return (off ^ ((i & 1) ? 64u : 0u)) + uint32_t(i) * 512u; }
};

__device__ __forceinline__ uint4 bf16x8_to_f16x8(uint4 w) {
    w.x = ptx::bf16x2_to_f16x2(w.x);  w.y = ptx::bf16x2_to_f16x2(w.y);
    w.z = ptx::bf16x2_to_f16x2(w.z);  w.w = ptx::bf16x2_to_f16x2(w.w);
    return w;
}

// A V warp's share of one staging round of Q: lane quarter vw % 4, half vw / 4 of the three chunks at `src` (12 16-byte
// columns of a row) to tensor-memory columns [dst, +96).
template <bool F16>
__device__ __forceinline__ void q_to_tmem(uint32_t src, uint32_t dst, int vw, int lane) {
    static_assert(kNumVWarps == 8 && kFirstVWarp % 4 == 0, "two warps per lane quarter");
    const int row = (vw & 1) * 32 + lane;
    const uint32_t base = src + uint32_t(row) * 128u, sw = uint32_t(row & 7) << 4, lanes = uint32_t((vw & 3) * 32) << 16;
#pragma unroll 1
    for (int i = 0; i < 4 * kQStageChunks; i += 2) {
        const int u = (vw >> 2) * 4 * kQStageChunks + i;
        const uint32_t chunk = base + uint32_t(u >> 3) * kQChunkBytes;
        uint4 x = ptx::lds_v4(chunk + ((uint32_t(u & 7) << 4) ^ sw)), y = ptx::lds_v4(chunk + ((uint32_t((u & 7) + 1) << 4) ^ sw));
        if constexpr (F16) { x = bf16x8_to_f16x8(x);  y = bf16x8_to_f16x8(y); }
        ptx::tmem_st8(dst + lanes + uint32_t(u) * 4u, x, y);
    }
}

template <int NCHUNK, int SRC>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kNumThreads, 1) decode_mma_kernel(const __grid_constant__ DecodeArgs a) {
    using L = SmemLayout<NCHUNK, SRC>;
    using R = RawLayout<SRC>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t smem_base = ptx::smem_u32(smem_raw);
    if (smem_base & 1023u) {                      // the operand layout needs it; the same answer in every block
        report_status(a.status, kStatusWaitQ, 5, -1);
        return;
    }
    const uint32_t q_base = smem_base + L::kQOff;
    const uint32_t q_stage = smem_base + L::kQStageOff;
    const uint32_t k_base = smem_base + L::kKOff;
    const uint32_t v_base = smem_base + L::kVOff;
    const uint32_t p_base = smem_base + L::kPOff;
    const uint32_t raw_base = smem_base + L::kRawOff;
    SmemMisc* misc = reinterpret_cast<SmemMisc*>(smem_raw + L::kMiscOff);

    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const int rank = int(blockIdx.x & 1u);        // = rank in the cluster pair
    const bool sched = a.sched_pair_begin != nullptr;
    const int rows = a.B * a.s_q;
    const uint32_t wait_ns = a.wait_ns;

    // ── this pair's items (known after set-up) ──
    int item_begin = 0, n_items = 1;
    auto get_item = [&](int k) -> Item {
        Item it;
        if (sched) {
            const int4* rec = reinterpret_cast<const int4*>(a.sched_items + int64_t(item_begin + k) * kItemWords);
            const int4 r0 = ptx::ld(rec), r1 = ptx::ld(rec + 1);
            it.n = r0.x;  it.hg = r0.y;  it.tile0 = r0.z;  it.ntiles = r0.w;
            it.slot = r1.x;  it.n_tok = r1.y;  it.kv_len_n = r1.z;
        } else {
            it.n = blockIdx.y;  it.hg = blockIdx.x >> 1;
            row_lengths<SRC>(a, it.n, it.n_tok, it.kv_len_n);
            const int split = blockIdx.z;
            const int tiles_total = (it.n_tok + kTileN - 1) / kTileN;
            const int tiles_per_split = (tiles_total + a.num_splits - 1) / a.num_splits;
            it.tile0 = min(split * tiles_per_split, tiles_total);
            it.ntiles = min(it.tile0 + tiles_per_split, tiles_total) - it.tile0;
            it.slot = a.num_splits > 1 ? split : -1;
        }
        return it;
    };

    // barriers of this block ...
    const uint32_t bar_raw_full = ptx::smem_u32(&misc->bar_raw_full[0]);
    const uint32_t bar_raw_free = ptx::smem_u32(&misc->bar_raw_free[0]);
    const uint32_t bar_id_full = ptx::smem_u32(&misc->bar_id_full[0][0]);
    const uint32_t bar_id_free = ptx::smem_u32(&misc->bar_id_free[0][0]);
    const uint32_t bar_q_full = ptx::smem_u32(&misc->bar_q_full[0]);
    const uint32_t bar_q_copied = ptx::smem_u32(&misc->bar_q_copied[0]);
    const uint32_t bar_tmem = ptx::smem_u32(&misc->bar_tmem);
    const uint32_t bar_s_full = ptx::smem_u32(&misc->bar_s_full[0]);
    const uint32_t bar_v_free = ptx::smem_u32(&misc->bar_v_free);
    const uint32_t bar_o_full = ptx::smem_u32(&misc->bar_o_full[0]);
    // ... and of the even one
    const uint32_t bar_q_ready = ptx::smem_u32(&misc->bar_q_ready);
    const uint32_t bar_k_full = ptx::smem_u32(&misc->bar_k_full[0]);
    const uint32_t bar_v_full = ptx::smem_u32(&misc->bar_v_full[0]);
    const uint32_t bar_p_full = ptx::smem_u32(&misc->bar_p_full[0]);
    auto arrive_even = [&](uint32_t bar) {
        if (rank == 0) ptx::mbar_arrive(bar);
        else ptx::mbar_arrive_remote(ptx::mapa(bar, 0));
    };

    // On the static grid a launch over 656-byte records sees to Q before anything is known of the row (top-k 2048, 64 requests: 62.5 -> 60.3 us).
    // The reference planes, with no lengths, indices or tables to wait for, have their first records before Q: 1 us of 45 slower with Q first.
    // Packed reference pages (40 ragged requests): 48.0 to 48.3 us either way.  On a schedule Q comes item by item; its first one early was not tried.
    const bool early_q = use_f16(SRC) && !sched;

    // ── set-up ──
    if (early_q && warp >= kFirstVWarp && warp < kSWarp) prefetch_start<NCHUNK, SRC>(a, blockIdx.y, blockIdx.x >> 1, rank, warp - kFirstVWarp, lane);
    if (warp == kSWarp && lane == 0) ptx::prefetch_tensormap(&a.q_map);
    if (!is_ref_layout(SRC) && warp == kFetchWarp && lane < 3 && a.num_pages > 0) ptx::prefetch_tensormap(&a.rec_map[0][lane]);
    if (tid == 0) {
        for (int i = 0; i < kStages; ++i) {
            ptx::mbar_init(bar_raw_full + 8 * i, 2);
            ptx::mbar_init(bar_raw_free + 8 * i, kNumKWarps + kNumVWarps);
        }
        for (int i = 0; i < 2 * kIdRing; ++i) {
            ptx::mbar_init(bar_id_full + 8 * i, 1);
            ptx::mbar_init(bar_id_free + 8 * i, 1);
        }
        ptx::sts_u32(failed_flag(), 0u);
        ptx::mbar_init(bar_tmem, 1);
        ptx::mbar_init(bar_v_free, 1);
        ptx::mbar_init(bar_q_ready, 2 * (early_q ? kNumVWarps + kNumKWarps : kNumVWarps));
        for (int i = 0; i < 2; ++i) {
            ptx::mbar_init(bar_q_full + 8 * i, 1);
            ptx::mbar_init(bar_q_copied + 8 * i, kNumVWarps);
            ptx::mbar_init(bar_k_full + 8 * i, 2 * kNumKWarps);
            ptx::mbar_init(bar_s_full + 8 * i, 1);
            ptx::mbar_init(bar_o_full + 8 * i, 1);
            ptx::mbar_init(bar_v_full + 8 * i, kNumVWarps);              // half of the warps of each block
            ptx::mbar_init(bar_p_full + 8 * i, 2 * kNumSoftmaxWarps);
        }
        ptx::fence_mbar_init();
    }
    // The barriers of both blocks are initialised before any role of either starts.
    __syncwarp();
    ptx::cluster_sync();
    ptx::pdl_wait();
    if (sched) {
        const int pair = blockIdx.x >> 1;
        item_begin = ptx::ld(a.sched_pair_begin + pair);
        n_items = ptx::ld(a.sched_pair_begin + pair + 1) - item_begin;
    }
    // All 512 columns are allocated, so tensor memory starts at address 0 (checked where it is allocated): as a constant it keeps the
    // operands of every tcgen05 instruction out of vector registers.
    constexpr uint32_t tmem = 0;
    auto wait_tmem = [&]() -> bool {
        const bool w = ptx::mbar_wait_warp(bar_tmem, 0u, wait_ns);
        ptx::tc_fence_after_sync();
        return w;
    };
    // Waits of a whole warp: the outcome is the same in all lanes (the warp-collective operations below need them all).
    auto wait_for = [&](uint32_t bar, uint32_t phase, int code, int role, int at) -> bool {
        const bool w = ptx::mbar_wait_warp(bar, phase & 1u, wait_ns);
        if (!w) wait_ran_out(a.status, code, role, at);
        return w;
    };

    // Running counters, the same in every role of both blocks: `g` counts the tiles the pair has gone through over all
    // its items, `qn` the items that had tiles.  Tile g is the g-th use of the K and V buffers, the (g / 2)-th of S and P
    // buffer g % 2 and the (g / 3)-th of raw stage g % 3.  A wait on a barrier never lags two of its phases (the next
    // phase always needs the waiter) and never runs ahead of it by more than one (every waiter goes through its
    // phases one by one).

    // one of eight warps' share of Q's chunks in shared memory, BF16 to FP16 (element-wise, so the swizzled layout is untouched)
    auto convert_q = [&](int w) {
        constexpr int kVecs = L::kQChunks * kQChunkBytes / 16 / (kNumVWarps * 32);
#pragma unroll 1
        for (int i = 0; i < kVecs; ++i) {
            const uint32_t at = q_base + uint32_t((i * kNumVWarps + w) * 32 + lane) * 16u;
            ptx::sts_v4(at, bf16x8_to_f16x8(ptx::lds_v4(at)));
        }
    };

    if (warp >= kFirstKWarp && warp < kFirstVWarp) {
        // ───────────── K warps ─────────────
        // K rows 4 kw .. +3 of this block, all columns.  (Refilling the first half of the tile while the S MMAs still read the
        // second gained nothing: a commit in the middle of a chain of MMAs into one accumulator arrives with the one at its
        // end.)
        const int kw = warp - kFirstKWarp;
        const uint32_t piece = uint32_t(loader_piece(lane, R::kOwnRow));
        const LoaderAddr ad(4 * kw, piece, lane);
        bool ok = true;
        if (early_q) {
            // (Q's chunks that stay in shared memory, before the first records are there)
            ok = wait_for(bar_q_full, 0u, kStatusWaitQ, 2, 0);
            if (ok) {
                convert_q(kw);
                ptx::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) arrive_even(bar_q_ready);
            }
        }
#pragma unroll 1
        for (uint32_t g = 0; ok; ++g) {
            const uint32_t st = g % kStages, raw = raw_base + st * R::kBytes;
            if (kw == 0 && lane == 0) trace_mark(a, 2, 8 * int(g));
            if (!wait_for(bar_raw_full + 8 * st, g / kStages, kStatusWaitRaw, 2, int(g))) break;
            const uint32_t meta = *reinterpret_cast<volatile uint32_t*>(&misc->meta[g % kTagRing]);
            if (!(meta & kMetaTile)) break;                              // the end of the stream
            const bool used = kw < tile_groups(meta_entries(meta));
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                uint4 x[2], rope;
                uint32_t sc[2];
                // (rows that are not in use hold whatever the ring held before: finite or not, their logits are masked)
                const uint32_t src = raw + R::own(ad.row) + uint32_t(h) * 256u + piece * 16u;
                x[0] = ptx::lds_v4(src);
                if (!is_ref_layout(SRC) || h == 0 || ad.flip == 0u) x[1] = ptx::lds_v4(src + 128u);       // (reference layouts: the last span ends with its first chunk)
                if constexpr (!is_ref_layout(SRC)) {
                    const uint2 s2 = ptx::lds_v2(raw + R::own(ad.row) + 512u + uint32_t(h) * 8u);
                    sc[0] = s2.x;  sc[1] = s2.y;
                } else {
                    const uint32_t at = raw + R::kScaleOff + (uint32_t(rank) * 32u + ad.row) * 8u + uint32_t(h) * 4u + ad.flip;
                    sc[0] = ptx::lds_u8(at);  sc[1] = ptx::lds_u8(at + 2u);
                }
                if (h) rope = ptx::lds_v4(raw + R::own_rope(ad.row) + piece * 16u);
                if (h) {
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(bar_raw_free + 8 * st);
                } else if (g > 0u) {
                    ok = wait_for(bar_s_full + 8 * ((g - 1u) & 1u), (g - 1u) >> 1, kStatusWaitKvFree, 2, int(g));
                    if (!ok) break;
                }
                if (used) {
                    const uint32_t dst = k_base + (4u * uint32_t(h) + ad.flip) * kKChunkBytes + ad.lat;
                    store_latent<SRC>(dst, x[0], sc[0]);
                    if (!is_ref_layout(SRC) || h == 0 || ad.flip == 0u) store_latent<SRC>(dst + 2u * kKChunkBytes, x[1], sc[1]);
                    if (h) ptx::sts_v4(k_base + uint32_t(NCHUNK - 1) * kKChunkBytes + ad.rope, use_f16(SRC) ? bf16x8_to_f16x8(rope) : rope);
                }
                ptx::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0 && !(a.dbg_drop_tile >= 0 && g == uint32_t(a.dbg_drop_tile))) arrive_even(bar_k_full + 8 * h);
            }
            if (!ok) break;
        }
    } else if (warp >= kFirstVWarp && warp < kSWarp) {
        // ───────────── V warps ─────────────
        // Warp (jj, hb, hr): rows 16 hr .. +15 of block hb, 128-column span jj of this block's value columns.  Also Q's set-up.
        const int vw = warp - kFirstVWarp, jj = vw >> 2, hb = (vw >> 1) & 1, hr = vw & 1, span = 2 * rank + jj;
        const bool mine = hb == rank;
        const uint32_t piece = uint32_t(loader_piece(lane, mine ? R::kOwnRow : R::half_row(rank)));
        const LoaderAddr ad(16 * hr, piece, lane);
        const uint32_t v_span = v_base + 2u * uint32_t(jj) * kVChunkBytes + uint32_t(hb) * (kRowsPerBlock * 128u);
        uint32_t qn = 0;
        // Q of an item has been sent for by the S warp (early: at once; else once the previous item's S MMAs had completed):
        // chunks 0-5 reach tensor memory through a staging area in two rounds, the others land at their place in
        // shared memory and are converted there.
        auto set_up_q = [&](uint32_t g) -> bool {
#pragma unroll 1
            for (int round = 0; round < 2; ++round) {
                if (!wait_for(bar_q_full + 8 * round, qn, kStatusWaitQ, 2, int(g)) || (qn == 0u && !wait_tmem())) return false;
                q_to_tmem<use_f16(SRC)>(round && qn == 0u ? v_base : q_stage, tmem + kTmemQ + 96 * round, vw, lane);
                if (use_f16(SRC) && round == 0 && !early_q) convert_q(vw);
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(bar_q_copied + 8 * round);
            }
            ptx::tmem_wait_st();
            ptx::tc_fence_before_sync();
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) arrive_even(bar_q_ready);
            // (the first item's second round was staged in the V tile)
            if (qn == 0u && !wait_for(bar_q_copied + 8, 0u, kStatusWaitQ, 2, int(g))) return false;
            ++qn;
            return true;
        };
        bool ok = !early_q || set_up_q(0u);
#pragma unroll 1
        for (uint32_t g = 0; ok; ++g) {
            const uint32_t st = g % kStages, raw = raw_base + st * R::kBytes;
            if (!wait_for(bar_raw_full + 8 * st, g / kStages, kStatusWaitRaw, 2, int(g))) break;
            const uint32_t meta = *reinterpret_cast<volatile uint32_t*>(&misc->meta[g % kTagRing]);
            if (!(meta & kMetaTile)) break;
            if (!early_q && (meta & kMetaFirst) && !set_up_q(g)) break;
            const int groups = tile_groups(meta_entries(meta)), rows = 16 * tile_ksteps(meta_entries(meta));
            const uint32_t valid = *reinterpret_cast<volatile uint32_t*>(&misc->mask[g % kTagRing][hb]);
            uint4 x[4], rope[is_ref_layout(SRC) ? 4 : 1];
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t row = ad.row + 4 * i;
                if (4 * hr + i < groups) {
                    const uint32_t c = 2u * uint32_t(span) + ad.flip;
                    if (!is_ref_layout(SRC) || c < 7u)
                        x[i] = ptx::lds_v4(raw + (mine ? R::own(row) + uint32_t(span) * 128u : R::half(row, rank) + uint32_t(jj) * 128u) + piece * 16u);
                    if constexpr (!is_ref_layout(SRC)) {
                        w[i] = ptx::lds_u32(raw + (mine ? R::own(row) + 512u : R::kScaleOff + (row >> 2) * 128u + (row & 3u) * 16u) + uint32_t(span) * 4u);
                    } else {
                        w[i] = ptx::lds_u8(raw + R::kScaleOff + (uint32_t(hb) * 32u + row) * 8u + c);
                        if (span == 3) rope[i] = ptx::lds_v4(raw + (mine ? R::own_rope(row) : R::half_rope(row)) + piece * 16u);
                    }
                }
                if (!((valid >> row) & 1u)) {
                    // an entry that takes no part: a zero row stays finite under the MMA whatever its probability holds
                    x[i] = make_uint4(0, 0, 0, 0);
                    w[i] = 0u;
                    if constexpr (is_ref_layout(SRC)) rope[i] = make_uint4(0, 0, 0, 0);
                }
            }
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(bar_raw_free + 8 * st);
            if (vw == 0 && lane == 0) trace_mark(a, 2, 8 * int(g) + 5);
            if (g > 0u && !wait_for(jj ? bar_o_full + 8 * ((g - 1u) & 1u) : bar_v_free, jj ? (g - 1u) >> 1 : g - 1u, kStatusWaitKvFree, 2, int(g))) break;
            if (vw == 0 && lane == 0) trace_mark(a, 2, 8 * int(g) + 6);
            if (16 * hr < rows) {                                        // else not read by the MMAs of this tile
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if constexpr (is_ref_layout(SRC)) {
                        if (span == 3) {
                            // chunk 6 is the end of the latent, chunk 7 the RoPE tail
                            ptx::sts_v4(v_span + kVChunkBytes + LoaderAddr::at(ad.rope, i), rope[i]);
                            if (ad.flip) continue;
                        }
                    }
                    store_latent<SRC>(v_span + ad.flip * kVChunkBytes + LoaderAddr::at(ad.lat, i), x[i], w[i]);
                }
            }
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) arrive_even(bar_v_full + 8 * jj);
            if (vw == 0 && lane == 0) trace_mark(a, 2, 8 * int(g) + 7);
        }
    } else if (warp == kSWarp) {
        // ───────────── tensor-memory allocation, Q load, S = Q . K^T ─────────────
        constexpr uint32_t kDescHi = ptx::smem_desc_hi(1024);        // 8-row groups 1 KB apart
        // Q rows of this block's 64 heads by TMA, one 64-column box per chunk, landing in the swizzled operand
        // layout.  Rows past the end of Q read as zero; rows of a following request (H < 128) are computed
        // but never written out.
        auto q_row = [&](int n, int hg) { return n * a.H + hg * kHeadsPerCta + rank * kHeadsPerBlock; };
        auto second_round = [&](uint32_t dst, int qrow0) {
            ptx::mbar_arrive_expect_tx(bar_q_full + 8, kQStageChunks * kQChunkBytes);
#pragma unroll
            for (int c = 0; c < kQStageChunks; ++c) ptx::tma_load_2d(dst + uint32_t(c) * kQChunkBytes, &a.q_map, (kQStageChunks + c) * 64, qrow0, bar_q_full + 8);
        };
        auto send_for_q = [&](int qrow0, bool first) {
            if (ptx::elect_one()) {
                ptx::mbar_arrive_expect_tx(bar_q_full, uint32_t(kQStageChunks + L::kQChunks) * kQChunkBytes);
#pragma unroll
                for (int c = 0; c < kQStageChunks; ++c) ptx::tma_load_2d(q_stage + uint32_t(c) * kQChunkBytes, &a.q_map, c * 64, qrow0, bar_q_full);
#pragma unroll
                for (int c = 0; c < L::kQChunks; ++c) ptx::tma_load_2d(q_base + uint32_t(c) * kQChunkBytes, &a.q_map, (kQTmemChunks + c) * 64, qrow0, bar_q_full);
                if (first) second_round(v_base, qrow0);                  // the V tile is still unused
            }
            __syncwarp();
        };
        // (the K and V warps wait for an early Q whether the row turns out empty or not)
        if (early_q) send_for_q(q_row(blockIdx.y, blockIdx.x >> 1), true);
        ptx::tmem2_alloc(ptx::smem_u32(&misc->tmem_base), kTmemCols);
        ptx::tmem2_relinquish();
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0 && *reinterpret_cast<volatile uint32_t*>(&misc->tmem_base) == tmem) ptx::mbar_arrive(bar_tmem);
        bool ok = wait_tmem();
        constexpr uint32_t idesc = use_f16(SRC) ? ptx::make_idesc_f16(128, kTileN, false, false) : ptx::make_idesc_bf16(128, kTileN, false, false);
        const uint32_t q_lo = ptx::smem_desc_lo(q_base, 16), k_lo = ptx::smem_desc_lo(k_base, 16);
        uint32_t gt = 0, qn = 0;
        Item cur = get_item(0);
#pragma unroll 1
        for (int k = 0; k < n_items && ok; ++k) {
            const int ntiles = cur.ntiles;
            if (ntiles > 0) {
                // every S MMA of the previous item must have completed before its Q is replaced
                if (gt > 0u && !wait_for(bar_s_full + 8 * ((gt - 1u) & 1u), (gt - 1u) >> 1, kStatusWaitSFull, 1, int(gt))) { ok = false;  break; }
                const int qrow0 = q_row(cur.n, cur.hg);
                if (!early_q) send_for_q(qrow0, qn == 0u);
                if (qn > 0u) {
                    if (!wait_for(bar_q_copied, qn, kStatusWaitQ, 1, int(gt))) { ok = false;  break; }
                    if (ptx::elect_one()) second_round(q_stage, qrow0);
                    __syncwarp();
                }
                if (rank == 0) {
#pragma unroll 1
                    for (int it = 0; it < ntiles; ++it) {
                        const uint32_t g = gt + uint32_t(it);
                        // the S buffer has been read by the softmax of the tile two before
                        if ((g >= 2u && !wait_for(bar_p_full + 8 * (g & 1u), (g - 2u) >> 1, kStatusWaitPFull, 1, int(g))) ||
                            !wait_for(bar_k_full, g, kStatusWaitKvFull, 1, int(g)) ||
                            (it == 0 && !wait_for(bar_q_ready, qn, kStatusWaitQ, 1, int(g)))) { ok = false;  break; }
                        ptx::tc_fence_after_sync();
                        if (lane == 0) trace_mark(a, 1, 4 * int(g));
                        // unrolled: 18 cycles an instruction to issue, 25 to 40 in a loop
                        const uint32_t d = tmem + kTmemS + (g & 1u) * 32u;
                        auto issue = [&](auto c0_tag, auto c1_tag) {
                            constexpr int C0 = decltype(c0_tag)::value, C1 = decltype(c1_tag)::value;
#pragma unroll
                            for (int c = C0; c < C1; ++c)
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    const uint32_t b_lo = k_lo + uint32_t((c * kKChunkBytes + k * 32) >> 4);
                                    if (c < kQTmemChunks) ptx::mma2_ts(d, tmem + kTmemQ + c * 32 + k * 8, b_lo, kDescHi, idesc, (c | k) ? 1u : 0u);
                                    else ptx::mma2_ss(d, q_lo + uint32_t(((c - kQTmemChunks) * kQChunkBytes + k * 32) >> 4), b_lo, kDescHi, idesc, 1u);
                                }
                        };
                        if (ptx::elect_one()) issue(std::integral_constant<int, 0>{}, std::integral_constant<int, 4>{});
                        __syncwarp();
                        if (!wait_for(bar_k_full + 8, g, kStatusWaitKvFull, 1, int(g))) { ok = false;  break; }
                        ptx::tc_fence_after_sync();
                        if (lane == 0) trace_mark(a, 1, 4 * int(g) + 1);
                        if (ptx::elect_one()) {
                            issue(std::integral_constant<int, 4>{}, std::integral_constant<int, NCHUNK>{});
                            ptx::mma2_commit(bar_s_full + 8 * (g & 1u));
                        }
                        __syncwarp();
                        if (lane == 0) trace_mark(a, 1, 4 * int(g) + 2);
                    }
                } else {
                    // The odd block only follows, phase by phase: a wait may not run ahead of its barrier by more than one.
#pragma unroll 1
                    for (int it = 0; it + 1 < ntiles; ++it) {
                        const uint32_t g = gt + uint32_t(it);
                        if (!wait_for(bar_s_full + 8 * (g & 1u), g >> 1, kStatusWaitSFull, 1, int(g))) { ok = false;  break; }
                    }
                }
                gt += uint32_t(ntiles);
                ++qn;
            }
            if (k + 1 < n_items) cur = get_item(k + 1);
        }
    } else if (warp == kOWarp) {
        // ───────────── O += P . V ─────────────
        if (rank == 0) {
            constexpr uint32_t kDescHi = ptx::smem_desc_hi(1024);
            bool ok = wait_tmem();
                constexpr uint32_t idesc = use_f16(SRC) ? ptx::make_idesc_f16(128, 256, false, true) : ptx::make_idesc_bf16(128, 256, false, true);
            // B = V[16 entries x 256 columns], MN-major: 64-column chunks 8 KB apart (leading offset), 8-entry groups 1 KB
            // apart; each block supplies 128 of the columns
            const uint32_t p_lo = ptx::smem_desc_lo(p_base, 16), v_lo = ptx::smem_desc_lo(v_base, kVChunkBytes);
            uint32_t g = 0;
            Item cur = get_item(0);
#pragma unroll 1
            for (int k = 0; k < n_items && ok; ++k) {
                const int ntiles = cur.ntiles;
#pragma unroll 1
                for (int it = 0; it < ntiles && ok; ++it, ++g) {
                    const int ksteps = tile_ksteps(cur.tile_entries(it));
                    // (the first P of an item is written after the softmax warps have read the previous item's O out of tensor
                    // memory, so the overwrite below needs no barrier of its own)
                    if (!wait_for(bar_p_full + 8 * (g & 1u), g >> 1, kStatusWaitPFull, 3, int(g))) { ok = false;  break; }
                    if (lane == 0) trace_mark(a, 3, 4 * int(g));
                    const uint32_t p_tile = p_lo + (g & 1u) * uint32_t(kQChunkBytes >> 4);
#pragma unroll 1
                    for (int jj = 0; jj < 2; ++jj) {
                        if (!wait_for(bar_v_full + 8 * jj, g, kStatusWaitKvFull, 3, int(g))) { ok = false;  break; }
                        ptx::tc_fence_after_sync();
                        if (lane == 0) trace_mark(a, 3, 4 * int(g) + 1 + jj);
                        if (ptx::elect_one()) {
#pragma unroll
                            for (int h = 0; h < 2; ++h)
#pragma unroll
                                for (int q = 0; q < 2; ++q)
                                    if (q < ksteps)
                                        ptx::mma2_ss(tmem + kTmemO + jj * 128, p_tile + uint32_t(((h * 2 + q) * 32) >> 4),
                                                     v_lo + uint32_t((2 * jj * kVChunkBytes + (h * kRowsPerBlock + q * 16) * 128) >> 4), kDescHi, idesc,
                                                     (it > 0 || h > 0 || q > 0) ? 1u : 0u);
                            ptx::mma2_commit(jj == 0 ? bar_v_free : bar_o_full + 8 * (g & 1u));
                        }
                        __syncwarp();
                    }
                }
                if (k + 1 < n_items) cur = get_item(k + 1);
            }
        }
        __syncwarp();
    } else if (warp >= kResolveWarp) {
        // ───────────── resolve warps: where does every entry live? ─────────────
        // Walk the pair's items in order; a lane owns K row `lane` of its block.  The dependent loads (index list -> block table)
        // are issued one step and looked at the next.
        const int p = warp - kResolveWarp, block = rank ^ p;
        const int slot = ((lane >> 2) << 3) | (block << 2) | (lane & 3);
        int ck = -1, ct = 0;
        Item ci{};
        auto next_tile = [&]() -> TileCtx {
            TileCtx c{};
            if (ck < 0 || ++ct >= ci.ntiles) {                           // on to the next item that has tiles
                ct = 0;
                ci.ntiles = 0;
#pragma unroll 1
                while (ck < n_items && ci.ntiles == 0)
                    if (++ck < n_items) ci = get_item(ck);
            }
            if (ck < n_items) {
                c.n = ci.n;  c.b = ci.n / a.s_q;  c.hg = ci.hg;  c.n_tok = ci.n_tok;  c.kv_len_n = ci.kv_len_n;
                c.v0 = (ci.tile0 + ct) * kTileN;
                c.meta = kMetaTile | (ct == 0 ? kMetaFirst : 0u) | uint32_t(ci.tile_entries(ct));
            }
            return c;
        };
        // A pipeline over the stream of tiles: of tile c2 the index value (CSA) is sent for, of c1 the block-table value, c0 is
        // finished and handed on.  (Reference layouts, no index list: of c2 the block-table value, of c1 the record number and
        // the scales.)
        TileCtx c0{}, c1{};
        int e1 = -1;               // c1's index value
        PendingId p0{kNoPage, 0u};
        uint32_t id0 = 0u;
        uint2 s0 = make_uint2(0u, 0u);
#pragma unroll 1
        for (uint32_t step = 0;; ++step) {
            const TileCtx c2 = next_tile(), cur = c0;
            uint32_t id;
            uint2 scales = s0;
            if constexpr (!is_ref_layout(SRC)) {
                const PendingId p1 = resolve_issue<SRC>(a, c1, e1, slot);
                if constexpr (SRC == kSrcCsa) e1 = resolve_index(a, c2, slot);
                id = resolve_finish<SRC>(a, p0);
                p0 = p1;
            } else {
                id = id0;
                id0 = resolve_finish<SRC>(a, p0);                        // c1's
                s0 = load_ref_scales<SRC>(a, id0);
                p0 = resolve_issue<SRC>(a, c2, -1, slot);
            }
            c0 = c1;
            c1 = c2;
            if (step < 2u) continue;
            const uint32_t t = step - 2u;
            const uint32_t i = t % kIdRing, bars = 8u * uint32_t(p * kIdRing) + 8u * i;
            if (t >= uint32_t(kIdRing) && !wait_for(bar_id_free + bars, t / kIdRing - 1u, kStatusWaitRaw, 4, int(t))) break;
            IdSlot& is = misc->id_ring[p][i];
            const uint32_t valid = __ballot_sync(0xFFFFFFFFu, (id & kIdValid) != 0u);
            const uint32_t second = __ballot_sync(0xFFFFFFFFu, (id & kIdSecond) != 0u);
            is.num[lane] = (id & kIdValid) ? int32_t(id & kIdNumber) : 0;
            if constexpr (is_ref_layout(SRC)) is.scales[lane] = scales;
            if (lane == 0) { is.valid = valid;  is.second = second;  is.meta = cur.meta; }
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(bar_id_full + bars);
            if (!(cur.meta & kMetaTile)) break;                          // that was the end mark
            if (!early_q && p == 0 && (c0.meta & kMetaFirst)) prefetch_q_l2<NCHUNK>(a, c0.n, c0.hg, rank, lane);
        }
        __syncwarp();
    } else if (warp >= kFetchWarp) {
        // ───────────── fetch warps ─────────────
        const int p = warp - kFetchWarp, block = rank ^ p;
#pragma unroll 1
        for (uint32_t t = 0;; ++t) {
            const uint32_t i = t % kIdRing, bars = 8u * uint32_t(p * kIdRing) + 8u * i;
            const uint32_t st = t % kStages, stage = raw_base + st * R::kBytes;
            if (!wait_for(bar_id_full + bars, t / kIdRing, kStatusWaitRaw, 4, int(t))) break;
            const IdSlot& is = misc->id_ring[p][i];
            const uint32_t meta = *reinterpret_cast<const volatile uint32_t*>(&is.meta);
            const uint32_t valid = *reinterpret_cast<const volatile uint32_t*>(&is.valid), second = *reinterpret_cast<const volatile uint32_t*>(&is.second);
            if (t >= uint32_t(kStages) && !wait_for(bar_raw_free + 8 * st, t / kStages - 1u, kStatusWaitRaw, 4, int(t))) break;
            if (lane == 0) {
                misc->mask[t % kTagRing][block] = valid;
                if (p == 0) misc->meta[t % kTagRing] = meta;
            }
            if (!(meta & kMetaTile)) {                                   // the end mark
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(bar_raw_full + 8 * st);
                break;
            }
            if constexpr (is_ref_layout(SRC)) {
                const uint2 sc = ptx::lds_v2(ptx::smem_u32(&is.scales[lane]));
                ptx::sts_v2(stage + R::kScaleOff + uint32_t(block * 32 + lane) * 8u, sc);
            }
            __syncwarp();
            fetch_raw<SRC>(a, is.num, valid, second, p, rank, stage, bar_raw_full + 8 * st, lane);
            if (lane == 0) ptx::mbar_arrive(bar_id_free + bars);
        }
        __syncwarp();
    } else {
        // ───────────── softmax + epilogue warps ─────────────
        // Thread tid owns head row tid % 64 of this block and, of its S row, the entries of block tid / 64; of its O row the value
        // columns [256 (tid / 64), +256).  The two threads of a row (same lane, warps w and w + 2) share one reference
        // maximum: they meet at a named barrier per tile, which tells whether any of its 64 threads wants to move it.
        const int r = tid & 63, colhalf = tid >> 6;
        const uint32_t lane_addr = uint32_t(warp * 32) << 16;
        const uint32_t pair_bar = 1u + uint32_t(warp & 1);
        bool ok = wait_tmem();
        if (!ok) wait_ran_out(a.status, kStatusWaitQ, 0, -1);
        // (where the wait ran out for one warp of a barrier only, the other would wait for it there, without a limit)
        ok = !ptx::bar_any(pair_bar, 64, !ok);
        // this thread's 64 bytes of a P row: 16-byte columns 4 colhalf .. +3 of row r; column c lives at (c ^ (r % 8)) << 4
        const uint32_t p_row = p_base + uint32_t(r) * 128u;
        const uint32_t p_sw = (uint32_t(4 * colhalf) ^ uint32_t(r & 7)) << 4;
        uint32_t gt = 0;
        Item cur = get_item(0);
#pragma unroll 1
        for (int k = 0; k < n_items && ok; ++k) {
            const int nb = cur.ntiles;
            const int n = cur.n, h0 = cur.hg * kHeadsPerCta + rank * kHeadsPerBlock, slot = cur.slot;
            const bool final_out = slot < 0;
            const bool write = h0 + r < a.H;
            // row of this block's head 0 in the partial areas
            const int64_t prow0 = final_out ? 0 : (sched ? int64_t(slot) * kHeadsPerCta + rank * kHeadsPerBlock : (int64_t(slot) * rows + n) * a.H + h0);
            __nv_bfloat16* const out_rows = final_out ? a.out + (int64_t(n) * a.H + h0) * 512 : reinterpret_cast<__nv_bfloat16*>(a.partial_o) + prow0 * 512;
            if (nb <= 0) {
                // Nothing to attend to: zero output, LSE = -inf.
#pragma unroll 1
                for (int i = tid; i < kHeadsPerBlock * 64; i += kNumSoftmaxWarps * 32)
                    if (h0 + (i >> 6) < a.H) *reinterpret_cast<uint4*>(out_rows + int64_t(i >> 6) * 512 + (i & 63) * 8) = make_uint4(0, 0, 0, 0);
                if (colhalf == 0 && write) {
                    if (!final_out) a.partial_lse[prow0 + r] = -CUDART_INF_F;
                    else if (a.lse != nullptr) a.lse[int64_t(n) * a.H + h0 + r] = -CUDART_INF_F;
                }
                if (k + 1 < n_items) cur = get_item(k + 1);
                continue;
            }
            float m_ref = -CUDART_INF_F;                   // reference maximum used in exp2 (log2 units)
            float l_sum = 0.f;                             // of this thread's entries
            bool left = false;
#pragma unroll 1
            for (int it = 0; it < nb; ++it) {
                const uint32_t g = gt + uint32_t(it);
                const uint32_t s_tmem = tmem + lane_addr + kTmemS + (g & 1u) * 32u;
                if (ok) ok = wait_for(bar_s_full + 8 * (g & 1u), g >> 1, kStatusWaitSFull, 0, int(g));
                ptx::tc_fence_after_sync();
                if (tid == 0) trace_mark(a, 0, 4 * int(g));
                const uint32_t vmask = *reinterpret_cast<volatile uint32_t*>(&misc->mask[g % kTagRing][colhalf]);
                uint32_t s0[32];
                ptx::tmem_ld32(s_tmem, s0);
                ptx::tmem_wait_ld();
                if (vmask != ~0u) {
                    // entries that do not take part (padding, the end of the list): -inf before the scale
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (!((vmask >> i) & 1u)) s0[i] = 0xFF800000u;
                }
                // maximum of the raw logits (the scale is positive), four chains
                float t4[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) t4[i] = fmaxf(__uint_as_float(s0[i]), __uint_as_float(s0[i + 4]));
#pragma unroll
                for (int i = 8; i < 32; i += 8)
#pragma unroll
                    for (int j = 0; j < 4; ++j) t4[j] = ptx::max3(t4[j], __uint_as_float(s0[i + 2 * j]), __uint_as_float(s0[i + 2 * j + 1]));
                // (of NaN logits only it is -inf: such a row moves no maximum and spoils itself alone, through its probabilities)
                const float tmax = ptx::max3(ptx::max3(t4[0], t4[1], t4[2]), t4[3], -CUDART_INF_F) * a.scale_log2;
                // Lazy reference maximum: move it only when the true maximum exceeds it by
                // more than the threshold (exp2 of the excess stays <= 2^threshold).  A warp whose wait ran out comes here too
                // and says so, so that both warps of the barrier leave the loop together.
                float alpha = 1.f;
                const bool moved = ptx::bar_any(pair_bar, 64, !ok || tmax > m_ref + kRescaleThreshold);
                if (moved) {
                    misc->exch[tid] = tmax;
                    // the failure travels with the barrier, apart from the data: no value of a logit can look like one
                    if (ptx::bar_any(pair_bar + 2u, 64, !ok)) { ok = false;  left = true;  break; }
                    const float rmax = fmaxf(tmax, misc->exch[tid ^ 64]);
                    if (rmax > m_ref + kRescaleThreshold) {       // also true for the first finite max; the same in both threads
                        alpha = (m_ref == -CUDART_INF_F) ? 0.f : ptx::ex2(m_ref - rmax);
                        m_ref = rmax;
                    }
                }
                const float neg_m = (m_ref == -CUDART_INF_F) ? 0.f : -m_ref;
                // p = 2^(s * scale - m): half a fused multiply-add and one exp2 per element; the packed pairs replace s
                const uint64_t scale2 = ptx::pack_f32x2(a.scale_log2, a.scale_log2), neg2 = ptx::pack_f32x2(neg_m, neg_m);
                uint64_t ps2[2] = {0ull, 0ull};
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float e0, e1;
                    ptx::unpack_f32x2(ptx::fma_f32x2(ptx::pack_f32x2(__uint_as_float(s0[2 * i]), __uint_as_float(s0[2 * i + 1])), scale2, neg2), e0, e1);
                    const float p0 = ptx::ex2(e0), p1 = ptx::ex2(e1);
                    ps2[i & 1] = ptx::add_f32x2(ps2[i & 1], ptx::pack_f32x2(p0, p1));
                    s0[i] = use_f16(SRC) ? ptx::pack_f16x2(p0, p1) : ptx::pack_bf16x2(p0, p1);
                }
                float ps_lo, ps_hi;
                ptx::unpack_f32x2(ptx::add_f32x2(ps2[0], ps2[1]), ps_lo, ps_hi);
                l_sum = l_sum * alpha + (ps_lo + ps_hi);
                // the P buffer has been read by the O MMAs of the tile two before
                if (g >= 2u && !(ok = wait_for(bar_o_full + 8 * (g & 1u), (g - 2u) >> 1, kStatusWaitOFull, 0, int(g)))) continue;      // leaves at the next barrier
                if (tid == 0) trace_mark(a, 0, 4 * int(g) + 1);
                if (it > 0 && moved && __any_sync(0xFFFFFFFFu, alpha != 1.f)) {
                    // O is written by the O MMAs of the previous tile: they must have finished
                    if (!(ok = wait_for(bar_o_full + 8 * ((g - 1u) & 1u), (g - 1u) >> 1, kStatusWaitOFull, 0, int(g)))) continue;
                    ptx::tc_fence_after_sync();
#pragma unroll 1
                    for (int c = 0; c < 8; ++c) {
                        uint32_t o[32];
                        ptx::tmem_ld32(tmem + lane_addr + kTmemO + c * 32, o);
                        ptx::tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        ptx::tmem_st32(tmem + lane_addr + kTmemO + c * 32, o);
                    }
                    ptx::tmem_wait_st();
                }
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    ptx::sts_v4(p_row + (g & 1u) * kQChunkBytes + (p_sw ^ (uint32_t(c) << 4)), make_uint4(s0[4 * c], s0[4 * c + 1], s0[4 * c + 2], s0[4 * c + 3]));
                ptx::fence_proxy_async_smem();
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) arrive_even(bar_p_full + 8 * (g & 1u));
                if (tid == 0) trace_mark(a, 0, 4 * int(g) + 2);
            }
            if (left) break;
            // ── epilogue ──
            gt += uint32_t(nb);
            if (k + 1 < n_items) cur = get_item(k + 1);      // the next item's record arrives while this one is written out
            if (ok) ok = wait_for(bar_o_full + 8 * ((gt - 1u) & 1u), (gt - 1u) >> 1, kStatusWaitOFull, 0, int(gt));
            if (ptx::bar_any(pair_bar, 64, !ok)) { ok = false;  break; }
            misc->exch[tid] = l_sum;
            ptx::bar_sync(pair_bar + 2u, 64);
            l_sum += misc->exch[tid ^ 64];
            ptx::tc_fence_after_sync();
            if (tid == 0) trace_mark(a, 0, 4 * int(gt - 1u) + 3);
            // The merge may be made resident once every block of this grid is here (or gone): by then no block of this grid is waiting for
            // an SM any more.  (Without a merge the successor may be another decode; its blocks, let in this early, cost 2 us of 63.)
            if (tid == 0 && k == n_items - 1 && (sched || a.num_splits > 1)) ptx::pdl_trigger();
            float denom = l_sum;
            if (final_out && a.attn_sink != nullptr && write) {
                const float s2 = ptx::ld(a.attn_sink + h0 + r) * 1.4426950408889634f;
                denom = (l_sum != 0.f) ? l_sum + ptx::ex2(s2 - m_ref) : 1.f;   // empty row: O is 0 anyway
            }
            const float inv = (l_sum != 0.f) ? 1.f / denom : 0.f;
            // O leaves through shared memory: each thread owns half a row in tensor memory, but rows are 1 KB apart in global
            // memory, so 64 columns at a time are laid down in this warp's own 64 bytes per row of each P buffer (swizzled like
            // P; the MMAs that read P have completed, and the next P there is written by this warp) and written
            // out 4 x 128 contiguous bytes per warp instruction.  Split partials are BF16 as well: the merge reads them
            // back at once, and at eight splits their traffic would otherwise exceed the KV bytes.
            const int row0 = (warp & 1) * 32;
            uint8_t* gbase = reinterpret_cast<uint8_t*>(out_rows + int64_t(row0) * 512 + colhalf * 256);
#pragma unroll 1
            for (int pass = 0; pass < 4; ++pass) {
#pragma unroll
                for (int hc = 0; hc < 2; ++hc) {
                    uint32_t o[32];
                    ptx::tmem_ld32(tmem + lane_addr + kTmemO + pass * 64 + hc * 32, o);
                    ptx::tmem_wait_ld();
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        uint4 w;
                        w.x = ptx::pack_bf16x2(__uint_as_float(o[8 * v + 0]) * inv, __uint_as_float(o[8 * v + 1]) * inv);
                        w.y = ptx::pack_bf16x2(__uint_as_float(o[8 * v + 2]) * inv, __uint_as_float(o[8 * v + 3]) * inv);
                        w.z = ptx::pack_bf16x2(__uint_as_float(o[8 * v + 4]) * inv, __uint_as_float(o[8 * v + 5]) * inv);
                        w.w = ptx::pack_bf16x2(__uint_as_float(o[8 * v + 6]) * inv, __uint_as_float(o[8 * v + 7]) * inv);
                        ptx::sts_v4(p_row + uint32_t(hc) * kQChunkBytes + (p_sw ^ (uint32_t(v) << 4)), w);
                    }
                }
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const uint32_t rl = uint32_t(q * 4 + (lane >> 3)), vc = uint32_t(lane & 7);
                    const uint32_t at = p_base + (vc >> 2) * kQChunkBytes + uint32_t(row0 + rl) * 128u + (((4u * colhalf + (vc & 3u)) ^ (rl & 7u)) << 4);
                    if (h0 + row0 + int(rl) < a.H)
                        *reinterpret_cast<uint4*>(gbase + int64_t(rl) * 1024 + pass * 128 + vc * 16u) = ptx::lds_v4(at);
                }
                __syncwarp();
            }
            if (write && colhalf == 0) {
                const float lse2 = (l_sum != 0.f) ? m_ref + log2f(l_sum) : -CUDART_INF_F;
                if (!final_out) a.partial_lse[prow0 + r] = lse2;
                else if (a.lse != nullptr) a.lse[int64_t(n) * a.H + h0 + r] = (l_sum != 0.f) ? lse2 * 0.6931471805599453f : -CUDART_INF_F;
            }
        }
    }

    // ── common exit: every thread of both blocks gets here, with or without an error: no MMA, commit or remote arrival of the
    // pair is then on its way to a block that has left ──
    __syncwarp();
    ptx::tc_fence_before_sync();
    ptx::cluster_sync();
    if (warp == kSWarp) {
        ptx::tc_fence_after_sync();
        if (ptx::lds_u32(failed_flag())) hold_block();
        ptx::tmem2_dealloc(misc->tmem_base, kTmemCols);
    }
}

}  // namespace dsv4
