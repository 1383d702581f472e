// warp_scan.cuh -- the one-query fused scan with one warp per row tile
// (device side; included by kernels.cu inside its anonymous namespace after
// pipe_scan.cuh, whose descriptors and helpers it shares).
//
// Replaces, for one query: ChunkDecompressor::step (core/comp.cuh:171-195)
// feeding pipeline_q1_lineorder (usecases/ssb/queries/01.cuh:27-54),
// pipeline_q2 (02.cuh:103), pipeline_q3 (03.cuh:119-170) or pipeline_q4
// (04.cuh:100), with the chunk pruning of MetaChecker
// (core/metadata.cuh:638-658) and the per-chunk worker loop of
// usecases/ssb/queries/01.hpp:350-424 folded into the same launch.
//
// Every warp is an independent worker: after two block-wide barriers at the
// start (chunk keep bits of the launch and their prefix counts, computed by
// each CTA) no warp waits for another; grouped plans have one more at the end,
// before the CTA's group table is flushed.  The 1024-row tiles of the surviving
// chunks form a dense rank space; warp w of the grid takes tiles w, w + W,
// w + 2W, ... (W warps), and the tiles of the last, incomplete round are cut
// into 256- or 512-row parts when there are warps to spare (so a pruned scan
// of a few hundred tiles uses the whole chip, and a long one ends level).
// Tiles are decided eight at a time (four for plans of more than 4 columns,
// steps or predicates):
//   * one decision round: lane (q << cl) + c reads column c's directory entry
//     and side-index entries for tile q (a cascaded page's header and up to 8
//     runs too) and writes to the warp's records in shared memory how the
//     column is read -- direct (raw rows or a 16-byte aligned LZ4 literal run:
//     the evaluator loads the rows from HBM itself), from the page's own bytes
//     (bit-packed values, two runs), constant (one value on the
//     tile), or decoded by the warp into its buffer (LZ4 ranges with matches:
//     groups of lanes per segment; other cascaded pages: run windows of 32
//     runs, one per lane).  The next round's directory lines are prefetched,
//     and the round's steps over constant columns decided, all in one chain of
//     loads;
//   * per tile: the decodes, then the plan's other steps over row groups of
//     128 rows (4 consecutive rows per lane, one 16-byte load per column).
//     Plans of the SSB shapes run a compile-time evaluator selected by their
//     signature (all values of its row groups loaded before any is used);
//     other plans read their steps at run time: with a group key in the same
//     evaluator, without one step by step over the tile (ws_eval_steps).
// Scalar sums stay in registers; grouped rows are collected per warp and
// added, 32 at a time, to the CTA's group table in shared memory (keys that
// find no slot go to the global table), flushed when the CTA is done.
// Join-table reads carry an L2 evict-last policy, so that the tables stay in
// L2 while the fact columns pass through it.
//
// What bounds it, and why it is built this way (B200, 148 SMs): a Q1 scan of
// 60M rows has to read 747 MB, 114 us at the measured copy rate, and a loop
// that only reads three columns in this tile pattern reaches 6.4 TB/s with 24
// warps per SM and two row groups of loads in flight per warp.  Staging tiles
// in shared memory held the kernel at 12 warps, waiting for its own copies:
// 180 us; rows read in place, decisions in shared memory instead of registers,
// row masks as predicates (1,450 -> 1,115 instructions per tile): 132 us.  The
// star joins are bound by random table reads; there one row group per warp,
// chains walked for all of a lane's rows together and dense group-table adds
// took the 200M-row join from 6.3 to 2.2 ms, the four-join profit query over
// 24M rows from 1.65 ms to 0.56 ms.  All-cascaded Q1 over 16M rows, values
// unpacked in registers instead of through a decode buffer: 626 -> 222 us.

constexpr uint32_t kWsLog2 = 10;
constexpr uint32_t kWsTile = 1u << kWsLog2;    // rows of one warp tile
constexpr uint32_t kWsNT = 128;                // threads per CTA (4 independent warps)
constexpr uint32_t kWsWarps = kWsNT / 32;
constexpr uint32_t kWsBatch = 128;             // rows of one row group (4 per lane)
constexpr uint32_t kWsGroups = kWsTile / kWsBatch;  // row groups of a tile
constexpr uint32_t kWsEvalGroups = 2;               // row groups an evaluator runs at once at most
constexpr uint32_t kWsPartRows = kWsBatch * kWsEvalGroups;  // smallest part of a tile a warp takes
constexpr uint32_t kWsMaxParts = kWsTile / kWsPartRows;
static_assert(kWsGroups % kWsEvalGroups == 0, "the evaluator's row-group batches cover the tile");
constexpr uint32_t kWsMaxCols = kPipeMaxCols;
constexpr uint32_t kWsGroupLog2 = 9;           // the CTA's group table: 512 slots
constexpr uint32_t kWsGroupSlots = 1u << kWsGroupLog2;
constexpr uint32_t kWsNone = 0xFFFFFFFFu;
constexpr uint32_t kWsMaxDynSmem = 220u << 10;  // dynamic shared memory of one CTA at most
constexpr uint32_t kWsMaxChunkWords = 1024;     // chunk keep bits of one launch: 32768 chunks
// per-warp words before the decode buffers: 32 column records of 8 words, 8
// tile records of 8 words, the dense join tables' {base, span} headers per
// step (16), the constant steps' group-key digits (32), the rows scanned (2,
// and 2 of padding)
constexpr uint32_t kWsHead = 32 * 8 + 8 * 8 + 2 * GX_MAX_STEPS + 32 + 4;
// LZ4 columns decoded with one lane per segment: segments of 32 to 128 rows,
// four words of padding after each; the staged compressed bytes of a tile
// (less than 7/8 of its rows' bytes, and the ends of the aligned copy)
constexpr uint32_t kWsLaneShift0 = 5, kWsLaneShift1 = 7;
constexpr uint32_t kWsStageWords = kWsTile * 7 / 8 + 16;
static_assert(4 * kWsStageWords >= 4 * kWsTile * 7 / 8 + 38 && kWsStageWords % 4 == 0, "a staged range fits");
constexpr uint32_t kWsQueueWords = (kWsBatch + 32) * 3;  // grouped plans: the warp's WsQueue, before its decode buffers
static_assert(kWsHead % 4 == 0, "decode buffers start 16-byte aligned");
static_assert(kWsTile == kCascTileRows, "simple cascaded pages are simple for the scan's tiles");
static_assert(kWsTile <= kCascPageRows && kCascPageRows % kWsTile == 0, "a warp tile lies in one cascaded page");

struct WsParams {
    ShQuery q;                      // steps index into cols
    gx_dcol cols[kWsMaxCols];
    uint32_t n_cols;
    uint32_t blocks_per_chunk, rows_per_chunk, rows_per_block, tiles_per_block;
    // division by the tiles per chunk and per block, for numerators below 2^31
    uint32_t pc_mul, pc_shift, tpb_mul, tpb_shift;
    uint32_t col_log2;              // decision rounds: 4 lanes per tile (at most 4 columns, steps, predicates) or 8
    uint32_t parts;                 // 1: tiles of the last round may be cut (no column needs an LZ4 decode)
    uint64_t n_rows;                // rows of the table
    uint32_t chunk_lo, chunk_hi;    // chunks [chunk_lo, chunk_hi) are scanned
    uint32_t buf_of[kWsMaxCols];    // decode buffer of column c (cascaded / LZ4 with matches): word in the warp's
                                    // areas, or kWsNone
    uint32_t lane_cols;             // LZ4 columns of short sequences (a lane per segment)
    uint32_t stage_of, n_stages;    // staging of their compressed ranges: first word, buffers of kWsStageWords
    uint32_t warp_words;            // shared memory words per warp
    uint32_t chunk_words;           // words of the chunk keep bitmap (and of its prefix counts)
    uint32_t grouped_tab;           // 1: the warp has a group table
    unsigned long long* rows_scanned;
};

// Column read modes of one tile.
// kWmDirect: the tile's rows lie in memory as they are (raw, or inside one
// 16-byte aligned LZ4 literal run) and the evaluator loads them itself.
// Cascaded pages that the evaluator reads from their own bytes, without a
// decode: kWmPack, bit-packed values without RLE or DELTA (four values of a
// lane from up to five words); kWmRuns2, a tile of a few-run page covered by
// two runs (value cval on tile rows [0, aux0), value aux1 from there).
// kWmRows: in shared memory, after the warp's decode.
enum : uint32_t {
    kWmDirect = 0, kWmConst = 1, kWmLz4 = 2, kWmCasc = 3, kWmBad = 4, kWmRuns2 = 5, kWmRows = 6, kWmPack = 7
};

// Inclusive warp scan (wrapping uint32 sum).
__device__ __forceinline__ uint32_t ws_scan(uint32_t x, uint32_t lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
        if (lane >= (uint32_t)d) x += y;
    }
    return x;
}

// Rows [h0, h0 + n) of a cascaded page decoded by one warp into out[0..n),
// or, when one run covers them, *cv = that value and 1 is returned (out is
// not written).  RLE pages are walked in windows of 32 runs (run j of the
// window in lane j: its value, start and end from warp scans that carry over
// from the previous windows); the rows of a window are written 32 at a time
// by the runs overlapping them.  Pages without RLE unpack their values
// directly; with DELTA the prefix up to row h0 is a warp reduction and the
// tile's rows a running warp scan.  Returns 0, 1 (constant) or kErrCorrupt
// (uniform over the warp).
__device__ __noinline__ int ws_casc_rows(const uint8_t* __restrict__ pg, uint32_t pg_bytes, uint32_t page_rows,
                                         uint32_t h0, uint32_t n, int32_t* out, int32_t* cv, uint32_t lane) {
    const casc_hdr h = casc_load_header(pg);
    if (!casc_header_ok(h, pg_bytes, page_rows) || h0 + n > page_rows) return kErrCorrupt;
    const bool rle = (h.flags & CASC_RLE) != 0, delta = (h.flags & CASC_DELTA) != 0;
    const uint32_t* vw = (const uint32_t*)(pg + h.vals_off);
    const uint32_t vb = h.val_bits, base = (uint32_t)h.val_base;
    if (!rle) {
        if (!delta) {
            for (uint32_t i = lane; i < n; i += 32) out[i] = (int32_t)(unpack_bits(vw, h0 + i, vb) + base);
            __syncwarp();
            return 0;
        }
        uint32_t pre = 0;  // entries 1 .. h0-1 (entry 0 is 0)
        for (uint32_t k = 1 + lane; k < h0; k += 32) pre += unpack_bits(vw, k, vb) + base;
        pre = __reduce_add_sync(0xFFFFFFFFu, pre);
        uint32_t run = (uint32_t)h.first + pre;
        for (uint32_t g = 0; g < n; g += 32) {
            const uint32_t i = h0 + g + lane;
            const uint32_t e = (i == 0 || g + lane >= n) ? 0u : unpack_bits(vw, i, vb) + base;
            const uint32_t x = ws_scan(e, lane);
            if (g + lane < n) out[g + lane] = (int32_t)(run + x);
            run += __shfl_sync(0xFFFFFFFFu, x, 31);
        }
        __syncwarp();
        return 0;
    }
    const uint32_t nr = h.n_runs;
    const uint32_t* lw = (const uint32_t*)(pg + h.lens_off);
    const uint32_t t0 = h0, t1 = h0 + n;
    uint32_t c_end = 0, c_val = 0;  // carried over the windows: rows and value deltas so far
    bool is_const = false;
    for (uint32_t w0 = 0; w0 < nr; w0 += 32) {
        const uint32_t j = w0 + lane;
        const bool in = j < nr;
        const uint32_t le = in ? unpack_bits(lw, j, h.len_bits) + h.len_base : 0u;
        const uint32_t ve = in ? ((delta && j == 0) ? 0u : unpack_bits(vw, j, vb) + base) : 0u;
        const uint32_t end = c_end + ws_scan(le, lane), start = end - le;
        const uint32_t val = delta ? (uint32_t)h.first + c_val + ws_scan(ve, lane) : ve;
        const uint32_t w_end = __shfl_sync(0xFFFFFFFFu, end, 31), w_start = c_end;
        c_end = w_end;
        if (delta) c_val += __reduce_add_sync(0xFFFFFFFFu, ve);
        // (every window is walked: the run lengths must add up to the page)
        if (is_const || w_end <= t0 || w_start >= t1) continue;
        // one run covering the whole tile: its value, nothing written
        const uint32_t cover = __ballot_sync(0xFFFFFFFFu, in && start <= t0 && end >= t1);
        if (cover) {
            *cv = (int32_t)__shfl_sync(0xFFFFFFFFu, val, __ffs(cover) - 1);
            is_const = true;
            continue;
        }
        const uint32_t r_lo = max(w_start, t0), r_hi = min(w_end, t1);
        for (uint32_t g = r_lo & ~31u; g < r_hi; g += 32) {
            const uint32_t r = g + lane;
            // runs of this window that overlap rows [g, g + 32)
            uint32_t m = __ballot_sync(0xFFFFFFFFu, in && le > 0 && start < g + 32 && end > g);
            int32_t v = 0;
            bool got = false;
            while (m) {
                const uint32_t k = __ffs(m) - 1;
                m &= m - 1;
                const uint32_t s = __shfl_sync(0xFFFFFFFFu, start, k), e = __shfl_sync(0xFFFFFFFFu, end, k);
                const uint32_t x = __shfl_sync(0xFFFFFFFFu, val, k);
                if (r >= s && r < e) {
                    v = (int32_t)x;
                    got = true;
                }
            }
            if (got && r >= r_lo && r < r_hi) out[r - t0] = v;
        }
    }
    if (c_end != page_rows) return kErrCorrupt;
    __syncwarp();
    return is_const ? 1 : 0;
}

// The warp's per-segment LZ4 decode of a tile: segments j0 .. j0+nseg-1 of
// the block that starts at address blk (blk_bytes compressed bytes; side
// index entries e) into out (segment t at out + t * seg_rows), groups of lanes
// per segment.  Returns 0 or kErrCorrupt (uniform).
__device__ __noinline__ int ws_lz4_rows(const uint8_t* blk, uint32_t blk_bytes, const uint32_t* e, uint32_t seg_shift,
                                        uint32_t rows, uint32_t r0, uint32_t n, uint32_t lo, uint32_t hi,
                                        uint32_t* out, bool steps, uint32_t lane) {
    const uint32_t seg_rows = 1u << seg_shift;
    const uint32_t j0 = r0 >> seg_shift, nseg = (n + seg_rows - 1) >> seg_shift;
    // payload addresses keep the payload offsets' alignment modulo 16
    const uintptr_t a_wb = ((uintptr_t)blk + lo) & ~(uintptr_t)15;
    const uint32_t* A = (const uint32_t*)a_wb;
    const uint32_t wbase = (uint32_t)(a_wb - (uintptr_t)blk);
    const uint32_t glog = seg_group_log2(nseg, 32);
    // the tile's compressed lines into L1 first, all in flight together
    for (uint32_t x = 128 * lane; x < hi - lo; x += 128 * 32) asm volatile("prefetch.global.L1 [%0];" ::"l"(A + x / 4));
    int err = 0;
    lz4_segs(steps, lane, 32, glog, j0, nseg, rows, seg_rows, A, wbase, lo, hi, blk_bytes, e + 2 * j0, out, 0, &err);
    __syncwarp();
    return __any_sync(0xFFFFFFFFu, err != 0) ? kErrCorrupt : 0;
}

// One row tile: block slot, first row in the block, rows, block rows, and
// the rows [a, b) of the tile that the warp evaluates (all of them, or the
// part of a tile cut for the last round).
struct __align__(16) WsTile {
    uint32_t slot, r0, n, rows, a, b;
    uint32_t steps;  // bit s: step s is over a constant column; kWsDecode, kWsDead, kWsMixed
    uint32_t pad;
};
constexpr uint32_t kWsDecode = 1u << 29;     // a column needs a decode, or is corrupt
constexpr uint32_t kWsDead = 1u << 30;       // a constant step drops every row
constexpr uint32_t kWsMixed = 1u << 31;      // a column is neither direct nor a loose step's that is not packed
constexpr uint32_t kWsHard = 1u << 28;       // ... nor decoded
static_assert(sizeof(WsTile) == 32, "tile records of 8 words");

// How one column of one tile is read.
struct __align__(16) WsCol {
    const uint8_t* src;   // direct, kWmRows: the rows; LZ4: the block; cascaded: the page; kWmPack: its values
    uint32_t mode;        // kWm*
    int32_t cval;         // kWmConst: the value; kWmRuns2: the first run's; kWmPack: the frame of reference
    uint32_t aux0, aux1;  // LZ4: [lo, hi) in the block; cascaded: page bytes, page rows; kWmRuns2: the first
                          // run's end, the second's value; kWmPack: bits per value; kWmRows: log2 of the rows
                          // between every four words of padding
    uint32_t bytes;       // LZ4: the block's compressed bytes; kWmPack: the tile's first row in the page
    uint32_t pad;
};
static_assert(sizeof(WsCol) == 32, "column records of 8 words");

// Four rows of a column read in place (16-byte aligned), without taking room
// in L1.  (volatile: the loads of a batch stay together at
// its start, also when a value is used only after the probes.)
__device__ __forceinline__ uint4 ws_ld_rows(const uint8_t* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

// The tile's LZ4 columns of short sequences (P.lane_cols; unless nearly all
// literals on this tile) decoded with one lane per segment: up to n_stages
// columns at a time, as many as have 32 segments on the tile together.  Their
// compressed ranges are staged, their rows land with four words between
// segments (cols[c].aux0 = log2 of the segment).  Returns the columns done;
// *err is set on a corrupt stream.
__device__ __noinline__ uint32_t ws_lz4_lanes(const WsParams& P, const gx_dcol* s_cols, const WsTile& T, WsCol* cols,
                                              uint32_t todo, uint32_t* areas, uint32_t lane, int* err) {
    uint32_t done = 0;
    // the columns that qualify: lane c decides column c
    bool q = false;
    if ((todo >> lane) & 1u) {
        q = (cols[lane].aux1 - cols[lane].aux0) * 8 < T.n * 4 * 7;
    }
    todo = __ballot_sync(0xFFFFFFFFu, q);
    while (todo) {
        // one pass: columns of one segment size
        const uint32_t shift = s_cols[__ffs(todo) - 1].seg_shift, nseg = (T.n + (1u << shift) - 1) >> shift;
        uint32_t pass = 0, cnt = 0, mine = kWsNone, my_stage = 0;
        for (uint32_t m = todo; m && cnt < P.n_stages && (cnt + 1) * nseg <= 32; m &= m - 1) {
            const uint32_t c = __ffs(m) - 1;
            if (s_cols[c].seg_shift != shift) continue;
            uint32_t* st = areas + P.stage_of + cnt * kWsStageWords;
            const uintptr_t a0 = ((uintptr_t)cols[c].src + cols[c].aux0) & ~(uintptr_t)15;
            const uintptr_t a1 = (uintptr_t)cols[c].src + cols[c].aux1;
            // (up to 23 bytes past the range: inside the payload's slack)
            for (uint32_t i = lane; i < (uint32_t)(a1 - a0 + 8 + 15) / 16; i += 32)
                ((uint4*)st)[i] = ws_ld_rows((const uint8_t*)a0 + 16 * i);
            if (lane / nseg == cnt) {
                mine = c;
                my_stage = smem_u32(st) + (uint32_t)((uintptr_t)cols[c].src + cols[c].aux0 - a0) - cols[c].aux0;
            }
            pass |= 1u << c;
            ++cnt;
        }
        const bool in = mine != kWsNone && lane < cnt * nseg;
        const uint32_t c = in ? mine : (uint32_t)__ffs(pass) - 1, t = in ? lane % nseg : 0u;
        const gx_dcol& col = s_cols[c];
        const uint32_t j = (T.r0 >> shift) + t, K = min(1u << shift, T.rows - (j << shift));
        const uint32_t* e = col.seg + (size_t)2 * col.S * T.slot + 2 * j;
        const uint32_t cp = __ldg(e), info = __ldg(e + 1), lo = cols[c].aux0, hi = cols[c].aux1;
        const bool range = cp >= lo && cp <= hi;
        __syncwarp();
        const bool ok = lz4_seg_lane(my_stage + (range ? cp : lo), my_stage + hi, my_stage + cols[c].bytes, info, K,
                                     smem_u32(areas + P.buf_of[c] + t * ((1u << shift) + 4)), in && range);
        if (__any_sync(0xFFFFFFFFu, in && !(ok && range))) *err = kErrCorrupt;
        __syncwarp();
        if (lane < 8 && ((pass >> lane) & 1u)) {
            cols[lane].mode = kWmRows;
            cols[lane].src = (const uint8_t*)(areas + P.buf_of[lane]);
            cols[lane].aux0 = shift;
        }
        __syncwarp();
        done |= pass;
        todo &= ~pass;
    }
    return done;
}

// The columns of a tile that need a decode (or are corrupt), by the whole warp:
// LZ4 columns of short sequences together, the others one at a time.  Returns
// 0 or the error.  Out of line: most tiles have none.
__device__ __noinline__ int ws_decode_tile(const WsParams& P, const gx_dcol* s_cols, const WsTile& T, WsCol* cols,
                                           uint32_t* areas, uint32_t lane) {
    const uint32_t ncols = P.n_cols;
    int terr = 0;
    const uint32_t lz = __ballot_sync(0xFFFFFFFFu, lane < ncols && cols[lane].mode == kWmLz4);
    if (lz & P.lane_cols) ws_lz4_lanes(P, s_cols, T, cols, lz & P.lane_cols, areas, lane, &terr);
    for (uint32_t c = 0; c < ncols && !terr; ++c) {
        const uint32_t m = cols[c].mode;
        if (m == kWmBad) return kErrCorrupt;
        if (m != kWmLz4 && m != kWmCasc) continue;
        uint32_t* buf = areas + P.buf_of[c];
        int32_t cv = 0;
        if (m == kWmCasc) {
            terr = ws_casc_rows(cols[c].src, cols[c].aux0, cols[c].aux1, T.r0 & (kCascPageRows - 1u), T.n,
                                (int32_t*)buf, &cv, lane);
            if (terr == 1) {  // one run covers the tile (a page of many runs): its value written out
                for (uint32_t i = lane; i < T.n; i += 32) buf[i] = (uint32_t)cv;
                terr = 0;
            }
        } else {
            const gx_dcol& col = s_cols[c];
            terr = ws_lz4_rows(cols[c].src, cols[c].bytes, col.seg + (size_t)2 * col.S * T.slot, col.seg_shift, T.rows,
                               T.r0, T.n, cols[c].aux0, cols[c].aux1, buf, col.lz4_steps != 0, lane);
        }
        __syncwarp();
        if (lane == 0) {
            cols[c].mode = kWmRows;
            cols[c].src = (const uint8_t*)buf;
            cols[c].aux0 = 31;  // no padding
        }
        __syncwarp();
    }
    return terr;
}

// Add of (key, val) to the CTA's group table in shared memory: sets of four
// slots, the key's set and the next one; a key that finds no slot there goes
// to the global table.  The sums are kept as 32-bit halves (a shared 64-bit
// add is a compare-and-swap loop): the low half's old value tells the carry.
__device__ __forceinline__ void ws_group_add(uint32_t gk, int64_t val, uint32_t* tkey, uint32_t* tlo, uint32_t* thi,
                                             int64_t* keys, int64_t* sums, uint32_t log2cap) {
    if (gk != kEmptyGKey) {
        const uint32_t s0 = hash_key32((int32_t)gk, kWsGroupLog2) & ~3u;
#pragma unroll 1
        for (uint32_t i = 0; i < 2; ++i) {
            const uint32_t b = (s0 + 4 * i) & (kWsGroupSlots - 1);
            uint32_t x[4];
            asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3])
                         : "r"(smem_u32(tkey + b))
                         : "memory");
            uint32_t slot = kWsNone;
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
                if (x[j] == gk) slot = b + j;
            if (slot == kWsNone) {
                // not there yet: the first free slot of the set (a slot another
                // thread takes meanwhile is passed over unless it took it for gk)
#pragma unroll 1
                for (uint32_t j = 0; j < 4 && slot == kWsNone; ++j) {
                    if (x[j] != kEmptyGKey) continue;
                    const uint32_t old = atomicCAS(&tkey[b + j], kEmptyGKey, gk);
                    if (old == kEmptyGKey || old == gk) slot = b + j;
                }
            }
            if (slot != kWsNone) {
                const uint32_t lo = (uint32_t)(uint64_t)val;
                const uint32_t old = atomicAdd(&tlo[slot], lo);
                const uint32_t hi = (uint32_t)((uint64_t)val >> 32) + (old + lo < old ? 1u : 0u);
                if (hi) atomicAdd(&thi[slot], hi);
                return;
            }
        }
    }
    if (!group_add_global(keys, sums, log2cap, (int64_t)gk, val)) raise_error(kErrCapacity);
}

// The grouped rows of a warp on their way to the group table: few rows of a
// row group survive a star join's probes, so they are collected in shared
// memory until 32 of them fill the warp's lanes (room for the rows of a batch and a
// rest of 31).
constexpr uint32_t kWsQueue = kWsBatch + 32;
struct WsQueue {
    int64_t val[kWsQueue];
    uint32_t key[kWsQueue];
};

// One row per lane (lanes with `on`).
__device__ __noinline__ void ws_group_add_lanes(bool on, uint32_t gk, int64_t val, uint32_t* tkey, int64_t* keys,
                                                int64_t* sums, uint32_t log2cap) {
    if (on) ws_group_add(gk, val, tkey, tkey + kWsGroupSlots, tkey + 2 * kWsGroupSlots, keys, sums, log2cap);
    __syncwarp();
}

// The queue's newest n rows (at most 32, qn of them after) into the table.
__device__ __noinline__ void ws_queue_flush(const WsQueue* wq, uint32_t qn, uint32_t n, uint32_t* tkey, int64_t* keys,
                                            int64_t* sums, uint32_t log2cap, uint32_t lane) {
    __syncwarp();
    if (lane < n)
        ws_group_add(wq->key[qn + lane], wq->val[qn + lane], tkey, tkey + kWsGroupSlots, tkey + 2 * kWsGroupSlots,
                     keys, sums, log2cap);
    __syncwarp();
}

// Position of the k-th set bit of m (k < popc(m)).
__device__ __forceinline__ uint32_t ws_select(uint32_t m, uint32_t k) {
    uint32_t pos = 0;
#pragma unroll
    for (uint32_t width = 16; width >= 1; width >>= 1) {
        const uint32_t low = __popc(m & ((1u << width) - 1u));
        if (k >= low) {
            k -= low;
            m >>= width;
            pos += width;
        }
    }
    return pos;
}

// n / d for n < 2^31, d's multiplier and shift computed by the host.
__device__ __forceinline__ uint32_t ws_div(uint32_t n, uint32_t mul, uint32_t shift) {
    return (uint32_t)(((uint64_t)n * mul) >> shift);
}

// The launch's work, the same for every warp: `first` is the first surviving
// chunk when they are neighbours (a range predicate on a sorted column, no
// pruning), else kWsNone and a chunk is found by its rank in the keep bits.
// t_end tiles go to W warps: `full` rounds of W whole tiles, then the tiles
// left over, cut into 1 << parts_log2 parts, one per warp.
struct WsWork {
    uint32_t first, t_end, W, full, rounds, parts_log2;
};

// Tile number t of the surviving chunks (chunk-major) -> its tile, whole;
// false when t is past the end or the chunk has no such rows.
__device__ __forceinline__ bool ws_locate(const WsParams& P, const uint32_t* s_kbits, const uint32_t* s_kpre,
                                          const WsWork& R, uint32_t t, WsTile& T) {
    if (t >= R.t_end) return false;
    const uint32_t tpb = P.tiles_per_block, bpc = P.blocks_per_chunk;
    const uint32_t k = ws_div(t, P.pc_mul, P.pc_shift), loc = t - k * (bpc * tpb);
    uint32_t chunk = R.first + k;
    if (R.first == kWsNone) {
        uint32_t lo = 0, hi = P.chunk_words - 1;  // the bitmap word holding the k-th surviving chunk
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if (s_kpre[mid] <= k) lo = mid; else hi = mid - 1;
        }
        chunk = P.chunk_lo + lo * 32 + ws_select(s_kbits[lo], k - s_kpre[lo]);
    }
    const uint32_t jb = ws_div(loc, P.tpb_mul, P.tpb_shift), tile = loc - jb * tpb;
    const uint64_t c_rows = min((uint64_t)P.rows_per_chunk, P.n_rows - (uint64_t)chunk * P.rows_per_chunk);
    const uint64_t jrow = (uint64_t)jb * P.rows_per_block;
    T.rows = jrow < c_rows ? (uint32_t)min((uint64_t)P.rows_per_block, c_rows - jrow) : 0u;
    T.r0 = tile * kWsTile;
    T.slot = chunk * bpc + jb;
    if (T.r0 >= T.rows) return false;
    T.n = min(kWsTile, T.rows - T.r0);
    T.a = 0;
    T.b = T.n;
    return true;
}

// Warp w's piece of round r.
__device__ __forceinline__ bool ws_piece(const WsParams& P, const uint32_t* s_kbits, const uint32_t* s_kpre,
                                         const WsWork& R, uint32_t w, uint32_t r, WsTile& T) {
    if (r < R.full) return ws_locate(P, s_kbits, s_kpre, R, r * R.W + w, T);
    if (r > R.full || !ws_locate(P, s_kbits, s_kpre, R, r * R.W + (w >> R.parts_log2), T)) return false;
    const uint32_t part = kWsTile >> R.parts_log2, p0 = (w & ((1u << R.parts_log2) - 1u)) * part;
    T.a = p0;
    T.b = min(T.n, p0 + part);
    return T.a < T.b;
}

// Column c's read decision for tile T (directory entry, side-index
// entries, a cascaded page's header: a single-run page needs no decode).
__device__ __forceinline__ WsCol ws_column(const WsParams& P, const gx_dcol& col, uint32_t c, const WsTile& T) {
    WsCol C;
    C.mode = kWmBad;
    C.src = nullptr;
    C.aux0 = C.aux1 = C.bytes = 0;
    C.cval = 0;
    const uint32_t slot = T.slot, r0 = T.r0, n = T.n, rows = T.rows;
    const uint4 dw = __ldg((const uint4*)(col.blocks + slot));
    const uint64_t d_off = ((uint64_t)dw.y << 32) | dw.x;
    const uint32_t d_bytes = dw.z, d_rows = dw.w;
    const bool dir_ok =
        d_rows == rows && d_off <= col.payload_bytes && (uint64_t)d_bytes + 32 <= col.payload_bytes - d_off;
    const uint8_t* blk = col.payload + d_off;
    if (col.codec == GX_CODEC_NONE) {
        if (dir_ok && d_bytes == rows * 4 && (d_off & 15u) == 0) {
            C.mode = kWmDirect;
            C.src = blk + 4ull * r0;
            C.aux0 = 31;
        }
    } else if (col.codec == GX_CODEC_LZ4) {
        const uint32_t sr = 1u << col.seg_shift;
        const uint32_t j0 = r0 >> col.seg_shift, nseg = (n + sr - 1) >> col.seg_shift;
        if ((r0 & (sr - 1u)) == 0 && j0 + nseg <= col.S) {
            const uint32_t* e = col.seg + (size_t)2 * col.S * slot;
            const uint32_t e0 = __ldg(e + 2 * j0), e1 = __ldg(e + 2 * j0 + 1);
            const uint32_t e2 = j0 + nseg < col.S ? __ldg(e + 2 * (j0 + nseg)) : 0u;
            const uint32_t hi = j0 + nseg < col.S ? e2 : d_bytes;
            if (dir_ok && e0 <= hi && hi <= d_bytes) {
                const bool lit = (e1 & 16u) && (e1 >> 5) >= 4 * n && hi - e0 == 4 * n;
                if (lit && ((d_off + e0) & 15u) == 0) {
                    C.mode = kWmDirect;
                    C.src = blk + e0;
                    C.aux0 = 31;
                } else if (P.buf_of[c] != kWsNone) {
                    C.mode = kWmLz4;
                    C.src = blk;
                    C.aux0 = e0;
                    C.aux1 = hi;
                    C.bytes = d_bytes;
                }
            }
        }
    } else if (col.codec == GX_CODEC_CASCADED) {
        const uint32_t page = r0 >> kCascPageLog2;
        if (page < col.S) {
            const uint32_t* e = col.seg + (size_t)2 * col.S * slot + 2 * page;
            const uint32_t po = __ldg(e), pb = __ldg(e + 1);
            if (dir_ok && (d_off & 15u) == 0 && (po & 15u) == 0 && (uint64_t)po + pb <= d_bytes && pb >= 32) {
                const uint8_t* pg = blk + po;
                if (P.buf_of[c] != kWsNone) C.mode = kWmCasc;
                C.src = pg;
                C.aux0 = pb;
                C.aux1 = min(kCascPageRows, rows - page * kCascPageRows);
                // pages that hold one value need no decode: zero-width values
                // without RLE (with DELTA: zero steps), or one run of the whole page
                const casc_hdr h = casc_load_header(pg);
                const bool rle = (h.flags & CASC_RLE) != 0, delta = (h.flags & CASC_DELTA) != 0;
                if (casc_header_ok(h, pb, C.aux1)) {
                    if (!rle && h.val_bits == 0 && (!delta || h.val_base == 0)) {
                        C.mode = kWmConst;
                        C.cval = delta ? h.first : h.val_base;
                    } else if (!rle && !delta) {
                        C.mode = kWmPack;
                        C.src = pg + h.vals_off;
                        C.cval = h.val_base;
                        C.aux0 = h.val_bits;
                        C.bytes = r0 & (kCascPageRows - 1u);
                    } else if (rle && h.n_runs <= kCascFewRuns) {
                        // a few runs (sorted columns): the run holding the tile's first
                        // row, and whether it also holds the last
                        const uint32_t* vw = (const uint32_t*)(pg + h.vals_off);
                        const uint32_t* lw = (const uint32_t*)(pg + h.lens_off);
                        const uint32_t h0 = r0 & (kCascPageRows - 1u), h1 = h0 + n;
                        uint32_t end = 0, val = 0;
                        for (uint32_t k = 0; k < h.n_runs; ++k) {
                            const uint32_t start = end;
                            end += unpack_bits(lw, k, h.len_bits) + h.len_base;
                            const uint32_t e =
                                (delta && k == 0) ? 0u : unpack_bits(vw, k, h.val_bits) + (uint32_t)h.val_base;
                            val = delta ? val + e : e;
                            if (start <= h0 && h0 < end) {
                                const uint32_t v0 = delta ? val + (uint32_t)h.first : val;
                                if (h1 <= end) {
                                    C.mode = kWmConst;
                                    C.cval = (int32_t)v0;
                                } else if (k + 1 < h.n_runs) {
                                    // the next run: when it covers the rest of the tile,
                                    // the tile is two runs
                                    const uint32_t end2 = end + unpack_bits(lw, k + 1, h.len_bits) + h.len_base;
                                    const uint32_t e2 = unpack_bits(vw, k + 1, h.val_bits) + (uint32_t)h.val_base;
                                    const uint32_t v1 = delta ? v0 + e2 : e2;
                                    if (h1 <= end2) {
                                        C.mode = kWmRuns2;
                                        C.cval = (int32_t)v0;
                                        C.aux0 = end - h0;
                                        C.aux1 = v1;
                                    }
                                }
                                break;
                            }
                        }
                    }
                }
            }
        }
    }
    return C;
}

// Decisions for warp w's pieces of the 32 >> cl rounds from r0 on at once (cl:
// WsParams::col_log2): lane (q << cl) + c decides column c of round r0 + q
// (and checks prune predicate c's zone map), so that eight tiles of a narrow
// plan or four of a wide one cost one chain of dependent loads, and the
// directory and side-index lines of the rounds after them are prefetched into
// L2.  The records go to tiles[q] and cols[(q << cl) + c]; returns the mask of
// the tiles to scan.  Out of line: its registers are not the evaluator's.
__device__ __noinline__ uint32_t ws_decide(const WsParams& P, const gx_dcol* s_cols, const uint32_t* s_kbits,
                                           const uint32_t* s_kpre, const WsWork& R, uint32_t w, uint32_t r0,
                                           uint32_t lane, WsTile* tiles, WsCol* cols) {
    const ShQuery& Q = P.q;
    const uint32_t cl = P.col_log2, q = lane >> cl, c = lane & ((1u << cl) - 1u), nq = 32u >> cl;
    WsTile T;
    const bool ok = ws_piece(P, s_kbits, s_kpre, R, w, r0 + q, T);
    bool zfail = false;
    if (ok && c < Q.n_prune) {
        const PrunePred& pr = Q.prune[c];
        if (pr.bmins) zfail = !(pr.lo <= __ldg(pr.bmaxs + T.slot) && pr.hi >= __ldg(pr.bmins + T.slot));
    }
    if (ok && c < P.n_cols) {
        const WsCol C = ws_column(P, s_cols[c], c, T);
        cols[lane] = C;
        if (C.mode == kWmPack) {  // the tile's packed values to L2 (inside the payload's slack)
            const uintptr_t p0 = ((uintptr_t)C.src + ((uint64_t)(C.bytes + T.a) * C.aux0) / 8) & ~(uintptr_t)15;
            const uintptr_t p1 = ((uintptr_t)C.src + ((uint64_t)(C.bytes + T.b) * C.aux0) / 8 + 15) & ~(uintptr_t)15;
            if (p1 > p0)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p0), "r"((uint32_t)(p1 - p0))
                             : "memory");
        }
    }
    if (ok && c == 0) tiles[q] = T;
    const uint32_t oks = __ballot_sync(0xFFFFFFFFu, ok), fails = __ballot_sync(0xFFFFFFFFu, zfail);
    uint32_t vm = 0;
    for (uint32_t g = 0; g < nq; ++g)
        if (((oks >> (g << cl)) & 1u) && ((fails >> (g << cl)) & ((1u << (1u << cl)) - 1u)) == 0) vm |= 1u << g;
    if (c < P.n_cols && r0 + nq + q < R.rounds && ws_piece(P, s_kbits, s_kpre, R, w, r0 + nq + q, T)) {
        const gx_dcol& col = s_cols[c];
        asm volatile("prefetch.global.L2 [%0];" ::"l"(col.blocks + T.slot));
        if (col.codec != GX_CODEC_NONE)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(col.seg + (size_t)2 * col.S * T.slot +
                                                          2 * (T.r0 >> col.seg_shift)));
    }
    __syncwarp();
    return vm;
}

// One key in a join table: dense tables through their cached header.
__device__ __forceinline__ bool ws_probe1(const ShStep& st, uint64_t hdr, int32_t v, int32_t* p, uint64_t pol_keep) {
    if (st.ht_layout != GX_HT_DENSE) return ht_probe_any(st.ht, st.ht_log2, st.ht_layout, v, p);
    const uint32_t u = (uint32_t)v - (uint32_t)hdr;
    if (v == kEmptyKey || u >= (uint32_t)(hdr >> 32)) return false;
    const unsigned long long e = ws_ld_slot((const unsigned long long*)st.ht + 1 + u, pol_keep);
    if ((int32_t)(uint32_t)e != v) return false;
    *p = (int32_t)(uint32_t)(e >> 32);
    return true;
}

// Plans of no known signature (below) are evaluated at run time: their
// "signatures" have no step count, and bit 6 for those with a group key.
constexpr uint32_t kSigRt = 0, kSigRtGroup = 1u << 6;
template <uint32_t SIG>
constexpr bool kWsRunTime = (SIG & 7) == 0;

// Steps whose column need not be direct in the flat evaluator (constant, of
// two runs or decoded will do): probes and the first step, when they neither
// carry nor are the last.
__device__ constexpr bool ws_loose_step(uint32_t s, uint32_t n_steps, bool probe, bool carry) {
    return (probe || s == 0) && !carry && s + 1 < n_steps;
}

// The steps over columns that hold one value on their tile, decided once per
// tile and for all tiles of the round together (their probes are one chain of
// loads): lane (q << cl) + s decides step s of tile q, leaves its group-key
// digit in sdig[lane] and tiles[q].steps says which steps are constant and
// whether one of them drops every row.
template <uint32_t SIG>
__device__ __forceinline__ void ws_const_steps(const WsParams& P, uint32_t vm, WsTile* tiles, const WsCol* cols,
                                               const uint64_t* whdr, uint32_t* sdig, uint64_t pol_keep,
                                               uint32_t lane) {
    const ShQuery& Q = P.q;
    const uint32_t cl = P.col_log2, q = lane >> cl, s = lane & ((1u << cl) - 1u);
    bool isc = false, ok = true, bad = false, mixed = false, hard = false, dec = false, digits = false;
    if (((vm >> q) & 1u) && s < P.n_cols) {  // as a column
        const uint32_t m = cols[lane].mode;
        dec = m == kWmLz4 || m == kWmCasc || m == kWmBad;
    }
    if (((vm >> q) & 1u) && s < Q.n_steps) {
        const ShStep& st = Q.steps[s];
        const WsCol& c = cols[(q << cl) + st.col];
        isc = c.mode == kWmConst;
        mixed = c.mode != kWmDirect &&
                (c.mode == kWmPack || !ws_loose_step(s, Q.n_steps, (st.flags & GX_STEP_PROBE) != 0,
                                                     (st.flags & GX_STEP_CARRY) != 0));
        hard = mixed && c.mode != kWmLz4 && c.mode != kWmCasc;
        if (isc) {
            const int32_t v = c.cval;
            int32_t pp = v;
            if (st.flags & GX_STEP_FILTER) ok = v >= st.lo && v <= st.hi;
            if (ok && (st.flags & GX_STEP_PROBE)) ok = ws_probe1(st, whdr[s], v, &pp, pol_keep);
            if (ok && st.digit_card) {
                const uint32_t dgt = (uint32_t)(pp - st.digit_base);
                bad = dgt >= st.digit_card;
                sdig[lane] = dgt;
            }
        }
        digits = bad || (SIG == kSigRtGroup && !isc && st.digit_card);
    }
    const uint32_t m0 = (1u << (1u << cl)) - 1u, sh = q << cl;
    const uint32_t cst = (__ballot_sync(0xFFFFFFFFu, isc) >> sh) & m0;
    const uint32_t fails = (__ballot_sync(0xFFFFFFFFu, isc && !ok) >> sh) & m0;
    const uint32_t bads = (__ballot_sync(0xFFFFFFFFu, bad) >> sh) & m0;
    const uint32_t digs = (__ballot_sync(0xFFFFFFFFu, digits) >> sh) & m0;
    const uint32_t decs = (__ballot_sync(0xFFFFFFFFu, dec) >> sh) & m0;
    const uint32_t mixes = (__ballot_sync(0xFFFFFFFFu, mixed) >> sh) & m0;
    const uint32_t hards = (__ballot_sync(0xFFFFFFFFu, hard) >> sh) & m0;
    if (s == 0 && ((vm >> q) & 1u)) {
        uint32_t f = cst | (mixes ? kWsMixed : 0u) | (hards ? kWsHard : 0u) | (fails ? kWsDead : 0u);
        // a digit out of range is an error for rows alive at its step: its tile's
        // steps are taken row by row (a step over rows before it may have dropped
        // them) unless a constant step before it drops the tile.  Run-time plans
        // also look at the digits of rows before they let a constant step drop
        // them; the compile-time ones leave such a tile unread
        const uint32_t before = fails ? (1u << (__ffs(fails) - 1)) - 1u : m0;
        if (((fails ? digs : bads) & before) != 0) f = kWsMixed | kWsHard;
        f |= decs ? kWsDecode : 0u;
        tiles[q].steps = f;
    }
    __syncwarp();
}

// ---- plan signatures: compile-time evaluators for the known query shapes
// A signature packs the step count (bits 0-2), the aggregate (3-5), grouped
// (6) and per step s a kind nibble at bit 7 + 4 s: 1 FILTER, 2 PROBE,
// 4 CARRY, 8 group-key digit.
constexpr uint32_t kWkF = 1, kWkP = 2, kWkC = 4, kWkD = 8;
constexpr uint32_t ws_sig(uint32_t ns, uint32_t agg, bool grouped, uint32_t k0, uint32_t k1 = 0, uint32_t k2 = 0,
                          uint32_t k3 = 0, uint32_t k4 = 0, uint32_t k5 = 0) {
    return ns | (agg << 3) | ((grouped ? 1u : 0u) << 6) | (k0 << 7) | (k1 << 11) | (k2 << 15) | (k3 << 19) |
           (k4 << 23) | (k5 << 27);
}
// pipeline_q1_lineorder: date probe, discount filter carried, quantity filter, price x discount
constexpr uint32_t kSigQ1 = ws_sig(4, GX_AGG_SUM_PRODUCT, false, kWkP, kWkF | kWkC, kWkF, 0);
// pipeline_q3: customer / supplier / date probes with digits, revenue grouped
constexpr uint32_t kSigQ3 = ws_sig(4, GX_AGG_SUM, true, kWkP | kWkD, kWkP | kWkD, kWkP | kWkD, 0);
// pipeline_q2: part probe (brand digit), supplier probe, date probe (year digit), revenue grouped
constexpr uint32_t kSigQ2 = ws_sig(4, GX_AGG_SUM, true, kWkP | kWkD, kWkP, kWkP | kWkD, 0);
// a group-by of one column over a range of another (dates): value grouped by a digit
constexpr uint32_t kSigGroup = ws_sig(3, GX_AGG_SUM, true, kWkF, kWkD, 0);
// pipeline_q4: customer (nation digit), supplier, date (year digit), part probes, supplycost carried, profit grouped
constexpr uint32_t kSigQ4 = ws_sig(6, GX_AGG_SUM_DIFF, true, kWkP | kWkD, kWkP, kWkP | kWkD, kWkP, kWkC, 0);

// The steps of a signature that run step by step: up to the last probe, and
// the first one (often the sort key's filter, decided for the whole tile).
constexpr uint32_t ws_probes_end(uint32_t sig) {
    uint32_t e = 1;
    for (uint32_t s = 0; s < (sig & 7); ++s)
        if ((sig >> (7 + 4 * s)) & kWkP) e = s + 1;
    return e;
}
template <uint32_t SIG>
constexpr uint32_t kWsProbesEnd = ws_probes_end(SIG);

// Elements i .. i + 3 of a bit-packed stream of width w (1..32), plus base:
// the words that hold them are shifted to the first one's bit once (s below,
// per lane), after which element k starts at bit k * w in every lane.  Reads
// at most four words past the last element's.
__device__ __forceinline__ uint4 ws_unpack4(const uint32_t* words, uint32_t i, uint32_t w, uint32_t base) {
    const uint32_t bit = i * w, s = bit & 31u;
    const uint32_t* p = words + (bit >> 5);
    const uint32_t mask = 0xFFFFFFFFu >> (32 - w);
    const uint32_t p0 = __ldg(p), p1 = __ldg(p + 1);
    const uint32_t a0 = __funnelshift_r(p0, p1, s);
    if (w <= 8)
        return make_uint4((a0 & mask) + base, ((a0 >> w) & mask) + base, ((a0 >> (2 * w)) & mask) + base,
                          ((a0 >> (3 * w)) & mask) + base);
    const uint32_t p2 = __ldg(p + 2), p3 = w > 16 ? __ldg(p + 3) : 0u, p4 = w > 24 ? __ldg(p + 4) : 0u;
    const uint32_t a1 = __funnelshift_r(p1, p2, s), a2 = __funnelshift_r(p2, p3, s), a3 = __funnelshift_r(p3, p4, s);
    auto at = [&](uint32_t off) {
        const uint32_t k = off >> 5;
        const uint32_t lo = k == 0 ? a0 : k == 1 ? a1 : k == 2 ? a2 : a3;
        const uint32_t hi = k == 0 ? a1 : k == 1 ? a2 : a3;
        return (__funnelshift_r(lo, hi, off & 31u) & mask) + base;
    };
    return make_uint4((a0 & mask) + base, at(w), at(2 * w), at(3 * w));
}

template <uint32_t R>
__device__ __forceinline__ void ws_put(uint32_t (&w)[R], uint32_t h, const uint4& x) {
    w[4 * h] = x.x;
    w[4 * h + 1] = x.y;
    w[4 * h + 2] = x.z;
    w[4 * h + 3] = x.w;
}

// Tile rows row .. row + 3 of a column of two runs.
__device__ __forceinline__ uint4 ws_runs2(const WsCol& d, uint32_t row) {
    const uint32_t e = d.aux0, v0 = (uint32_t)d.cval, v1 = d.aux1;
    return make_uint4(row < e ? v0 : v1, row + 1 < e ? v0 : v1, row + 2 < e ? v0 : v1, row + 3 < e ? v0 : v1);
}

// Tile rows row .. row + 3 of a decoded column.
__device__ __forceinline__ uint4 ws_decoded(const WsCol& d, uint32_t row) {
    return *(const uint4*)(d.src + 4 * (row + ((row >> d.aux0) << 2)));
}

// Tile rows row .. row + 3 of a direct or decoded column (generic address).
__device__ __forceinline__ uint4 ws_ld_any(const WsCol& d, uint32_t row) {
    uint4 v;
    asm volatile("ld.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(d.src + 4 * (row + ((row >> d.aux0) << 2))));
    return v;
}

// Tile rows row .. row + 3 of a column, however it is read.
__device__ __forceinline__ uint4 ws_quad(const WsCol& d, uint32_t row) {
    const uint32_t mode = d.mode;
    if (mode == kWmDirect) return ws_ld_rows(d.src + 4 * row);
    if (mode == kWmPack) return ws_unpack4((const uint32_t*)d.src, d.bytes + row, d.aux0, (uint32_t)d.cval);
    const uint32_t v0 = (uint32_t)d.cval;
    if (mode == kWmConst) return make_uint4(v0, v0, v0, v0);
    if (mode == kWmRuns2) return ws_runs2(d, row);
    return ws_decoded(d, row);  // kWmRows
}

enum class WsForm { kAny, kFlat, kRows };

// Tile rows [a, b) evaluated through the plan's steps, H 128-row groups at a
// time (a is a multiple of kWsPartRows): the lane's rows of group j are
// 128 j + 4 lane + i (i < 4), row r = 4 h + i of the batch; bit r of m is its
// mask.  A compile-time signature loads all columns of the batch before any
// is used and unrolls its steps: up to the last probe step by step, the
// filters after it and the aggregate row by row, where a row's mask is a
// predicate.  Run-time plans with a group key load a column at its step.  kFlat:
// [a, b) is whole batches and every column is direct or a loose step's that is
// not packed (a sorted date), so that a batch's loads are unconditional and all
// in flight together; kRows: the same with decoded columns among them, every
// quad from a generic address (as kAny, where a quad's read mode is looked up
// first, four batches of a tile took 14,000 cycles, which a pruned scan of a few
// such tiles waits for).  Steps over constant columns were decided by
// ws_const_steps.
// Returns the scalar part; grouped sums go to the CTA's group table through
// the warp's queue.
template <uint32_t SIG, WsForm FORM>
__device__ __forceinline__ int64_t ws_eval(const ShQuery& Q, const WsCol* cols, uint32_t cst, const uint32_t* sdig,
                                           uint32_t a, uint32_t b, uint32_t* tkey, WsQueue* wq, uint32_t& qn,
                                           uint64_t pol_keep, const uint64_t* s_hdr,
                                           uint32_t lane) {
    constexpr bool RT = kWsRunTime<SIG>, FLAT = FORM != WsForm::kAny, ROWS = FORM == WsForm::kRows;
    constexpr bool GR = ((SIG >> 6) & 1) != 0;  // grouped: the queue holds one row group
    constexpr uint32_t H = GR ? 1 : kWsEvalGroups;
    constexpr uint32_t R = 4 * H;
    constexpr uint32_t NS = RT ? 1 : (SIG & 7);
    constexpr uint32_t PE = RT ? 0 : kWsProbesEnd<SIG>;  // steps [0, PE) run step by step
    const uint32_t ns = RT ? Q.n_steps : NS;
    const uint32_t agg = RT ? Q.agg : (SIG >> 3) & 7;
    int64_t acc = 0;
    const uint8_t* src[NS];  // FLAT: the lane's quad of each step's column
    uint32_t some = ~0u;     // signatures: 0 when a filter after the probes has an empty range
    if (!RT) {
#pragma unroll
        for (uint32_t s = 0; s < NS; ++s) {
            src[s] = FLAT && !ROWS ? cols[Q.steps[s].col].src + (a + 4 * lane) * 4 : nullptr;
            if (s + 1 > PE && ((SIG >> (7 + 4 * s)) & kWkF) && Q.steps[s].lo > Q.steps[s].hi) some = 0;
        }
    }
#pragma unroll 1
    for (uint32_t j0 = a; j0 < b; j0 += H * kWsBatch) {
        const uint32_t row = j0 + 4 * lane;
        uint32_t m = (1u << R) - 1u;
        if (!FLAT && j0 + H * kWsBatch > b) {
            m = 0;
#pragma unroll
            for (uint32_t r = 0; r < R; ++r)
                if (row + kWsBatch * (r / 4) + r % 4 < b) m |= 1u << r;
        }
        uint32_t w[NS][R];
        uint32_t g[R], carry[R];
#pragma unroll
        for (uint32_t r = 0; r < R; ++r) g[r] = carry[r] = 0;
        if (!RT) {
            // (values of rows that are not wanted are not used: any will do.  A quad with one
            // wanted row ends at most 12 bytes after its block, inside the payload)
#pragma unroll
            for (uint32_t s = 0; s < NS; ++s) {
                const uint32_t K = (SIG >> (7 + 4 * s)) & 15u;
                const bool loose = ws_loose_step(s, NS, (K & kWkP) != 0, (K & kWkC) != 0);
                const bool skip = loose && ((cst >> s) & 1u);
#pragma unroll
                for (uint32_t h = 0; h < H; ++h) {
                    uint4 x;
                    asm("" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w));
                    if (FLAT) {
                        const WsCol& d = cols[Q.steps[s].col];
                        if (loose && !skip && d.mode == kWmRuns2)
                            x = ws_runs2(d, row + kWsBatch * h);
                        else if (ROWS && !skip)
                            x = ws_ld_any(d, row + kWsBatch * h);
                        else if (loose && !skip && d.mode == kWmRows)
                            x = ws_decoded(d, row + kWsBatch * h);
                        else if (!skip)
                            x = ws_ld_rows(src[s] + kWsBatch * 4 * h);
                    } else if (cols[Q.steps[s].col].mode == kWmDirect && row + kWsBatch * h < b) {
                        x = ws_ld_rows(cols[Q.steps[s].col].src + (row + kWsBatch * h) * 4);
                    }
                    ws_put(w[s], h, x);
                }
                if (FLAT && !ROWS) src[s] += H * kWsBatch * 4;
            }
            if (!FLAT) {
#pragma unroll
                for (uint32_t s = 0; s < NS; ++s) {
                    const WsCol& d = cols[Q.steps[s].col];
                    if (d.mode == kWmDirect) continue;
#pragma unroll
                    for (uint32_t h = 0; h < H; ++h)
                        if (row + kWsBatch * h < b) ws_put(w[s], h, ws_quad(d, row + kWsBatch * h));
                }
            }
        }
        // one step over the batch: v = the lane's rows of its column
        auto step = [&](uint32_t s, uint32_t K, const uint32_t (&v)[R]) {
            const ShStep& stp = Q.steps[s];
            const bool decided = ((cst >> s) & 1u) != 0;
            if ((K & kWkF) && !decided) {
                // lo <= v <= hi as one unsigned comparison of v - lo with hi - lo
                // (an empty range, hi < lo, keeps nothing)
                const uint32_t lo = (uint32_t)stp.lo, span = (uint32_t)stp.hi - lo;
                if (stp.lo > stp.hi) m = 0;
#pragma unroll
                for (uint32_t r = 0; r < R; ++r)
                    if (v[r] - lo > span) m &= ~(1u << r);
            }
            uint32_t pp[R];
#pragma unroll
            for (uint32_t r = 0; r < R; ++r) pp[r] = v[r];
            if ((K & kWkP) && !decided) m = ht_probe_rows<R>(stp.ht, stp.ht_log2, stp.ht_layout, s_hdr[s], v, m, pp, pol_keep);
            if (K & kWkD) {
                const uint32_t dcard = stp.digit_card, dbase = (uint32_t)stp.digit_base, cdig = sdig[s];
                if (decided) {
#pragma unroll
                    for (uint32_t r = 0; r < R; ++r) g[r] = g[r] * dcard + cdig;
                } else {
                    uint32_t bad = 0;
#pragma unroll
                    for (uint32_t r = 0; r < R; ++r) {
                        const uint32_t dgt = pp[r] - dbase;
                        if (dgt >= dcard) bad |= 1u << r;
                        g[r] = g[r] * dcard + dgt;
                    }
                    if (bad & m) {
                        raise_error(kErrInvalid);
                        m &= ~bad;
                    }
                }
            }
            if (K & kWkC) {
#pragma unroll
                for (uint32_t r = 0; r < R; ++r) carry[r] = v[r];
            }
        };
        uint32_t val[R];  // the last column
        if constexpr (!RT) {
#pragma unroll
            for (uint32_t s = 0; s < NS; ++s) {
                const uint32_t K = (SIG >> (7 + 4 * s)) & 15u;
                if (s < PE || (K & kWkD)) step(s, K, w[s]);
                else if (K & kWkC) {
#pragma unroll
                    for (uint32_t r = 0; r < R; ++r) carry[r] = w[s][r];
                }
            }
            m &= some;
#pragma unroll
            for (uint32_t r = 0; r < R; ++r) val[r] = w[NS - 1][r];
        } else {
#pragma unroll
            for (uint32_t r = 0; r < R; ++r) val[r] = 0;
#pragma unroll 1
            for (uint32_t s = 0; s < ns; ++s) {
                if (!__any_sync(0xFFFFFFFFu, m)) break;
                const ShStep& stp = Q.steps[s];
                const WsCol& d = cols[stp.col];
#pragma unroll
                for (uint32_t h = 0; h < H; ++h) {
                    uint4 x = make_uint4(0, 0, 0, 0);
                    if (row + kWsBatch * h < b) x = ws_quad(d, row + kWsBatch * h);
                    ws_put(val, h, x);
                }
                const uint32_t f = stp.flags;
                step(s, ((f & GX_STEP_FILTER) ? kWkF : 0u) | ((f & GX_STEP_PROBE) ? kWkP : 0u) |
                            ((f & GX_STEP_CARRY) ? kWkC : 0u) | (stp.digit_card ? kWkD : 0u), val);
            }
        }
        // the filters after the probes and the aggregate, row by row
        auto kept = [&](uint32_t r) {
            bool k = ((m >> r) & 1u) != 0;
            if (!RT) {
#pragma unroll
                for (uint32_t s = PE; s < NS; ++s)
                    if ((SIG >> (7 + 4 * s)) & kWkF) {
                        const uint32_t lo = (uint32_t)Q.steps[s].lo, span = (uint32_t)Q.steps[s].hi - lo;
                        k = k && w[s][r] - lo <= span;
                    }
            }
            return k;
        };
        auto value = [&](uint32_t r) -> int64_t {
            const int32_t x = (int32_t)val[r], c = (int32_t)carry[r];
            return agg == GX_AGG_SUM_PRODUCT ? (int64_t)x * c
                   : agg == GX_AGG_SUM_DIFF  ? (int64_t)x - c
                   : agg == GX_AGG_COUNT     ? 1
                                             : (int64_t)x;
        };
        if (!GR) {
#pragma unroll
            for (uint32_t r = 0; r < R; ++r) {
                if constexpr (SIG == kSigQ1) {
                    // both filters and the multiply-add as one predicate chain
                    asm("{\n .reg .pred p;\n .reg .u32 d, e;\n sub.u32 d, %1, %2;\n sub.u32 e, %4, %5;\n"
                        " setp.ne.u32 p, %7, 0;\n setp.le.and.u32 p, d, %3, p;\n setp.le.and.u32 p, e, %6, p;\n"
                        " @p mad.wide.s32 %0, %8, %9, %0;\n}"
                        : "+l"(acc)
                        : "r"(w[1][r]), "r"(Q.steps[1].lo), "r"((uint32_t)Q.steps[1].hi - (uint32_t)Q.steps[1].lo),
                          "r"(w[2][r]), "r"(Q.steps[2].lo), "r"((uint32_t)Q.steps[2].hi - (uint32_t)Q.steps[2].lo),
                          "r"(m & (1u << r)), "r"(w[3][r]), "r"(w[1][r]));
                } else if (kept(r)) {
                    acc += value(r);
                }
            }
        } else {
            const uint32_t below = (1u << lane) - 1u;
#pragma unroll
            for (uint32_t r = 0; r < R; ++r) {
                const bool on = kept(r);
                const uint32_t bal = __ballot_sync(0xFFFFFFFFu, on);
                if (__popc(bal) >= 24) {  // most lanes have a row: no detour through the queue
                    ws_group_add_lanes(on, g[r], value(r), tkey, Q.g_keys, Q.g_sums, Q.g_log2);
                    continue;
                }
                if (on) {
                    const uint32_t at = qn + __popc(bal & below);
                    wq->key[at] = g[r];
                    wq->val[at] = value(r);
                }
                qn += __popc(bal);
            }
            while (qn >= 32) {
                qn -= 32;
                ws_queue_flush(wq, qn, 32, tkey, Q.g_keys, Q.g_sums, Q.g_log2, lane);
            }
        }
    }
    return acc;
}

// A run-time plan without a group key over tile rows [a, b), step by step: a
// step issues the loads of four quads (512 rows of the warp) together, those of
// rows still kept, and leaves the rows it keeps in a mask (bit 4 j + i: row
// 128 j + 4 lane + i); probes go two quads at a time, and a carried column is
// read again beside the last step's.  What kind of step it is, how its column
// is read and the aggregate are so decided once per 512 rows: row group by row
// group (as ws_eval takes grouped plans, whose keys live in registers) these
// decisions and one load in flight per step bound the scan: over 20M rows a sum
// 91 us, a filtered sum 144 us, a date probe with a filter and a sum 174 us;
// 21, 38 and 54 us here.  Returns the lane's part of the sum.
__device__ __forceinline__ int64_t ws_eval_steps(const ShQuery& Q, const WsCol* cols, uint32_t cst, uint32_t a,
                                                 uint32_t b, uint64_t pol_keep, const uint64_t* s_hdr,
                                                 uint32_t lane) {
    uint32_t keep = ~0u;
    if (a != 0 || b != kWsTile) {
        keep = 0;
        for (uint32_t j = a / kWsBatch; j * kWsBatch < b; ++j) {
            const uint32_t row = j * kWsBatch + 4 * lane, n = row < b ? min(4u, b - row) : 0u;
            keep |= ((1u << n) - 1u) << (4 * j);
        }
    }
    // quads j .. j + 3 of a column (those with a row kept)
    auto load = [&](const WsCol& d, uint32_t j, uint32_t k, uint32_t (&x)[16]) {
        const uint32_t row = j * kWsBatch + 4 * lane;
        if (d.mode == kWmDirect) {
            const uint8_t* p = d.src + 4 * row;
#pragma unroll
            for (uint32_t h = 0; h < 4; ++h)
                if ((k >> (4 * h)) & 15u) ws_put(x, h, ws_ld_rows(p + 4 * kWsBatch * h));
        } else {
#pragma unroll
            for (uint32_t h = 0; h < 4; ++h)
                if ((k >> (4 * h)) & 15u) ws_put(x, h, ws_quad(d, row + kWsBatch * h));
        }
    };
    const uint32_t ns = Q.n_steps, agg = Q.agg, j_end = (b + kWsBatch - 1) / kWsBatch;
    const WsCol* carried = nullptr;
    int64_t acc = 0;
#pragma unroll 1
    for (uint32_t s = 0; s < ns; ++s) {
        const ShStep& stp = Q.steps[s];
        const WsCol& d = cols[stp.col];
        const uint32_t f = stp.flags;
        const bool last = s + 1 == ns, decided = ((cst >> s) & 1u) != 0;
        if (f & GX_STEP_CARRY) carried = &d;
        const bool filt = (f & GX_STEP_FILTER) && !decided;
        if (filt && stp.lo > stp.hi) return 0;
        const uint32_t lo = (uint32_t)stp.lo, span = (uint32_t)stp.hi - lo;
        if ((f & GX_STEP_PROBE) && !decided) {
#pragma unroll 1
            for (uint32_t j = a / kWsBatch; j < j_end; j += 2) {
                uint32_t k = (keep >> (4 * j)) & 255u, m = k;
                if (!__any_sync(0xFFFFFFFFu, k)) continue;
                uint32_t v[8], pay[8];
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h)
                    if ((k >> (4 * h)) & 15u) ws_put(v, h, ws_quad(d, (j + h) * kWsBatch + 4 * lane));
                if (filt) {
#pragma unroll
                    for (uint32_t r = 0; r < 8; ++r)
                        if (v[r] - lo > span) m &= ~(1u << r);
                }
                m = ht_probe_rows<8>(stp.ht, stp.ht_log2, stp.ht_layout, s_hdr[s], v, m, pay, pol_keep);
                keep &= ~((k & ~m) << (4 * j));
            }
        }
        const bool here = filt && !(f & GX_STEP_PROBE);
        if (here || last) {
            const bool both = agg == GX_AGG_SUM_PRODUCT || agg == GX_AGG_SUM_DIFF;
#pragma unroll 1
            for (uint32_t j = a / kWsBatch; j < j_end; j += 4) {
                uint32_t k = (keep >> (4 * j)) & 0xFFFFu;
                if (!__any_sync(0xFFFFFFFFu, k)) continue;
                uint32_t x[16], c[16];
                if (here || agg != GX_AGG_COUNT) load(d, j, k, x);
                if (last && both) load(*carried, j, k, c);
                if (here) {
                    uint32_t m = k;
#pragma unroll
                    for (uint32_t r = 0; r < 16; ++r)
                        if (x[r] - lo > span) m &= ~(1u << r);
                    keep &= ~((k & ~m) << (4 * j));
                    k = m;
                }
                if (!last) continue;
                if (agg == GX_AGG_SUM_PRODUCT) {
#pragma unroll
                    for (uint32_t r = 0; r < 16; ++r)
                        if ((k >> r) & 1u) acc += (int64_t)(int32_t)x[r] * (int32_t)c[r];
                } else if (agg == GX_AGG_COUNT) {
                    acc += __popc(k);
                } else {
#pragma unroll
                    for (uint32_t r = 0; r < 16; ++r)
                        if ((k >> r) & 1u) acc += (int32_t)x[r];
                    if (agg == GX_AGG_SUM_DIFF) {
#pragma unroll
                        for (uint32_t r = 0; r < 16; ++r)
                            if ((k >> r) & 1u) acc -= (int32_t)c[r];
                    }
                }
            }
        }
        if (!__any_sync(0xFFFFFFFFu, keep)) break;
    }
    return acc;
}

// The signatures with a kRows evaluator: scalar ones.  (One more instance in the
// kernel of the grouped star join cost it 2.6 %.)
template <uint32_t SIG>
constexpr bool kWsRows = !kWsRunTime<SIG> && ((SIG >> 6) & 1) == 0;

// The other evaluators out of line: tiles with decoded columns; ragged tiles,
// other columns that are not direct, run-time plans.
template <uint32_t SIG, WsForm FORM>
__device__ __noinline__ int64_t ws_eval_any(const ShQuery& Q, const WsCol* cols, uint32_t cst, const uint32_t* sdig,
                                            uint32_t a, uint32_t b, uint32_t* tkey, WsQueue* wq, uint32_t* qn,
                                            uint64_t pol_keep, const uint64_t* s_hdr,
                                            uint32_t lane) {
    uint32_t n = *qn;
    const int64_t acc = ws_eval<SIG, FORM>(Q, cols, cst, sdig, a, b, tkey, wq, n, pol_keep, s_hdr, lane);
    *qn = n;
    return acc;
}

// CTAs per SM each form is built for.  Scalar signatures (two row groups and
// their columns in registers) keep 96 registers: five CTAs, 20 warps, scan Q1
// over 60M rows in 132 us where four take 165 us (too few loads in flight) and
// six 150 us (spills); scalar run-time plans likewise (a filtered sum over 20M
// rows 38 us, with four 43, with six 38 but a pruned one 13.7 for 12.6).
// Grouped ones (one row group, probes) take six: the 200M-row star join 2.17 ms,
// 2.26 with five, 2.35 with seven; more shared memory costs them L1, which holds
// their reads in flight: 2048 group slots instead of 512, 4.2 ms).  The group-by
// without joins waits on group-table adds and takes eight (30M rows into 1.4M
// groups: 585 us, 674 with six; as a run-time plan 782).  Grouped run-time plans
// take seven (20M rows counted into 50 groups 171 us, with eight 195; summed into
// 550 groups 468 us, 488 with eight and 502 with six).
constexpr int ws_ctas(uint32_t sig) {
    return sig == kSigGroup ? 8 : sig == kSigRtGroup ? 7 : ((sig >> 6) & 1) ? 6 : 5;
}

template <uint32_t SIG>
__global__ void __launch_bounds__(kWsNT, ws_ctas(SIG)) warp_scan_kernel(const __grid_constant__ WsParams P) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ gx_dcol s_cols[kWsMaxCols];
    __shared__ WsWork s_work;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t ncols = P.n_cols;
    const ShQuery& Q = P.q;
    uint32_t* const s_kbits = (uint32_t*)smem;               // chunk keep bits of [chunk_lo, chunk_hi)
    uint32_t* const s_kpre = s_kbits + P.chunk_words;        // surviving chunks before each word
    uint32_t* const wmem = s_kpre + P.chunk_words + (size_t)warp * P.warp_words;
    WsCol* const wcols = (WsCol*)wmem;                       // column records of the round's tiles
    WsTile* const wtiles = (WsTile*)(wmem + 32 * 8);         // their tile records
    uint64_t* const whdr = (uint64_t*)(wmem + 40 * 8);  // dense join tables' headers, per step
    uint32_t* const wdig = wmem + 40 * 8 + 2 * GX_MAX_STEPS;  // constant steps' group-key digits
    unsigned long long* const wrows = (unsigned long long*)(wdig + 32);  // rows scanned
    WsQueue* const wq = (WsQueue*)(wmem + kWsHead);          // grouped: rows on their way to the group table
    uint32_t* const areas = wmem + kWsHead + (P.grouped_tab ? kWsQueueWords : 0u);  // the decode buffers
    // grouped: the CTA's group table (keys, low halves, high halves of the sums) after the warps' regions
    uint32_t* const tkey = s_kpre + P.chunk_words + (size_t)kWsWarps * P.warp_words;
    const uint64_t pol_keep = ws_policy_keep();

    // The launch may overlap the kernel before it on the stream (programmatic
    // dependent launch): until a thread has passed griddep_wait it reads only
    // the columns (payload, directory, side index, min/max, zone maps: never
    // written by kernels), and every read of join tables, keep_in, and every
    // global write (results, keep_out, group tables) comes after its wait.
    bool waited = false;
    if (Q.keep_in) {  // keep flags may come from the kernel before
        griddep_wait();
        waited = true;
    }
    // a warp's first evaluation: the wait, then the dense join tables' headers
    auto await_tables = [&]() {
        if (!waited) griddep_wait();
        waited = true;
        if (lane < GX_MAX_STEPS) {
            const ShStep& st = Q.steps[lane];
            whdr[lane] = (lane < Q.n_steps && (st.flags & GX_STEP_PROBE) && st.ht_layout == GX_HT_DENSE)
                             ? __ldcg((const unsigned long long*)st.ht)
                             : 0ull;
        }
        __syncwarp();
    };
    bool tables = false;  // whdr loaded
    for (uint32_t i = tid; i < ncols * (uint32_t)(sizeof(gx_dcol) / 4); i += kWsNT)
        ((uint32_t*)s_cols)[i] = ((const uint32_t*)P.cols)[i];
    // chunk keep (keep_in and the prune predicates' chunk min/max, the
    // reference's granularity), one ballot word per 32 chunks; CTA 0 writes
    // keep_out from them at the end
    const uint32_t n_range = P.chunk_hi - P.chunk_lo;
    for (uint32_t wb = warp * 32; wb < P.chunk_words * 32; wb += kWsNT) {
        const uint32_t i = wb + lane, chunk = P.chunk_lo + i;
        bool ck = i < n_range;
        if (ck) {
            if (Q.keep_in) ck = __ldg(Q.keep_in + chunk) != 0;
            for (uint32_t p = 0; p < Q.n_prune; ++p) {
                const PrunePred& pr = Q.prune[p];
                ck = ck && pr.lo <= __ldg(pr.maxs + chunk) && pr.hi >= __ldg(pr.mins + chunk);
            }
        }
        const uint32_t word = __ballot_sync(0xFFFFFFFFu, ck);
        if (lane == 0) s_kbits[wb / 32] = word;
    }
    if (P.grouped_tab) {
        for (uint32_t i = tid; i < kWsGroupSlots; i += kWsNT) {
            tkey[i] = kEmptyGKey;
            tkey[kWsGroupSlots + i] = 0;
            tkey[2 * kWsGroupSlots + i] = 0;
        }
    }
    __syncthreads();
    if (warp == 0) {  // exclusive prefix of the popcounts: per lane a run of words, then a warp scan
        const uint32_t per = (P.chunk_words + 31) / 32, w0 = min(P.chunk_words, lane * per),
                       w1 = min(P.chunk_words, w0 + per);
        uint32_t cnt = 0, first = kWsNone, last = 0;  // surviving chunks of the lane's words: count, first, last
        for (uint32_t i = w0; i < w1; ++i) {
            const uint32_t m = s_kbits[i];
            cnt += __popc(m);
            if (m) {
                first = min(first, i * 32 + (__ffs(m) - 1));
                last = i * 32 + (31 - __clz(m));
            }
        }
        uint32_t run = ws_scan(cnt, lane) - cnt;
        for (uint32_t i = w0; i < w1; ++i) {
            s_kpre[i] = run;
            run += __popc(s_kbits[i]);
        }
        first = __reduce_min_sync(0xFFFFFFFFu, first);
        last = __reduce_max_sync(0xFFFFFFFFu, last);
        if (lane == 31) {
            WsWork R;
            R.first = run && last - first + 1 == run ? P.chunk_lo + first : kWsNone;
            R.t_end = run * P.blocks_per_chunk * P.tiles_per_block;  // the launch keeps tile indices below 2^31
            R.W = gridDim.x * kWsWarps;
            R.full = R.t_end / R.W;
            const uint32_t left = R.t_end - R.full * R.W;
            R.rounds = R.full + (left ? 1u : 0u);
            R.parts_log2 = 0;
            if (P.parts)  // as many parts as there are warps for
                while ((1u << R.parts_log2) < kWsMaxParts && (left << (R.parts_log2 + 1)) <= R.W) ++R.parts_log2;
            s_work = R;
        }
    }
    __syncthreads();  // the last block-wide barrier: warps are independent from here on

    const uint32_t w = blockIdx.x * kWsWarps + warp, rounds = s_work.rounds;
    int64_t local = 0;
    uint32_t qn = 0;  // rows in the warp's queue
    if (lane == 0) *wrows = 0;
    const uint32_t cl = P.col_log2, nq = 32u >> cl;
    for (uint32_t r0 = 0; r0 < rounds; r0 += nq) {
        const uint32_t vm = ws_decide(P, s_cols, s_kbits, s_kpre, s_work, w, r0, lane, wtiles, wcols);
        if (!vm) continue;
        if (!tables) {
            await_tables();
            tables = true;
        }
        ws_const_steps<SIG>(P, vm, wtiles, wcols, whdr, wdig, pol_keep, lane);
        for (uint32_t q = 0; q < nq; ++q) {
            if (!((vm >> q) & 1u)) continue;
            const WsTile& T = wtiles[q];
            WsCol* const cols = wcols + (q << cl);
            int terr = 0;
            if (T.steps & kWsDecode) terr = ws_decode_tile(P, s_cols, T, cols, areas, lane);
            if (terr) {
                if (lane == 0) raise_error(terr);
                continue;
            }
            if (lane == 0) *wrows += T.b - T.a;
            // ---- evaluation
            const uint32_t st = T.steps;
            if (!(st & kWsDead)) {
                // whole row batches of direct columns: the flat form
                const uint32_t* const dig = wdig + (q << cl);
                if constexpr (SIG == kSigRt)
                    local += ws_eval_steps(Q, cols, st, T.a, T.b, pol_keep, whdr, lane);
                else if (!kWsRunTime<SIG> && !(st & kWsMixed) && ((T.b - T.a) & (kWsPartRows - 1u)) == 0)
                    local += ws_eval<SIG, kWsRunTime<SIG> ? WsForm::kAny : WsForm::kFlat>(
                        Q, cols, st, dig, T.a, T.b, tkey, wq, qn, pol_keep, whdr, lane);
                else if (kWsRows<SIG> && !(st & kWsHard) && ((T.b - T.a) & (kWsPartRows - 1u)) == 0)
                    local += ws_eval_any<SIG, kWsRows<SIG> ? WsForm::kRows : WsForm::kAny>(
                        Q, cols, st, dig, T.a, T.b, tkey, wq, &qn, pol_keep, whdr, lane);
                else
                    local += ws_eval_any<SIG, WsForm::kAny>(Q, cols, st, dig, T.a, T.b, tkey, wq, &qn, pol_keep, whdr,
                                                            lane);
            }
            __syncwarp();  // every lane is done with the tile's buffers and records before they are overwritten
        }
        __syncwarp();
    }
    // ---- results: the CTA's group table once every warp is done, else the warp's sum
    if (qn) ws_queue_flush(wq, 0, qn, tkey, Q.g_keys, Q.g_sums, Q.g_log2, lane);
    __syncwarp();
    if (!waited) griddep_wait();
    if (blockIdx.x == 0 && Q.keep_out)
        for (uint32_t i = tid; i < n_range; i += kWsNT) Q.keep_out[P.chunk_lo + i] = (s_kbits[i / 32] >> (i % 32)) & 1u;
    if (Q.grouped && P.grouped_tab) {
        __syncthreads();
        for (uint32_t i = tid; i < kWsGroupSlots; i += kWsNT) {
            const uint32_t key = tkey[i];
            const uint64_t sum = ((uint64_t)tkey[2 * kWsGroupSlots + i] << 32) | tkey[kWsGroupSlots + i];
            if (key != kEmptyGKey && !group_add_global(Q.g_keys, Q.g_sums, Q.g_log2, (int64_t)key, (int64_t)sum))
                raise_error(kErrCapacity);
        }
    } else if (!Q.grouped) {
        const uint64_t u = warp_sum_u64((uint64_t)local);
        if (lane == 0 && u && Q.result) atomicAdd((unsigned long long*)Q.result, (unsigned long long)u);
    }
    if (lane == 0 && P.rows_scanned && *wrows) atomicAdd(P.rows_scanned, *wrows);
}
