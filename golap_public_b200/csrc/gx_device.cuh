// gx_device.cuh -- sm_100a device building blocks: block decoders (segmented
// LZ4, generic LZ4, cascaded), TMA bulk staging, join-table probing and
// group-table updates.  Included by kernels.cu only.
//
// Reference counterparts: the nvCOMP decompressors behind
// ChunkDecompressor::step (core/comp.cuh:186), HashMap::probe
// (core/dev_structs.cuh:105-113) and HashAggregate::add
// (core/dev_structs.cuh:210-244).  Unlike HashAggregate::add, no wait here
// is unbounded: every probe loop is capped by the table size and every
// mbarrier wait by an iteration count.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "gx_internal.h"

namespace gx {

constexpr int kErrCorrupt = 2;   // == GX_ERR_CORRUPT
constexpr int kErrCapacity = 3;  // == GX_ERR_CAPACITY
constexpr int kErrTimeout = 4;   // == GX_ERR_TIMEOUT
constexpr int kErrInvalid = 6;   // == GX_ERR_INVALID
constexpr uint64_t kEmptySlot = (uint64_t)(uint32_t)kEmptyKey;  // {key=INT32_MIN, payload=0}
constexpr uint32_t kEmptyGKey = 0xFFFFFFFFu;                    // shared-memory group table

// ---------------------------------------------------------- byte access
__device__ __forceinline__ uint32_t ldb(const uint8_t* p) { return (uint32_t)__ldg(p); }

// Global-memory byte source (read-only path) for the generic LZ4 decoder.
struct GlobalSrc {
    const uint8_t* p;
    __device__ __forceinline__ uint32_t b(uint32_t i) const { return ldb(p + i); }
};
// Byte source over a block staged in shared memory.
struct SharedSrc {
    const uint8_t* p;
    __device__ __forceinline__ uint32_t b(uint32_t i) const { return p[i]; }
};

// ------------------------------------------------ TMA bulk copy + mbarrier
// One-dimensional cp.async.bulk (no multicast) from global memory into this
// CTA's shared memory, completed on an mbarrier.  Source, destination and
// size must be 16-byte aligned / multiples of 16.
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* m, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(m)), "r"(count) : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// Orders this thread's earlier generic-proxy accesses of shared memory
// before later async-proxy (TMA) writes to it.
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tma_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* m) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(m)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(m))
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* m, uint32_t phase) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(m)), "r"(phase)
        : "memory");
    return ok != 0;
}

// try_wait that may suspend the thread until the phase completes or about
// `ns` nanoseconds pass: waiting threads sleep instead of spinning through
// issue slots while a bulk copy is in flight.
__device__ __forceinline__ bool mbar_try_wait_sleep(uint64_t* m, uint32_t phase, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(m)), "r"(phase), "r"(ns)
        : "memory");
    return ok != 0;
}

// Bounded wait for the phase to complete (never waits forever: at most
// kMbarWaitCap tries of at most 1 us each).
constexpr uint32_t kMbarWaitCap = 1u << 21;
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* m, uint32_t phase) {
    for (uint32_t i = 0; i < kMbarWaitCap; ++i)
        if (mbar_try_wait_sleep(m, phase, 1000u)) return true;
    return false;
}

// Programmatic dependent launch: a kernel launched with programmatic stream
// serialization may start while the kernel before it on the stream still
// runs; griddep_wait blocks the calling thread until that kernel has
// completed and its writes are visible (at once when there is none), and
// griddep_launch lets the kernel that follows start early once every CTA of
// this one has issued it.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" :::); }

// L2 cache policy of join tables: they stay (evict last).
__device__ __forceinline__ uint64_t ws_policy_keep() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
// A join-table slot read under policy pol (read-only path).
__device__ __forceinline__ unsigned long long ws_ld_slot(const unsigned long long* a, uint64_t pol) {
    unsigned long long v;
    asm("ld.global.nc.L2::cache_hint.b64 %0, [%1], %2;" : "=l"(v) : "l"(a), "l"(pol));
    return v;
}
// ------------------------------------------------- segmented LZ4
// 4 bytes at byte offset r of a staged window (little endian, any alignment).
__device__ __forceinline__ uint32_t fetch4(const uint32_t* __restrict__ A, uint32_t r) {
    const uint32_t w = r >> 2;
    return __funnelshift_r(A[w], A[w + 1], (r & 3u) * 8);
}

// LZ4 length extension at stream position pos: adds bytes to len until one
// below 255 has been added, four bytes per step (per-byte equality with 255
// by __vcmpeq4).  Consumes no byte at or past hi (returns false then).
__device__ __forceinline__ bool lz4_len_ext(const uint32_t* __restrict__ A, uint32_t wbase, uint32_t& pos,
                                            uint32_t hi, uint32_t& len) {
    while (true) {
        if (pos >= hi) return false;
        const uint32_t x = fetch4(A, pos - wbase);
        const uint32_t ff = __vcmpeq4(x, 0xFFFFFFFFu);
        if (ff == 0xFFFFFFFFu) {
            len += 4 * 255;
            pos += 4;
            continue;
        }
        const uint32_t nfull = (uint32_t)(__ffs(~ff) - 1) >> 3;  // leading bytes equal to 255
        len += 255 * nfull + ((x >> (8 * nfull)) & 255u);
        pos += nfull + 1;
        return pos <= hi;
    }
}

// Decodes one segment of a segmented LZ4 block with a group of G lanes
// (G a power of two <= 32, the group's lanes adjacent in one warp; gmask =
// the group's lanes, gl = this lane's index in the group).  Every lane of the
// group parses the same sequence headers (broadcast shared loads), so the
// group stays converged; literal runs and matches are copied G words per
// step.  A match's words are all computed from output before the match:
// out[k + i] = out[k - offw + (i mod offw)] (LZ4 overlap semantics), so one
// __syncwarp before each match orders it after every earlier write of the
// group.  A = the words from byte wbase (staged, or in place), [lo, hi) the
// tile's compressed range, K output words.  Returns 0 or kErrCorrupt (the same
// for every lane of the group).
__device__ __forceinline__ int lz4_seg_group(const uint32_t* __restrict__ A, uint32_t wbase, uint32_t lo,
                                             uint32_t hi, uint32_t block_end, uint32_t comp_pos, uint32_t info,
                                             uint32_t K, uint32_t* __restrict__ out, uint32_t gl, uint32_t G,
                                             uint32_t gmask) {
    if (comp_pos < lo || comp_pos > hi) return kErrCorrupt;
    uint32_t pos = comp_pos, k = 0, litw = 0, mnib = 0;
    bool tok_next = true;
    if (info & 16u) {  // the segment starts inside a sequence
        const uint32_t lit = info >> 5;
        if (lit & 3u) return kErrCorrupt;
        litw = lit >> 2;
        mnib = info & 15u;
        tok_next = false;
    }
    while (true) {
        if (tok_next) {
            if (k >= K) break;
            if (pos >= hi) return kErrCorrupt;
            const uint32_t x = fetch4(A, pos - wbase);
            uint32_t lit = (x >> 4) & 15u;
            mnib = x & 15u;
            ++pos;
            if (lit == 15 && !lz4_len_ext(A, wbase, pos, hi, lit)) return kErrCorrupt;
            if (lit & 3u) return kErrCorrupt;
            litw = lit >> 2;
        }
        const uint32_t n = min(litw, K - k);
        if ((uint64_t)pos + 4ull * n > hi) return kErrCorrupt;
        {
            const uint32_t r = pos - wbase, w = r >> 2, sh = (r & 3u) * 8;
            for (uint32_t i = gl; i < n; i += G) out[k + i] = __funnelshift_r(A[w + i], A[w + i + 1], sh);
        }
        k += n;
        pos += 4 * n;
        if (k >= K) break;  // the segment ends inside or right after the literals
        // literals done: the block may end here (then the segment is short)
        if (pos == block_end || (uint64_t)pos + 2 > hi) return kErrCorrupt;
        const uint32_t off = fetch4(A, pos - wbase) & 0xFFFFu;
        pos += 2;
        uint32_t ml = mnib + 4;
        if (mnib == 15 && !lz4_len_ext(A, wbase, pos, hi, ml)) return kErrCorrupt;
        if ((off & 3u) || (ml & 3u) || off == 0) return kErrCorrupt;
        const uint32_t offw = off >> 2, mw = ml >> 2;
        if (offw > k || mw > K - k) return kErrCorrupt;
        __syncwarp(gmask);
        const uint32_t* src = out + (k - offw);
        if (offw >= mw) {
            for (uint32_t i = gl; i < mw; i += G) out[k + i] = src[i];
        } else if (offw == 1) {
            const uint32_t v = src[0];
            for (uint32_t i = gl; i < mw; i += G) out[k + i] = v;
        } else {
            uint32_t r = gl % offw;
            const uint32_t step = G % offw;
            for (uint32_t i = gl; i < mw; i += G) {
                out[k + i] = src[r];
                r += step;
                if (r >= offw) r -= offw;
            }
        }
        k += mw;
        tok_next = true;
    }
    return 0;
}

// As lz4_seg_group, with the groups of a warp in step: one sequence each per
// round, for columns of short sequences.  Called by whole warps; lanes of a
// group without a segment pass active = false.
// What bounds it: the chain of dependent instructions of a sequence (100 or
// so, 6 to 8 cycles each with few warps resident), of which a segment of small
// integers has nearly one per row.  A round of short sequences therefore reads
// token, offset and one literal extension byte from one unaligned word and
// fetches the next token before the copy, and the groups stay in step (their
// own loops drifted apart and ran one after another).  Q1 over 10M rows of such
// columns 665 -> 570 us, decoding 24M discount rows 353 -> 330; a column known
// to hold many short sequences takes lz4_seg_lane in the scan.  Sequences longer
// than such a round pay for looking (LzGroups below).
__device__ __forceinline__ int lz4_seg_step(const uint32_t* __restrict__ A, uint32_t wbase, uint32_t lo, uint32_t hi,
                                            uint32_t block_end, uint32_t comp_pos, uint32_t info, uint32_t K,
                                            uint32_t* __restrict__ out, uint32_t gl, uint32_t G, bool active) {
    uint32_t pos = comp_pos, k = 0, litw = 0, mnib = 0;
    bool ok = comp_pos >= lo && comp_pos <= hi, run = active && ok;
    bool tok = true;  // the next thing is a token
    if (run && (info & 16u)) {  // the segment starts inside a sequence
        ok = ((info >> 5) & 3u) == 0;
        litw = info >> 7;
        mnib = info & 15u;
        tok = false;
    }
    run = run && ok && (k < K || !tok);
    if (!run) pos = lo;  // lanes without work read some word of the range
    uint32_t x = fetch4(A, pos - wbase);
    while (__any_sync(0xFFFFFFFFu, run)) {
        const uint32_t tl = (x >> 4) & 15u, tm = x & 15u;
        const bool ext = tl == 15u && ((x >> 8) & 255u) == 255u;  // longer literals than one extension byte gives
        if (!__any_sync(0xFFFFFFFFu, run && (!tok || ext || tm == 15u))) {
            // ---- a round of short sequences: at most 67 literal words, at most 4 match words
            const uint32_t lit = tl == 15u ? 15u + ((x >> 8) & 255u) : tl, q0 = pos + (tl == 15u ? 2u : 1u);
            const uint32_t lw = lit >> 2, n = min(lw, K - k), q = q0 - wbase, kk = k + n;
            const bool more = lw < K - k;  // the segment goes on with the match
            uint32_t off = x >> 8;
            bool good = (lit & 3u) == 0 && q0 + 4 * n <= hi;
            if (__any_sync(0xFFFFFFFFu, run && lit)) {
                if (run && good)
                    for (uint32_t i = gl; i < n; i += G) out[k + i] = fetch4(A, q + 4 * i);
                if (lit && run && good && more) off = fetch4(A, q + lit);
            }
            off &= 0xFFFFu;
            const uint32_t offw = off >> 2, mw = more ? (tm >> 2) + 1 : 0u;
            const uint32_t p1 = q0 + lit;
            if (more)
                good = good && p1 != block_end && p1 + 2 <= hi && ((off | tm) & 3u) == 0 && offw - 1u < kk && mw <= K - kk;
            if (run && !good) ok = run = false;
            __syncwarp();
            const uint32_t nx = run && more ? fetch4(A, p1 + 2 - wbase) : x;  // the next token, ahead of the copy
            if (run)
                for (uint32_t i = gl; i < mw; i += G) {
                    uint32_t r = i;
                    if (offw < 4) r = offw == 1 ? 0u : offw == 2 ? (i & 1u) : (i == 3 ? 0u : i);
                    out[kk + i] = out[kk - offw + r];
                }
            if (run) {
                k = kk + mw;
                pos = p1 + 2;
                x = nx;
            }
            run = run && more && k < K;
            __syncwarp();
            continue;
        }
        // ---- the general round
        if (run && tok) {
            ok = pos < hi;
            if (ok) {
                uint32_t lit = tl;
                mnib = tm;
                ++pos;
                if (lit == 15) ok = lz4_len_ext(A, wbase, pos, hi, lit);
                ok = ok && (lit & 3u) == 0;
                litw = lit >> 2;
            }
            run = ok;
        }
        uint32_t n = run ? min(litw, K - k) : 0u;
        if (run && (uint64_t)pos + 4ull * n > hi) {
            ok = run = false;
            n = 0;
        }
        {
            const uint32_t r = pos - wbase, w = r >> 2, sh = (r & 3u) * 8;
            for (uint32_t i = gl; i < n; i += G) out[k + i] = __funnelshift_r(A[w + i], A[w + i + 1], sh);
        }
        k += n;
        pos += 4 * n;
        run = run && k < K;  // else the segment ends inside or right after the literals
        // the match (the block may not end before it: then the segment is short)
        uint32_t offw = 1, mw = 0;
        if (run) {
            ok = pos != block_end && (uint64_t)pos + 2 <= hi;
            if (ok) {
                const uint32_t off = fetch4(A, pos - wbase) & 0xFFFFu;
                pos += 2;
                uint32_t ml = mnib + 4;
                if (mnib == 15) ok = lz4_len_ext(A, wbase, pos, hi, ml);
                ok = ok && (off & 3u) == 0 && (ml & 3u) == 0 && off != 0;
                offw = off >> 2;
                mw = ml >> 2;
                ok = ok && offw <= k && mw <= K - k;
            }
            run = ok;
            if (!ok) mw = 0;
        }
        __syncwarp();
        {
            const bool wrap = offw < mw;
            uint32_t r = gl, st = G;
            if (wrap && offw != 1) {
                r = gl % offw;
                st = G % offw;
            }
            const uint32_t* src = out + (k - offw);
            if (offw == 1) {
                const uint32_t v = mw ? src[0] : 0u;
                for (uint32_t i = gl; i < mw; i += G) out[k + i] = v;
            } else {
                for (uint32_t i = gl; i < mw; i += G) {
                    out[k + i] = src[r];
                    r += st;
                    if (wrap && r >= offw) r -= offw;
                }
            }
        }
        k += mw;
        tok = true;
        run = run && k < K;
        if (run) x = fetch4(A, pos - wbase);
        __syncwarp();
    }
    return active && !ok ? kErrCorrupt : 0;
}

// Which of the two a column takes: groups in step (gx_dcol::lz4_steps) when at
// least three in four of its sequences fit a round of short ones (the groups of
// a warp have to have one at the same time), whatever the number of sequences.
// Measured on both sides of that line, groups in step against each on its own
// (time of decompressing / a pipelined / a shared scan of 8M rows): 90 to 100 %
// short 0.88 to 1.02 / 0.75 to 0.84 / 0.80 to 0.96; up to 23 % short 0.96 to
// 1.16 / 1.02 to 1.12 / 1.02 to 1.09.
enum class LzGroups { kEither, kAlone, kInStep };  // the decoders an instance holds

// nseg segments (block segments j0 ..; entries at seg) by the tid-th of NT
// threads, 1 << glog lanes each, from the words A on; segment t goes to buf + t *
// (seg_rows + pad).  Records an error in *err.  (Each decoder with a loop of its
// own: with one loop around both, a shared scan of long sequences took 5 % more.)
template <LzGroups LZ = LzGroups::kEither>
__device__ __forceinline__ void lz4_segs(bool steps, uint32_t tid, uint32_t NT, uint32_t glog, uint32_t j0,
                                         uint32_t nseg, uint32_t rows, uint32_t seg_rows,
                                         const uint32_t* __restrict__ A, uint32_t wbase, uint32_t lo, uint32_t hi,
                                         uint32_t block_end, const uint32_t* seg, uint32_t* buf, uint32_t pad,
                                         int* err) {
    const uint32_t G = 1u << glog, gl = tid & (G - 1u), lane = tid & 31u;
    if (LZ == LzGroups::kInStep || (LZ == LzGroups::kEither && steps)) {
        for (uint32_t t0 = (tid & ~31u) >> glog; t0 < nseg; t0 += (NT >> glog)) {  // whole warps go round together
            const uint32_t t = t0 + (lane >> glog);
            const bool in = t < nseg;
            const uint32_t ts = in ? t : 0u, K = min(seg_rows, rows - (j0 + ts) * seg_rows);
            const int r2 = lz4_seg_step(A, wbase, lo, hi, block_end, seg[2 * ts], seg[2 * ts + 1], K,
                                        buf + ts * (seg_rows + pad), gl, G, in);
            if (r2 && gl == 0) *err = r2;
        }
    } else {
        const uint32_t gmask = G >= 32 ? 0xFFFFFFFFu : (((1u << G) - 1u) << (lane & ~(G - 1u)));
        for (uint32_t t = tid >> glog; t < nseg; t += (NT >> glog)) {
            const uint32_t K = min(seg_rows, rows - (j0 + t) * seg_rows);
            const int r2 = lz4_seg_group(A, wbase, lo, hi, block_end, seg[2 * t], seg[2 * t + 1], K,
                                         buf + t * (seg_rows + pad), gl, G, gmask);
            if (r2 && gl == 0) *err = r2;
        }
    }
}

// ---- one lane per segment, from staged bytes
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// 4 bytes at shared-memory address a, any alignment.
__device__ __forceinline__ uint32_t lds32u(uint32_t a) {
    const uint32_t b = a & ~3u;
    return __funnelshift_r(lds32(b), lds32(b + 4), a * 8);  // (the shift counts modulo 32)
}
// Decodes one segment of a segmented LZ4 block per lane, two output words of a
// sequence per round, for segments of many short sequences.  p = shared-memory address of
// the byte at the segment's entry position, hi and block_end those of the ends
// of the staged range and of the block; info and K as in lz4_seg_step; out =
// shared-memory address of the segment's words (segments a multiple of four
// words apart, not of 32: neighbouring lanes store to different banks).
// Called by whole warps (active = false: no segment).  Returns false on a
// corrupt stream.
// Why: a sequence of small integers is a word or two long, so the work is the
// parse of its header, whichever lanes are idle.  With a group of 4 lanes per
// segment (lz4_seg_step) a warp parses 8 at a time, with one lane up to 32; a
// header's token and offset are read at once (the offset's place follows from
// the token), conditions are combined without branches, and literal and match
// words take one path, so that the lanes stay together.  Length extensions of
// more than two bytes: a match ends in its segment of at most 128 words and has
// none; literals of more than 131 words go on past the segment, which ends in
// them, so that they are left to the end (read in the loop, they cost it 2 %).
__device__ __forceinline__ bool lz4_seg_lane(uint32_t p, uint32_t hi, uint32_t block_end, uint32_t info, uint32_t K,
                                             uint32_t out, bool active) {
    uint32_t L = 0, M = 0;      // literal and match words left of the sequence
    uint32_t lp = p, src = out; // where they are
    uint32_t bad = p > hi ? 1u : 0u;
    constexpr uint32_t kLong = 1u << 31;  // a literal run of more words than the segment has left
    // the match of a sequence whose token nibble is mn and whose literals end at
    // q, L words from output word k on; p = the next token
    auto match = [&](uint32_t q, uint32_t mn, uint32_t k) {
        const uint32_t y = lds32u(min(q, hi)), off = y & 0xFFFFu, rem = K - k;
        uint32_t ml = mn + 4, q2 = q + 2, b = 0;
        if (mn == 15) {
            const uint32_t e = (y >> 16) & 255u, f = e == 255u ? y >> 24 : 0u;
            ml += e + f;
            q2 += e == 255u ? 2u : 1u;
            b = f == 255u ? 1u : 0u;
        }
        M = ml >> 2;
        b |= (q == block_end ? 1u : 0u) | (q2 > hi ? 1u : 0u) | ((off | ml) & 3u) | (off - 1u >= 4 * (k + L) ? 1u : 0u) |
             (M > rem - L ? 1u : 0u);
        bad |= L < rem ? b : 0u;  // (else the segment ends inside or right after the literals)
        src = out + 4 * L - off;
        p = q2;
    };
    if (info & 16u) {  // the segment starts inside a sequence
        const uint32_t lit = info >> 5;
        L = lit >> 2;
        bad |= (lit & 3u) | (p + 4 * min(L, K) > hi ? 1u : 0u);
        L = min(L, K);
        if (active && !bad) match(p + 4 * L, info & 15u, 0);
    }
    bool run = active && !bad;
    uint32_t k = 0;
    while (__any_sync(0xFFFFFFFFu, run)) {
        if (run && (L | M) == 0) {
            const uint32_t x = lds32u(p), tok = x & 255u;
            uint32_t lit = tok >> 4, q = p + 1;
            bad = p >= hi ? 1u : 0u;
            if (lit == 15) {
                const uint32_t e = (x >> 8) & 255u, f = e == 255u ? (x >> 16) & 255u : 0u;
                lit += e + f;
                q += e == 255u ? 2u : 1u;
                bad |= f == 255u ? kLong : 0u;
            }
            lp = q;
            L = min(lit >> 2, K - k);
            bad |= (lit & 3u) | (q + 4 * L > hi ? 1u : 0u);
            match(q + lit, tok & 15u, k);
            run = bad == 0;
        }
        if (run) {
            // (a segment that ends inside a sequence's literals has M words it does not take)
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i) {
                const bool lt = L != 0;
                if ((lt || M != 0) && k < K) {
                    sts32(out, lds32u(lt ? lp : src));
                    lp += lt ? 4u : 0u;
                    src += lt ? 0u : 4u;
                    L -= lt ? 1u : 0u;
                    M -= lt ? 0u : 1u;
                    out += 4;
                    ++k;
                }
            }
            run = k < K;
        }
    }
    if (bad & kLong) {  // the segment ends in it: the rest of its length, then words to the end
        uint32_t lit = 15 + 255 + 255, f = 255;
        while (f == 255u && lp < hi) {
            f = lds32u(lp) & 255u;
            lit += f;
            ++lp;
        }
        bad = (f == 255u ? 1u : 0u) | (lit & 3u) | (lp + 4 * (K - k) > hi ? 1u : 0u);
        if (!bad)
            for (; k < K; ++k, lp += 4, out += 4) sts32(out, lds32u(lp));
    }
    return !active || bad == 0;
}

// log2 of the lanes per segment for `nseg` segments on NT threads: the
// largest power of two G <= 32 with nseg * G <= NT (at least 1).
__device__ __forceinline__ uint32_t seg_group_log2(uint32_t nseg, uint32_t NT) {
    const uint32_t q = nseg ? NT / nseg : NT;
    return q <= 1 ? 0u : min(5u, 31u - (uint32_t)__clz(q));
}

// ------------------------------------------------ generic LZ4, one warp
// Decodes a complete LZ4 block (any conforming encoder, byte granular) into
// `out` (out_size bytes expected).  All 32 lanes call it; every lane sees the
// same control flow.  Returns 0 or kErrCorrupt (uniform across the warp).
template <class Src>
__device__ __noinline__ int lz4_warp_block(const Src in, uint32_t in_size, uint8_t* __restrict__ out,
                                           uint32_t out_size, uint32_t lane) {
    uint32_t pos = 0, o = 0;
    int err = 0;
    while (true) {
        if (pos >= in_size) { err = kErrCorrupt; break; }
        uint32_t tok = in.b(pos++);
        uint32_t lit = tok >> 4;
        if (lit == 15) {
            uint32_t b;
            do {
                if (pos >= in_size) { err = kErrCorrupt; break; }
                b = in.b(pos++);
                lit += b;
            } while (b == 255);
            if (err) break;
        }
        if ((uint64_t)pos + lit > in_size || (uint64_t)o + lit > out_size) { err = kErrCorrupt; break; }
        for (uint32_t i = lane; i < lit; i += 32) out[o + i] = (uint8_t)in.b(pos + i);
        o += lit;
        pos += lit;
        if (pos == in_size) break;  // last sequence: literals only
        if (pos + 2 > in_size) { err = kErrCorrupt; break; }
        uint32_t off = in.b(pos) | (in.b(pos + 1) << 8);
        pos += 2;
        uint32_t ml = (tok & 15u) + 4;
        if ((tok & 15u) == 15) {
            uint32_t b;
            do {
                if (pos >= in_size) { err = kErrCorrupt; break; }
                b = in.b(pos++);
                ml += b;
            } while (b == 255);
            if (err) break;
        }
        if (off == 0 || off > o || (uint64_t)o + ml > out_size) { err = kErrCorrupt; break; }
        __syncwarp();
        const uint32_t src = o - off;
        if (off >= ml) {
            for (uint32_t i = lane; i < ml; i += 32) out[o + i] = out[src + i];
        } else {
            for (uint32_t i = lane; i < ml; i += 32) out[o + i] = out[src + (i % off)];
        }
        __syncwarp();
        o += ml;
    }
    __syncwarp();
    if (!err && o != out_size) err = kErrCorrupt;
    return err;
}

// ------------------------------------------------------ block-wide scans
// Barrier of a group of NT threads: BAR == 0 is the whole CTA
// (__syncthreads), otherwise named barrier BAR of exactly NT threads (the
// consumer warps of a warp-specialised kernel).
template <int NT, int BAR>
__device__ __forceinline__ void grp_sync() {
    if constexpr (BAR == 0) {
        __syncthreads();
    } else {
        asm volatile("bar.sync %0, %1;" ::"n"(BAR), "n"(NT) : "memory");
    }
}

// Inclusive scan (wrapping uint32 addition) of a[0..n) in shared memory by
// the NT threads of a group (tid = index in the group); thread t owns the
// contiguous range [t*per, (t+1)*per).  `tmp` has >= NT/32 words.  Must be
// called by all NT threads.
template <int NT, int BAR = 0>
__device__ __forceinline__ void block_inclusive_scan(uint32_t* a, uint32_t n, uint32_t* tmp,
                                                     uint32_t tid = threadIdx.x) {
    const uint32_t lane = tid & 31, warp = tid >> 5;
    const uint32_t per = (n + NT - 1) / NT;
    const uint32_t b = min(n, tid * per), e = min(n, b + per);
    uint32_t s = 0;
    for (uint32_t i = b; i < e; ++i) s += a[i];
    uint32_t x = s;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
        if (lane >= (uint32_t)d) x += y;
    }
    if (lane == 31) tmp[warp] = x;
    grp_sync<NT, BAR>();
    if (warp == 0) {
        uint32_t w = lane < NT / 32 ? tmp[lane] : 0;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, d);
            if (lane >= (uint32_t)d) w += y;
        }
        if (lane < NT / 32) tmp[lane] = w;
    }
    grp_sync<NT, BAR>();
    uint32_t run = (x - s) + (warp ? tmp[warp - 1] : 0);
    for (uint32_t i = b; i < e; ++i) {
        run += a[i];
        a[i] = run;
    }
    grp_sync<NT, BAR>();
}

// ------------------------------------------------------- cascaded pages
__device__ __forceinline__ bool casc_header_ok(const casc_hdr& h, uint32_t pg_bytes, uint32_t rows) {
    const bool rle = (h.flags & CASC_RLE) != 0;
    if (pg_bytes < 32 || h.n_rows != rows || h.val_bits > 32 || h.len_bits > 32) return false;
    if (rle ? (h.n_runs == 0 || h.n_runs > kCascPageMaxRuns) : h.n_runs != rows) return false;
    if (h.vals_off < 32 || (h.vals_off & 3) ||
        (uint64_t)h.vals_off + 4ull * (((uint64_t)h.n_runs * h.val_bits + 31) / 32 + 1) > pg_bytes)
        return false;
    if (rle && ((h.lens_off & 3) || h.lens_off < 32 ||
                (uint64_t)h.lens_off + 4ull * (((uint64_t)h.n_runs * h.len_bits + 31) / 32 + 1) > pg_bytes))
        return false;
    return true;
}

// Header of a page (16-byte aligned; global or shared memory).
__device__ __forceinline__ casc_hdr casc_load_header(const uint8_t* pg) {
    const uint4* hw = (const uint4*)pg;
    const uint4 a = hw[0], b = hw[1];
    casc_hdr h;
    h.n_rows = a.x;
    h.n_runs = a.y;
    h.flags = (uint8_t)(a.z & 255u);
    h.val_bits = (uint8_t)((a.z >> 8) & 255u);
    h.len_bits = (uint8_t)((a.z >> 16) & 255u);
    h.pad = (uint8_t)(a.z >> 24);
    h.first = (int32_t)a.w;
    h.val_base = (int32_t)b.x;
    h.len_base = b.y;
    h.vals_off = b.z;
    h.lens_off = b.w;
    return h;
}

// Decodes one cascaded page of `rows` rows (<= kCascPageRows; global or
// shared memory, 16-byte aligned) into out[0..rows) in shared memory, plain
// row order.  RLE pages go through run tables run_val / run_end (shared,
// kCascPageMaxRuns entries each): run values (with a delta scan), run ends
// (an inclusive scan of the lengths), then each thread expands a contiguous
// range of rows from the run that holds its first row (binary search).
// Called by the NT threads of a group (barrier BAR, tid = index in the
// group).  Returns 0 or kErrCorrupt (uniform over the group).
// With FINAL_SYNC false the values are complete only after the caller's
// next barrier of the group (callers that place one right after save one).
template <int NT, int BAR = 0, bool FINAL_SYNC = true>
__device__ __forceinline__ int casc_decode_page(const uint8_t* __restrict__ pg, uint32_t pg_bytes, uint32_t rows,
                                                int32_t* out, int32_t* run_val, uint32_t* run_end, uint32_t* tmp,
                                                uint32_t tid = threadIdx.x) {
    if (pg_bytes < 32) return kErrCorrupt;
    const casc_hdr h = casc_load_header(pg);
    if (!casc_header_ok(h, pg_bytes, rows)) return kErrCorrupt;
    const bool rle = (h.flags & CASC_RLE) != 0, delta = (h.flags & CASC_DELTA) != 0;
    const uint32_t* vw = (const uint32_t*)(pg + h.vals_off);
    if (!rle) {
        for (uint32_t i = tid; i < rows; i += NT)
            out[i] = (int32_t)((i == 0 && delta) ? 0u : unpack_bits(vw, i, h.val_bits) + (uint32_t)h.val_base);
        if (delta) {
            grp_sync<NT, BAR>();
            block_inclusive_scan<NT, BAR>((uint32_t*)out, rows, tmp, tid);
            for (uint32_t i = tid; i < rows; i += NT) out[i] = (int32_t)((uint32_t)out[i] + (uint32_t)h.first);
        }
        if (FINAL_SYNC) grp_sync<NT, BAR>();
        return 0;
    }
    const uint32_t nr = h.n_runs;
    const uint32_t* lw = (const uint32_t*)(pg + h.lens_off);
    if (nr <= 32) {
        // few runs (sorted or low-cardinality pages): one warp builds the run
        // table with shuffle scans, one barrier publishes it
        if (tid < 32) {
            const bool in = tid < nr;
            uint32_t v = in ? ((tid == 0 && delta) ? 0u : unpack_bits(vw, tid, h.val_bits) + (uint32_t)h.val_base) : 0u;
            uint32_t e = in ? unpack_bits(lw, tid, h.len_bits) + h.len_base : 0u;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t pv = __shfl_up_sync(0xFFFFFFFFu, v, d), pe = __shfl_up_sync(0xFFFFFFFFu, e, d);
                if (tid >= (uint32_t)d) {
                    if (delta) v += pv;
                    e += pe;
                }
            }
            if (in) {
                run_val[tid] = (int32_t)(delta ? v + (uint32_t)h.first : v);
                run_end[tid] = e;
            }
        }
        grp_sync<NT, BAR>();
    } else {
        for (uint32_t i = tid; i < nr; i += NT) {
            run_val[i] = (int32_t)((i == 0 && delta) ? 0u : unpack_bits(vw, i, h.val_bits) + (uint32_t)h.val_base);
            run_end[i] = unpack_bits(lw, i, h.len_bits) + h.len_base;
        }
        grp_sync<NT, BAR>();
        if (delta) {
            block_inclusive_scan<NT, BAR>((uint32_t*)run_val, nr, tmp, tid);
            for (uint32_t i = tid; i < nr; i += NT) run_val[i] = (int32_t)((uint32_t)run_val[i] + (uint32_t)h.first);
        }
        block_inclusive_scan<NT, BAR>(run_end, nr, tmp, tid);
    }
    if (run_end[nr - 1] != rows) return kErrCorrupt;  // uniform: every thread reads the same word
    const uint32_t per = (rows + NT - 1) / NT;
    const uint32_t r_begin = min(rows, tid * per), r_stop = min(rows, r_begin + per);
    if (r_begin < r_stop) {
        uint32_t lo = 0, hi = nr - 1;  // first run ending after r_begin
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (run_end[mid] <= r_begin) lo = mid + 1; else hi = mid;
        }
        uint32_t k = lo, e = run_end[k];
        int32_t v = run_val[k];
        for (uint32_t r = r_begin; r < r_stop; ++r) {
            while (r >= e && k + 1 < nr) {
                ++k;
                e = run_end[k];
                v = run_val[k];
            }
            out[r] = v;
        }
    }
    if (FINAL_SYNC) grp_sync<NT, BAR>();
    return 0;
}

// --------------------------------------------------------- join tables
__device__ __forceinline__ bool ht_probe(const uint64_t* __restrict__ slots, uint32_t log2cap, int32_t key,
                                         int32_t* payload) {
    if (key == kEmptyKey) return false;
    const uint32_t mask = (1u << log2cap) - 1;
    uint32_t s = hash_key32(key, log2cap);
    for (uint32_t i = 0; i <= mask; ++i) {
        uint64_t e = __ldg((const unsigned long long*)slots + s);
        int32_t k = (int32_t)(uint32_t)e;
        if (k == key) {
            *payload = (int32_t)(uint32_t)(e >> 32);
            return true;
        }
        if (k == kEmptyKey) return false;
        s = (s + 1) & mask;
    }
    return false;
}

// Bucketized layout: 2^log2cap slots grouped in buckets of 8 (64 bytes); a
// key hashes to a bucket, is placed in its first free slot, and spills to
// the next bucket when the bucket is full.
constexpr uint32_t kBucketSlots = 8;

__device__ __forceinline__ bool ht_probe_bucket(const uint64_t* __restrict__ slots, uint32_t log2cap, int32_t key,
                                                int32_t* payload) {
    if (key == kEmptyKey || log2cap < 3) return false;
    const uint32_t lb = log2cap - 3, bmask = (1u << lb) - 1;
    uint32_t bkt = hash_key32(key, lb);
    for (uint32_t i = 0; i <= bmask; ++i) {
        const ulonglong2* bp = (const ulonglong2*)(slots + (size_t)bkt * kBucketSlots);
        const ulonglong2 a = __ldg(bp), b = __ldg(bp + 1), c = __ldg(bp + 2), d = __ldg(bp + 3);
        const unsigned long long e[8] = {a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y};
        bool any_empty = false;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int32_t k = (int32_t)(uint32_t)e[j];
            if (k == key) {
                *payload = (int32_t)(uint32_t)(e[j] >> 32);
                return true;
            }
            any_empty |= (k == kEmptyKey);
        }
        if (any_empty) return false;
        bkt = (bkt + 1) & bmask;
    }
    return false;
}

// Dense layout: slot 0 = {base, span}; the key's entry at slot 1 + (key - base).
__device__ __forceinline__ bool ht_probe_dense(const uint64_t* __restrict__ slots, int32_t key, int32_t* payload) {
    const uint64_t h = __ldg((const unsigned long long*)slots);
    const uint32_t u = (uint32_t)key - (uint32_t)h;
    if (key == kEmptyKey || u >= (uint32_t)(h >> 32)) return false;
    const uint64_t e = __ldg((const unsigned long long*)slots + 1 + u);
    if ((int32_t)(uint32_t)e != key) return false;
    *payload = (int32_t)(uint32_t)(e >> 32);
    return true;
}

__device__ __forceinline__ bool ht_probe_any(const uint64_t* __restrict__ slots, uint32_t log2cap, uint32_t layout,
                                             int32_t key, int32_t* payload) {
    if (layout == GX_HT_DENSE) return ht_probe_dense(slots, key, payload);
    return layout ? ht_probe_bucket(slots, log2cap, key, payload) : ht_probe(slots, log2cap, key, payload);
}

// A join-table probe of R rows per lane (hdr: a dense table's header): rows whose bit
// in m is set and whose key is found keep their bit, with their payload in
// pay.  All rows' reads of a round are in flight together, a round reads two
// neighbouring slots (16 bytes, one sector) and goes on with the rows whose
// chain is not settled.  The three layouts are one walk: linear tables from
// the key's hash slot, bucket tables from the first slot of its bucket (keys
// fill a bucket's slots in order, then the next bucket's), dense tables one
// slot.  A pair's slot before the key's own can hold the key only in a dense
// table's header (its base), so the slot at or after it is preferred.
template <uint32_t R>
__device__ __forceinline__ uint32_t ht_probe_rows(const uint64_t* __restrict__ ht, uint32_t log2cap, uint32_t lay,
                                                  uint64_t hdr, const uint32_t (&v)[R], uint32_t m,
                                                  uint32_t (&pay)[R], uint64_t pol) {
    const uint32_t mask = (1u << log2cap) - 1u;
    const bool dense = lay == GX_HT_DENSE;
    uint32_t slot[R];
#pragma unroll
    for (uint32_t r = 0; r < R; ++r) {
        bool out = v[r] == (uint32_t)kEmptyKey;
        if (dense) {
            const uint32_t u = v[r] - (uint32_t)hdr;
            out = out || u >= (uint32_t)(hdr >> 32);
            slot[r] = 1u + u;
        } else if (lay == GX_HT_BUCKET) {
            slot[r] = hash_key32((int32_t)v[r], log2cap - 3) * kBucketSlots;
        } else {
            slot[r] = hash_key32((int32_t)v[r], log2cap);
        }
        if (out) m &= ~(1u << r);
    }
    uint32_t u = m;  // rows whose chain is not settled
#pragma unroll 1
    for (uint32_t t = 0; u && t <= mask / 2 + 1; ++t) {
        ulonglong2 e[R];
#pragma unroll
        for (uint32_t r = 0; r < R; ++r) {
            asm("" : "=l"(e[r].x), "=l"(e[r].y));  // rows not read keep any value: masked below
            if ((u >> r) & 1u)
                asm("ld.global.nc.L2::cache_hint.v2.b64 {%0, %1}, [%2], %3;"
                    : "=l"(e[r].x), "=l"(e[r].y)
                    : "l"(ht + (slot[r] & ~1u)), "l"(pol));
        }
#pragma unroll
        for (uint32_t r = 0; r < R; ++r) {
            const uint32_t bit = 1u << r, kx = (uint32_t)e[r].x, ky = (uint32_t)e[r].y;
            const bool hit = kx == v[r] || ky == v[r];
            const bool open = !hit && !dense && ky != (uint32_t)kEmptyKey &&
                              (kx != (uint32_t)kEmptyKey || (slot[r] & 1u));
            if ((u & bit) && hit) pay[r] = ky == v[r] ? (uint32_t)(e[r].y >> 32) : (uint32_t)(e[r].x >> 32);
            if ((u & bit) && !hit && !open) m &= ~bit;
            if (!open) u &= ~bit;
            slot[r] = ((slot[r] | 1u) + 1u) & mask;
        }
    }
    return m & ~u;
}

// --------------------------------------------------------- group tables
// Global open-addressing group table: keys int64 (kEmptyGroup = free), sums int64.
__device__ __forceinline__ bool group_add_global(int64_t* keys, int64_t* sums, uint32_t log2cap, int64_t key,
                                                 int64_t v) {
    const uint32_t mask = (1u << log2cap) - 1;
    uint32_t s = hash_key64(key, log2cap);
    for (uint32_t i = 0; i <= mask; ++i) {
        // A slot's key is written once (free -> key) and never changes, so a plain
        // (possibly cached, possibly stale) read that shows a key is final: the
        // common case -- the key already there -- costs a read and a fire-and-forget
        // add, and only a slot that reads free takes the compare-and-swap.
        long long cur;
        asm volatile("ld.global.ca.b64 %0, [%1];" : "=l"(cur) : "l"(keys + s));
        if (cur == (long long)key) {
            atomicAdd((unsigned long long*)&sums[s], (unsigned long long)v);
            return true;
        }
        if (cur == (long long)kEmptyGroup) {
            const unsigned long long old = atomicCAS((unsigned long long*)&keys[s], (unsigned long long)kEmptyGroup,
                                                     (unsigned long long)key);
            if (old == (unsigned long long)kEmptyGroup || old == (unsigned long long)key) {
                atomicAdd((unsigned long long*)&sums[s], (unsigned long long)v);
                return true;
            }
        }
        s = (s + 1) & mask;
    }
    return false;
}

// Shared-memory partial group table (uint32 keys).  Returns false when full.
__device__ __forceinline__ bool group_add_smem(uint32_t* keys, unsigned long long* sums, uint32_t log2cap,
                                               uint32_t key, uint64_t v) {
    const uint32_t mask = (1u << log2cap) - 1;
    uint32_t s = hash_key32((int32_t)key, log2cap);
    for (uint32_t i = 0; i <= mask; ++i) {
        uint32_t old = atomicCAS(&keys[s], kEmptyGKey, key);
        if (old == kEmptyGKey || old == key) {
            atomicAdd(&sums[s], (unsigned long long)v);
            return true;
        }
        s = (s + 1) & mask;
    }
    return false;
}

// Sum of a 64-bit value over all 32 lanes (non-members pass 0).  Exact:
// four 16-bit limbs are reduced separately and recombined modulo 2^64.
__device__ __forceinline__ uint64_t warp_sum_u64(uint64_t u) {
    uint32_t p0 = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)(u & 0xFFFF));
    uint32_t p1 = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)((u >> 16) & 0xFFFF));
    uint32_t p2 = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)((u >> 32) & 0xFFFF));
    uint32_t p3 = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)(u >> 48));
    return (uint64_t)p0 + ((uint64_t)p1 << 16) + ((uint64_t)p2 << 32) + ((uint64_t)p3 << 48);
}

}  // namespace gx
