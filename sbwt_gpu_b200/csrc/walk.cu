// walk.cu -- the forward walk: searches of batches of reads (and of the runs of
// a positions array) by walking each run of consecutive k-mers from left to
// right.  Same answers as the reference's per-k-mer search
// (include/gpu/search_kernel.hpp:61-104); no reference counterpart.
//
// What is known of a run decides how its next k-mers are found:
//  * probe: a k-mer with a q-mer (q letters, by the index's size: walk_q, 16
//    and k at most) that no indexed k-mer contains is absent, and so is every
//    other k-mer that contains that q-mer.  One bit per possible q-mer
//    (WalkView.qbits, L2-resident) tells.  The q-mers are probed from the right
//    end of the k-mer, so that an absent one at offset o settles the o + 1
//    k-mers from the current one on; random letters are settled k-q+1 k-mers at
//    a time with no access to the index proper.
//  * lookup, when the probed q-mers are all present: the nodes whose labels end
//    with the k-mer's last p letters are the presearch interval of those
//    letters, and labels are sorted, so a search by halves over the keys of
//    that interval (one 32-byte group of four per step) finds the node or shows
//    that there is none: two or three gathers instead of k-p rank pairs.
//  * extend, from a found k-mer's node: the read's letters are compared with
//    those of the path through the node, 32 at a time, and the nodes of the
//    k-mers that match follow each other in memory: 4 bytes per k-mer read in
//    order, copied by the whole warp.
//  * step, where the letters or the path's segment end: the k-mer y.c after the
//    node v follows iff the group of v has an edge c, and its node is C[c] +
//    rank_c of that group's first column (one line, one word of group marks).
//    Without an edge the letter is in no indexed k-mer after those before it,
//    so the next probes take the q-mers that contain it.
//
// Probing and walking alternate in phases, each with (nearly) all lanes of a
// warp busy on the same code: probing until a batch of runs has passed, then
// looking up, stepping and extending those; runs change hands in a pool in
// shared memory.  One loop in which every lane had its own state ran all of the
// bodies each time, for 12 active lanes on average, and was 1.6 times slower.
#include <algorithm>

#include "device.cuh"
#include "internal.h"
#include "launch.cuh"
#include "mlp_kernels.cuh"
#include "rank.cuh"
#include "stream.cuh"

namespace sbwt {
namespace {

using namespace dev;

constexpr u32 kFull = 0xffffffffu;
constexpr u32 kWarps = 4;  // 128-thread blocks
// A warp's pool of runs in progress, in shared memory: runs to probe grow from
// its start, runs to look up or step from its end.  Runs enter only when fewer
// than 32 wait to be probed (32 at most), with 32 in the lanes and fewer
// than kBatch waiting for a walk: 31 + 32 + 32 + kBatch - 1 <= kPool.
constexpr u32 kBatch = 32;
constexpr u32 kPool = 96 + kBatch;
constexpr u32 kTake = 8;     // idle lanes that take new runs to probe
// Stretches of at most so many answers are copied by their lanes, all at once; longer ones by the whole warp, one after
// the other.  In the smallest batches every stretch is one k-mer: 16 reads, 18.4 -> 13.5 us (2, 4 and 8 alike).  Two
// or four long stretches at a time gave nothing and took registers (10 blocks per SM instead of 12).
constexpr u32 kOwn = 4;
constexpr u32 kPiece = 256;  // k-mers per run at most: reads of 250 letters stay whole
// Batches of fewer k-mers are filled with absent answers by the walk itself: the fill kernel's launch would cost
// more than it gains.
constexpr u64 kFillAhead = 8ull << 20;

// What is left of one run: k-mer j (letters from pos on) and `left` k-mers
// after it.  hint: 0, or 1 + offset in k-mer j of the letter that ended the
// stretch found last.  at: 0, or the path position of k-mer j if its letters go
// on along the path of that stretch (after a substituted letter they do).
template <class IX> struct Run {
    IX pos, j;
    uint16_t left, hint;
    u32 at;
};

// Node of a k-mer (first letter at the top, letters past k ignored), or kNoNode.
__device__ __forceinline__ u32 lookup(const SearchArgs &a, u64 kmer) {
    const u32 k = a.k, p = a.p;
    u32 l = 0, r = a.wv.n - 1u;
    if (p) {
        const u64 idx = (kmer >> (64u - 2u * k)) & ((1ull << (2u * p)) - 1ull);  // its last p letters
        const uint2 e = ld_gather_u32x2(static_cast<const uint2 *>(a.pre) + idx, a.ef_pre, l2_evict_first_policy());
        l = e.x;
        r = e.y;
        if (l > r) return kNoNode;
    }
    const u64 key = letters_reverse(kmer) << (64u - 2u * k) | (k < 32u ? 1ull : 0ull);
    for (;;) {
        // the group of four keys in the middle of [l, r]; keys ascend over all columns
        const u32 g = (l + (r - l) / 2u) & ~3u;
        const ulonglong4 w = ld_line(reinterpret_cast<const ulonglong4 *>(a.wv.labels + g));
        if (key < w.x) {
            if (g <= l) return kNoNode;
            r = g - 1u;
        } else if (key > w.w) {
            if (g + 3u >= r) return kNoNode;
            l = g + 4u;
        } else {
            if (key != w.x && key != w.y && key != w.z && key != w.w) return kNoNode;
            u32 v = g + (key == w.w ? 3u : key == w.z ? 2u : key == w.y ? 1u : 0u);
            if (k == 32u) {  // keys have no room for the bit of labels without $: the last equal one has none, or all do
                v = min(v, a.wv.n - 1u);  // the padding equals the key of 32 T
                while (v + 1u < a.wv.n && __ldg(a.wv.labels + v + 1u) == key) v++;
                if (__ldg(a.wv.labels + v) != key || !((__ldg(a.sv.node + (v >> 1)) >> ((v & 1u) << 2)) & 7u))
                    return kNoNode;
            }
            return v;
        }
    }
}

// The 32 letters of the batch from pos on (search_kernel.hpp:66-68).
__device__ __forceinline__ u64 letters_at(const SearchArgs &a, u64 pos) {
    const u64 b = min(pos, a.max_pos) << 1;
    const u64 w0 = __ldg(a.words + (b >> 6)), w1 = __ldg(a.words + (b >> 6) + 1);
    const u32 sh = (u32)(b & 63u);
    return (w0 << sh) | (shr_clamp(w1, 63u - sh) >> 1);
}

// Node of the k-mer that follows the k-mer of node v with letter c, or kNoNode.
__device__ __forceinline__ u32 step(const SearchArgs &a, const LinesRanker &rk, const u32 *C, u32 v, u32 c) {
    const ulonglong4 *lines = rk.lines + (u64)c * rk.lpc;
    const u32 line = v / kLineBits;
    ulonglong4 w = ld_line(lines + line);
    const u32 u0 = group_start(__ldg(a.wv.marks + v / kMarkCols), v);
    const u32 line0 = u0 / kLineBits;
    if (line0 != line) w = ld_line(lines + line0);
    u32 bit;
    const u32 x = sums_rank(line_sums(w), u0 - line0 * kLineBits, bit);
    return bit ? C[c] + x : kNoNode;
}

// How many of the path's nodes from position i on follow the read's letters from
// pos on, in the same segment, at most `limit`.  closed: the letter after them
// continues no indexed k-mer.
__device__ __forceinline__ u32 extend(const SearchArgs &a, u32 i, u64 pos, u32 limit, bool &closed) {
    u32 n = 0;
    closed = false;
    while (n < limit) {
        const u32 sh = (i + n) & 31u;
        const ulonglong2 b = ld_nc2(a.wv.path + ((i + n) >> 5));
        const u64 diff = (b.x << (2u * sh)) ^ letters_at(a, pos + n);
        const u32 same = min((u32)__clzll((long long)diff) >> 1, 32u - sh);
        const u32 good = min(same, (u32)__clz((int)((u32)(b.y >> 32) << sh)));
        n += good;
        if (good < 32u - sh) {
            closed = n < limit && !((b.y >> (31u - sh - good)) & 1u);
            break;
        }
    }
    return min(n, limit);
}

// Whether path position x is the node of this k-mer: the k path letters up to x are its own and follow each other.
__device__ __forceinline__ bool on_path(const SearchArgs &a, u32 x, u64 kmer) {
    const u32 k = a.k;
    if (x < k - 1u || x >= a.wv.n) return false;
    const u32 i = x - (k - 1u), sh = i & 31u;
    const ulonglong2 b0 = ld_nc2(a.wv.path + (i >> 5)), b1 = ld_nc2(a.wv.path + (i >> 5) + 1);
    const u64 letters = (b0.x << (2u * sh)) | (shr_clamp(b1.x, 63u - 2u * sh) >> 1);
    const u32 starts = __funnelshift_l((u32)(b1.y >> 32), (u32)(b0.y >> 32), sh);
    return ((letters ^ kmer) >> (64u - 2u * k)) == 0 && ((starts << 1) >> (33u - k)) == 0;
}

// 16 letters from pos on (at least the first `need`), the first at the top: from half words of 16 letters, a
// word's first half at the higher address; the third half word is read only where `need` letters reach into it.
template <class IX>
__device__ __forceinline__ u32 half_words(const SearchArgs &a, IX pos, u32 need) {
    const u32 sh = (u32)(pos & 15u);
    const uint2 w = __ldg(reinterpret_cast<const uint2 *>(a.words) + (pos >> 5));
    u32 x = w.y, y = w.x;
    if (pos & 16u) {
        x = w.x;
        if (sh + need > 16u) y = __ldg(reinterpret_cast<const u32 *>(a.words) + 2u * ((pos >> 5) + 1u) + 1u);
    }
    return __funnelshift_l(y, x, 2u * sh);
}

__device__ __forceinline__ bool q_present(const SearchArgs &a, u32 code) {
    return (__ldg(a.wv.qbits + (code >> 5)) >> (code & 31u)) & 1u;
}

// Bits j .. j + count - 1 of the membership bitmap.
__device__ __forceinline__ void set_bits(uint32_t *member, u64 j, u32 count) {
    for (;;) {
        const u32 b = (u32)j & 31u, c = min(count, 32u - b);
        atomicOr(member + (j >> 5), (kFull >> (32u - c)) << b);
        if (count == c) return;
        j += c;
        count -= c;
    }
}

// IX: type of the k-mer and letter indices (u32 where the batch allows it, run32_ok).  12 blocks per SM (40 registers)
// for u32: 1M own reads, membership only, 323 us against 347 at 10; 14 blocks (36 registers) within 2 % either way.
// The u64 form would spill there.
template <class IX>
__global__ void __launch_bounds__(kWarps * 32, sizeof(IX) == 4 ? 12 : 10) walk_kernel(const LinesRanker rk, const SearchArgs a) {
    // kernel contract: the run count is on the device; too few runs and the per-k-mer search takes the call
    const u64 n_rows = a.runs_dev ? *a.runs_dev : a.n_rows;
    if (a.runs_dev && !runs_usable(n_rows, a.n_kmers)) return;
    __shared__ Run<IX> pools[kWarps][kPool];
    __shared__ u32 sC[4];
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const u32 lt = (1u << lane) - 1u;
    const u32 k = a.k;
    if (threadIdx.x < 4) sC[threadIdx.x] = (u32)a.C[threadIdx.x];
    __syncthreads();
    const IX n_eff = (IX)min(a.n_kmers, a.kstart[n_rows]);
    Run<IX> *const pool = pools[warp];
    u32 nr = 0, nw = 0;  // runs to probe, runs to walk (warp-uniform)
    bool more = true;
    IX cj = 0, ce = 0, crow = 0;  // the warp's chunk: next k-mer to cut into runs, end, a row at or before cj's

    for (;;) {
        // ======== probe: until kBatch runs wait for a walk, or none is left to probe
        {
            const u32 o_max = k - a.wv.q, qs = 32u - 2u * a.wv.q;
            const u32 two = a.wv.q < 16u ? 1u : 0u;  // 16 letters hold two q-mers
            // Rounds of a k-mer whose q-mers are present: its right end, its middle, its left end, so that no letter
            // of it stays unprobed: one substituted letter among the first k - 2 q costs two rounds instead of a failed
            // look-up for each k-mer that holds it.  Two rounds against three: 10,000 reads, half own, 77 and 65 us;
            // 230,000 uneven reads 1957 and 1805; 1M own reads, membership only, 323 and 302; four 69, 1845, 323.  In
            // the smallest batches a run is one k-mer, and a third round only waits (13.0 and 14.3 us for 16 reads).
            const u32 rounds = a.piece > 1u ? 3u : 2u;
            const IX max_pos = (IX)a.max_pos;
            bool act = false;
            IX pos = 0, J = 0;
            u32 left = 0, at = 0, hint = 0;
            u32 tries = 0;  // pairs of q-mers of k-mer J found present
            for (;;) {
                if (more && nr < 32u) {
                    if (cj >= ce) {
                        unsigned long long base = 0;
                        if (lane == 0) base = atomicAdd(a.counter, (unsigned long long)a.chunk);
                        base = __shfl_sync(kFull, base, 0);
                        if (base >= n_eff) {
                            more = false;
                        } else {
                            cj = (IX)base;
                            ce = (IX)min((u64)base + a.chunk, (u64)n_eff);
                            crow = a.chunk_row[base / a.chunk];
                            if (a.answers && !a.found_only && a.n_kmers < kFillAhead)
                                for (u64 t = base + lane; t < ce; t += 32u) a.answers[t] = ~0ull;
                            if (a.member)  // base is a multiple of 32
                                for (u64 t = base / 32u + lane; t < ((u64)ce + 31u) / 32u; t += 32u) a.member[t] = 0u;
                        }
                    }
                    if (more) {
                        // the next 32 rows' k-mers of the chunk, in equal pieces of at most a.piece k-mers:
                        // up to 32 pieces become runs
                        const IX r = crow + lane;
                        const IX ks = r < (IX)n_rows ? (IX)a.kstart[r] : ce;
                        const IX b0 = max(ks, cj), b1 = r < (IX)n_rows ? min((IX)a.kstart[r + 1], ce) : ce;
                        const u32 len = b0 < b1 ? (u32)(b1 - b0) : 0u;  // rows shorter than k hold no k-mers
                        const u32 np = (len + a.piece - 1u) / a.piece;
                        u32 inc = np;
#pragma unroll
                        for (u32 d = 1; d < 32u; d <<= 1) {
                            const u32 x = __shfl_up_sync(kFull, inc, d);
                            if (lane >= d) inc += x;
                        }
                        const u32 total = min(__shfl_sync(kFull, inc, 31), 32u);
                        u32 own = 0;  // the lane whose row holds piece `lane`
#pragma unroll
                        for (u32 d = 16; d; d >>= 1)
                            if (__shfl_sync(kFull, inc, own + d - 1u) <= lane) own += d;
                        own = min(own, 31u);
                        const u32 o_np = __shfl_sync(kFull, np, own), o_len = __shfl_sync(kFull, len, own);
                        const u32 idx = lane - (__shfl_sync(kFull, inc, own) - o_np);
                        const IX o_b0 = __shfl_sync(kFull, b0, own), o_ks = __shfl_sync(kFull, ks, own);
                        IX stop = 0;
                        if (lane < total) {
                            const u32 size = (o_len + o_np - 1u) / o_np;
                            const u32 from = min(idx * size, o_len), to = min(from + size, o_len);
                            stop = o_b0 + to;
                            const IX j = o_b0 + from;
                            pool[nr + lane] = Run<IX>{(IX)((IX)a.row_starts[crow + own] + (j - o_ks)), j,
                                                      (uint16_t)(to - from - 1u), 0, 0};
                        }
                        nr += total;
                        if (total) {
                            cj = __shfl_sync(kFull, stop, total - 1u);
                            crow += __shfl_sync(kFull, own, total - 1u);
                        } else {
                            crow += 32u;
                            if (crow >= (IX)n_rows) cj = ce;  // a row table that does not add up: never a wait for its rows
                        }
                    }
                    __syncwarp();
                    if (more && nr < 32u) continue;
                }
                const u32 idle = __ballot_sync(kFull, !act);
                const u32 take = min((u32)__popc(idle), nr);
                if (take >= kTake || (take && take == nr)) {
                    const u32 i = __popc(idle & lt);
                    if (!act && i < take) {
                        const Run<IX> e = pool[nr - 1u - i];
                        pos = e.pos;
                        J = e.j;
                        left = e.left;
                        hint = e.hint;
                        at = e.at;
                        tries = 0;
                        act = true;
                    }
                    nr -= take;
                    __syncwarp();
                } else if (idle == kFull) {
                    if (more) continue;
                    break;
                }
                // ---- one round: q-mers at offsets o and o - d of the current k-mer
                bool pass = false;
                if (act) {
                    // the letter that ended a stretch is in no indexed k-mer after those before it: the q-mers that
                    // hold it are probed from the right one on; otherwise the right end, the middle and the left end
                    const u32 last = hint ? min(hint - 1u, o_max) : o_max;
                    const u32 o = hint ? last - 2u * tries : tries == 0u ? o_max : tries == 1u ? o_max / 2u : min(two, o_max);
                    const u32 d = o ? two : 0u;
                    const u32 x = half_words(a, min(pos + (o - d), max_pos), a.wv.q + d);
                    u32 adv = o + 1u;
                    bool in = q_present(a, (x << (2u * d)) >> qs);
                    if (in) {
                        in = q_present(a, x >> qs);
                        adv -= d;
                    }
                    if (in) {
                        tries++;
                        pass = tries >= (hint ? 3u : rounds) || (hint && (o < 2u || o + a.wv.q < hint + 2u));
                    } else if (adv > left) {
                        act = false;
                    } else {
                        left -= adv;
                        pos += adv;
                        J += adv;
                        if (at) at += adv;
                        pass = hint && hint <= adv && at;  // behind that letter the read most likely goes on along its path
                        hint = hint > adv ? hint - adv : 0u;
                        tries = 0;
                    }
                }
                if (const u32 pm = __ballot_sync(kFull, pass)) {
                    if (pass) {
                        pool[kPool - 1u - nw - __popc(pm & lt)] = Run<IX>{pos, J, (uint16_t)left, (uint16_t)hint, at};
                        act = false;
                    }
                    nw += __popc(pm);
                }
                if (nw >= kBatch) break;
            }
            const u32 am = __ballot_sync(kFull, act);
            if (act) pool[nr + __popc(am & lt)] = Run<IX>{pos, J, (uint16_t)left, (uint16_t)hint, at};
            nr += __popc(am);
            __syncwarp();
        }
        if (nw == 0) break;  // nothing left to probe either
        // ======== walk: look up, step and extend until every run is settled or has to be probed again
        {
            IX pos = 0, J = 0;  // of the next k-mer
            u32 left = 0;
            u32 v = kNoNode;  // node of k-mer J - 1, or kNoNode: look J up
            u32 at = 0;       // v == kNoNode: path position to try first, unless hint says that k-mer J left the path
            u32 hint = 0;
            bool act = false;
            for (;;) {
                const u32 idle = __ballot_sync(kFull, !act);
                if (nw) {
                    const u32 take = min((u32)__popc(idle), nw), rank = __popc(idle & lt);
                    if (!act && rank < take) {
                        const Run<IX> e = pool[kPool - nw + rank];
                        pos = e.pos;
                        J = e.j;
                        left = e.left;
                        v = kNoNode;
                        at = e.at;
                        hint = e.hint;
                        act = true;
                    }
                    nw -= take;
                } else if (idle == kFull) {
                    break;
                }
                u32 count = 0;     // found k-mers from J on, the first one at path position `at`
                bool miss = false; // the k-mer after those is absent: the rest goes back to be probed
                if (act) {
                    const u64 kmer = letters_at(a, pos);
                    const u32 was = hint;
                    hint = 0;
                    if (v != kNoNode) {
                        v = step(a, rk, sC, v, (u32)(kmer >> (64u - 2u * k)) & 3u);
                        if (v == kNoNode) hint = k;  // the letter of the missing edge
                        else at = __ldg(a.wv.node_pos + v);
                    } else if (was || !at || !on_path(a, at, kmer)) {
                        v = lookup(a, kmer);
                        if (v == kNoNode) hint = was;
                        if (!was) at = 0;
                        if (v != kNoNode) at = __ldg(a.wv.node_pos + v);
                    } else {
                        v = ~0u;  // found
                    }
                    bool closed = false;
                    if (v != kNoNode) count = 1u + extend(a, at + 1u, (u64)pos + k, left, closed);
                    miss = v == kNoNode || closed;
                    if (closed) hint = k;
                }
                // the taken runs are read before other lanes write over their places below; convergence alone (the
                // ballots) orders no memory
                __syncwarp();
                if (a.answers) {
                    if (count && count <= kOwn) {
                        u32 x[kOwn];
#pragma unroll
                        for (u32 t = 0; t < kOwn; t++) x[t] = t < count ? __ldg(a.wv.path_node + at + t) : 0u;
#pragma unroll
                        for (u32 t = 0; t < kOwn; t++)
                            if (t < count) a.answers[J + t] = (u64)x[t];
                    }
                    __syncwarp();
                    for (u32 m = __ballot_sync(kFull, count > kOwn); m; m &= m - 1u) {
                        const int src = __ffs(m) - 1;
                        const u32 c = __shfl_sync(kFull, count, src), f = __shfl_sync(kFull, at, src);
                        u64 *const out = a.answers + __shfl_sync(kFull, J, src);
#pragma unroll 1  // unrolled, lanes with a different trip count would take another path
                        for (u32 t = lane; t < (c + 31u) / 32u * 32u; t += 32u)
                            if (t < c) out[t] = (u64)__ldg(a.wv.path_node + f + t);
                    }
                }
                bool back = false;
                if (act) {
                    if (count && a.member) set_bits(a.member, J, count);
                    const u32 adv = count + (miss ? 1u : 0u);  // settled from J on, at most left + 1
                    act = adv <= left;
                    back = act && miss;
                    if (act && !miss) v = __ldg(a.wv.path_node + at + count - 1u);
                    if (at) at += adv;  // where k-mer J + adv lies if the read goes on along this path
                    if (hint) hint--;   // k-mer J + adv is the one after the absent one
                    left -= adv;
                    pos += adv;
                    J += adv;
                    act = act && !miss;
                }
                const u32 bm = __ballot_sync(kFull, back);
                if (back) pool[nr + __popc(bm & lt)] = Run<IX>{pos, J, (uint16_t)left, (uint16_t)hint, at};
                nr += __popc(bm);
                __syncwarp();
            }
        }
    }
}

}  // namespace

namespace {

// ---------------------------------------------------- lists of k-mers
//
// K-mers without neighbours (a list, or the positions of the kernel contract
// that form no runs): each is probed for q-mers that no indexed k-mer contains,
// at its two ends, and looked up if both are present.  The probes of kListSlots
// k-mers a lane overlap; those that pass are collected per warp and looked up 32
// at a time, so that the few present ones do not idle the other lanes.
constexpr u32 kListSlots = 4;
constexpr u32 kListPool = 32 * kListSlots + 31;

__global__ void __launch_bounds__(kWarps * 32, 10) list_kernel(const SearchArgs a) {
    if (a.runs_dev && runs_usable(*a.runs_dev, a.n_kmers)) return;  // the run walk takes this kernel-contract call
    struct Item {
        u64 kmer, j;
    };
    __shared__ Item pools[kWarps][kListPool];
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const u32 lt = (1u << lane) - 1u;
    const u32 q = a.wv.q, o_max = a.k - q;
    const mlp::Bloom bloom{a.bloom_bits, a.bloom_mask, a.bloom_hashes};
    Item *const pool = pools[warp];
    const u64 step = (u64)gridDim.x * kWarps * (32u * kListSlots);
    u64 base = ((u64)blockIdx.x * kWarps + warp) * (32u * kListSlots);
    u32 np = 0;
    for (;;) {
        const bool more = base < a.n_kmers;
        if (more) {
            u64 km[kListSlots];
            bool in[kListSlots];
            u32 n_skip = 0;
#pragma unroll
            for (u32 u = 0; u < kListSlots; u++) {
                const u64 j = base + u * 32u + lane;
                in[u] = j < a.n_kmers;
                km[u] = 0;
                if (in[u]) km[u] = a.kmer_list ? __ldg(a.kmer_list + j) : letters_at(a, a.positions[j]);
            }
            if (a.logits) {  // learned-Bloom sandwich: answered "absent" only if both reject
#pragma unroll
                for (u32 u = 0; u < kListSlots; u++) {
                    const u64 j = base + u * 32u + lane;
                    if (in[u] && __ldg(a.logits + j) < a.tau && !bloom.probe(mlp::kmer_key(km[u], a.k))) {
                        in[u] = false;
                        n_skip++;
                    }
                }
                n_skip = __reduce_add_sync(kFull, n_skip);
                if (a.skipped && lane == 0 && n_skip) atomicAdd(a.skipped, (unsigned long long)n_skip);
            }
#pragma unroll
            for (u32 u = 0; u < kListSlots; u++)
                if (in[u]) in[u] = q_present(a, (u32)(km[u] >> (64u - 2u * q)));
#pragma unroll
            for (u32 u = 0; u < kListSlots; u++)
                if (in[u]) in[u] = q_present(a, (u32)((km[u] << (2u * o_max)) >> (64u - 2u * q)));
#pragma unroll
            for (u32 u = 0; u < kListSlots; u++) {
                const u64 j = base + u * 32u + lane;
                const u32 m = __ballot_sync(kFull, in[u]);
                if (in[u]) pool[np + __popc(m & lt)] = Item{km[u], j};
                else if (j < a.n_kmers) a.answers[j] = ~0ull;
                np += __popc(m);
            }
            base += step;
            __syncwarp();
        }
        while (np >= 32u || (np && !more)) {
            const u32 take = min(np, 32u);
            np -= take;
            if (lane < take) {
                const Item it = pool[np + lane];
                const u32 v = lookup(a, it.kmer);
                a.answers[it.j] = v != kNoNode ? (u64)v : ~0ull;
            }
        }
        __syncwarp();
        if (!more) break;
    }
}

// answers[0 .. n) = absent, ahead of the walk.  Written by the walk as it settles absent k-mers, the same bytes
// pushed the q-mer bitmap out of L2 (it then missed at every probe) and did not overlap with the probing: 1.2G
// k-mers, nine tenths of the reads foreign, 100M columns: 4.18 ms a call against 4.85 (4.94 with each warp filling
// its chunk first).  Four 32-byte stores a thread, blocks in order: 7.6 TB/s for 9.6 GB; a grid-stride loop of as many
// threads as the device holds 6.3.
constexpr u32 kFillThreads = 512, kFillStores = 4;
__global__ void __launch_bounds__(kFillThreads) fill_kernel(u64 *__restrict__ answers, u64 n, const u64 *runs_dev,
                                                            const u64 *__restrict__ kstart, u64 n_rows) {
    if (runs_dev && !runs_usable(*runs_dev, n)) return;  // the answers still hold the positions of the per-k-mer search
    if (!runs_dev) n = min(n, kstart[n_rows]);
    const u64 head = min(n, (u64)((32u - (reinterpret_cast<uintptr_t>(answers) & 31u)) & 31u) / 8u);
    const u64 quads = (n - head) / 4u, tail = n - head - 4u * quads;
    const u64 b = (u64)blockIdx.x * (kFillThreads * kFillStores) + threadIdx.x;
#pragma unroll
    for (u32 i = 0; i < kFillStores; i++) {
        const u64 t = b + i * kFillThreads;
        if (t < quads)
            asm volatile("st.global.v4.u64 [%0], {%1, %1, %1, %1};" ::"l"(answers + head + 4u * t), "l"(~0ull) : "memory");
    }
    if (blockIdx.x == 0) {
        if (threadIdx.x < head) answers[threadIdx.x] = ~0ull;
        if (threadIdx.x < tail) answers[head + 4u * quads + threadIdx.x] = ~0ull;
    }
}

}  // namespace

// K-mers a warp takes at a time (a power of two): 32 times the index's window
// (KernelShape.window), or as many as the batch gives each resident warp when
// that is less, so that a small batch is spread over all of them.
u32 walk_chunk(const sbwt_index *ix, u64 n_kmers) {
    const u64 warps = (u64)ix->num_sms * 10u * kWarps;
    const u32 top = 32u * (ix->shape.layout == SBWT_LAYOUT_LINES && ix->shape.window ? ix->shape.window : 128u);
    u32 c = 32u;
    while (c < top && (u64)c * warps < n_kmers) c *= 2u;
    return c;
}

bool walk_fills(const SearchArgs &a) { return a.walk && a.answers && !a.found_only && a.n_kmers >= kFillAhead; }

int launch_list(const sbwt_index *ix, SearchArgs &a, cudaStream_t s) {
    int per_sm = 0;
    SBWT_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, list_kernel, kWarps * 32, 0));
    const u64 per = (u64)kWarps * 32u * kListSlots, need = (a.n_kmers + per - 1) / per;
    const u32 blocks = (u32)std::min<u64>((u64)std::max(per_sm, 1) * (u64)ix->num_sms, need);
    list_kernel<<<blocks, kWarps * 32, 0, s>>>(a);
    SBWT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

int launch_walk(const sbwt_index *ix, SearchArgs &a, cudaStream_t s, uint32_t *blocks_out) {
    auto kern = run32_ok(a) ? walk_kernel<u32> : walk_kernel<u64>;
    int per_sm = 0;
    SBWT_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kWarps * 32, 0));
    if (per_sm < 1) per_sm = 1;
    if (ix->shape.blocks_per_sm && (int)ix->shape.blocks_per_sm < per_sm) per_sm = (int)ix->shape.blocks_per_sm;
    // longest run: one k-mer in the smallest chunks
    a.piece = a.chunk > 32u ? std::min(a.chunk / 16u, kPiece) : 1u;
    const u64 need = (a.n_kmers + (u64)a.chunk * kWarps - 1) / ((u64)a.chunk * kWarps);
    const u32 blocks = (u32)std::min<u64>((u64)per_sm * (u64)ix->num_sms, need);
    if (blocks_out) *blocks_out = blocks;
    if (!a.cleared) SBWT_CHECK_CUDA(cudaMemsetAsync(a.counter, 0, sizeof(unsigned long long), s));
    if (walk_fills(a)) {
        const u64 per = 4ull * kFillThreads * kFillStores;
        fill_kernel<<<(unsigned)((a.n_kmers + per - 1) / per), kFillThreads, 0, s>>>(a.answers, a.n_kmers, a.runs_dev, a.kstart, a.n_rows);
        SBWT_CHECK_CUDA(cudaGetLastError());
    }
    return launch_kernel(kern, blocks, kWarps * 32, s, ix, LinesRanker{ix->d_lines, ix->lpc}, a);
}

}  // namespace sbwt
