// stream.cu -- builds the walk's structures (stream.cuh): sorted labels, path
// text, q-mer bitmap and group marks of the forward walk, select samples and
// node nibbles of the backward step, on the GPU from the index's lines alone,
// so that indexes loaded from the reference's files get them
// too.  No reference counterpart.
//
// First letters and groups come from the labels: with pred(v) = the first
// node of the group of v's predecessor (stream.cuh), the last letter of
// pred^t(v) is label(v)[k-1-t] for t < k, and the chain reaches the all-$
// root exactly where the label's $ padding starts.  Labels roll along the paths
// (write_segment) into
//   code(v) = sum_t lastletter(pred^t(v)) << 2t,  len(v) = letters before the root
// Then first letter = letter k-1 (or $ if len < k), and v starts a group iff
// its last k-1 letters (and how many of them are real) differ from v-1's.
#include <algorithm>
#include <cstring>
#include <vector>

#include <cub/cub.cuh>

#include "internal.h"
#include "stream.cuh"

namespace sbwt {
namespace {

using namespace dev;

// sel_c[s] = line holding the one of rank 64 s of vector c.
__global__ void select_samples_kernel(const ulonglong4 *__restrict__ lines, u32 lpc, u32 *__restrict__ sel,
                                      u32 n_samples) {
    const u32 t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= lpc) return;
    const ulonglong4 w = lines[t];
    const u32 cnt = (u32)(w.x >> 32);
    const u32 ones = __popcll(w.x & 0xffffffffull) + __popcll(w.y) + __popcll(w.z) + __popcll(w.w);
    if (!ones) return;
    const u32 s_lo = (cnt + 63u) >> kSelLog, s_hi = (cnt + ones - 1u) >> kSelLog;
    for (u32 s = s_lo; s <= s_hi && s < n_samples; s++) sel[s] = t;
}

// ---- paths: each column's first outgoing edge links it to one successor (the
// root's none: it has no letter), and every node but the root has one incoming
// edge, so the links form chains and cycles.  They are cut into segments at the
// nodes without a link to them and at one node in kSegment (by a hash), so that
// one thread per segment walks it: once to size it, once to write it together
// with the labels, which roll along the segment from its first node's (k select
// steps back).  In between the segments are put in order by pointer doubling, so
// that those of one chain adjoin and a read runs on over the cuts: with every cut
// a path's end, a quarter of the stretches of 150-letter reads ended there and
// took a rank step each.

constexpr u32 kSegment = 256;

__device__ __forceinline__ bool cut_here(u32 v) { return v * 0x9E3779B1u < 0xffffffffu / kSegment; }

// succ[v] = node of v's first outgoing edge (0: none); the other edges' nodes get
// their bit in `head`, and v its bit in `fork` if there are any.  counts[0] +=
// upper bound of the number of segments.
__global__ void succ_kernel(const StreamView sv, u32 *__restrict__ succ, u32 *__restrict__ head, u32 *__restrict__ fork,
                            unsigned long long *__restrict__ counts) {
    const u32 v = blockIdx.x * blockDim.x + threadIdx.x;
    u32 heads = 0;
    if (v < sv.n) {
        const u32 line = v / kLineBits, t = v - line * kLineBits + 32u;
        u32 s = 0;
        heads = v == 0 || cut_here(v);
        for (u32 c = 0; c < 4u; c++) {
            const ulonglong4 w = ld_line(sv.lines + (u64)c * sv.lpc + line);
            if (!((sector_word(w, t >> 6) >> (63u - (t & 63u))) & 1ull)) continue;
            const u32 x = sv.C[c] + line_rank_from(w, t - 32u);
            if (s == 0 && v) {
                s = x;
            } else {
                atomicOr(head + (x >> 5), 1u << (x & 31u));
                atomicOr(fork + (v >> 5), 1u << (v & 31u));
                heads++;
            }
        }
        succ[v] = s;
    }
    heads = __reduce_add_sync(0xffffffffu, heads);
    if ((threadIdx.x & 31u) == 0 && heads) atomicAdd(counts, (unsigned long long)heads);
}

// The segments' first nodes, in any order.
__global__ void heads_kernel(u32 n, const u32 *__restrict__ head, u32 *__restrict__ first,
                             unsigned long long *__restrict__ count) {
    const u32 v = blockIdx.x * blockDim.x + threadIdx.x;
    const bool is = v < n && (v == 0 || cut_here(v) || ((head[v >> 5] >> (v & 31u)) & 1u));
    const u32 m = __ballot_sync(0xffffffffu, is);
    if (!m) return;
    unsigned long long base = 0;
    if ((threadIdx.x & 31u) == 0) base = atomicAdd(count, (unsigned long long)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (is) first[base + __popc(m & ((1u << (threadIdx.x & 31u)) - 1u))] = v;
}

constexpr u32 kNoSeg = ~0u;

// pos[first node of segment i] = i, for the links between segments
__global__ void segment_ids_kernel(u32 n_seg, const u32 *__restrict__ first, u32 *__restrict__ pos,
                                   u32 *__restrict__ prev) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_seg) return;
    pos[first[i]] = i;
    prev[i] = kNoSeg;
}

__global__ void segment_len_kernel(u32 n_seg, const u32 *__restrict__ first, const u32 *__restrict__ succ,
                                   const u32 *__restrict__ pos, u32 *__restrict__ len, u32 *__restrict__ prev) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_seg) return;
    u32 l = 0, v = first[i];
    do {
        v = succ[v];
        l++;
    } while (v && !cut_here(v));
    len[i] = l;
    if (v) prev[pos[v]] = i;
}

// Per segment i: before = nodes of the segments between i and ptr (both
// excluded), head = the farthest of them (i if there is none), low = the
// smallest of i and them.
struct SegRank {
    u32 ptr, before, head, low;
};

__global__ void rank_init_kernel(u32 n_seg, const u32 *__restrict__ prev, SegRank *__restrict__ r) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n_seg) r[i] = SegRank{prev[i], 0u, i, i};
}

// One doubling round.
__global__ void rank_double_kernel(u32 n_seg, const u32 *__restrict__ len, const SegRank *__restrict__ r,
                                   SegRank *__restrict__ out) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_seg) return;
    SegRank x = r[i];
    if (x.ptr != kNoSeg) {
        const SegRank y = r[x.ptr];
        x = SegRank{y.ptr, x.before + len[x.ptr] + y.before, y.head, min(x.low, y.low)};
    }
    out[i] = x;
}

// After all rounds a segment that still has a ptr lies on a cycle: the smallest of each becomes its first.
__global__ void open_cycles_kernel(u32 n_seg, const SegRank *__restrict__ r, u32 *__restrict__ prev,
                                   unsigned long long *__restrict__ opened) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_seg || r[i].ptr == kNoSeg || r[i].low != i) return;
    prev[i] = kNoSeg;
    atomicAdd(opened, 1ull);
}

// total[first segment of a chain] = nodes of the chain (0 for the other segments, and at n_seg).
__global__ void chain_len_kernel(u32 n_seg, const SegRank *__restrict__ r, const u32 *__restrict__ len,
                                 u32 *__restrict__ total) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n_seg) atomicMax(total + r[i].head, r[i].before + len[i]);
}

struct PathArrays {
    u32 *node, *pos;    // path_node, node_pos
    ulonglong2 *path;
    u64 *code;          // letter t from the end of the label at bits 2t, 2t+1 (t < k)
    uint8_t *len;       // letters of the label before its $ padding, at most k
};

// The segment of `count` nodes that starts at v goes to positions off .. off + count - 1; starts: no other one
// leads into it.
__device__ void write_segment(const StreamView &sv, u32 k, const u32 *succ, u32 v, u32 off, u32 count, bool starts,
                              const PathArrays &a, unsigned long long *bad) {
    const u64 mask = k < 32u ? (1ull << (2u * k)) - 1ull : ~0ull;
    u64 code = 0;
    u32 l = 0;
    for (u32 u = v; l < k && u; l++) {
        code |= (u64)sv.last_letter(u) << (2u * l);
        u = sv.pred(u);
        if (u >= sv.n) {  // not an SBWT: record it, stop at the root
            atomicAdd(bad, 1ull);
            u = 0;
        }
    }
    if (starts) atomicOr((unsigned long long *)&a.path[off >> 5].y, 1ull << (63u - (off & 31u)));
    for (u32 i = 0; i < count; i++) {
        a.node[off + i] = v;
        a.pos[v] = off + i;
        a.code[v] = code;
        a.len[v] = (uint8_t)l;
        v = succ[v];
        code = ((code << 2) | sv.last_letter(v)) & mask;
        l = min(l + 1u, k);
    }
}

__global__ void segment_write_kernel(const StreamView sv, u32 k, u32 n_seg, const u32 *__restrict__ first,
                                     const u32 *__restrict__ succ, const u32 *__restrict__ len,
                                     const SegRank *__restrict__ r, const u32 *__restrict__ chain_off,
                                     const PathArrays a, unsigned long long *__restrict__ bad) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_seg) return;
    const SegRank x = r[i];
    write_segment(sv, k, succ, first[i], chain_off[x.head] + x.before, len[i], x.head == i, a, bad);
}

// Cycles that no cut falls on (short ones): the thread of a cycle's smallest node writes it.
__global__ void cycles_kernel(const StreamView sv, u32 k, const u32 *__restrict__ succ, const PathArrays a,
                              u32 *__restrict__ reached, unsigned long long *__restrict__ bad) {
    const u32 v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= sv.n || *(volatile u32 *)(a.pos + v) != ~0u) return;
    u32 x = succ[v], count = 1;
    for (; x > v; x = succ[x]) count++;
    if (x == v) write_segment(sv, k, succ, v, atomicAdd(reached, count), count, true, a, bad);
}

// The last letters of the path's nodes, 32 positions a thread, and the positions that cannot be judged by the
// letters alone: segment starts, and the positions after a node with more than one edge.
__global__ void path_letters_kernel(const StreamView sv, const u32 *__restrict__ node, const u32 *__restrict__ fork,
                                    ulonglong2 *__restrict__ path, u32 blocks) {
    const u32 b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= blocks) return;
    u64 x = 0, starts = path[b].y, open = 0;
    u32 u = b && (u64)b * 32u <= sv.n ? node[(u64)b * 32u - 1u] : 0u;  // the node before position 32 b
    for (u32 t = 0; t < 32u; t++) {
        const u64 i = (u64)b * 32u + t;
        if ((fork[u >> 5] >> (u & 31u)) & 1u) open |= 1ull << (31u - t);
        if (i < sv.n) {
            u = node[i];
            x |= (u64)sv.last_letter(u) << (62u - 2u * t);
        } else {
            starts |= 1ull << (63u - t);  // the last segment ends here
        }
    }
    path[b].x = x;
    path[b].y = starts | starts >> 32 | open;
}

// One thread per byte: the nibbles of nodes 2t and 2t+1.
__global__ void node_nibbles_kernel(u32 n, u32 k, const u64 *__restrict__ code, const uint8_t *__restrict__ len,
                                   uint8_t *__restrict__ node) {
    const u32 t = blockIdx.x * blockDim.x + threadIdx.x;
    if ((u64)t * 2u >= n) return;
    const u64 mask = (1ull << (2u * (k - 1u))) - 1ull;  // the last k-1 letters (k <= 32)
    u32 byte = 0;
    for (u32 h = 0; h < 2u; h++) {
        const u32 v = 2u * t + h;
        if (v >= n) break;
        const u32 l = len[v];
        const u64 c = code[v];
        const u32 first = l >= k ? (u32)((c >> (2u * (k - 1u))) & 3u) + 1u : 0u;
        bool start = v == 0;
        if (!start) {
            const u32 lp = len[v - 1];
            start = ((c ^ code[v - 1]) & mask) != 0 || min(l, k - 1u) != min(lp, k - 1u);
        }
        byte |= (first | (start ? kGroupStart : 0u)) << (4u * h);
    }
    node[t] = (uint8_t)byte;
}

// ---- structures of the forward walk (WalkView, stream.cuh)

// The q-mer bitmap: one atomic per distinct q-mer (labels are sorted, so equal
// suffixes of q letters are neighbours).
__global__ void qbits_kernel(u32 n, u32 q, const u64 *__restrict__ code, const uint8_t *__restrict__ len,
                             u32 *__restrict__ qbits) {
    const u32 v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n || len[v] < q) return;
    const u64 x = code[v] & ((1ull << (2u * q)) - 1ull);  // q <= 16
    if (v && len[v - 1] >= q && (code[v - 1] & ((1ull << (2u * q)) - 1ull)) == x) return;
    atomicOr(qbits + (x >> 5), 1u << (x & 31u));
}

__global__ void marks_kernel(u32 n, const uint8_t *__restrict__ node, u32 *__restrict__ marks, u32 words) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= words) return;
    u32 w = 0;
    for (u32 b = 0; b < 32u; b++) {
        const int64_t v = (int64_t)i * kMarkCols - 4 + b;
        if (v < 0 || v >= (int64_t)n) continue;
        if ((node[v >> 1] >> ((v & 1) * 4)) & kGroupStart) w |= 1u << b;
    }
    marks[i] = w;
}

// code[v] -> the node's key, in place; ~0 past the last node.
__global__ void keys_kernel(u32 n, u32 n_pad, u32 k, u64 *__restrict__ code, const uint8_t *__restrict__ len) {
    const u32 v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n_pad) return;
    u64 x = ~0ull;
    if (v < n) {
        x = letters_reverse(code[v]);
        if (k < 32u) {
            x &= ~0ull << (64u - 2u * k);
            if (len[v] >= k) x |= 1ull;
        }
    }
    code[v] = x;
}

// What the forward walk relies on, for every column: keys ascend, strictly
// between labels without $; only group starts have outgoing edges; a group has
// at most 5 members.  With a smaller k than the index's this fails where two
// labels agree in their last k letters.  Where none do, and with a larger k,
// labels, groups and edges stay consistent (a label is what the edges spell
// backwards, as in the search), and the forward walk serves that k.
__global__ void walk_check_kernel(u32 n, u32 k, const u64 *__restrict__ keys, const uint8_t *__restrict__ node,
                                  const u32 *__restrict__ marks, const ulonglong4 *__restrict__ lines, u32 lpc,
                                  unsigned long long *__restrict__ bad) {
    const u32 v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    const u32 f = (u32)(node[v >> 1] >> ((v & 1u) * 4u)) & 15u;
    bool ok = true;
    if (v + 1u < n) {
        const u64 a = keys[v], b = keys[v + 1u];
        const u32 g = (u32)(node[(v + 1u) >> 1] >> (((v + 1u) & 1u) * 4u)) & 15u;
        ok = a < b || (a == b && !((f & 7u) && (g & 7u)));
    }
    if (!(f & kGroupStart)) {
        ok = ok && v - group_start(marks[v / kMarkCols], v) < 5u;
        const u32 line = v / kLineBits, t = v - line * kLineBits + 32u;
        for (u32 c = 0; c < 4u; c++)
            ok = ok && !((sector_word(lines[(u64)c * lpc + line], t >> 6) >> (63u - (t & 63u))) & 1ull);
    }
    if (!ok) atomicAdd(bad, 1ull);
}

// Letters of the q-mers: the smallest q with 4^q >= 16 n, so that at most one in
// 16 q-mers of random letters is present, as long as the bitmap (4^q bits) is no
// larger than 32 MiB (q = 14), where it still hits L2; larger indexes keep q = 14
// up to 4^14 columns, then take the smallest q with 4^q >= n.  Measured at 1M
// columns with the limit at 2 n or 4 n (q = 11), 8 n or 16 n (q = 12) and 64 n
// (q = 13): 100M single k-mers 949 / 844 / 802 us, uneven reads 2092 / 1955 /
// 1951, 10,000 reads 95 / 87 / 89; at 4M columns (13 for 16 n, 14 for 64 n) 284 /
// 300.
u32 walk_q(u64 n, u32 k) {
    u32 q = 1;
    while (q < 14u && (1ull << (2u * q)) < 16ull * n) q++;
    while (q < 16u && (1ull << (2u * q)) < n) q++;
    return q < k ? q : k;
}

}  // namespace

WalkView walk_view(const sbwt_index *ix) {
    WalkView w;
    w.labels = ix->d_labels;
    w.qbits = ix->d_qbits;
    w.marks = ix->d_marks;
    w.path_node = ix->d_path_node;
    w.node_pos = ix->d_node_pos;
    w.path = ix->d_path;
    w.q = ix->walk_q;
    w.n = (u32)ix->n;
    return w;
}

StreamView stream_view(const sbwt_index *ix) {
    StreamView sv;
    std::memset(&sv, 0, sizeof(sv));
    sv.lines = ix->d_lines;
    sv.lpc = ix->lpc;
    sv.sel = ix->d_sel;
    for (int c = 0; c < 4; c++) {
        sv.sel_off[c] = ix->sel_off[c];
        sv.sel_n[c] = ix->sel_n[c];
        sv.C[c] = (u32)ix->C[c];
    }
    sv.node = ix->d_node;
    sv.n = (u32)ix->n;
    return sv;
}

// One allocation behind several arrays: `put` places them, first to size it, then in it.  With a cudaMalloc for each
// of the twenty arrays and a cudaFree for each of the thirteen of scratch, building the structures took 3.75 ms at 1M
// columns, 11.6 at 20M and 20.3 at 50M; with four of the one and two of the other 2.3, 7.3 and 15.2.
struct Arena {
    uint8_t *base = nullptr;
    size_t bytes = 0;
    template <class T> void put(T *&p, size_t count) {
        p = reinterpret_cast<T *>(base + bytes);
        bytes += (std::max<size_t>(count, 1) * sizeof(T) + 255) / 256 * 256;
    }
};

// place(arena) puts the arrays; base: the allocation.
template <class F> cudaError_t alloc_arena(void **base, F place) {
    Arena size;
    place(size);
    const cudaError_t e = cudaMalloc(base, size.bytes);
    Arena in;
    if (e == cudaSuccess) {
        in.base = static_cast<uint8_t *>(*base);
        place(in);
    }
    return e;
}

void free_walk(sbwt_index *ix) {
    cudaFree(ix->walk_mem);
    ix->walk_mem = nullptr;
    ix->d_labels = nullptr;
    ix->d_qbits = nullptr;
    ix->d_marks = nullptr;
    ix->d_path_node = nullptr;
    ix->d_node_pos = nullptr;
    ix->d_path = nullptr;
    ix->walk_q = 0;
}

void free_stream(sbwt_index *ix) {
    free_walk(ix);
    cudaFree(ix->stream_mem);
    ix->stream_mem = nullptr;
    ix->d_node = nullptr;
    ix->d_sel = nullptr;
}

int build_stream(sbwt_index *ix, cudaStream_t s) {
    if (ix->stream_ok) return 0;
    if (!ix->lines_ok) return set_error("the walk needs the line layout");
    if (ix->k > 32 || ix->k < 2) return set_error("k out of range");
    const u32 n = (u32)ix->n, k = ix->k;
    u64 total = 0;
    for (int c = 0; c < 4; c++) {
        const u64 ones = ix->C[c + 1] - ix->C[c];
        ix->sel_off[c] = (u32)total;
        ix->sel_n[c] = (u32)((ones + 63) >> kSelLog);
        total += ix->sel_n[c] + 1;
    }
    const u32 n_pad = (n + 3u) / 4u * 4u + 4u;
    const u32 q = walk_q(n, k), mark_words = n / kMarkCols + 1u, path_blocks = n / 32u + 2u;
    const size_t qwords = std::max<size_t>(1, (size_t)((1ull << (2u * q)) / 32u));
    const u32 blocks = (n + 255) / 256;
    // scratch: first successors, head bits, label lengths, segments; counters: segments (upper bound),
    // segments, nodes without a predecessor, columns the forward walk cannot take, cycles of segments
    u32 *succ = nullptr, *head = nullptr, *fork = nullptr, *first = nullptr, *off = nullptr;
    u32 *seg_len = nullptr, *prev = nullptr;
    SegRank *rank[2] = {nullptr, nullptr};
    uint8_t *len = nullptr, *tmp = nullptr;
    void *col_mem = nullptr, *seg_mem = nullptr;  // the arrays above, per column and per segment
    unsigned long long *cnt = nullptr, h_cnt[5] = {0, 0, 0, 0, 0};
    cudaError_t e = cudaSuccess;
    auto ok = [&](cudaError_t x) {
        if (e == cudaSuccess) e = x;
        return e == cudaSuccess;
    };
    int rc = 0;
    do {
        if (!ok(alloc_arena(&ix->stream_mem,
                            [&](Arena &a) {
                                a.put(ix->d_sel, total);
                                a.put(ix->d_node, (size_t)n / 2 + 16);
                            })) ||
            !ok(alloc_arena(&ix->walk_mem,
                            [&](Arena &a) {
                                a.put(ix->d_labels, n_pad);
                                a.put(ix->d_qbits, qwords);
                                a.put(ix->d_marks, mark_words);
                                a.put(ix->d_path_node, n);
                                a.put(ix->d_node_pos, n);
                                a.put(ix->d_path, path_blocks);
                            })) ||
            !ok(alloc_arena(&col_mem, [&](Arena &a) {
                a.put(succ, n);
                a.put(head, (size_t)n / 32 + 1);
                a.put(fork, (size_t)n / 32 + 1);
                a.put(len, n);
                a.put(cnt, sizeof h_cnt / sizeof h_cnt[0]);
            })))
            break;
        cudaMemsetAsync(ix->d_sel, 0, total * sizeof(u32), s);
        cudaMemsetAsync(ix->d_qbits, 0, qwords * sizeof(u32), s);
        cudaMemsetAsync(ix->d_path, 0, (size_t)path_blocks * sizeof(ulonglong2), s);
        cudaMemsetAsync(head, 0, ((size_t)n / 32 + 1) * sizeof(u32), s);
        cudaMemsetAsync(fork, 0, ((size_t)n / 32 + 1) * sizeof(u32), s);
        cudaMemsetAsync(cnt, 0, sizeof h_cnt, s);
        for (int c = 0; c < 4; c++)
            if (ix->sel_n[c])
                select_samples_kernel<<<(ix->lpc + 255) / 256, 256, 0, s>>>(
                    ix->d_lines + (u64)c * ix->lpc, ix->lpc, ix->d_sel + ix->sel_off[c], ix->sel_n[c]);
        const StreamView sv = stream_view(ix);
        succ_kernel<<<blocks, 256, 0, s>>>(sv, succ, head, fork, cnt);
        if (!ok(cudaMemcpyAsync(h_cnt, cnt, sizeof h_cnt, cudaMemcpyDeviceToHost, s)) || !ok(cudaStreamSynchronize(s)))
            break;
        const u32 max_seg = (u32)h_cnt[0];
        size_t tmp_bytes = 0;
        if (!ok(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, off, off, (int64_t)max_seg + 1, s)) ||
            !ok(alloc_arena(&seg_mem, [&](Arena &a) {
                a.put(first, max_seg);
                a.put(off, (size_t)max_seg + 1);
                a.put(seg_len, max_seg);
                a.put(prev, max_seg);
                a.put(rank[0], max_seg);
                a.put(rank[1], max_seg);
                a.put(tmp, tmp_bytes);
            })))
            break;
        heads_kernel<<<blocks, 256, 0, s>>>(n, head, first, cnt + 1);
        if (!ok(cudaMemcpyAsync(h_cnt, cnt, sizeof h_cnt, cudaMemcpyDeviceToHost, s)) || !ok(cudaStreamSynchronize(s)))
            break;
        const u32 n_seg = (u32)h_cnt[1], seg_blocks = (n_seg + 127) / 128;
        segment_ids_kernel<<<seg_blocks, 128, 0, s>>>(n_seg, first, ix->d_node_pos, prev);
        segment_len_kernel<<<seg_blocks, 128, 0, s>>>(n_seg, first, succ, ix->d_node_pos, seg_len, prev);
        int cur = 0;
        for (int pass = 0; pass < 2; pass++) {
            rank_init_kernel<<<seg_blocks, 128, 0, s>>>(n_seg, prev, rank[cur]);
            for (u64 reach = 1; reach < 2ull * n_seg; reach *= 2, cur ^= 1)
                rank_double_kernel<<<seg_blocks, 128, 0, s>>>(n_seg, seg_len, rank[cur], rank[cur ^ 1]);
            if (pass) break;
            open_cycles_kernel<<<seg_blocks, 128, 0, s>>>(n_seg, rank[cur], prev, cnt + 4);
            if (!ok(cudaMemcpyAsync(h_cnt, cnt, sizeof h_cnt, cudaMemcpyDeviceToHost, s)) || !ok(cudaStreamSynchronize(s)))
                break;
            if (h_cnt[4] == 0) break;
        }
        if (e != cudaSuccess) break;
        cudaMemsetAsync(off, 0, ((size_t)n_seg + 1) * sizeof(u32), s);
        chain_len_kernel<<<seg_blocks, 128, 0, s>>>(n_seg, rank[cur], seg_len, off);
        if (!ok(cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, off, off, (int64_t)n_seg + 1, s)) ||
            !ok(cudaMemsetAsync(ix->d_node_pos, 0xff, (size_t)n * sizeof(u32), s)))
            break;
        const PathArrays pa{ix->d_path_node, ix->d_node_pos, ix->d_path, ix->d_labels, len};
        segment_write_kernel<<<seg_blocks, 128, 0, s>>>(sv, k, n_seg, first, succ, seg_len, rank[cur], off, pa, cnt + 2);
        cycles_kernel<<<blocks, 256, 0, s>>>(sv, k, succ, pa, off + n_seg, cnt + 2);
        path_letters_kernel<<<(path_blocks + 255) / 256, 256, 0, s>>>(sv, ix->d_path_node, fork, ix->d_path,
                                                                         path_blocks);
        node_nibbles_kernel<<<(n / 2 + 1 + 255) / 256, 256, 0, s>>>(n, k, ix->d_labels, len, ix->d_node);
        qbits_kernel<<<blocks, 256, 0, s>>>(n, q, ix->d_labels, len, ix->d_qbits);
        marks_kernel<<<(mark_words + 255) / 256, 256, 0, s>>>(n, ix->d_node, ix->d_marks, mark_words);
        keys_kernel<<<(n_pad + 255) / 256, 256, 0, s>>>(n, n_pad, k, ix->d_labels, len);
        walk_check_kernel<<<blocks, 256, 0, s>>>(n, k, ix->d_labels, ix->d_node, ix->d_marks, ix->d_lines, ix->lpc,
                                                 cnt + 3);
        if (!ok(cudaGetLastError()) || !ok(cudaMemcpyAsync(h_cnt, cnt, sizeof h_cnt, cudaMemcpyDeviceToHost, s)) ||
            !ok(cudaStreamSynchronize(s)))
            break;
        if (h_cnt[2]) rc = set_error("the bit vectors are not an SBWT: %llu nodes have no predecessor", h_cnt[2]);
    } while (false);
    if (e != cudaSuccess)
        rc = set_error("CUDA error while building the walk's structures: %s", cudaGetErrorString(e));
    cudaFree(col_mem);
    cudaFree(seg_mem);
    if (rc || h_cnt[3]) free_walk(ix);  // with h_cnt[3], reads are searched without the forward walk
    else ix->walk_q = q;
    if (rc) {
        free_stream(ix);
        return rc;
    }
    ix->stream_ok = true;
    ix->gen++;
    return 0;
}

}  // namespace sbwt

using namespace sbwt;

extern "C" int sbwt_node_bytes_export(sbwt_index *ix, uint8_t *out, uint64_t count) {
    clear_error();
    if (!ix || !out) return set_error("NULL argument");
    if (count != ix->n) return set_error("count must be the number of columns (%llu)", (unsigned long long)ix->n);
    SBWT_CHECK_CUDA(cudaSetDevice(ix->device));
    SBWT_TRY(build_stream(ix, 0));
    std::vector<uint8_t> packed(count / 2 + 1);
    SBWT_CHECK_CUDA(cudaMemcpy(packed.data(), ix->d_node, count / 2 + (count & 1), cudaMemcpyDeviceToHost));
    for (u64 v = 0; v < count; v++) out[v] = (uint8_t)((packed[v >> 1] >> ((v & 1) * 4)) & 15u);
    return 0;
}
