// ingest.cu -- query ingest on the GPU: 2-bit packing, the per-row k-mer
// table, the chunk->row table of the search kernel, and the membership bitmap.
#include "device.cuh"
#include "internal.h"
#include "scan.cuh"

namespace sbwt {
namespace {

using namespace dev;

// Four letters (byte 0 first) -> one byte holding their 2-bit codes, first
// letter in bits 7..6.  A/a->0 C/c->1 G/g->2 T/t->3, any other byte -> 0, as
// the LUT of include/gpu/create_kmer_string.hpp:18-20.  (x | 0x20) folds case;
// only 'C'/'c' become 0x63, 'G'/'g' 0x67, 'T'/'t' 0x74.  The multiply by
// 0x40100401 moves the code of byte i to bits 30-2i..31-2i without carries
// into the top byte.
__device__ __forceinline__ u32 pack4_any(u32 x) {
    const u32 lo = x | 0x20202020u;
    const u32 codes = (__vcmpeq4(lo, 0x63636363u) & 0x01010101u) | (__vcmpeq4(lo, 0x67676767u) & 0x02020202u) |
                      (__vcmpeq4(lo, 0x74747474u) & 0x03030303u);
    return (codes * 0x40100401u) >> 24;
}

// The same where all four are ACGT or acgt: their low three bits (1, 3, 7, 4)
// select the code and the letter they then have to be from two 8-byte tables
// held in registers.  bad != 0 afterwards: some byte is none of them.
__device__ __forceinline__ u32 pack4(u32 x, u32 &bad) {
    const u32 t = x & 0x07070707u;
    const u32 sel = __byte_perm(t | (t >> 4), 0, 0x4420);  // the four indices as nibbles
    bad |= __byte_perm(0x630061ffu, 0x67ffff74u, sel) ^ (x | 0x20202020u);
    return (__byte_perm(0x01000000u, 0x02000003u, sel) * 0x40100401u) >> 24;
}

__device__ __forceinline__ u64 pack32(const uint4 &v0, const uint4 &v1) {
    const u32 in[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    u32 bad = 0;
    u64 x = 0;
#pragma unroll
    for (u32 i = 0; i < 8u; i++) x |= (u64)pack4(in[i], bad) << (56u - 8u * i);
    if (bad) {
        x = 0;
#pragma unroll
        for (u32 i = 0; i < 8u; i++) x |= (u64)pack4_any(in[i]) << (56u - 8u * i);
    }
    return x;
}

// kPackWords output words (32 letters each) per thread, a block apart.  ALIGN:
// the letters' alignment, 32 (one load a word), 16 (two) or 1; the words that
// hold the end, the padding after it and all unaligned ones are assembled byte
// by byte (bytes past n_letters are 0, i.e. 'A', as the reference's zero
// padding, kmer_search.hpp:292-301).  HBM-bound: 1.25 bytes a letter.  1.5G
// letters: 0.28 ms (6.8 TB/s) with 32-byte loads and the table form of pack4,
// 0.31 with two 16-byte loads and one word a thread; byte compares for every
// letter took 0.47.
constexpr u32 kPackThreads = 256, kPackWords = 4;

// `block` of blocks of THREADS threads.
template <int ALIGN, u32 THREADS>
__device__ __forceinline__ void pack_block(const uint8_t *__restrict__ letters, u64 n_letters, u64 *__restrict__ words,
                                           u64 n_words, u64 block) {
    const u64 w0 = block * (THREADS * kPackWords) + threadIdx.x;
    const u64 whole = n_letters / 32u;  // words inside the letters
    uint4 v[kPackWords][2];
#pragma unroll
    for (u32 i = 0; i < kPackWords; i++) {
        const u64 w = w0 + i * THREADS;
        if (ALIGN == 1 || w >= whole) continue;
        const uint4 *p = reinterpret_cast<const uint4 *>(letters + w * 32u);
        if constexpr (ALIGN == 32) {
            asm("ld.global.nc.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                : "=r"(v[i][0].x), "=r"(v[i][0].y), "=r"(v[i][0].z), "=r"(v[i][0].w), "=r"(v[i][1].x), "=r"(v[i][1].y),
                  "=r"(v[i][1].z), "=r"(v[i][1].w)
                : "l"(p));
        } else {
            v[i][0] = __ldg(p);
            v[i][1] = __ldg(p + 1);
        }
    }
#pragma unroll
    for (u32 i = 0; i < kPackWords; i++) {
        const u64 w = w0 + i * THREADS;
        if (ALIGN != 1 && w < whole) {
            words[w] = pack32(v[i][0], v[i][1]);
        } else if (w < n_words) {
            u64 x = 0;
            for (u32 g = 0; g < 8; g++) {
                u32 c = 0;
                for (u32 b = 0; b < 4; b++) {
                    const u64 j = w * 32u + g * 4u + b;
                    c |= (j < n_letters ? (u32)letters[j] : 0u) << (8 * b);
                }
                x |= (u64)pack4_any(c) << (56 - 8 * g);
            }
            words[w] = x;
        }
    }
}

template <int ALIGN>
__global__ void __launch_bounds__(kPackThreads) pack_kernel(const uint8_t *__restrict__ letters, u64 n_letters,
                                                            u64 *__restrict__ words, u64 n_words) {
    pack_block<ALIGN, kPackThreads>(letters, n_letters, words, n_words, blockIdx.x);
}

struct KstartScan {
    const u64 *row_starts;
    u64 *kstart;
    u32 k;
    struct Item {
        u64 v;
    };
    __device__ __forceinline__ Item load(u64 r) const {
        const u64 len = row_starts[r + 1] - row_starts[r];
        return Item{len >= k ? len - k + 1ull : 0ull};
    }
    __device__ __forceinline__ u64 value(const Item &it) const { return it.v; }
    __device__ __forceinline__ void emit(u64 r, u64 prefix, const Item &) const { kstart[r] = prefix; }
};

// chunk_row[c] = the row holding k-mer c*chunk: the first r with
// kstart[r+1] > c*chunk (rows without k-mers are skipped).
__global__ void chunk_rows_kernel(const u64 *kstart, u64 n_rows, u64 n_chunks, u32 chunk, u32 *chunk_row) {
    const u64 c = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_chunks) return;
    const u64 j = c * chunk;
    u64 lo = 0, hi = n_rows;
    while (lo < hi) {
        const u64 mid = (lo + hi) >> 1;
        if (kstart[mid + 1] <= j) lo = mid + 1; else hi = mid;
    }
    chunk_row[c] = (u32)lo;
}

// ---- small batches: everything before the search in one launch
//
// The first block makes the row table (first k-mer of each row, the row of each
// chunk's first k-mer) in shared memory and clears the search's counter, the
// others pack.  As pack, three scan kernels, chunk rows and a memset the same took
// six launches of 3-8 us each: 10,000 reads 87 us a call, 75 in one; 16 reads 44,
// 26.
constexpr u32 kPrepThreads = 1024, kPrepRowsPerThread = 11;
constexpr u32 kPrepRows = kPrepThreads * kPrepRowsPerThread - 1;
constexpr u64 kPrepKmers = 16ull << 20;

template <int ALIGN>
__global__ void __launch_bounds__(kPrepThreads) prep_kernel(const uint8_t *__restrict__ letters, u64 n_letters,
                                                            u64 *__restrict__ words, u64 n_words,
                                                            const u64 *__restrict__ row_starts, u32 n_rows, u32 k,
                                                            u64 *__restrict__ kstart, u32 n_chunks, u32 chunk,
                                                            u32 *__restrict__ chunk_row, unsigned long long *counter) {
    if (blockIdx.x) {
        pack_block<ALIGN, kPrepThreads>(letters, n_letters, words, n_words, blockIdx.x - 1u);
        return;
    }
    __shared__ u32 ks[kPrepRows + 1];
    if (threadIdx.x == 0) *counter = 0;
    // each thread's rows adjoin; lengths through shared memory, so that the loads coalesce
    for (u32 r = threadIdx.x; r < n_rows; r += kPrepThreads) {
        const u64 len = row_starts[r + 1] - row_starts[r];
        ks[r] = len >= k ? (u32)(len - k + 1u) : 0u;
    }
    __syncthreads();
    const u32 per = (n_rows + kPrepThreads - 1u) / kPrepThreads, r0 = min(threadIdx.x * per, n_rows), r1 = min(r0 + per, n_rows);
    u64 sum = 0, total;
    for (u32 r = r0; r < r1; r++) sum += ks[r];
    u64 at = block_exclusive_scan(sum, &total);
    for (u32 r = r0; r < r1; r++) {
        const u32 len = ks[r];
        ks[r] = (u32)at;
        at += len;
    }
    if (threadIdx.x == 0) ks[n_rows] = (u32)total;
    __syncthreads();
    for (u32 r = threadIdx.x; r <= n_rows; r += kPrepThreads) kstart[r] = ks[r];
    for (u32 c = threadIdx.x; c < n_chunks; c += kPrepThreads) {
        u32 lo = 0, hi = n_rows;
        while (lo < hi) {
            const u32 mid = (lo + hi) >> 1;
            if (ks[mid + 1] <= c * chunk) lo = mid + 1; else hi = mid;
        }
        chunk_row[c] = lo;
    }
}

// out[t] = the MSB-first 64-bit window of k-mer j0 + t of a batch of reads
// (search_kernel.hpp:66-68 on the per-row k-mer table), t < count.
__global__ void kmer_list_kernel(const u64 *__restrict__ words, const u64 *__restrict__ row_starts,
                                 const u64 *__restrict__ kstart, const u32 *__restrict__ chunk_row, u32 chunk,
                                 u64 max_pos, u64 j0, u64 count, u64 *__restrict__ out) {
    const u64 t = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count) return;
    const u64 j = j0 + t;
    u64 r = chunk_row[j / chunk];
    while (kstart[r + 1] <= j) r++;  // rows shorter than k hold no k-mers
    const u64 b = min(row_starts[r] + (j - kstart[r]), max_pos) << 1;
    const u64 w0 = words[b >> 6], w1 = words[(b >> 6) + 1];
    const u32 sh = (u32)(b & 63u);
    out[t] = (w0 << sh) | (dev::shr_clamp(w1, 63u - sh) >> 1);
}

__global__ void member_bits_kernel(const u64 *__restrict__ answers, u64 n, uint32_t *__restrict__ bits) {
    const u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    const bool hit = i < n && answers[i] != ~0ull;
    const u32 m = __ballot_sync(0xffffffffu, hit);
    if ((threadIdx.x & 31u) == 0 && (i >> 5) < (n + 31) / 32) bits[i >> 5] = m;
}

}  // namespace

int launch_pack(const uint8_t *d_letters, uint64_t n_letters, uint64_t *d_words, cudaStream_t s) {
    const u64 n_words = (n_letters + 32u + 31u) / 32u;  // ceil((n+32)/32), kmer_search.hpp:294
    const uintptr_t at = (uintptr_t)d_letters;
    const auto kern = at % 32u == 0 ? pack_kernel<32> : at % 16u == 0 ? pack_kernel<16> : pack_kernel<1>;
    const u64 per = kPackThreads * kPackWords;
    kern<<<(unsigned)((n_words + per - 1) / per), kPackThreads, 0, s>>>(d_letters, n_letters, d_words, n_words);
    SBWT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

// Packs the letters and makes the row table of a batch; *cleared: the counter has been zeroed too.
int launch_prep(const uint8_t *d_letters, uint64_t n_letters, uint64_t *d_words, const uint64_t *d_row_starts,
                uint64_t n_rows, uint32_t k, uint64_t *d_kstart, uint64_t *d_scan, uint64_t n_kmers, uint32_t chunk,
                uint32_t *d_chunk_row, unsigned long long *d_counter, bool *cleared, cudaStream_t s) {
    // letters bound the k-mers: a row table that adds up to more than n_kmers still fits 32 bits
    *cleared = n_rows <= kPrepRows && n_kmers <= kPrepKmers && n_letters <= 2ull * kPrepKmers;
    if (!*cleared) {
        SBWT_TRY(launch_pack(d_letters, n_letters, d_words, s));
        SBWT_TRY(launch_kstart(d_row_starts, n_rows, k, d_kstart, d_scan, s));
        return launch_chunk_rows(d_kstart, n_rows, n_kmers, chunk, d_chunk_row, s);
    }
    const u64 n_words = (n_letters + 32u + 31u) / 32u, per = kPrepThreads * kPackWords;
    const uintptr_t at = (uintptr_t)d_letters;
    const auto kern = at % 32u == 0 ? prep_kernel<32> : at % 16u == 0 ? prep_kernel<16> : prep_kernel<1>;
    kern<<<1u + (unsigned)((n_words + per - 1) / per), kPrepThreads, 0, s>>>(
        d_letters, n_letters, d_words, n_words, d_row_starts, (u32)n_rows, k, d_kstart,
        (u32)((n_kmers + chunk - 1) / chunk), chunk, d_chunk_row, d_counter);
    SBWT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

uint64_t scan_scratch_words(uint64_t n_items) { return scan_blocks(n_items) + 2; }

int launch_kstart(const uint64_t *d_row_starts, uint64_t n_rows, uint32_t k, uint64_t *d_kstart, uint64_t *d_scan,
                  cudaStream_t s) {
    KstartScan f{d_row_starts, d_kstart, k};
    cudaError_t e = device_scan(f, n_rows, d_scan, d_kstart + n_rows, s);
    if (e != cudaSuccess) return set_error("k-mer table scan failed: %s", cudaGetErrorString(e));
    return 0;
}

int launch_chunk_rows(const uint64_t *d_kstart, uint64_t n_rows, uint64_t n_kmers, uint32_t chunk,
                      uint32_t *d_chunk_row, cudaStream_t s) {
    const u64 n_chunks = (n_kmers + chunk - 1) / chunk;
    if (n_chunks == 0) return 0;
    chunk_rows_kernel<<<(unsigned)((n_chunks + 255) / 256), 256, 0, s>>>(d_kstart, n_rows, n_chunks, chunk,
                                                                         d_chunk_row);
    SBWT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

int launch_kmer_list(const SearchArgs &a, uint64_t j0, uint64_t count, uint64_t *d_out, cudaStream_t s) {
    if (count == 0) return 0;
    kmer_list_kernel<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(a.words, a.row_starts, a.kstart, a.chunk_row,
                                                                     a.chunk, a.max_pos, j0, count, d_out);
    SBWT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

int launch_member_bits(const uint64_t *d_answers, uint64_t n, uint32_t *d_bits, cudaStream_t s) {
    if (n == 0) return 0;
    const u64 threads = (n + 31) / 32 * 32;
    member_bits_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(d_answers, n, d_bits);
    SBWT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace sbwt
