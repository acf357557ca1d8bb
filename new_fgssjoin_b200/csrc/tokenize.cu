// tokenize.cu -- text -> token sets on the GPU.
//
// Semantics follow the reference's preprocessing and its shipped fixture:
//   lines            src/io.cpp:8-26 (split on '\n', empty lines skipped)
//   lower-case       src/preprocess/string/data.cpp:36-40 (ASCII A-Z only)
//   q-grams          src/preprocess/string/qgram.cpp:20-49 (unpadded; every
//                    repeat becomes its own token "gram"+occurrence); padding
//                    and distinct-gram modes are options
//   term ids         src/preprocess_cli.cpp:266-340: ascending document
//                    frequency; ties by first occurrence (line, position) as
//                    test/data/string/small.txt.3gram.bin shows
//   record layout    ids ascending per record, records by ascending size
//                    (ties by line) in a .bin, i.e. the reverse in memory
// Keys are exact: q <= 8 bytes are packed into 64 bits (the reference hashes
// the gram string with sdbm, src/util.cpp:146-157, which can collide); longer
// grams use a 64-bit FNV-1a hash.  k-mer mode packs canonical k-mers (k <= 32)
// of A/C/G/T into 2k bits, skipping windows with any other byte.
//
// Two pipelines.  tokenize_lines, for lines of at most kMaxLineGrams grams whose
// gram fits 63 bits: line bounds in two passes over the text -> per line, a warp
// numbers the occurrences of its grams in a shared-memory table (count, then fill)
// -> one sort by key' of (key', token number), runs = terms, df = run length, the
// first element = the first occurrence -> terms in first-occurrence order (marked
// tokens, scanned) sorted by df = term ids -> ids scattered back to the tokens ->
// records by size -> each record's tokens sorted by id in shared memory and
// written at its place.  tokenize_sorted, for the rest: the same steps as global
// stable sorts (gram, line, key', line and id).
//
// What bounds tokenize_lines is the copies of the text in and of the tokens and
// positions out (8 bytes a token over the link); on the device, the table and the
// sort of each line in shared memory and the one global sort.  The global-sort form
// moves 16-byte records through 9 to 11 radix passes and 8-byte keys through 16 to
// 20 more.  Call times, global sorts and lines (the sort passes the same, results
// copied whole), lines with the results in parts, and the copies out and in by
// themselves: 200,000 titles 7.2, 4.4, 4.1 (1.9 + 0.7) ms, 60,000 heavy-tailed records
// with occurrences 4.6, 3.8, 3.5 (1.2 + 0.5), 200,000 reads 23.6, 11.1, 10.2 (3.8 + 1.6).
#include <string.h>

#include <vector>

#include "ctx.h"
#include "pinned.h"
#include "prims.cuh"
#include "tokenize.h"

namespace fgss {

namespace {

__device__ __forceinline__ unsigned char lower_ascii(unsigned char c) {
    return (c <= 'Z' && c >= 'A') ? (unsigned char)(c - ('Z' - 'z')) : c;
}

__global__ void k_flag_newlines(const unsigned char* __restrict__ text, uint64_t n, uint32_t* __restrict__ flag) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        flag[i] = text[i] == '\n';
}

// Line k spans [start, end); line starts are 0 and every newline + 1.
__global__ void k_newlines(const uint32_t* __restrict__ flag, const uint32_t* __restrict__ scan, uint64_t n,
                        uint32_t n_lines, uint64_t* __restrict__ nl_pos) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        if (flag[i]) nl_pos[scan[i]] = i;
    (void)n_lines;
}

// Per raw line: bounds, non-empty flag.
__global__ void k_line_bounds(const uint64_t* __restrict__ nl_pos, uint32_t n_nl, uint64_t n_bytes,
                              uint64_t* __restrict__ lstart, uint32_t* __restrict__ llen,
                              uint32_t* __restrict__ nonempty) {
    const uint32_t nl = n_nl + 1;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nl; k += gridDim.x * blockDim.x) {
        uint64_t s = k == 0 ? 0 : nl_pos[k - 1] + 1;
        uint64_t e = k < n_nl ? nl_pos[k] : n_bytes;
        lstart[k] = s;
        llen[k] = (uint32_t)(e - s);
        nonempty[k] = e > s ? 1u : 0u;
    }
}

__global__ void k_compact_lines(const uint64_t* __restrict__ lstart, const uint32_t* __restrict__ llen,
                                const uint32_t* __restrict__ nonempty, const uint32_t* __restrict__ off, uint32_t nl,
                                uint64_t* __restrict__ ostart, uint32_t* __restrict__ olen) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nl; k += gridDim.x * blockDim.x)
        if (nonempty[k]) {
            ostart[off[k]] = lstart[k];
            olen[off[k]] = llen[k];
        }
}

__device__ __forceinline__ int base2(unsigned char c) {
    switch (lower_ascii(c)) {
        case 'a': return 0;
        case 'c': return 1;
        case 'g': return 2;
        case 't': return 3;
        default: return -1;
    }
}

// Grams per (non-empty) line.
__global__ void k_gram_count(const unsigned char* __restrict__ text, const uint64_t* __restrict__ ls,
                             const uint32_t* __restrict__ ll, uint32_t nlines, TokParams p, uint32_t* __restrict__ g) {
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; l < nlines; l += warps) {
        int64_t len = ll[l];
        if (p.mode == 0) {
            int64_t c = p.pad ? len + p.q - 1 : len - p.q + 1;
            if (lane_id() == 0) g[l] = c > 0 ? (uint32_t)c : 0u;
            continue;
        }
        // k-mers: windows of k bytes that are all A/C/G/T
        const unsigned char* t = text + ls[l];
        uint32_t cnt = 0;
        for (int64_t s = lane_id(); s + p.q <= len; s += 32) {
            bool ok = true;
            for (int i = 0; i < p.q && ok; i++) ok = base2(t[s + i]) >= 0;
            cnt += ok;
        }
        cnt = warp_sum(cnt);
        if (lane_id() == 0) g[l] = cnt;
    }
}

__device__ __forceinline__ unsigned char padded_at(const unsigned char* t, int64_t len, int64_t i, const TokParams& p) {
    // i indexes the padded line: [pad x (q-1)] line [pad x (q-1)]
    int64_t np = p.pad ? p.q - 1 : 0;
    int64_t j = i - np;
    if (j < 0 || j >= len) return (unsigned char)p.pad_char;
    unsigned char c = t[j];
    return p.lower ? lower_ascii(c) : c;
}

// Gram keys (line-major, position order) and their (line, position) tags.
__global__ void k_gram_fill(const unsigned char* __restrict__ text, const uint64_t* __restrict__ ls,
                            const uint32_t* __restrict__ ll, uint32_t nlines, TokParams p,
                            const uint32_t* __restrict__ goff, uint64_t* __restrict__ key, uint64_t* __restrict__ tag) {
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; l < nlines; l += warps) {
        int64_t len = ll[l];
        const unsigned char* t = text + ls[l];
        uint32_t o = goff[l];
        if (p.mode == 0) {
            int64_t g = p.pad ? len + p.q - 1 : len - p.q + 1;
            for (int64_t s = lane_id(); s < g; s += 32) {
                uint64_t k;
                if (p.q <= 8) {
                    k = 0;
                    for (int i = 0; i < p.q; i++) k = (k << 8) | padded_at(t, len, s + i, p);
                } else {
                    k = 1469598103934665603ULL;
                    for (int i = 0; i < p.q; i++) {
                        k ^= padded_at(t, len, s + i, p);
                        k *= 1099511628211ULL;
                    }
                }
                key[o + s] = k;
                tag[o + s] = ((uint64_t)l << 32) | (uint32_t)s;
            }
        } else {
            // k-mers: windows are written in position order with a warp-wide compaction
            uint32_t base = o;
            for (int64_t s0 = 0; s0 + p.q <= len; s0 += 32) {
                int64_t s = s0 + lane_id();
                bool ok = s + p.q <= len;
                uint64_t f = 0, r = 0;
                for (int i = 0; i < p.q && ok; i++) {
                    int c = base2(t[s + i]);
                    if (c < 0) { ok = false; break; }
                    f = (f << 2) | (uint64_t)c;
                    r |= (uint64_t)(3 - c) << (2 * i);
                }
                uint32_t m = __ballot_sync(kFull, ok);
                if (ok) {
                    uint32_t d = base + __popc(m & lanemask_lt());
                    key[d] = f < r ? f : r;
                    tag[d] = ((uint64_t)l << 32) | (uint32_t)s;
                }
                base += __popc(m);
            }
        }
    }
}

// After sorting by (line, gram, position): occurrence number (suffix mode) or
// first-of-run flag (distinct mode).  In suffix mode the key becomes
// gram << 16 | occurrence (q <= 6 keeps it within 64 bits).
__global__ void k_occurrence(const uint64_t* __restrict__ key, const uint64_t* __restrict__ tag, uint64_t n,
                             int suffix, uint64_t* __restrict__ key2, uint32_t* __restrict__ keep) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t k = key[i];
        uint32_t line = (uint32_t)(tag[i] >> 32);
        uint64_t j = i;
        while (j > 0 && key[j - 1] == k && (uint32_t)(tag[j - 1] >> 32) == line) j--;
        uint64_t occ = i - j;
        if (suffix) {
            key2[i] = (k << 16) | (occ < 0xffffu ? occ : 0xffffu);
            keep[i] = 1;
        } else {
            key2[i] = k;
            keep[i] = occ == 0;
        }
    }
}

__global__ void k_compact_tok(const uint64_t* __restrict__ key, const uint64_t* __restrict__ tag,
                              const uint32_t* __restrict__ keep, const uint32_t* __restrict__ off, uint64_t n,
                              uint64_t* __restrict__ okey, uint64_t* __restrict__ otag) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        if (keep[i]) {
            okey[off[i]] = key[i];
            otag[off[i]] = tag[i];
        }
}

// tag (line << 32 | pos) -> a 32-bit number that ascends with (line, pos), for the
// first-occurrence order: the gram's index, but of k-mers the window's place in the text (ls:
// the lines' starts; windows with other bytes are skipped, so goff does not count positions).
__global__ void k_tag_index(const uint64_t* __restrict__ tag, const uint32_t* __restrict__ goff,
                            const uint64_t* __restrict__ ls, int kmers, uint64_t n, uint32_t* __restrict__ gidx,
                            const uint32_t* __restrict__ err) {
    if (gave_up(err)) return;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t t = tag[i];
        gidx[i] = (kmers ? (uint32_t)ls[t >> 32] : goff[t >> 32]) + (uint32_t)t;
    }
}

// Runs of equal key (sorted): run-start flags
__global__ void k_run_flags(const uint64_t* __restrict__ key, uint64_t n, uint32_t* __restrict__ flag) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        flag[i] = (i == 0 || key[i] != key[i - 1]) ? 1u : 0u;
}

// Run id of every element (exclusive scan of the run-start flags) and the
// start index of every run.
__global__ void k_run_start(const uint32_t* __restrict__ flag, uint32_t* __restrict__ rid, uint64_t n,
                            uint32_t* __restrict__ rstart, const uint32_t* __restrict__ err) {
    if (gave_up(err)) return;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t r = rid[i] + flag[i] - 1;
        rid[i] = r;
        if (flag[i]) rstart[r] = (uint32_t)i;
    }
}

__global__ void k_run_keys2(const uint32_t* __restrict__ rstart, const uint32_t* __restrict__ gidx, uint64_t n,
                            uint32_t nruns, uint64_t* __restrict__ rkey, uint32_t* __restrict__ rval) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < nruns; r += gridDim.x * blockDim.x) {
        uint32_t s = rstart[r];
        uint32_t e = r + 1 < nruns ? rstart[r + 1] : (uint32_t)n;
        uint64_t df = e - s;
        rkey[r] = (df << 32) | gidx[s];  // sorted input: first element of a run is its first occurrence
        rval[r] = r;
    }
}

// rank of every run after the (df, first) sort -> term id per run
__global__ void k_run_ids(const uint32_t* __restrict__ rval_sorted, uint32_t nruns, uint32_t* __restrict__ id_of_run,
                          const uint32_t* __restrict__ err) {
    if (gave_up(err)) return;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nruns; k += gridDim.x * blockDim.x)
        id_of_run[rval_sorted[k]] = k;
}

// tokens -> (line << 32 | id) keys with the position as value
__global__ void k_line_id_keys(const uint32_t* __restrict__ rid, const uint32_t* __restrict__ id_of_run,
                               const uint64_t* __restrict__ tag, uint64_t n, uint64_t* __restrict__ k2,
                               uint32_t* __restrict__ pos) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t t = tag[i];
        k2[i] = (t & 0xffffffff00000000ull) | id_of_run[rid[i]];
        pos[i] = (uint32_t)t;
    }
}

// tokens per line (sorted by line): sizes via run boundaries
__global__ void k_line_bounds2(const uint64_t* __restrict__ k2, uint64_t n, uint32_t* __restrict__ lend,
                               uint32_t* __restrict__ loff, const uint32_t* __restrict__ err) {
    if (gave_up(err)) return;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t l = (uint32_t)(k2[i] >> 32);
        if (i == 0 || (uint32_t)(k2[i - 1] >> 32) != l) loff[l] = (uint32_t)i;
        if (i + 1 == n || (uint32_t)(k2[i + 1] >> 32) != l) lend[l] = (uint32_t)(i + 1);
    }
}

__global__ void k_line_sizes(const uint32_t* __restrict__ lend, const uint32_t* __restrict__ loff, uint32_t nlines,
                             uint32_t* __restrict__ lsz) {
    for (uint32_t l = blockIdx.x * blockDim.x + threadIdx.x; l < nlines; l += gridDim.x * blockDim.x)
        lsz[l] = lend[l] - loff[l];  // both zero for a line without tokens
}

// record sort keys: lines with tokens, key = (size << 32 | line); value = line
__global__ void k_rec_keys(const uint32_t* __restrict__ lsz, uint32_t nlines, uint64_t* __restrict__ rk,
                           uint32_t* __restrict__ rv) {
    for (uint32_t l = blockIdx.x * blockDim.x + threadIdx.x; l < nlines; l += gridDim.x * blockDim.x) {
        rk[l] = ((uint64_t)lsz[l] << 32) | l;
        rv[l] = l;
    }
}

// memory order i = file order reversed; file order = ascending (size, line)
// (empty records sort first in file order and are cut off at the end)
__global__ void k_rec_out(const uint32_t* __restrict__ rv_sorted, const uint32_t* __restrict__ lsz, uint32_t nlines,
                          uint32_t nempty, uint32_t* __restrict__ mline, uint32_t* __restrict__ mid,
                          uint32_t* __restrict__ mlen, const uint32_t* __restrict__ err) {
    if (gave_up(err)) return;
    const uint32_t nrec = nlines - nempty;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nrec; i += gridDim.x * blockDim.x) {
        uint32_t l = rv_sorted[nlines - 1 - i];
        mline[i] = l;
        mid[i] = l + 1;  // 1-based line number among the non-empty lines
        mlen[i] = lsz[l];
    }
}

__global__ void k_gather_rec(const uint32_t* __restrict__ mline, const uint32_t* __restrict__ moff, uint32_t nrec,
                             const uint32_t* __restrict__ loff, const uint32_t* __restrict__ lsz,
                             const uint64_t* __restrict__ k2, const uint32_t* __restrict__ pos,
                             uint32_t* __restrict__ otok, uint32_t* __restrict__ oloc,
                             const uint32_t* __restrict__ err) {
    if (gave_up(err)) return;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nrec; i += warps) {
        uint32_t l = mline[i], src = loff[l], n = lsz[l], dst = moff[i];
        for (uint32_t j = lane_id(); j < n; j += 32) {
            otok[dst + j] = (uint32_t)k2[src + j];
            oloc[dst + j] = pos[src + j];
        }
    }
}

__global__ void k_count_zero(const uint32_t* __restrict__ lsz, uint32_t n, uint32_t* out) {
    uint32_t c = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) c += lsz[i] == 0;
    c = warp_sum(c);
    if (lane_id() == 0 && c) atomicAdd(out, c);
}

int key_bits(const TokParams& p) {
    if (p.mode == 1) return 2 * p.q;
    if (p.q <= 8) return 8 * p.q;
    return 64;
}

int bits_for32(uint64_t v) {
    int b = 1;
    while (b < 64 && (1ull << b) < v) b++;
    return b;
}

// ------------------------------------------------------------ line by line

constexpr uint32_t kTextTile = 4096;       // text bytes per CTA of the line passes, 16 per thread
constexpr uint32_t kMaxLineGrams = 8192;   // grams of a line of tokenize_lines
constexpr uint64_t kPartTokens = 1 << 20;  // tokens from which a result is copied in parts
// Classes of lines by grams (a warp each; tables of 512 and 2048 slots at eight and
// four warps per CTA, beyond that of twice the longest line at one warp per CTA) and
// of records by tokens (a warp, 256 and 1024 threads each).
constexpr uint32_t kSmallLine = 256, kMidLine = 1024;

// Counters of one call, read back together.
struct TokCounts {
    uint32_t n_lines, max_grams, n_mid, n_long, max_occ, max_size, n_empty, n_tokens;
    uint32_t present[8];  // byte values that occur (after lower-casing)
};

// Bits of a thread's 16 bytes: non-empty lines start (byte after a newline or
// at the text's start that is no newline) and end (newline after another byte).
__device__ __forceinline__ void line_flags(const unsigned char* __restrict__ text, uint64_t base, uint64_t n,
                                           uint32_t (&w)[4], uint32_t& starts, uint32_t& ends) {
    const uint4 v = base < n ? *reinterpret_cast<const uint4*>(text + base) : make_uint4(0, 0, 0, 0);
    w[0] = v.x;
    w[1] = v.y;
    w[2] = v.z;
    w[3] = v.w;
    bool prev_nl = base == 0 || base > n || text[base - 1] == '\n';
    starts = ends = 0;
#pragma unroll
    for (uint32_t i = 0; i < 16; i++) {
        const bool in = base + i < n, nl = ((w[i >> 2] >> (8 * (i & 3))) & 0xffu) == '\n';
        if (in && !nl && prev_nl) starts |= 1u << i;
        if (in && nl && !prev_nl) ends |= 1u << i;
        prev_nl = nl;
    }
}

// Line starts per tile and the byte values that occur.
__global__ void __launch_bounds__(256) k_text_count(const unsigned char* __restrict__ text, uint64_t n, int lower,
                                                    uint32_t* __restrict__ tile_starts, TokCounts* cnt) {
    __shared__ uint32_t s_mask[8], s_wsum[33];
    if (threadIdx.x < 8) s_mask[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t base = (uint64_t)blockIdx.x * kTextTile + threadIdx.x * 16;
    uint32_t w[4], starts, ends;
    line_flags(text, base, n, w, starts, ends);
    uint32_t m[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (uint32_t i = 0; i < 16; i++) {
        if (base + i >= n) break;
        unsigned char c = (unsigned char)(w[i >> 2] >> (8 * (i & 3)));
        if (lower) c = lower_ascii(c);
#pragma unroll
        for (uint32_t k = 0; k < 8; k++)
            if (c >> 5 == k) m[k] |= 1u << (c & 31);
    }
#pragma unroll
    for (uint32_t k = 0; k < 8; k++) {
        const uint32_t all = __reduce_or_sync(kFull, m[k]);
        if (lane_id() == 0 && all) atomicOr(&s_mask[k], all);
    }
    uint32_t total;
    block_excl_scan<uint32_t>(__popc(starts), s_wsum, &total);
    if (threadIdx.x == 0) tile_starts[blockIdx.x] = total;
    if (threadIdx.x < 8 && s_mask[threadIdx.x] & ~cnt->present[threadIdx.x])
        atomicOr(&cnt->present[threadIdx.x], s_mask[threadIdx.x]);
}

// Bounds of the non-empty lines (the k-th start belongs to the k-th end).
__global__ void __launch_bounds__(256) k_text_lines(const unsigned char* __restrict__ text, uint64_t n,
                                                    const uint32_t* __restrict__ tile_off, uint32_t* __restrict__ lstart,
                                                    uint32_t* __restrict__ lend, const uint32_t* __restrict__ err) {
    __shared__ uint32_t s_wsum[33];
    if (gave_up(err)) return;
    const uint64_t base = (uint64_t)blockIdx.x * kTextTile + threadIdx.x * 16;
    uint32_t w[4], starts, ends, total;
    line_flags(text, base, n, w, starts, ends);
    uint32_t k = tile_off[blockIdx.x] + block_excl_scan<uint32_t>(__popc(starts), s_wsum, &total);
#pragma unroll
    for (uint32_t i = 0; i < 16; i++) {
        if (ends >> i & 1u) lend[k - 1] = (uint32_t)(base + i);
        if (starts >> i & 1u) lstart[k++] = (uint32_t)(base + i);
        if (base + i + 1 == n && ((w[i >> 2] >> (8 * (i & 3))) & 0xffu) != '\n') lend[k - 1] = (uint32_t)n;
    }
}

__device__ __forceinline__ uint32_t line_grams(uint32_t len, const TokParams& p) {  // windows of q bytes
    const int64_t g = p.mode == 0 && p.pad ? (int64_t)len + p.q - 1 : (int64_t)len - p.q + 1;
    return g > 0 ? (uint32_t)g : 0u;
}

// The largest line, and the lists of the lines of more than kSmallLine grams (mid
// from the front, long ones from the back).
__global__ void k_line_classes(const uint32_t* __restrict__ lstart, const uint32_t* __restrict__ lend, TokParams p,
                               TokCounts* cnt, uint32_t* __restrict__ list, uint32_t list_cap,
                               const uint32_t* __restrict__ err) {
    if (gave_up(err)) return;
    const uint32_t nl = cnt->n_lines;
    uint32_t mx = 0;
    for (uint32_t l = blockIdx.x * blockDim.x + threadIdx.x; l < nl; l += gridDim.x * blockDim.x) {
        const uint32_t g = line_grams(lend[l] - lstart[l], p);
        mx = max(mx, g);
        if (g > kMidLine) list[list_cap - 1 - atomicAdd(&cnt->n_long, 1u)] = l;
        else if (g > kSmallLine) list[atomicAdd(&cnt->n_mid, 1u)] = l;
    }
    mx = __reduce_max_sync(kFull, mx);
    if (lane_id() == 0 && mx) atomicMax(&cnt->max_grams, mx);
}

// Grams of line l in rows of 32 positions, a warp per line: f(position, key,
// valid) for every row (all lanes).  q-grams: the dense codes of q bytes.
// k-mers: canonical = the smaller of the window and its reverse complement as
// (high bits, low bits) of the two-bit codes, taken from the row's ballots.
template <typename K, typename F>
__device__ __forceinline__ void for_grams(const unsigned char* __restrict__ t, uint32_t len, const TokParams& p,
                                          const uint8_t* lut, int cb, F&& f) {
    const uint32_t lane = lane_id(), g = line_grams(len, p);
    if (p.mode == 1) {
        const uint32_t mk = p.q == 32 ? 0xffffffffu : (1u << p.q) - 1u;
        uint32_t b0 = 0, b1 = 0, ok = 0;
        auto load = [&](uint32_t s0, uint32_t& x0, uint32_t& x1, uint32_t& v) {
            const int c = s0 + lane < len ? base2(t[s0 + lane]) : -1;
            x0 = __ballot_sync(kFull, c & 1);
            x1 = __ballot_sync(kFull, c & 2);
            v = __ballot_sync(kFull, c >= 0);
        };
        load(0, b0, b1, ok);
        for (uint32_t s0 = 0; s0 < g; s0 += 32) {
            uint32_t n0, n1, nk;
            load(s0 + 32, n0, n1, nk);
            const uint32_t lo = __funnelshift_r(b0, n0, lane) & mk, hi = __funnelshift_r(b1, n1, lane) & mk;
            const bool valid = s0 + lane < g && (__funnelshift_r(ok, nk, lane) & mk) == mk;
            const uint32_t rlo = __brev(~lo) >> (32 - p.q), rhi = __brev(~hi) >> (32 - p.q);
            const K a = (K)((uint64_t)hi << p.q | lo), b = (K)((uint64_t)rhi << p.q | rlo);
            f(s0 + lane, a < b ? a : b, valid);
            b0 = n0;
            b1 = n1;
            ok = nk;
        }
        return;
    }
    const int32_t np = p.pad ? p.q - 1 : 0;
    auto code = [&](uint32_t s) -> uint32_t {  // of byte s of the padded line
        const int32_t j = (int32_t)s - np;
        return lut[j >= 0 && j < (int32_t)len ? t[j] : (unsigned char)p.pad_char + 256u];
    };
    uint32_t c = code(lane);
    for (uint32_t s0 = 0; s0 < g; s0 += 32) {
        const uint32_t nx = code(s0 + 32 + lane);
        K k = (K)c;
        for (int i = 1; i < p.q; i++) {
            const uint32_t src = lane + i, u = __shfl_sync(kFull, c, src & 31u), v = __shfl_sync(kFull, nx, src & 31u);
            k = k << cb | (K)(src < 32 ? u : v);
        }
        f(s0 + lane, k, s0 + lane < g);
        c = nx;
    }
}

template <typename K>
__device__ __forceinline__ K shared_cas(K* p, K cmp, K v);
template <>
__device__ __forceinline__ uint32_t shared_cas(uint32_t* p, uint32_t cmp, uint32_t v) {
    return atomicCAS(p, cmp, v);
}
template <>
__device__ __forceinline__ uint64_t shared_cas(uint64_t* p, uint64_t cmp, uint64_t v) {
    return atomicCAS(reinterpret_cast<unsigned long long*>(p), (unsigned long long)cmp, (unsigned long long)v);
}
__device__ __forceinline__ uint32_t gram_hash(uint32_t k) { return k * 0x9E3779B1u; }
__device__ __forceinline__ uint32_t gram_hash(uint64_t k) {
    return (uint32_t)((k * 0x9E3779B97F4A7C15ull) >> 32);
}

// A warp's open-addressing table for one line: gram -> first position (distinct
// mode) or occurrences so far (suffix mode); `slots` is at least twice the grams.
// fill: writes key' (gram << ob | occurrence), token number and position of the
// kept grams, in position order, from token o; else only counts.  Returns the
// kept grams.
template <typename K, typename KO>
__device__ __forceinline__ uint32_t line_tokens(const unsigned char* __restrict__ t, uint32_t len, const TokParams& p,
                                                const uint8_t* lut, int cb, K* tab, uint32_t* val, uint32_t slots,
                                                bool fill, int ob, uint32_t o, KO* __restrict__ key,
                                                uint32_t* __restrict__ num, uint32_t* __restrict__ pos,
                                                uint32_t& max_occ) {
    const uint32_t lane = lane_id(), lt = lanemask_lt();
    const bool suffix = p.mode == 0 && p.suffix;
    const K none = ~K(0);
    for (uint32_t i = lane; i < slots; i += 32) {
        tab[i] = none;
        val[i] = suffix ? 0u : 0xffffffffu;
    }
    __syncwarp();
    const int sh = 32 - (31 - __clz((int)slots));
    uint32_t kept = 0;
    for_grams<K>(t, len, p, lut, cb, [&](uint32_t s, K k, bool valid) {
        uint32_t h = gram_hash(k) >> sh;
        if (valid) {
            for (uint32_t i = 0; i < slots; i++) {  // (half the slots stay free: one is found)
                const K old = shared_cas(&tab[h], none, k);
                if (old == none || old == k) break;
                h = (h + 1) & (slots - 1);
            }
        }
        uint32_t occ = 0;
        bool keep = valid;
        if (suffix) {
            const uint32_t peers = __match_any_sync(kFull, valid ? h : slots + lane);
            const uint32_t before = valid ? val[h] : 0u;
            __syncwarp();
            if (valid && (peers & lt) == 0) val[h] = before + __popc(peers);
            occ = before + __popc(peers & lt);
            if (valid) max_occ = max(max_occ, occ);
        } else {
            if (valid) atomicMin(&val[h], s);
            __syncwarp();
            keep = valid && val[h] == s;
        }
        const uint32_t m = __ballot_sync(kFull, keep);
        if (fill && keep) {
            const uint32_t at = o + kept + __popc(m & lt);
            key[at] = (KO)k << ob | (KO)occ;
            num[at] = at;
            pos[at] = s;
        }
        kept += __popc(m);
        __syncwarp();
    });
    return kept;
}

// Warp per line: list == nullptr: every line of at most kSmallLine grams, else the
// n listed ones.  Table of `slots` at most (dynamic shared memory).
template <typename K, typename KO>
__global__ void k_lines(const unsigned char* __restrict__ text, const uint32_t* __restrict__ lstart,
                        const uint32_t* __restrict__ lend, const uint32_t* __restrict__ list, uint32_t n, TokParams p,
                        const uint8_t* __restrict__ glut, int cb, uint32_t slots, bool fill, int ob,
                        uint32_t* __restrict__ lsz, const uint32_t* __restrict__ loff, KO* __restrict__ key,
                        uint32_t* __restrict__ num, uint32_t* __restrict__ pos, TokCounts* cnt) {
    extern __shared__ __align__(16) unsigned char s_tab[];
    __shared__ uint8_t lut[512];  // code of a byte; of the padding byte from 256 on
    for (uint32_t i = threadIdx.x; i < 512; i += blockDim.x) lut[i] = glut[i];
    __syncthreads();
    const uint32_t nw = blockDim.x >> 5, wid = threadIdx.x >> 5;
    K* tab = reinterpret_cast<K*>(s_tab) + (size_t)wid * slots;
    uint32_t* val = reinterpret_cast<uint32_t*>(reinterpret_cast<K*>(s_tab) + (size_t)nw * slots) + (size_t)wid * slots;
    uint32_t max_occ = 0, max_size = 0, n_empty = 0;
    for (uint32_t i = blockIdx.x * nw + wid; i < n; i += gridDim.x * nw) {
        const uint32_t l = list ? list[i] : i, a = lstart[l], len = lend[l] - a, g = line_grams(len, p);
        if (!list && g > kSmallLine) continue;
        uint32_t use = 64;
        while (use < 2 * g) use <<= 1;
        const uint32_t kept = g == 0 ? 0u : line_tokens<K, KO>(text + a, len, p, lut, cb, tab, val, use, fill, ob,
                                                               fill ? loff[l] : 0u, key, num, pos, max_occ);
        if (!fill && lane_id() == 0) {
            lsz[l] = kept;
            max_size = max(max_size, kept);
            n_empty += kept == 0;
        }
        __syncwarp();
    }
    if (fill) return;
    max_occ = __reduce_max_sync(kFull, max_occ);
    if (lane_id() == 0) {
        if (max_occ) atomicMax(&cnt->max_occ, max_occ);
        if (max_size) atomicMax(&cnt->max_size, max_size);
        if (n_empty) atomicAdd(&cnt->n_empty, n_empty);
    }
}

template <typename KO>
__global__ void k_key_flags(const KO* __restrict__ key, uint32_t n, uint32_t* __restrict__ flag) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        flag[i] = (i == 0 || key[i] != key[i - 1]) ? 1u : 0u;
}

// Marks every term's first token with the term's run + 1.
__global__ void k_mark_first(const uint32_t* __restrict__ rstart, const uint32_t* __restrict__ num, uint32_t nruns,
                             uint32_t* __restrict__ mark) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < nruns; r += gridDim.x * blockDim.x)
        mark[num[rstart[r]]] = r + 1;
}

__global__ void k_nonzero(const uint32_t* __restrict__ mark, uint32_t n, uint32_t* __restrict__ flag) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) flag[i] = mark[i] != 0;
}

// Terms in first-occurrence order: their df and run.
__global__ void k_term_order(const uint32_t* __restrict__ mark, const uint32_t* __restrict__ rank, uint32_t n,
                             const uint32_t* __restrict__ rstart, uint32_t nruns, uint32_t* __restrict__ df,
                             uint32_t* __restrict__ run, const uint32_t* __restrict__ err) {
    if (gave_up(err)) return;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (mark[i] == 0) continue;
        const uint32_t r = mark[i] - 1, e = r + 1 < nruns ? rstart[r + 1] : n;
        df[rank[i]] = e - rstart[r];
        run[rank[i]] = r;
    }
}

// Term id of every token, in token order.
__global__ void k_token_ids(const uint32_t* __restrict__ rid, const uint32_t* __restrict__ id_of_run,
                            const uint32_t* __restrict__ num, uint32_t n, uint32_t* __restrict__ id) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        id[num[i]] = id_of_run[rid[i]];
}

__global__ void k_size_keys(const uint32_t* __restrict__ lsz, uint32_t n, uint32_t* __restrict__ key,
                            uint32_t* __restrict__ val) {
    for (uint32_t l = blockIdx.x * blockDim.x + threadIdx.x; l < n; l += gridDim.x * blockDim.x) {
        key[l] = lsz[l];
        val[l] = l;
    }
}

// Ascending bitonic sort of v[0 .. n) by `threads` threads (t of them); every
// comparison orders its pair the same way, so a pair with an element past n is
// skipped as if that were larger than all.
template <typename S, typename Sync>
__device__ __forceinline__ void sort_shared(S* v, uint32_t n, uint32_t t, uint32_t threads, Sync&& sync) {
    uint32_t m = 1;
    while (m < n) m <<= 1;
    for (uint32_t k = 2; k <= m; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t x = t; x < m / 2; x += threads) {
                const uint32_t a = (x / j) * 2 * j + (x & (j - 1));
                const uint32_t b = 2 * j == k ? (a | (k - 1)) - (a & (k - 1)) : a + j;  // first step of a merge: mirrored
                if (b < n) {
                    const S p = v[a], q = v[b];
                    if (q < p) {
                        v[a] = q;
                        v[b] = p;
                    }
                }
            }
            sync();
        }
    }
}

// Records [first, end) of (lo, hi] tokens: tokens sorted by id, written at the record's
// place (records are in descending size, so each class is a run of them).  S:
// id << pb | position, 32 bits where that fits.  WARP: a warp per record, else a CTA.
template <typename S, bool WARP>
__global__ void k_records(const uint32_t* __restrict__ mline, const uint32_t* __restrict__ mlen,
                          const uint32_t* __restrict__ moff, uint32_t first, uint32_t end, uint32_t lo,
                          uint32_t hi, const uint32_t* __restrict__ loff, const uint32_t* __restrict__ id,
                          const uint32_t* __restrict__ pos, int pb, uint32_t* __restrict__ otok,
                          uint32_t* __restrict__ oloc, const uint32_t* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char s_rec[];
    if (gave_up(err)) return;
    const uint32_t nw = WARP ? blockDim.x >> 5 : 1, wid = WARP ? threadIdx.x >> 5 : 0;
    const uint32_t t = WARP ? lane_id() : threadIdx.x, nt = WARP ? 32 : blockDim.x;
    S* v = reinterpret_cast<S*>(s_rec) + (size_t)wid * hi;
    auto sync = [] {
        if (WARP) __syncwarp();
        else __syncthreads();
    };
    const S pm = ((S)1 << pb) - 1;
    for (uint32_t i = first + blockIdx.x * nw + wid; i < end; i += gridDim.x * nw) {
        const uint32_t n = mlen[i];
        if (n <= lo) break;  // shorter ones only from here on
        if (n > hi) continue;
        const uint32_t src = loff[mline[i]], dst = moff[i];
        for (uint32_t j = t; j < n; j += nt) v[j] = (S)id[src + j] << pb | (S)pos[src + j];
        sync();
        sort_shared(v, n, t, nt, sync);
        for (uint32_t j = t; j < n; j += nt) {
            otok[dst + j] = (uint32_t)(v[j] >> pb);
            oloc[dst + j] = (uint32_t)(v[j] & pm);
        }
        sync();
    }
}

uint32_t read_u32(Ctx& c, const uint32_t* d) {
    uint32_t* h = c.pinnedT<uint32_t>("tk.h", 4);
    FGSS_CK(cudaMemcpyAsync(h, d, 4, cudaMemcpyDeviceToHost, c.stream));
    c.sync();
    return *h;
}

}  // namespace

namespace {

// The records in device memory to the caller's host arrays.
void copy_out(Ctx& c, fgss_sets* out, uint32_t nrec, uint64_t T, uint32_t V, const uint32_t* mid, const uint32_t* mlen,
              const uint32_t* moff, const uint32_t* otok, const uint32_t* oloc) {
    out->n_sets = nrec;
    out->n_tokens = T;
    out->n_terms = V;
    alloc_host_sets(out, nrec, T, true);
    if (nrec) {
        FGSS_CK(cudaMemcpyAsync(out->id, mid, (uint64_t)nrec * 4, cudaMemcpyDeviceToHost, c.stream));
        FGSS_CK(cudaMemcpyAsync(out->len, mlen, (uint64_t)nrec * 4, cudaMemcpyDeviceToHost, c.stream));
        FGSS_CK(cudaMemcpyAsync(out->pos, moff, (uint64_t)nrec * 4, cudaMemcpyDeviceToHost, c.stream));
    }
    FGSS_CK(cudaMemcpyAsync(out->tokens, otok, T * 4, cudaMemcpyDeviceToHost, c.stream));
    FGSS_CK(cudaMemcpyAsync(out->loc, oloc, T * 4, cudaMemcpyDeviceToHost, c.stream));
    c.sync();
    out->max_len = nrec ? out->len[0] : 0;  // descending sizes
}

// One class of lines (k_lines): warps per CTA and table slots per warp sized for
// `grams` grams at most.
template <typename K, typename KO>
void launch_lines(Ctx& c, const unsigned char* text, const uint32_t* lstart, const uint32_t* lend, const uint32_t* list,
                  uint32_t n, const TokParams& p, const uint8_t* lut, int cb, uint32_t grams, int warps, bool fill, int ob,
                  uint32_t* lsz, const uint32_t* loff, KO* key, uint32_t* num, uint32_t* pos, TokCounts* cnt) {
    if (n == 0) return;
    uint32_t slots = 64;
    while (slots < 2 * grams) slots <<= 1;
    const size_t smem = (size_t)warps * slots * (sizeof(K) + 4);
    // Every launch sets the largest table of any class, not its own: the limit belongs to the
    // function, which all contexts of a device share, and a thread that lowered it between
    // another one's setting and launch would have that launch refused.
    constexpr int kMost = (int)(2 * kMaxLineGrams * (sizeof(K) + 4));
    static_assert(8 * 2 * kSmallLine <= 2 * kMaxLineGrams && 4 * 2 * kMidLine <= 2 * kMaxLineGrams, "largest table");
    if (smem + 1024 > 48 * 1024)  // (with the static code table)
        FGSS_CK(cudaFuncSetAttribute(k_lines<K, KO>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
    k_lines<K, KO><<<grid_for(n, warps, c.num_sms * 16), warps * 32, smem, c.stream>>>(
        text, lstart, lend, list, n, p, lut, cb, slots, fill, ob, lsz, loff, key, num, pos, cnt);
    FGSS_LAUNCH_CK();
}

// tokenize_lines from the kept grams on: K' = KO keys of kbits bits.
template <typename K, typename KO>
void tokenize_terms(Ctx& c, const unsigned char* dtext, const uint32_t* lstart, const uint32_t* lend, const TokParams& p,
                    const uint8_t* lut, int cb, uint32_t lcap, const uint32_t* list, const TokCounts& h, int ob, int kbits,
                    uint32_t* lsz, uint32_t* loff, TokCounts* cnt, fgss_sets* out) {
    const uint32_t nl = h.n_lines, T = h.n_tokens;
    KO* key = c.devT<KO>("tl.key", (uint64_t)T + 1);
    uint32_t* num = c.devT<uint32_t>("tl.num", (uint64_t)T + 1);
    uint32_t* pos = c.devT<uint32_t>("tl.pos", (uint64_t)T + 1);
    launch_lines<K, KO>(c, dtext, lstart, lend, nullptr, nl, p, lut, cb, kSmallLine, 8, true, ob, lsz, loff, key, num,
                        pos, cnt);
    launch_lines<K, KO>(c, dtext, lstart, lend, list, h.n_mid, p, lut, cb, kMidLine, 4, true, ob, lsz, loff, key, num,
                        pos, cnt);
    launch_lines<K, KO>(c, dtext, lstart, lend, list + (lcap - h.n_long), h.n_long, p, lut, cb, h.max_grams, 1, true, ob,
                        lsz, loff, key, num, pos, cnt);
    // terms: runs of equal key' after a stable sort
    radix_sort<KO, uint32_t>(c, key, num, T, nullptr, 0, kbits, "tl.sort");
    uint32_t* flag = c.devT<uint32_t>("tl.flag", (uint64_t)T + 1);
    uint32_t* rid = c.devT<uint32_t>("tl.rid", (uint64_t)T + 1);
    uint32_t* rstart = c.devT<uint32_t>("tl.rstart", (uint64_t)T + 1);
    uint32_t* tot = c.devT<uint32_t>("tl.tot", 2);
    const unsigned gT = grid_for(T, 256, c.num_sms * 32);
    k_key_flags<KO><<<gT, 256, 0, c.stream>>>(key, T, flag);
    FGSS_LAUNCH_CK();
    exclusive_scan<uint32_t>(c, flag, rid, T, nullptr, tot, "tl.s.run");
    k_run_start<<<gT, 256, 0, c.stream>>>(flag, rid, T, rstart, c.err_dev);
    FGSS_LAUNCH_CK();
    const uint32_t V = read_u32(c, tot);
    // term ids: first-occurrence order, then a stable sort by document frequency
    uint32_t* mark = c.devT<uint32_t>("tl.mark", (uint64_t)T + 1);
    uint32_t* df = c.devT<uint32_t>("tl.df", (uint64_t)V + 1);
    uint32_t* run = c.devT<uint32_t>("tl.run", (uint64_t)V + 1);
    uint32_t* id_of_run = c.devT<uint32_t>("tl.idrun", (uint64_t)V + 1);
    const unsigned gV = grid_for(V, 256, c.num_sms * 32);
    FGSS_CK(cudaMemsetAsync(mark, 0, (uint64_t)T * 4, c.stream));
    k_mark_first<<<gV, 256, 0, c.stream>>>(rstart, num, V, mark);
    FGSS_LAUNCH_CK();
    k_nonzero<<<gT, 256, 0, c.stream>>>(mark, T, flag);
    FGSS_LAUNCH_CK();
    exclusive_scan<uint32_t>(c, flag, flag, T, nullptr, (uint32_t*)nullptr, "tl.s.first");
    k_term_order<<<gT, 256, 0, c.stream>>>(mark, flag, T, rstart, V, df, run, c.err_dev);
    FGSS_LAUNCH_CK();
    radix_sort<uint32_t, uint32_t>(c, df, run, V, nullptr, 0, bits_for32((uint64_t)nl + 1), "tl.dfsort");
    k_run_ids<<<gV, 256, 0, c.stream>>>(run, V, id_of_run, c.err_dev);
    FGSS_LAUNCH_CK();
    uint32_t* id = mark;  // (the marks are done with)
    k_token_ids<<<gT, 256, 0, c.stream>>>(rid, id_of_run, num, T, id);
    FGSS_LAUNCH_CK();
    // records by (size, line), memory order = descending
    uint32_t* rk = c.devT<uint32_t>("tl.rk", (uint64_t)nl + 1);
    uint32_t* rv = c.devT<uint32_t>("tl.rv", (uint64_t)nl + 1);
    k_size_keys<<<grid_for(nl, 256), 256, 0, c.stream>>>(lsz, nl, rk, rv);
    FGSS_LAUNCH_CK();
    radix_sort<uint32_t, uint32_t>(c, rk, rv, nl, nullptr, 0, bits_for32((uint64_t)h.max_size + 1), "tl.recsort");
    const uint32_t nrec = nl - h.n_empty;
    uint32_t* mline = c.devT<uint32_t>("tl.mline", (uint64_t)nrec + 1);
    uint32_t* mid = c.devT<uint32_t>("tl.mid", (uint64_t)nrec + 1);
    uint32_t* mlen = c.devT<uint32_t>("tl.mlen", (uint64_t)nrec + 1);
    uint32_t* moff = c.devT<uint32_t>("tl.moff", (uint64_t)nrec + 1);
    k_rec_out<<<grid_for(nrec, 256), 256, 0, c.stream>>>(rv, lsz, nl, h.n_empty, mline, mid, mlen, c.err_dev);
    FGSS_LAUNCH_CK();
    exclusive_scan<uint32_t>(c, mlen, moff, nrec, nullptr, (uint32_t*)nullptr, "tl.s.rec");
    uint32_t* otok = c.devT<uint32_t>("tl.otok", (uint64_t)T + 1);
    uint32_t* oloc = c.devT<uint32_t>("tl.oloc", (uint64_t)T + 1);
    const int pb = bits_for32((uint64_t)h.max_grams + 1);
    auto records = [&](auto tag, uint32_t a, uint32_t b) {
        using S = decltype(tag);
        k_records<S, true><<<grid_for(b - a, 8, c.num_sms * 16), 256, 8 * kSmallLine * sizeof(S), c.stream>>>(
            mline, mlen, moff, a, b, 0, kSmallLine, loff, id, pos, pb, otok, oloc, c.err_dev);
        FGSS_LAUNCH_CK();
        // (sizes descend: the longer ones are among the first)
        if (h.max_size > kSmallLine && a < h.n_mid + h.n_long) {
            k_records<S, false><<<grid_for(h.n_mid + h.n_long - a, 1, c.num_sms * 8), 256, kMidLine * sizeof(S), c.stream>>>(
                mline, mlen, moff, a, b, kSmallLine, kMidLine, loff, id, pos, pb, otok, oloc, c.err_dev);
            FGSS_LAUNCH_CK();
        }
        if (h.max_size > kMidLine && a < h.n_long) {
            const size_t smem = (size_t)h.max_size * sizeof(S);
            FGSS_CK(cudaFuncSetAttribute(k_records<S, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(kMaxLineGrams * sizeof(S))));
            k_records<S, false><<<grid_for(h.n_long - a, 1, c.num_sms * 2), 1024, smem, c.stream>>>(
                mline, mlen, moff, a, b, kMidLine, h.max_size, loff, id, pos, pb, otok, oloc, c.err_dev);
            FGSS_LAUNCH_CK();
        }
    };
    const bool narrow = bits_for32((uint64_t)V + 1) + pb <= 32;
    auto part = [&](uint32_t a, uint32_t b) {
        if (narrow) records(uint32_t(), a, b);
        else records(uint64_t(), a, b);
    };
    // A large result goes to the host in parts, each while the next one's records are sorted:
    // 200,000 reads of 27 M tokens 11.3 -> 10.2 ms of the call, 200,000 titles 4.85 -> 4.28, 60,000
    // heavy-tailed texts 4.13 -> 3.72 (in four equal parts, the first the longest: 10.6, 4.33, 3.92).
    // Below 2^20 tokens (8 MB) the copies take no longer than the extra launches and events.
    if (T < kPartTokens || nrec < Ctx::kCopyParts) {
        part(0, nrec);
        copy_out(c, out, nrec, T, V, mid, mlen, moff, otok, oloc);
        return;
    }
    out->n_sets = nrec;
    out->n_tokens = T;
    out->n_terms = V;
    alloc_host_sets(out, nrec, T, true);
    c.copy_lane();
    struct Settle {  // no copy is in flight when the call returns or fails
        Ctx& c;
        ~Settle() {
            if (cudaStreamSynchronize(c.copy_stream) != cudaSuccess) (void)cudaGetLastError();
        }
    } settle{c};
    constexpr int kParts = Ctx::kCopyParts;
    uint32_t cut[kParts + 1], *hcut = c.pinnedT<uint32_t>("tl.hcut", kParts + 1);
    // the first part's sort is the one that no copy hides, and its records are the longest
    for (int i = 0; i <= kParts; i++) cut[i] = (uint32_t)((uint64_t)nrec * ((1u << i) - 1) / ((1u << kParts) - 1));
    for (int i = 1; i < kParts; i++)
        FGSS_CK(cudaMemcpyAsync(hcut + i, moff + cut[i], 4, cudaMemcpyDeviceToHost, c.stream));
    FGSS_CK(cudaEventRecord(c.copy_ev[kParts], c.stream));
    for (int i = 0; i < kParts; i++) {
        part(cut[i], cut[i + 1]);
        FGSS_CK(cudaEventRecord(c.copy_ev[i], c.stream));
    }
    FGSS_CK(cudaEventSynchronize(c.copy_ev[kParts]));
    c.check_waits();  // before the parts' bounds are used
    hcut[0] = 0;
    hcut[kParts] = T;
    cudaStream_t cs = c.copy_stream;
    FGSS_CK(cudaMemcpyAsync(out->id, mid, (uint64_t)nrec * 4, cudaMemcpyDeviceToHost, cs));
    FGSS_CK(cudaMemcpyAsync(out->len, mlen, (uint64_t)nrec * 4, cudaMemcpyDeviceToHost, cs));
    FGSS_CK(cudaMemcpyAsync(out->pos, moff, (uint64_t)nrec * 4, cudaMemcpyDeviceToHost, cs));
    for (int i = 0; i < kParts; i++) {
        const uint64_t o = hcut[i], n = hcut[i + 1] - o;
        FGSS_CK(cudaStreamWaitEvent(cs, c.copy_ev[i], 0));
        FGSS_CK(cudaMemcpyAsync(out->tokens + o, otok + o, n * 4, cudaMemcpyDeviceToHost, cs));
        FGSS_CK(cudaMemcpyAsync(out->loc + o, oloc + o, n * 4, cudaMemcpyDeviceToHost, cs));
    }
    FGSS_CK(cudaStreamSynchronize(cs));
    c.sync();
    out->max_len = out->len[0];  // descending sizes
}

void tokenize_sorted(Ctx& c, const unsigned char* dtext, uint64_t nb, const TokParams& p, fgss_sets* out);

// Lines, their classes and the tokens of each; false when the text needs
// tokenize_sorted (a longer line, or grams of more bits).
bool tokenize_lines(Ctx& c, const unsigned char* dtext, uint64_t nb, const TokParams& p, fgss_sets* out) {
    if (p.mode == 0 && p.q > 8) return false;
    const uint32_t ntiles = (uint32_t)((nb + kTextTile - 1) / kTextTile), lcap = (uint32_t)(nb / 2 + 1);
    TokCounts* cnt = c.devT<TokCounts>("tl.cnt", 1);
    TokCounts* h = c.pinnedT<TokCounts>("tl.h", 1);
    uint32_t* toff = c.devT<uint32_t>("tl.toff", (uint64_t)ntiles + 1);
    uint32_t* lstart = c.devT<uint32_t>("tl.lstart", lcap);
    uint32_t* lend = c.devT<uint32_t>("tl.lend", lcap);
    uint32_t* list = c.devT<uint32_t>("tl.list", lcap);
    FGSS_CK(cudaMemsetAsync(cnt, 0, sizeof(TokCounts), c.stream));
    k_text_count<<<ntiles, 256, 0, c.stream>>>(dtext, nb, p.mode == 0 && p.lower, toff, cnt);
    FGSS_LAUNCH_CK();
    exclusive_scan<uint32_t>(c, toff, toff, ntiles, nullptr, &cnt->n_lines, "tl.s.tile");
    k_text_lines<<<ntiles, 256, 0, c.stream>>>(dtext, nb, toff, lstart, lend, c.err_dev);
    FGSS_LAUNCH_CK();
    k_line_classes<<<grid_for(lcap, 256, c.num_sms * 8), 256, 0, c.stream>>>(lstart, lend, p, cnt, list, lcap,
                                                                                c.err_dev);
    FGSS_LAUNCH_CK();
    FGSS_CK(cudaMemcpyAsync(h, cnt, sizeof(TokCounts), cudaMemcpyDeviceToHost, c.stream));
    c.sync();
    const uint32_t nl = h->n_lines;
    if (nl == 0 || h->max_grams == 0) return true;
    if (h->max_grams > kMaxLineGrams || nb + (uint64_t)nl * (p.mode == 0 && p.pad ? p.q - 1 : 0) >= 0xffffffffull)
        return false;
    // dense codes of the bytes that occur; the padding byte's from index 256 on
    uint8_t* hlut = c.pinnedT<uint8_t>("tl.hlut", 512);
    memset(hlut, 0, 512);
    int gbits = 2 * p.q, cb = 2;
    if (p.mode == 0) {
        if (p.pad) h->present[(p.pad_char & 0xff) >> 5] |= 1u << (p.pad_char & 31);
        uint32_t code[256], ncode = 0;
        for (int b = 0; b < 256; b++) {
            code[b] = ncode;
            ncode += h->present[b >> 5] >> (b & 31) & 1u;
        }
        for (int b = 0; b < 256; b++) {
            const int x = p.lower && b >= 'A' && b <= 'Z' ? b + ('a' - 'A') : b;
            hlut[b] = (uint8_t)code[x];
            hlut[256 + b] = (uint8_t)code[b];
        }
        cb = bits_for32(ncode);
        gbits = cb * p.q;
        if (gbits > 63) return false;
    }
    uint8_t* lut = c.devT<uint8_t>("tl.lut", 512);
    FGSS_CK(cudaMemcpyAsync(lut, hlut, 512, cudaMemcpyHostToDevice, c.stream));
    uint32_t* lsz = c.devT<uint32_t>("tl.lsz", (uint64_t)nl + 1);
    uint32_t* loff = c.devT<uint32_t>("tl.loff", (uint64_t)nl + 1);
    // grams of up to 31 bits leave the 32-bit table its empty mark; canonical k-mers never have all bits set
    const bool narrow = gbits <= 31 || (p.mode == 1 && gbits <= 32);
    const uint32_t* longs = list + (lcap - h->n_long);
    auto count = [&](auto tag) {
        using K = decltype(tag);
        launch_lines<K, uint32_t>(c, dtext, lstart, lend, nullptr, nl, p, lut, cb, kSmallLine, 8, false, 0, lsz, loff,
                                  nullptr, nullptr, nullptr, cnt);
        launch_lines<K, uint32_t>(c, dtext, lstart, lend, list, h->n_mid, p, lut, cb, kMidLine, 4, false, 0, lsz, loff,
                                  nullptr, nullptr, nullptr, cnt);
        launch_lines<K, uint32_t>(c, dtext, lstart, lend, longs, h->n_long, p, lut, cb, h->max_grams, 1, false, 0, lsz,
                                  loff, nullptr, nullptr, nullptr, cnt);
    };
    if (narrow) count(uint32_t());
    else count(uint64_t());
    exclusive_scan<uint32_t>(c, lsz, loff, nl, nullptr, &cnt->n_tokens, "tl.s.line");
    FGSS_CK(cudaMemcpyAsync(h, cnt, sizeof(TokCounts), cudaMemcpyDeviceToHost, c.stream));
    c.sync();
    if (h->n_tokens == 0) return true;
    const int ob = p.mode == 0 && p.suffix && h->max_occ ? bits_for32((uint64_t)h->max_occ + 1) : 0;
    const TokCounts hc = *h;
    if (narrow && gbits + ob <= 32)
        tokenize_terms<uint32_t, uint32_t>(c, dtext, lstart, lend, p, lut, cb, lcap, list, hc, ob, gbits + ob, lsz, loff,
                                           cnt, out);
    else if (narrow)
        tokenize_terms<uint32_t, uint64_t>(c, dtext, lstart, lend, p, lut, cb, lcap, list, hc, ob, gbits + ob, lsz, loff,
                                           cnt, out);
    else
        tokenize_terms<uint64_t, uint64_t>(c, dtext, lstart, lend, p, lut, cb, lcap, list, hc, ob, gbits + ob, lsz, loff,
                                           cnt, out);
    return true;
}

}  // namespace

void tokenize_device(Ctx& c, const char* text, uint64_t n_bytes, const TokParams& p, fgss_sets* out) {
    if (p.q < 1 || p.q > 1024) fail(FGSS_ERR_INVALID, "q must be in [1, 1024] (preprocess_cli.cpp:41,86)");
    if (p.mode == 1 && p.q > 32) fail(FGSS_ERR_INVALID, "k-mers need k <= 32");
    if (p.mode == 0 && p.suffix && p.q > 6)
        fail(FGSS_ERR_UNSUPPORTED, "occurrence-suffix mode supports q <= 6 (gram and occurrence share 64 bits)");
    if (n_bytes >= (1ull << 32)) fail(FGSS_ERR_UNSUPPORTED, "text of 4 GiB or more");
    memset(out, 0, sizeof *out);
    unsigned char* dtext = c.devT<unsigned char>("tk.text", n_bytes + 16);
    if (n_bytes == 0) return;
    FGSS_CK(cudaMemcpyAsync(dtext, text, n_bytes, cudaMemcpyHostToDevice, c.stream));
    if (!tokenize_lines(c, dtext, n_bytes, p, out)) tokenize_sorted(c, dtext, n_bytes, p, out);
}

namespace {

void tokenize_sorted(Ctx& c, const unsigned char* dtext, uint64_t nb, const TokParams& p, fgss_sets* out) {
    // 1. lines
    uint32_t* flag = c.devT<uint32_t>("tk.flag", nb + 1);
    uint32_t* scan = c.devT<uint32_t>("tk.scan", nb + 1);
    uint32_t* tot = c.devT<uint32_t>("tk.tot", 8);
    FGSS_CK(cudaMemsetAsync(tot, 0, 32, c.stream));
    uint32_t n_nl = 0;
    if (nb) {
        k_flag_newlines<<<grid_for(nb, 256, c.num_sms * 32), 256, 0, c.stream>>>(dtext, nb, flag);
        FGSS_LAUNCH_CK();
        exclusive_scan<uint32_t>(c, flag, scan, nb, nullptr, tot, "tk.s1");
        n_nl = read_u32(c, tot);
    }
    uint64_t* nl_pos = c.devT<uint64_t>("tk.nlpos", (uint64_t)n_nl + 1);
    if (n_nl) {
        k_newlines<<<grid_for(nb, 256, c.num_sms * 32), 256, 0, c.stream>>>(flag, scan, nb, n_nl, nl_pos);
        FGSS_LAUNCH_CK();
    }
    const uint32_t nraw = n_nl + 1;
    uint64_t* lstart = c.devT<uint64_t>("tk.lstart", nraw);
    uint32_t* llen = c.devT<uint32_t>("tk.llen", nraw);
    uint32_t* nonempty = c.devT<uint32_t>("tk.ne", nraw);
    uint32_t* noff = c.devT<uint32_t>("tk.noff", nraw);
    k_line_bounds<<<grid_for(nraw, 256), 256, 0, c.stream>>>(nl_pos, n_nl, nb, lstart, llen, nonempty);
    FGSS_LAUNCH_CK();
    exclusive_scan<uint32_t>(c, nonempty, noff, nraw, nullptr, tot + 1, "tk.s2");
    const uint32_t nlines = read_u32(c, tot + 1);
    if (nlines == 0) return;
    uint64_t* ls = c.devT<uint64_t>("tk.ls", nlines);
    uint32_t* ll = c.devT<uint32_t>("tk.ll", nlines);
    k_compact_lines<<<grid_for(nraw, 256), 256, 0, c.stream>>>(lstart, llen, nonempty, noff, nraw, ls, ll);
    FGSS_LAUNCH_CK();
    // 2. grams
    uint32_t* gcnt = c.devT<uint32_t>("tk.gcnt", nlines + 1);
    uint32_t* goff = c.devT<uint32_t>("tk.goff", nlines + 1);
    k_gram_count<<<grid_for((uint64_t)nlines * 32, 256, c.num_sms * 32), 256, 0, c.stream>>>(dtext, ls, ll, nlines, p,
                                                                                            gcnt);
    FGSS_LAUNCH_CK();
    exclusive_scan<uint32_t>(c, gcnt, goff, nlines, nullptr, tot + 2, "tk.s3");
    const uint64_t G = read_u32(c, tot + 2);
    if (G == 0) return;
    uint64_t* key = c.devT<uint64_t>("tk.key", G);
    uint64_t* tag = c.devT<uint64_t>("tk.tag", G);
    k_gram_fill<<<grid_for((uint64_t)nlines * 32, 256, c.num_sms * 32), 256, 0, c.stream>>>(dtext, ls, ll, nlines, p,
                                                                                           goff, key, tag);
    FGSS_LAUNCH_CK();
    const int kb = key_bits(p);
    const int lb = bits_for32(nlines);
    // 3. (line, gram, position) order: stable by gram, then by line
    radix_sort<uint64_t, uint64_t>(c, key, tag, G, nullptr, 0, kb, "tk.sortA");
    {
        // sort by line: the line sits in tag's high half; sort (tag, key) by bits [32, 32+lb)
        radix_sort<uint64_t, uint64_t>(c, tag, key, G, nullptr, 32, 32 + lb, "tk.sortB");
    }
    const bool suffix = p.mode == 0 && p.suffix;
    uint64_t* key2 = c.devT<uint64_t>("tk.key2", G);
    uint32_t* keep = c.devT<uint32_t>("tk.keep", G + 1);
    k_occurrence<<<grid_for(G, 256, c.num_sms * 32), 256, 0, c.stream>>>(key, tag, G, suffix ? 1 : 0, key2, keep);
    FGSS_LAUNCH_CK();
    uint64_t Tn = G;
    uint64_t* tkey = key2;
    uint64_t* ttag = tag;
    if (!suffix) {
        uint32_t* koff = c.devT<uint32_t>("tk.koff", G + 1);
        exclusive_scan<uint32_t>(c, keep, koff, G, nullptr, tot + 3, "tk.s4");
        Tn = read_u32(c, tot + 3);
        tkey = c.devT<uint64_t>("tk.ckey", Tn + 1);
        ttag = c.devT<uint64_t>("tk.ctag", Tn + 1);
        k_compact_tok<<<grid_for(G, 256, c.num_sms * 32), 256, 0, c.stream>>>(key2, tag, keep, koff, G, tkey, ttag);
        FGSS_LAUNCH_CK();
    }
    // 4. terms: stable sort by key' keeps (line, position) order inside a run
    const int kb2 = suffix ? kb + 16 : kb;
    radix_sort<uint64_t, uint64_t>(c, tkey, ttag, Tn, nullptr, 0, kb2 > 64 ? 64 : kb2, "tk.sortC");
    uint32_t* gidx = c.devT<uint32_t>("tk.gidx", Tn + 1);
    k_tag_index<<<grid_for(Tn, 256, c.num_sms * 32), 256, 0, c.stream>>>(ttag, goff, ls, p.mode, Tn, gidx,
                                                                             c.err_dev);
    FGSS_LAUNCH_CK();
    uint32_t* rflag = c.devT<uint32_t>("tk.rflag", Tn + 1);
    uint32_t* rid = c.devT<uint32_t>("tk.rid", Tn + 1);
    k_run_flags<<<grid_for(Tn, 256, c.num_sms * 32), 256, 0, c.stream>>>(tkey, Tn, rflag);
    FGSS_LAUNCH_CK();
    exclusive_scan<uint32_t>(c, rflag, rid, Tn, nullptr, tot + 4, "tk.s5");
    const uint32_t V = read_u32(c, tot + 4);
    uint32_t* rstart = c.devT<uint32_t>("tk.rstart", (uint64_t)V + 1);
    k_run_start<<<grid_for(Tn, 256, c.num_sms * 32), 256, 0, c.stream>>>(rflag, rid, Tn, rstart, c.err_dev);
    FGSS_LAUNCH_CK();
    uint64_t* rkey = c.devT<uint64_t>("tk.rkey", (uint64_t)V + 1);
    uint32_t* rval = c.devT<uint32_t>("tk.rval", (uint64_t)V + 1);
    k_run_keys2<<<grid_for(V, 256, c.num_sms * 32), 256, 0, c.stream>>>(rstart, gidx, Tn, V, rkey, rval);
    FGSS_LAUNCH_CK();
    radix_sort<uint64_t, uint32_t>(c, rkey, rval, V, nullptr, 0, 32 + bits_for32((uint64_t)nlines + 1), "tk.sortD");
    uint32_t* id_of_run = c.devT<uint32_t>("tk.idrun", (uint64_t)V + 1);
    k_run_ids<<<grid_for(V, 256, c.num_sms * 32), 256, 0, c.stream>>>(rval, V, id_of_run, c.err_dev);
    FGSS_LAUNCH_CK();
    // 5. (line, id) order
    uint64_t* k2 = c.devT<uint64_t>("tk.k2", Tn + 1);
    uint32_t* pos = c.devT<uint32_t>("tk.pos", Tn + 1);
    k_line_id_keys<<<grid_for(Tn, 256, c.num_sms * 32), 256, 0, c.stream>>>(rid, id_of_run, ttag, Tn, k2, pos);
    FGSS_LAUNCH_CK();
    radix_sort<uint64_t, uint32_t>(c, k2, pos, Tn, nullptr, 0, bits_for32((uint64_t)V + 1), "tk.sortE");
    radix_sort<uint64_t, uint32_t>(c, k2, pos, Tn, nullptr, 32, 32 + lb, "tk.sortF");
    // 6. per-line sizes, records by (size, line)
    uint32_t* lsz = c.devT<uint32_t>("tk.lsz", nlines + 1);
    uint32_t* loff = c.devT<uint32_t>("tk.loff", nlines + 1);
    uint32_t* lend = c.devT<uint32_t>("tk.lend", nlines + 1);
    FGSS_CK(cudaMemsetAsync(loff, 0, (uint64_t)nlines * 4, c.stream));
    FGSS_CK(cudaMemsetAsync(lend, 0, (uint64_t)nlines * 4, c.stream));
    k_line_bounds2<<<grid_for(Tn, 256, c.num_sms * 32), 256, 0, c.stream>>>(k2, Tn, lend, loff, c.err_dev);
    FGSS_LAUNCH_CK();
    k_line_sizes<<<grid_for(nlines, 256, c.num_sms * 8), 256, 0, c.stream>>>(lend, loff, nlines, lsz);
    FGSS_LAUNCH_CK();
    k_count_zero<<<grid_for(nlines, 256, c.num_sms * 8), 256, 0, c.stream>>>(lsz, nlines, tot + 5);
    FGSS_LAUNCH_CK();
    uint64_t* rk = c.devT<uint64_t>("tk.rk", nlines + 1);
    uint32_t* rv = c.devT<uint32_t>("tk.rv", nlines + 1);
    k_rec_keys<<<grid_for(nlines, 256), 256, 0, c.stream>>>(lsz, nlines, rk, rv);
    FGSS_LAUNCH_CK();
    radix_sort<uint64_t, uint32_t>(c, rk, rv, nlines, nullptr, 0, lb, "tk.sortG");
    radix_sort<uint64_t, uint32_t>(c, rk, rv, nlines, nullptr, 32, 64, "tk.sortH");
    const uint32_t nempty = read_u32(c, tot + 5);
    const uint32_t nrec = nlines - nempty;
    uint32_t* mline = c.devT<uint32_t>("tk.mline", nrec + 1);
    uint32_t* mid = c.devT<uint32_t>("tk.mid", nrec + 1);
    uint32_t* mlen = c.devT<uint32_t>("tk.mlen", nrec + 1);
    uint32_t* moff = c.devT<uint32_t>("tk.moff", nrec + 1);
    if (nrec) {
        k_rec_out<<<grid_for(nrec, 256), 256, 0, c.stream>>>(rv, lsz, nlines, nempty, mline, mid, mlen, c.err_dev);
        FGSS_LAUNCH_CK();
        exclusive_scan<uint32_t>(c, mlen, moff, nrec, nullptr, tot + 6, "tk.s6");
    }
    uint32_t* otok = c.devT<uint32_t>("tk.otok", Tn + 1);
    uint32_t* oloc = c.devT<uint32_t>("tk.oloc", Tn + 1);
    if (nrec) {
        k_gather_rec<<<grid_for((uint64_t)nrec * 32, 256, c.num_sms * 32), 256, 0, c.stream>>>(
            mline, moff, nrec, loff, lsz, k2, pos, otok, oloc, c.err_dev);
        FGSS_LAUNCH_CK();
    }
    copy_out(c, out, nrec, Tn, V, mid, mlen, moff, otok, oloc);
}

}  // namespace

}  // namespace fgss
