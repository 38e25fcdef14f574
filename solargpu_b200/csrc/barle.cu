// ba-RLE writer on the GPU, byte-exact to the reference host encoder
// (src/barle_compression.cpp:156-187, format in include/barle_compression.h:7-44):
//   ids sorted descending (the lists are already unique), deltas with the
//   first value absolute, width classes 4/8/16/24/32 bits, maximal
//   same-width runs, the two-pass run optimiser, runs split at 255, then
//   blocks of <= 8 runs: 3 big-endian bytes of 3-bit codes (pad 7), one
//   length byte per run, then payload (4-bit deltas two per byte, high nibble
//   first; wider deltas big-endian).
//
// One warp per voxel.  Lists of up to 1024 ids (almost all) are encoded in one
// pass, in registers (k_barle_encode): a lane holds 8, 16 or 32 consecutive
// ids, sorted bitonically over lanes by shuffles, and every step after the sort
// is a short loop over a lane's own ids with one scan over the warp.  That needs
// the run optimiser without its sequential fixpoint:
//
//   A pass merges a run of one id into the run before it when that is one class
//   wider, going on after the merged one.  So run r is merged if that holds for
//   (r - 1, r) and r - 1 was not merged itself, a chain of at most four classes.
//   No later pass finds more: a run that was not merged keeps the run before it
//   or, if that was merged, meets the one before that, two classes wider or more.
//   A merged run has one id, so merging means giving the id the next class; the
//   final runs are the maximal ones of these classes.
//
// The stream goes after the sorted list in the voxel's row, a scan turns the
// sizes into offsets, and k_barle_copy moves the streams there.  Longer lists (up
// to one id a direction) take two passes with the reference's own loop on one
// lane: k_barle_size (sizes; sorted list and, room permitting, its runs left in
// the row) and k_barle_write.
//
// Bound: instructions (the sort's shuffles first); the one-lane loops and the
// run-by-run writes of the two passes were latency.  Sizes, offsets and streams:
// 160^2 town (35,840 voxels) 0.86 -> 0.24 ms, 512^2 city 9.2 -> 2.0 (3.0 with every
// loop unrolled, see sort_desc, and a warp a row looking for long lists).
#include "sgb_internal.cuh"

#include <algorithm>

namespace sgb {
namespace {

constexpr int kEncWarps = 4;        // the two passes for long lists
constexpr int kIdsCap = 4096;
constexpr int kRunsCap = 2624;
constexpr int kSmallIds = 1024;     // lists encoded in registers
constexpr int kCopyWarps = 8;
constexpr int kW4 = 0, kEnd = 7;

__device__ __forceinline__ int width_class(uint32_t x)
{
    return x <= 15u ? 0 : x <= 255u ? 1 : x <= 65535u ? 2 : x <= 16777215u ? 3 : 4;
}

__device__ __forceinline__ uint32_t delta_at(const uint32_t* ids, int i)
{
    return i == 0 ? ids[0] : ids[i - 1] - ids[i];
}

__device__ __forceinline__ uint32_t pack_run(int w, int len) { return ((uint32_t)w << 24) | (uint32_t)len; }
__device__ __forceinline__ int run_w(uint32_t r) { return (int)(r >> 24); }
__device__ __forceinline__ int run_len(uint32_t r) { return (int)(r & 0xFFFFFFu); }

// Descending bitonic sort of s[0..n2) (n2 a power of two >= 32), warp-wide.
__device__ void warp_sort_desc(uint32_t* s, int n2, int lane)
{
    for (int size = 2; size <= n2; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int t = lane; t < (n2 >> 1); t += 32) {
                const int i = 2 * t - (t & (stride - 1));
                const int j = i + stride;
                const bool desc = (i & size) == 0;
                const uint32_t a = s[i], b = s[j];
                if ((a < b) == desc) { s[i] = b; s[j] = a; }
            }
            __syncwarp();
        }
    }
}

// Builds the optimised run list of a sorted id list into runs[]; returns the
// run count (warp-uniform).  runs[r] = pack_run(width, len).
__device__ int build_runs(const uint32_t* ids, int k, uint32_t* runs, int lane)
{
    // 1. maximal same-width runs (detect_runs, barle_compression.cpp:90-105)
    int nr = 0;
    for (int base = 0; base < k; base += 32) {
        const int i = base + lane;
        int w = -1;
        bool start = false;
        if (i < k) {
            w = width_class(delta_at(ids, i));
            start = (i == 0) || (w != width_class(delta_at(ids, i - 1)));
        }
        const unsigned bal = __ballot_sync(0xFFFFFFFFu, start);
        if (start) runs[nr + __popc(bal & ((1u << lane) - 1u))] = pack_run(w, i);   // len slot holds start
        nr += __popc(bal);
    }
    __syncwarp();
    // starts -> lengths
    for (int r0 = 0; r0 < nr; r0 += 32) {
        const int r = r0 + lane;
        uint32_t cur = 0, nxt_start = (uint32_t)k;
        if (r < nr) {
            cur = runs[r];
            if (r + 1 < nr) nxt_start = (uint32_t)run_len(runs[r + 1]);
        }
        __syncwarp();
        if (r < nr) runs[r] = pack_run(run_w(cur), (int)nxt_start - run_len(cur));
        __syncwarp();
    }
    // 2. optimize_runs (barle_compression.cpp:112-152), sequential on lane 0
    if (lane == 0 && nr >= 2) {
        bool changed = true, single = false;
        while (changed) {
            changed = false;
            int nn = 0, i = 0;
            while (i < nr - 1) {
                const uint32_t a = runs[i], b = runs[i + 1];
                if (run_len(b) == 1 && run_w(b) + 1 == run_w(a)) {
                    changed = true;
                    runs[nn++] = pack_run(run_w(a), run_len(a) + 1);
                    i += 2;
                } else {
                    runs[nn++] = a;
                    ++i;
                }
            }
            if (i < nr) runs[nn++] = runs[i];
            if (nn == 1) { nr = 1; single = true; break; }
            nr = nn;   // unchanged passes rewrite the same list
        }
        if (!single) {
            int nn = 0, i = 0;
            while (i < nr) {
                const int w = run_w(runs[i]);
                int len = run_len(runs[i]);
                int j = i + 1;
                while (j < nr && run_w(runs[j]) == w) { len += run_len(runs[j]); ++j; }
                runs[nn++] = pack_run(w, len);
                i = j;
            }
            nr = nn;
        }
    }
    nr = __shfl_sync(0xFFFFFFFFu, nr, 0);
    __syncwarp();
    return nr;
}

__device__ __forceinline__ int payload_bytes(int w, int len)
{
    return w == kW4 ? (len + 1) >> 1 : len * w;
}

__device__ int load_sorted(const int* row, int k, uint32_t* ids, int lane, bool sort)
{
    int n2 = 32;
    while (n2 < k) n2 <<= 1;
    for (int i = lane; i < n2; i += 32) ids[i] = i < k ? (uint32_t)row[i] : 0u;
    __syncwarp();
    if (sort) warp_sort_desc(ids, n2, lane);
    return n2;
}

// ---- lists of up to kSmallIds ids -------------------------------------------------

constexpr unsigned kAll = 0xFFFFFFFFu;

// Bytes of the longest stream of k ids, and its room (whole 16-byte pieces).
__host__ __device__ constexpr int stream_bytes(int k) { return 4 * k + k + 3 * ((k + 7) / 8); }
__host__ __device__ constexpr int stream_room(int k) { return (stream_bytes(k) + 15) / 16 * 16; }
// Where the stream of a list of k ids starts in its row (in ints).
__device__ __forceinline__ int stream_at(int k) { return (k + 3) & ~3; }

__device__ __forceinline__ void swap_desc(uint32_t& a, uint32_t& b)
{
    const uint32_t hi = max(a, b), lo = min(a, b);
    a = hi;
    b = lo;
}

// Sorts 32 E ids descending, lane l holding the places [l E, (l + 1) E).  Every
// merge starts with a mirrored step, so all comparisons point the same way.
template <int E>
__device__ __forceinline__ void sort_desc(uint32_t (&x)[E], int lane)
{
#pragma unroll
    for (int size = 2; size <= E; size <<= 1) {
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const int m = (j & ~(size - 1)) + size - 1 - (j & (size - 1));
            if (j < m) swap_desc(x[j], x[m]);
        }
#pragma unroll
        for (int stride = size >> 2; stride > 0; stride >>= 1)
#pragma unroll
            for (int j = 0; j < E; ++j)
                if ((j & stride) == 0) swap_desc(x[j], x[j + stride]);
    }
    // The merges over lanes are not unrolled: with all of them in line the kernels
    // waited on instructions most of the time.
#pragma unroll 1
    for (int lanes = 2; lanes <= 32; lanes <<= 1) {
        const bool above = (lane & (lanes >> 1)) != 0;
#pragma unroll
        for (int j = 0; j < E / 2; ++j) {
            const uint32_t a = __shfl_xor_sync(kAll, x[E - 1 - j], lanes - 1);
            const uint32_t b = __shfl_xor_sync(kAll, x[j], lanes - 1);
            x[j] = above ? min(x[j], a) : max(x[j], a);
            x[E - 1 - j] = above ? min(x[E - 1 - j], b) : max(x[E - 1 - j], b);
        }
#pragma unroll 1
        for (int apart = lanes >> 2; apart > 0; apart >>= 1) {
            const bool upper = (lane & apart) != 0;
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const uint32_t a = __shfl_xor_sync(kAll, x[j], apart);
                x[j] = upper ? min(x[j], a) : max(x[j], a);
            }
        }
#pragma unroll
        for (int stride = E >> 1; stride > 0; stride >>= 1)
#pragma unroll
            for (int j = 0; j < E; ++j)
                if ((j & stride) == 0) swap_desc(x[j], x[j + stride]);
    }
}

// Encodes k ids (sorted, as sort_desc leaves them) into st; pieces: k words,
// deltas: 32 (E + 1).  Returns the stream's bytes.
template <int E>
__device__ __forceinline__ int encode_sorted(uint32_t (&x)[E], int k, unsigned char* st, uint32_t* pieces,
                                             uint32_t* deltas, int lane)
{
    constexpr int kNone = 15;   // class past the list's end
    const int base = lane * E, n = min(max(k - base, 0), E);   // this lane's ids
    const uint32_t before = __shfl_up_sync(kAll, x[E - 1], 1);
#pragma unroll
    for (int j = E - 1; j > 0; --j) x[j] = x[j - 1] - x[j];
    if (lane > 0) x[0] = before - x[0];   // x: deltas from here on
    int w[E];
#pragma unroll
    for (int j = 0; j < E; ++j) w[j] = j < n ? width_class(x[j]) : kNone;
    // ids that join the wider run before them
    int wl = __shfl_up_sync(kAll, w[E - 1], 1), wr = __shfl_down_sync(kAll, w[0], 1);
    if (lane == 0) wl = kNone;
    if (lane == 31) wr = kNone;
    unsigned c = 0;
#pragma unroll
    for (int j = 0; j < E; ++j) {
        const int l = j ? w[j - 1] : wl, r = j + 1 < E ? w[j + 1] : wr;
        if (l == w[j] + 1 && r != w[j] && l < kNone) c |= 1u << j;
    }
    const unsigned cl = __shfl_up_sync(kAll, c, 1);
    const auto at = [&](int j) { return ((cl >> j) & 1u) != 0; };
    bool joined = lane > 0 && at(E - 1) && !(at(E - 2) && !(at(E - 3) && !at(E - 4)));
#pragma unroll
    for (int j = 0; j < E; ++j) {
        joined = ((c >> j) & 1u) != 0 && !joined;
        if (joined) ++w[j];
    }
    // starts of runs
    wl = __shfl_up_sync(kAll, w[E - 1], 1);
    if (lane == 0) wl = kNone;
    int start = -1;
#pragma unroll
    for (int j = 0; j < E; ++j)
        if (w[j] != (j ? w[j - 1] : wl)) start = base + j;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kAll, start, o);
        if (lane >= o) start = max(start, y);
    }
    start = __shfl_up_sync(kAll, start, 1);   // the last start before this lane (lane 0 has one of its own)
    // pieces: runs split every 255 ids; two 4-bit deltas share a byte
    unsigned first = 0, odd = 0;
    int bytes = 0;
#pragma unroll
    for (int j = 0; j < E; ++j) {
        if (w[j] != (j ? w[j - 1] : wl)) start = base + j;
        int rel = base + j - start;
        while (rel >= 255) rel -= 255;
        if (j < n) {
            if (rel == 0) first |= 1u << j;
            if (rel & 1) odd |= 1u << j;
            bytes += w[j] ? w[j] : 1 - (rel & 1);
        }
    }
    int sum = bytes | (__popc(first) << 16);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kAll, sum, o);
        if (lane >= o) sum += y;
    }
    const int total = __shfl_sync(kAll, sum, 31), np = total >> 16, payload = total & 0xFFFF;
    sum -= bytes | (__popc(first) << 16);
    int b = sum & 0xFFFF, p = (sum >> 16) - 1;   // bytes before this id, its piece
    const uint32_t xr = __shfl_down_sync(kAll, x[0], 1);
    const int apart = __shfl_down_sync(kAll, (n == 0 || (first & 1u)) ? 1 : 0, 1);
    const bool ends = lane == 31 || apart != 0;   // the next lane's first id is in another piece, or past the end
    // the writes, a loop (see sort_desc): deltas in shared memory, classes 4 bits each
    unsigned long long wp[(E + 15) / 16];
#pragma unroll
    for (int j = 0; j < E; ++j) {
        deltas[32 * j + lane] = x[j];
        if (j % 16 == 0) wp[j / 16] = 0ull;
        wp[j / 16] |= (unsigned long long)w[j] << (4 * (j % 16));
    }
    deltas[32 * E + lane] = xr;   // a lane reads only what it wrote
#pragma unroll 1
    for (int j = 0; j < n; ++j) {
        const int wj = (int)((E > 16 && j >= 16 ? wp[(E - 1) / 16] : wp[0]) >> (4 * (j & 15))) & 15;
        const uint32_t xj = deltas[32 * j + lane];
        if ((first >> j) & 1u) {
            ++p;
            pieces[p] = ((uint32_t)b << 14) | (uint32_t)((base + j) << 3) | (uint32_t)wj;
        }
        // blocks of 8 pieces: 3 bytes of codes and the lengths come before a piece's payload
        const int q = (p >> 3) + 1;
        unsigned char* d = st + b + 3 * q + min(np, 8 * q);
        if (wj == kW4) {
            if (((odd >> j) & 1u) == 0) {
                const bool alone = j + 1 < E ? (j + 1 >= n || ((first >> (j + 1)) & 1u)) : ends;
                *d = (unsigned char)((xj << 4) | (alone ? 0u : deltas[32 * (j + 1) + lane] & 0x0Fu));
                ++b;
            }
        } else {
            for (int i = 0; i < wj; ++i) d[i] = (unsigned char)(xj >> (8 * (wj - 1 - i)));
            b += wj;
        }
    }
    __syncwarp();
    for (int p0 = 0; p0 < np; p0 += 32) {
        const int i = p0 + lane;
        const uint32_t pc = i < np ? pieces[i] : 0u;
        const int next = i + 1 < np ? (int)((pieces[i + 1] >> 3) & 0x7FFu) : k;
        const int q = i >> 3, j = i & 7;
        unsigned char* blk = st + (__shfl_sync(kAll, pc, lane & ~7) >> 14) + 11 * q;
        uint32_t bits = (i < np ? pc & 7u : (uint32_t)kEnd) << ((7 - j) * 3);
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) bits |= __shfl_xor_sync(kAll, bits, o);
        if (i < np) blk[3 + j] = (unsigned char)(next - (int)((pc >> 3) & 0x7FFu));
        if (j < 3 && 8 * q < np) blk[j] = (unsigned char)(bits >> (16 - 8 * j));
    }
    __syncwarp();
    return payload + np + 3 * ((np + 7) / 8);
}

// The list of a row, a lane's ids side by side: sorted, written back, encoded.
template <int E>
__device__ __forceinline__ int encode_row(int* row, int k, unsigned char* st, uint32_t* pieces, uint32_t* deltas, int lane)
{
    uint32_t x[E];
#pragma unroll
    for (int j = 0; j < E; ++j) x[j] = 32 * j + lane < k ? (uint32_t)row[32 * j + lane] : 0u;
    sort_desc<E>(x, lane);
#pragma unroll
    for (int j = 0; j < E / 4; ++j) {   // whole pieces: the stream starts on the next one
        const int i = lane * E + 4 * j;
        if (i < k) *reinterpret_cast<uint4*>(row + i) = make_uint4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
    }
    return encode_sorted<E>(x, k, st, pieces, deltas, lane);
}

// A warp's rows whose lists have more than lo ids: f(row, voxel, ids) for each.  It
// looks 32 rows over at a time, a count a lane, as far apart as there are warps
// (long lists are neighbours; side by side, one warp had them all: 160^2 lists 0.56 ms).
template <typename F>
__device__ __forceinline__ void for_long_rows(int chunk_count, const int* __restrict__ counts,
                                              const int* __restrict__ map, int warps, int lane, int lo, F&& f)
{
    const int w = blockIdx.x * warps + (threadIdx.x >> 5), apart = gridDim.x * warps;
    for (long long base = w; base < chunk_count; base += 32LL * apart) {
        const long long r = base + (long long)lane * apart;
        const int u = r < chunk_count ? (map ? __ldg(map + r) : (int)r) : 0;
        const int k = r < chunk_count ? __ldg(counts + u) : 0;
        unsigned left = __ballot_sync(kAll, k > lo);
        for (; left; left &= left - 1u) {
            const int i = __ffs(left) - 1;
            f((int)base + i * apart, __shfl_sync(kAll, u, i), __shfl_sync(kAll, k, i));
            __syncwarp();
        }
    }
}

// The stream of a row's list, of up to 32 E ids: its size, and the stream itself in the row
// after the sorted list.
template <int E, bool HALF>
__device__ __forceinline__ void encode_list(int* row, int k, int* size, unsigned char* st, uint32_t* pieces,
                                            uint32_t* deltas, int lane)
{
    const int bytes = HALF && k <= 16 * E ? encode_row<E / 2>(row, k, st, pieces, deltas, lane)
                                          : encode_row<E>(row, k, st, pieces, deltas, lane);
    if (lane == 0) *size = bytes;
    uint4* dst = reinterpret_cast<uint4*>(row + stream_at(k));
    for (int i = lane; i < (bytes + 15) / 16; i += 32) dst[i] = reinterpret_cast<const uint4*>(st)[i];
}

template <int E, int WARPS>
struct EncodeRoom {
    uint4 st[WARPS][stream_room(32 * E) / 16];
    uint32_t pieces[WARPS][32 * E], deltas[WARPS][32 * (E + 1)];
};
constexpr int kEncodeWarps = 8, kMidWarps = 4;

// Lists of up to 512 ids, a warp a row.
__global__ void __launch_bounds__(kEncodeWarps * 32)
k_barle_encode(int chunk_count, int D, int* __restrict__ raw, const int* __restrict__ counts, int* __restrict__ sizes,
               int* __restrict__ err, const int* __restrict__ perm)
{
    extern __shared__ __align__(16) unsigned char s_enc[];
    auto& room = *reinterpret_cast<EncodeRoom<16, kEncodeWarps>*>(s_enc);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lv = blockIdx.x * kEncodeWarps + warp;   // row
    if (lv >= chunk_count) return;
    const int u = perm ? perm[lv] : lv;                // voxel of the row
    const int k = counts[u];
    if (k > 512) return;
    if (k <= 0 || k > D) {
        if (lane == 0) {
            sizes[u] = 0;
            if (k > D) atomicOr(err, kErrListCapacity);
        }
        return;
    }
    encode_list<16, true>(raw + (size_t)lv * D, k, sizes + u, reinterpret_cast<unsigned char*>(room.st[warp]),
                          room.pieces[warp], room.deltas[warp], lane);
}

// Lists of 513 to 1024 ids (D is more, see launch_barle_size).
__global__ void __launch_bounds__(kMidWarps * 32)
k_barle_encode_mid(int chunk_count, int D, int* raw, const int* __restrict__ counts, int* sizes,
                   const int* __restrict__ perm)
{
    extern __shared__ __align__(16) unsigned char s_enc[];
    auto& room = *reinterpret_cast<EncodeRoom<32, kMidWarps>*>(s_enc);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for_long_rows(chunk_count, counts, perm, kMidWarps, lane, 512, [&](int lv, int u, int k) {
        if (k > kSmallIds) return;
        encode_list<32, false>(raw + (size_t)lv * D, k, sizes + u, reinterpret_cast<unsigned char*>(room.st[warp]),
                               room.pieces[warp], room.deltas[warp], lane);
    });
}

// The streams of k_barle_encode to their places: whole words there, from pairs
// of words here.
__global__ void __launch_bounds__(kCopyWarps * 32)
k_barle_copy(int chunk_count, int D, const int* __restrict__ raw, const int* __restrict__ counts,
             const long long* __restrict__ offsets, unsigned char* __restrict__ out, const int* __restrict__ inv)
{
    const int lane = threadIdx.x & 31;
    const int lv = blockIdx.x * kCopyWarps + (threadIdx.x >> 5);
    if (lv >= chunk_count) return;
    const int k = counts[lv];
    if (k <= 0 || k > kSmallIds) return;
    const long long o = offsets[lv];
    const int size = (int)(offsets[lv + 1] - o);
    const uint32_t* src = reinterpret_cast<const uint32_t*>(raw + (size_t)(inv ? inv[lv] : lv) * D + stream_at(k));
    unsigned char* dst = out + o;
    const int head = min(size, (int)((0u - (unsigned)reinterpret_cast<uintptr_t>(dst)) & 3u));
    const int words = (size - head) >> 2, tail = size - head - 4 * words;
    if (lane < head) dst[lane] = (unsigned char)(src[0] >> (8 * lane));
    uint32_t* dw = reinterpret_cast<uint32_t*>(dst + head);
    for (int i = lane; i < words; i += 32) dw[i] = __funnelshift_r(src[i], src[i + 1], 8 * head);   // head = 0: src[i]
    if (lane < tail) {
        const int at = size - tail + lane;
        dst[at] = (unsigned char)(src[at >> 2] >> (8 * (at & 3)));
    }
}

// ---- longer lists -----------------------------------------------------------------

__global__ void __launch_bounds__(kEncWarps * 32)
k_barle_size(int chunk_count, int D, int* __restrict__ raw, const int* __restrict__ counts,
             int* __restrict__ sizes, int* __restrict__ err, const int* __restrict__ perm)
{
    extern __shared__ uint32_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t* ids = smem + warp * (kIdsCap + kRunsCap);
    uint32_t* runs = ids + kIdsCap;
    for_long_rows(chunk_count, counts, perm, kEncWarps, lane, kSmallIds, [&](int lv, int u, int k) {
        if (k > D || k > kRunsCap) { if (lane == 0) { sizes[u] = 0; atomicOr(err, kErrListCapacity); } return; }
        int* row = raw + (size_t)lv * D;
        load_sorted(row, k, ids, lane, true);
        for (int i = lane; i < k; i += 32) row[i] = (int)ids[i];   // keep the sorted list for the write pass
        const int nr = build_runs(ids, k, runs, lane);
        // and, where the row has room after the list, its optimised runs (the
        // write pass then skips build_runs): row[k] = run count, runs after it
        if (k < D) {
            const bool fits = k + 1 + nr <= D;
            if (lane == 0) row[k] = fits ? nr : -1;
            if (fits)
                for (int r = lane; r < nr; r += 32) row[k + 1 + r] = (int)runs[r];
        }
        int pieces = 0, payload = 0;
        for (int r = lane; r < nr; r += 32) {
            const int w = run_w(runs[r]), len = run_len(runs[r]);
            const int full = len / 255, rem = len % 255;
            pieces += full + (rem > 0);
            payload += full * payload_bytes(w, 255) + payload_bytes(w, rem);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            pieces += __shfl_xor_sync(0xFFFFFFFFu, pieces, o);
            payload += __shfl_xor_sync(0xFFFFFFFFu, payload, o);
        }
        if (lane == 0) sizes[u] = 3 * ((pieces + 7) / 8) + pieces + payload;
    });
}

__global__ void __launch_bounds__(kEncWarps * 32)
k_barle_write(int chunk_count, int D, const int* __restrict__ raw, const int* __restrict__ counts,
              const long long* __restrict__ offsets, unsigned char* __restrict__ out,
              int* __restrict__ err, const int* __restrict__ inv)
{
    extern __shared__ uint32_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t* ids = smem + warp * (kIdsCap + kRunsCap);
    uint32_t* runs = ids + kIdsCap;
    for_long_rows(chunk_count, counts, nullptr, kEncWarps, lane, kSmallIds, [&](int lv, int, int k) {
        if (k > D || k > kRunsCap) return;
        const int* row = raw + (size_t)(inv ? inv[lv] : lv) * D;
        load_sorted(row, k, ids, lane, false);   // already sorted by k_barle_size
        // the runs k_barle_size left after the list, else built again
        int nr = k < D ? row[k] : -1;
        if (nr >= 0 && k + 1 + nr <= D) {
            for (int r = lane; r < nr; r += 32) runs[r] = (uint32_t)row[k + 1 + r];
            __syncwarp();
        } else {
            nr = build_runs(ids, k, runs, lane);
        }
        // split_long_runs (barle_compression.cpp:29-44), expanded in place from the back
        if (lane == 0) {
            int ns = 0;
            for (int r = 0; r < nr; ++r) ns += (run_len(runs[r]) + 254) / 255;
            int pos = ns;
            for (int r = nr - 1; r >= 0; --r) {
                const int w = run_w(runs[r]), len = run_len(runs[r]);
                const int np = (len + 254) / 255;
                pos -= np;
                for (int p = np - 1; p >= 0; --p) {
                    const int pl = (p == np - 1) ? len - 255 * (np - 1) : 255;
                    runs[pos + p] = pack_run(w, pl);
                }
            }
            nr = ns;
        }
        nr = __shfl_sync(0xFFFFFFFFu, nr, 0);
        __syncwarp();
        unsigned char* dst = out + offsets[lv];
        const long long limit = offsets[lv + 1] - offsets[lv];
        long long boff = 0;
        int estart = 0;
        for (int p = 0; p < nr; ++p) {
            if ((p & 7) == 0) {
                const int cnt = min(8, nr - p);
                if (lane == 0) {
                    uint32_t bits = 0;
                    for (int j = 0; j < 8; ++j) {
                        const int code = (j < cnt) ? run_w(runs[p + j]) : kEnd;
                        bits |= (uint32_t)(code & 7) << ((7 - j) * 3);
                    }
                    if (boff + 3 + cnt <= limit) {
                        dst[boff] = (unsigned char)(bits >> 16);
                        dst[boff + 1] = (unsigned char)(bits >> 8);
                        dst[boff + 2] = (unsigned char)bits;
                    }
                }
                if (lane < cnt && boff + 3 + cnt <= limit) dst[boff + 3 + lane] = (unsigned char)run_len(runs[p + lane]);
                boff += 3 + cnt;
            }
            const int w = run_w(runs[p]), len = run_len(runs[p]);
            const int nb = payload_bytes(w, len);
            if (boff + nb > limit) { if (lane == 0) atomicOr(err, kErrListCapacity); return; }
            if (w == kW4) {
                for (int b = lane; b < nb; b += 32) {
                    const int e = estart + 2 * b;
                    const uint32_t v1 = delta_at(ids, e);
                    const uint32_t v2 = (2 * b + 1 < len) ? delta_at(ids, e + 1) : 0u;
                    dst[boff + b] = (unsigned char)((v1 << 4) | (v2 & 0x0Fu));
                }
            } else {
                for (int i = lane; i < len; i += 32) {
                    const uint32_t x = delta_at(ids, estart + i);
                    unsigned char* q = dst + boff + (long long)i * w;
                    for (int b = 0; b < w; ++b) q[b] = (unsigned char)(x >> (8 * (w - 1 - b)));
                }
            }
            boff += nb;
            estart += len;
        }
    });
}

}  // namespace

// Blocks (of 4 warps) of the kernels for long lists: a warp for 32 rows, and small
// scenes fill the GPU.  A warp a row took 0.45 ms at 512^2 to find none above 1024.
static int long_blocks(int rows)
{
    static_assert(kEncWarps == 4 && kMidWarps == 4, "blocks of 4 warps");
    return std::max(std::min((rows + 3) / 4, 3 * 148), (rows + 127) / 128);
}

cudaError_t launch_barle_size(int chunk_count, int D, int* raw, const int* counts, int* sizes, int* err,
                              const int* perm, cudaStream_t st)
{
    if (chunk_count <= 0) return cudaSuccess;
    // a row holds the list and the stream of up to kSmallIds ids, and starts on 16 bytes
    if (D % 4 != 0 || 4 * D < 4 * kSmallIds + stream_room(kSmallIds)) return cudaErrorInvalidValue;
    constexpr size_t room = sizeof(EncodeRoom<16, kEncodeWarps>), mid = sizeof(EncodeRoom<32, kMidWarps>);
    constexpr size_t smem = (size_t)kEncWarps * (kIdsCap + kRunsCap) * sizeof(uint32_t);
    cudaError_t e = cudaFuncSetAttribute(k_barle_encode, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_barle_encode_mid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mid);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_barle_size, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_barle_encode<<<(chunk_count + kEncodeWarps - 1) / kEncodeWarps, kEncodeWarps * 32, room, st>>>(
        chunk_count, D, raw, counts, sizes, err, perm);
    k_barle_encode_mid<<<long_blocks(chunk_count), kMidWarps * 32, mid, st>>>(
        chunk_count, D, raw, counts, sizes, perm);
    k_barle_size<<<long_blocks(chunk_count), kEncWarps * 32, smem, st>>>(chunk_count, D, raw, counts, sizes, err, perm);
    return cudaGetLastError();
}

cudaError_t launch_barle_write(int chunk_count, int D, const int* raw, const int* counts,
                               const long long* offsets, unsigned char* out, int* err, const int* inv,
                               cudaStream_t st)
{
    if (chunk_count <= 0) return cudaSuccess;
    k_barle_copy<<<(chunk_count + kCopyWarps - 1) / kCopyWarps, kCopyWarps * 32, 0, st>>>(chunk_count, D, raw, counts,
                                                                                         offsets, out, inv);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    constexpr size_t smem = (size_t)kEncWarps * (kIdsCap + kRunsCap) * sizeof(uint32_t);
    e = cudaFuncSetAttribute(k_barle_write, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_barle_write<<<long_blocks(chunk_count), kEncWarps * 32, smem, st>>>(
        chunk_count, D, raw, counts, offsets, out, err, inv);
    return cudaGetLastError();
}

cudaError_t launch_barle_size(int chunk_count, int D, int* raw, const int* counts,
                              int* sizes, int* err, cudaStream_t st)
{
    return launch_barle_size(chunk_count, D, raw, counts, sizes, err, nullptr, st);
}

cudaError_t launch_barle_write(int chunk_count, int D, const int* raw, const int* counts,
                               const long long* offsets, unsigned char* out, int* err,
                               cudaStream_t st)
{
    return launch_barle_write(chunk_count, D, raw, counts, offsets, out, err, nullptr, st);
}

}  // namespace sgb
