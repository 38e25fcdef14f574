// Stage 1: hemispherical DDA viewshed over the heightmap.
//
// The per-ray arithmetic follows the reference kernel
// calc_kernel_hemispherical_viewshed_GPU (src/cuda/kernels/viewshed_kernels.cu:7-59)
// operation for operation, with explicit round-to-nearest intrinsics so the
// hit cell is bit-identical: the ray height oz + Cdir.z * t is one fused
// multiply-add, exactly as nvcc contracts it in the reference build.
//
// The B200 layout differs from the reference:
//   * one launch traces all 2592 directions (the reference launches once per
//     direction and synchronises after each);
//   * a warp holds 32 consecutive voxels that walk the same direction in
//     lockstep, so height loads of neighbouring rays share cache lines;
//   * hits go to a per-voxel raw row [chunk][D] written 16 directions at a
//     time as 64-byte vectors; the first-occurrence dedupe (the reference's
//     O(k) global-memory scan per hit, viewshed_kernels.cu:49-55) is a
//     separate warp-per-voxel pass with a shared-memory hash set and
//     ballot/popc compaction that keeps direction order;
//   * shadow bits are packed 32 per word, voxel-major ([N][words32]), and
//     written once per word;
//   * an upper ray also ends, with no hit, once it rises above every cell it
//     can still reach (the early-exit tables of cone.cu): the reference's
//     result with fewer steps.
#include "dda.cuh"

#include <algorithm>
#include <cstdlib>

namespace sgb {
namespace {

constexpr int kTraceBlock = 128;
constexpr int kDirParts = 32;      // blocks per voxel block, each 1/32 of the directions (16: +0.6% at 1024^2)
constexpr int kDedupeWarps = 4;
constexpr int kHashSlots = 4096;   // > 2592 possible distinct hits per voxel
constexpr int kDedupeBatch = 3;    // 2592 directions: 7 batches of 3 rounds of 128

// 16 blocks of 128 threads per SM: at most 32 registers a thread, so the SM
// holds 64 warps of rays (measured 116.4 -> 109.7 ms at 1024^2 against 38
// registers and 12 blocks).
__global__ void __launch_bounds__(kTraceBlock, 16)
k_trace(DevScene s, const DirEntry* __restrict__ dirs, int D, int words32,
        int voxel_offset, int chunk_count, int* __restrict__ raw, uint32_t* __restrict__ shadow,
        const int* __restrict__ perm, int* __restrict__ err)
{
    __shared__ int stage[kRawGroup][kTraceBlock];
    const int lv = blockIdx.x * kTraceBlock + threadIdx.x;
    const bool active = lv < chunk_count;
    // Row lv traces voxel voxel_offset + perm[lv] (visiting order: Morton-
    // adjacent lanes walk similar rays) or voxel_offset + lv.
    const int v = voxel_offset + (perm ? __ldg(perm + (active ? lv : 0)) : (active ? lv : 0));
    const int top = __ldg(s.pix_parent + v);
    const int gx = top % s.W;
    const int gy = top / s.W;
    const float base_z = (v < s.T) ? __ldg(s.grid + top) : __ldg(s.wall_z + (v - s.T));

    // this block's directions: groups [gb, ge) of kRawGroup
    const int ngroups = (D + kRawGroup - 1) / kRawGroup;
    const int gb = (int)((long long)ngroups * blockIdx.y / gridDim.y);
    const int ge = (int)((long long)ngroups * (blockIdx.y + 1) / gridDim.y);
    uint32_t acc = 0;
    int cur_word = -1;
    int* row = raw + (size_t)(active ? lv : 0) * D;
    for (int g0 = gb * kRawGroup; g0 < ge * kRawGroup; g0 += kRawGroup) {
        for (int k = 0; k < kRawGroup; ++k) {
            const DirEntry d = dirs[g0 + k];
            // up/down and the table are the same for the whole warp (one direction at a time)
            int hit = 0;
            Ray r;
            if (active && ray_start(s.W, s.H, gx, gy, base_z, d, r)) {
                if (!((d.meta >> 16) & 1))
                    hit = ray_walk<false, false>(s.gpad, nullptr, s.W, s.H, s.maxz, r, d);
                else if (s.cone)
                    hit = ray_walk<true, true>(s.gpad, s.cone + s.cone_stride * ((d.meta >> 17) & (kMaxConeTables - 1)),
                                               s.W, s.H, s.maxz, r, d);
                else
                    hit = ray_walk<true, false>(s.gpad, nullptr, s.W, s.H, s.maxz, r, d);
            }
            if (hit < 0) {
                atomicOr(err, kErrTraceBounds);
                hit = 0;
            }
            stage[k][threadIdx.x] = hit;
            const int dense = (d.meta & 0xFFFF) - 1;   // warp-uniform
            if (dense >= 0) {
                const int w = dense >> 5;
                if (w != cur_word) {
                    // a word may be shared with the neighbouring direction part
                    if (active && acc) atomicOr(shadow + (size_t)v * words32 + cur_word, acc);
                    acc = 0;
                    cur_word = w;
                }
                if (hit) acc |= 1u << (dense & 31);
            }
        }
        if (active) {
            int4* dst = reinterpret_cast<int4*>(row + g0);
#pragma unroll
            for (int q = 0; q < kRawGroup / 4; ++q)
                dst[q] = make_int4(stage[4 * q][threadIdx.x], stage[4 * q + 1][threadIdx.x],
                                   stage[4 * q + 2][threadIdx.x], stage[4 * q + 3][threadIdx.x]);
        }
    }
    if (active && acc && cur_word >= 0) atomicOr(shadow + (size_t)v * words32 + cur_word, acc);
}

__global__ void k_pad_grid(const float* __restrict__ grid, int W, int H, float* __restrict__ gpad)
{
    const int Wp = W + 2;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)Wp * (H + 2)) return;
    const int x = (int)(i % Wp) - 1, y = (int)(i / Wp) - 1;
    // the load is clamped into the grid, so it stays in bounds however the
    // select below is compiled
    const float h = grid[(size_t)min(max(y, 0), H - 1) * W + min(max(x, 0), W - 1)];
    gpad[i] = (x >= 0 && x < W && y >= 0 && y < H) ? h : __int_as_float(0x7f800000);
}

__device__ __forceinline__ uint32_t hash_slot(uint32_t x, int bits)
{
    x *= 0x9E3779B1u;
    return x >> (32 - bits);
}

// One warp per voxel: keeps the first occurrence of each hit id in direction
// order and compacts the row in place; counts[perm[lv]] = list length.
//
// Directions without a hit and hits equal to the previous direction's leave
// first, 128 directions a round; what is left queues up in shared memory in
// direction order and meets the hash set 32 ids at a time.
//
// SLOTS is the warp's shared-memory hash set.  The first pass uses a small
// set (4 KB a warp, so many warps fit an SM) and gives up on a voxel whose
// insert needs more than kProbes probes: it then writes nothing of the 32 ids
// it is at and records the row in `ovf`.  The ids before them were compacted in
// place; these and the later ones stand behind the compacted prefix, untouched,
// since at least as many directions come before an id as ids.  So every other
// entry behind the prefix repeats an id of it, and the second pass (4096
// slots, more than the 2592 possible distinct ids) run over the whole row gives
// the same first-occurrence list.
//
// Bound: instructions.  With every direction going through the set 82% of the issue
// slots were used and the rows' bytes took a quarter of the time: 1024^2 8.82 -> 4.93
// ms, 512^2 2.24 -> 1.25, 160^2 0.28 -> 0.17, 64^2 0.056 -> 0.037.
constexpr int kSmallSlots = 1024;
constexpr int kProbes = 32;   // default probe bound of the first pass (SGB_DEDUPE_PROBES overrides it)

template <int SLOTS, bool FIRST>
__global__ void __launch_bounds__(kDedupeWarps * 32)
k_dedupe(int chunk_count, int D, int* __restrict__ raw, int* __restrict__ counts, int* __restrict__ err,
         const int* __restrict__ perm, int* __restrict__ ovf, int probes)
{
    constexpr int kBits = SLOTS == 4096 ? 12 : SLOTS == 1024 ? 10 : 0;
    static_assert(kBits > 0, "hash set of 1024 or 4096 slots");
    extern __shared__ uint32_t tab_all[];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    uint32_t* tab = tab_all + warp * SLOTS;
    __shared__ int s_queue[kDedupeWarps][128 + 32];
    int* queue = s_queue[warp];
    const unsigned lt = (1u << lane) - 1u;
    // FIRST: row lv; else rows listed in ovf[1..ovf[0]], grid-strided
    const int w0 = blockIdx.x * kDedupeWarps + warp;
    const int nrows = FIRST ? chunk_count : ovf[0];
    for (int wi = w0; wi < nrows; wi += FIRST ? nrows : gridDim.x * kDedupeWarps) {
        const int lv = FIRST ? wi : ovf[1 + wi];
        uint4* t4 = reinterpret_cast<uint4*>(tab);
        for (int i = lane; i < SLOTS / 4; i += 32) t4[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
        int* row = raw + (size_t)lv * D;
        int n = 0, queued = 0, last = 0;
        // 32 ids (0: none) against the set; the new ones are written in order.  False: it gave up.
        const auto insert = [&](int h) {
            const unsigned same = __match_any_sync(0xFFFFFFFFu, h);
            const bool leader = (__ffs(same) - 1) == lane;
            bool fresh = false, full = false;
            if (h != 0 && leader) {
                uint32_t slot = hash_slot((uint32_t)h, kBits);
                const int bound = FIRST ? probes : SLOTS;
                int probe = 0;
                for (; probe < bound; ++probe) {
                    const uint32_t old = atomicCAS(&tab[slot], 0u, (uint32_t)h);
                    if (old == 0u) { fresh = true; break; }
                    if (old == (uint32_t)h) break;
                    slot = (slot + 1) & (SLOTS - 1);
                }
                full = probe == bound;
            }
            if (__any_sync(0xFFFFFFFFu, full)) {
                if (lane == 0) {
                    if (FIRST) ovf[1 + atomicAdd(ovf, 1)] = lv;
                    else atomicOr(err, kErrHashFull);
                }
                return false;
            }
            const unsigned bal = __ballot_sync(0xFFFFFFFFu, fresh);
            // below the directions read so far: no more ids than directions
            if (fresh) row[n + __popc(bal & lt)] = h;
            n += __popc(bal);
            return true;
        };
        bool ok = true;
        for (int base = 0; base < D / 4 && ok; base += 32 * kDedupeBatch) {
            int4 hv[kDedupeBatch];
#pragma unroll
            for (int u = 0; u < kDedupeBatch; ++u) {
                const int d = base + 32 * u + lane;
                hv[u] = d < D / 4 ? reinterpret_cast<const int4*>(row)[d] : make_int4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < kDedupeBatch && ok; ++u) {
                const int4 a = hv[u];
                int before = __shfl_up_sync(0xFFFFFFFFu, a.w, 1);
                if (lane == 0) before = last;
                last = __shfl_sync(0xFFFFFFFFu, a.w, 31);
                const bool c0 = a.x != 0 && a.x != before, c1 = a.y != 0 && a.y != a.x;
                const bool c2 = a.z != 0 && a.z != a.y, c3 = a.w != 0 && a.w != a.z;
                const unsigned m0 = __ballot_sync(0xFFFFFFFFu, c0), m1 = __ballot_sync(0xFFFFFFFFu, c1);
                const unsigned m2 = __ballot_sync(0xFFFFFFFFu, c2), m3 = __ballot_sync(0xFFFFFFFFu, c3);
                if ((m0 | m1 | m2 | m3) == 0u) continue;
                int at = queued + __popc(m0 & lt) + __popc(m1 & lt) + __popc(m2 & lt) + __popc(m3 & lt);
                if (c0) queue[at++] = a.x;
                if (c1) queue[at++] = a.y;
                if (c2) queue[at++] = a.z;
                if (c3) queue[at] = a.w;
                queued += __popc(m0) + __popc(m1) + __popc(m2) + __popc(m3);
                __syncwarp();
                int done = 0;
                for (; ok && queued - done >= 32; done += 32) ok = insert(queue[done + lane]);
                if (done == 0) continue;
                queued -= done;
                const int rest = lane < queued ? queue[done + lane] : 0;
                __syncwarp();
                if (lane < queued) queue[lane] = rest;
                __syncwarp();
            }
        }
        if (ok && queued > 0) ok = insert(lane < queued ? queue[lane] : 0);
        if (ok && lane == 0) counts[perm ? perm[lv] : lv] = n;
        __syncwarp();
        if (FIRST) break;
    }
}

// ---- exclusive scan of int counts into int64 offsets (3 phases) ----------
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ long long warp_incl_scan(long long x, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// Block-wide exclusive scan; returns this thread's exclusive prefix and the block total.
__device__ long long block_excl_scan(long long x, long long* total)
{
    __shared__ long long warp_sums[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long inc = warp_incl_scan(x, lane);
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        long long ws = lane < nw ? warp_sums[lane] : 0;
        ws = warp_incl_scan(ws, lane);
        if (lane < nw) warp_sums[lane] = ws;
    }
    __syncthreads();
    const long long before = warp > 0 ? warp_sums[warp - 1] : 0;
    *total = warp_sums[(blockDim.x >> 5) - 1];
    __syncthreads();
    return before + inc - x;
}

__global__ void __launch_bounds__(kScanThreads)
k_scan_tiles(const int* __restrict__ counts, int n, long long* __restrict__ offsets,
             long long* __restrict__ tile_sums)
{
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    long long v[kScanItems];
    long long local = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        v[i] = (base + i < n) ? counts[base + i] : 0;
        local += v[i];
    }
    long long total;
    long long run = block_excl_scan(local, &total);
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        if (base + i < n) offsets[base + i] = run;
        run += v[i];
    }
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads)
k_scan_tile_sums(long long* __restrict__ tile_sums, int ntiles, long long base,
                 long long* __restrict__ offsets, int n)
{
    long long carry = base;
    for (int i0 = 0; i0 < ntiles; i0 += kScanThreads) {
        const int i = i0 + threadIdx.x;
        const long long x = i < ntiles ? tile_sums[i] : 0;
        long long total;
        const long long ex = block_excl_scan(x, &total);
        if (i < ntiles) tile_sums[i] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) offsets[n] = carry;
}

__global__ void k_scan_add(long long* __restrict__ offsets, int n, const long long* __restrict__ tile_sums)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) offsets[i] += tile_sums[i / kScanTile];
}

__global__ void __launch_bounds__(256)
k_gather_csr(int chunk_count, int D, const int* __restrict__ raw, const long long* __restrict__ offsets,
             int* __restrict__ csr_ids, const int* __restrict__ inv)
{
    const int lv = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (lv >= chunk_count) return;
    const long long o = offsets[lv];
    const int k = (int)(offsets[lv + 1] - o);
    const int* row = raw + (size_t)(inv ? inv[lv] : lv) * D;
    for (int i = lane; i < k; i += 32) csr_ids[o + i] = row[i];
}

// Scans of up to kScanOne counts in one block: one launch for three (64^2 runs have
// five such scans: 884 -> 860 us).
constexpr int kScanOne = 16 * kScanThreads;

__global__ void __launch_bounds__(kScanThreads)
k_scan_one(const int* __restrict__ counts, int n, long long base, long long* __restrict__ offsets)
{
    constexpr int kItems = kScanOne / kScanThreads;
    const int per = (n + kScanThreads - 1) / kScanThreads, at = threadIdx.x * per;
    int v[kItems];
    long long local = 0;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        v[i] = i < per && at + i < n ? counts[at + i] : 0;
        local += v[i];
    }
    long long total;
    long long run = base + block_excl_scan(local, &total);
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        if (i < per && at + i < n) offsets[at + i] = run;
        run += v[i];
    }
    if (threadIdx.x == 0) offsets[n] = base + total;
}

}  // namespace

cudaError_t launch_pad_grid(const float* grid, int W, int H, float* gpad, cudaStream_t st)
{
    const long long n = (long long)(W + 2) * (H + 2);
    if (n <= 0) return cudaSuccess;
    k_pad_grid<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(grid, W, H, gpad);
    return cudaGetLastError();
}

cudaError_t launch_trace(const DevScene& s, const DirEntry* dirs, int D, int words32,
                         int voxel_offset, int chunk_count, int* raw, uint32_t* shadow,
                         const int* perm, int* err, cudaStream_t st)
{
    if (chunk_count <= 0) return cudaSuccess;
    if (!s.gpad) return cudaErrorInvalidValue;
    // D is a multiple of kRawGroup (rows are written kRawGroup directions at a time)
    if (D % kRawGroup != 0) return cudaErrorInvalidValue;
    const dim3 grid((chunk_count + kTraceBlock - 1) / kTraceBlock, kDirParts);
    k_trace<<<grid, kTraceBlock, 0, st>>>(s, dirs, D, words32, voxel_offset, chunk_count, raw, shadow, perm, err);
    return cudaGetLastError();
}

cudaError_t launch_dedupe(int chunk_count, int D, int* raw, int* counts, int* err, const int* perm, int* ovf,
                          cudaStream_t st)
{
    if (chunk_count <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(ovf, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    const size_t small = (size_t)kDedupeWarps * kSmallSlots * sizeof(uint32_t);
    const int grid = (chunk_count + kDedupeWarps - 1) / kDedupeWarps;
    // The probe bound only decides which rows go to the second pass (the
    // lists are the same either way); tests lower it to exercise that pass.
    int probes = kProbes;
    if (const char* env = std::getenv("SGB_DEDUPE_PROBES")) probes = std::max(1, std::min(kSmallSlots, std::atoi(env)));
    k_dedupe<kSmallSlots, true><<<grid, kDedupeWarps * 32, small, st>>>(chunk_count, D, raw, counts, err, perm, ovf,
                                                                         probes);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // the rows the first pass gave up on (usually none: the grid exits at once)
    const size_t big = (size_t)kDedupeWarps * kHashSlots * sizeof(uint32_t);
    e = cudaFuncSetAttribute(k_dedupe<kHashSlots, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)big);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    k_dedupe<kHashSlots, false><<<3 * sms, kDedupeWarps * 32, big, st>>>(chunk_count, D, raw, counts, err, perm, ovf,
                                                                          kHashSlots);
    return cudaGetLastError();
}

size_t scan_scratch_elems(int n)
{
    return (size_t)((n + kScanTile - 1) / kScanTile) + 1;
}

cudaError_t launch_scan_counts(const int* counts, int n, long long base, long long* offsets,
                               long long* block_sums, int* /*unused*/, cudaStream_t st)
{
    if (n > 0 && n <= kScanOne) {
        k_scan_one<<<1, kScanThreads, 0, st>>>(counts, n, base, offsets);
        return cudaGetLastError();
    }
    const int ntiles = (n + kScanTile - 1) / kScanTile;
    if (n > 0) k_scan_tiles<<<ntiles, kScanThreads, 0, st>>>(counts, n, offsets, block_sums);
    k_scan_tile_sums<<<1, kScanThreads, 0, st>>>(block_sums, ntiles, base, offsets, n);
    if (n > 0) k_scan_add<<<(n + 255) / 256, 256, 0, st>>>(offsets, n, block_sums);
    return cudaGetLastError();
}

cudaError_t launch_scan_sums(long long* sums, int n, cudaStream_t st)
{
    k_scan_tile_sums<<<1, kScanThreads, 0, st>>>(sums, n, 0, sums, n);
    return cudaGetLastError();
}

cudaError_t launch_gather_csr(int chunk_count, int D, const int* raw, const long long* offsets,
                              int* csr_ids, const int* inv, cudaStream_t st)
{
    if (chunk_count <= 0) return cudaSuccess;
    const long long threads = (long long)chunk_count * 32;
    k_gather_csr<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(chunk_count, D, raw, offsets, csr_ids, inv);
    return cudaGetLastError();
}

namespace {
__global__ void k_invert(const int* __restrict__ perm, int n, int* __restrict__ inv)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) inv[perm[i]] = i;
}
}  // namespace

namespace {
__global__ void k_chunk_flags(const int* __restrict__ order, int N, int v0, int n, int* __restrict__ flag)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < N) flag[p] = (unsigned)(order[p] - v0) < (unsigned)n ? 1 : 0;
}

__global__ void k_chunk_scatter(const int* __restrict__ order, int N, int v0, const int* __restrict__ flag,
                                const long long* __restrict__ pos, int* __restrict__ perm)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < N && flag[p]) perm[pos[p]] = order[p] - v0;
}
}  // namespace

cudaError_t launch_chunk_order(const int* order, int N, int v0, int n, int* flag, long long* pos,
                               long long* scan_tmp, int* perm, cudaStream_t st)
{
    if (N <= 0 || n <= 0) return cudaSuccess;
    const unsigned grid = (unsigned)((N + 255) / 256);
    k_chunk_flags<<<grid, 256, 0, st>>>(order, N, v0, n, flag);
    cudaError_t e = launch_scan_counts(flag, N, 0, pos, scan_tmp, nullptr, st);
    if (e != cudaSuccess) return e;
    k_chunk_scatter<<<grid, 256, 0, st>>>(order, N, v0, flag, pos, perm);
    return cudaGetLastError();
}

cudaError_t launch_invert(const int* perm, int n, int* inv, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    k_invert<<<(n + 255) / 256, 256, 0, st>>>(perm, n, inv);
    return cudaGetLastError();
}

}  // namespace sgb
