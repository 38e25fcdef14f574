// Hour-block reflection on the tensor cores (tcgen05).
//
// R[v, h] = sum_g w(v, g) I[g, h] is, for a group of 128 voxels that are
// close in the visiting order, a dense product over the union U of their
// neighbor cells:  D[128 voxels][256 hours] = W[128][U] x I[U][256].  W is
// sparse (a voxel sees ~7-10% of its group's union), but the tensor cores run
// the dense product faster than CUDA cores run the sparse one, and every
// slab row staged for the group feeds 128 voxels at once.
//
// That holds for the cells that many voxels of the group see.  On the 256^2
// city 71% of a union's cells are seen by at most 8 of the 128 voxels and hold
// 20% of the weights.  A dense row costs its share of a chunk's 1024 cycles, 16 and more,
// a weight 2 of an SM's FP32 lanes.  So these light cells stay out of the union:
//   light    every light weight goes to its cell's list; a warp keeps 16 weights
//            and their sums in registers, streams the cell's row through (each
//            8-hour piece is converted once for all 16) and multiplies hour by
//            hour on packed FP32 pairs, over all blocks of the slab (k_light).
//            The weights stay in FP32; every sum has a place of its own, and a
//            voxel's are added in a fixed order (k_mma_accumulate).
// At most 2 entries a light cell: 1024^2 run 119 ms, 4: 108, 6: 103.9, 8: 103.2, 10:
// 103.6, 13: 109 (144 without light cells).
//
// Once per run (hour-independent):
//   union    each aligned group of 128 visiting positions: its distinct cells
//            (shared-memory hash set, with the entries of each), the light
//            ones left out, sorted descending; every weighted entry gets its
//            slot (index in the union);
//   layout   the union is cut into chunks of 64 rows (the MMA K per stage);
//            per chunk, its entries are stored as (byte offset in the
//            shared-memory W tile, fp16 hi, fp16 lo): the weights of voxel t
//            are scaled by 2^-e_t (e_t: the exponent of its largest weight)
//            and split as w = hi + lo, so the two fp16 MMAs carry ~22 bits of
//            each weight; 2^e_t is kept per position for the epilogue.
//
// One launch for all hour blocks (B = 256 hours) that the slab has room for; a
// persistent CTA walks its (hour block, group) items:
//   producers (4 warps)  copy each chunk's 64 union rows of the fp16 slab
//                        (I[g][256 hours], 512 B a row) with 16-byte cp.async
//                        straight into the MN-major 128-byte-swizzled layout
//                        the MMA reads (B operand, N = hours) -- 4 slab
//                        stages, the copies of 3 chunks in flight -- then
//                        fence the async proxy and arrive on the stage's
//                        full barrier;
//   builders (3 x 3 warps) zero one of 3 W stages (K-major, 128-byte swizzle,
//                        A operand, M = voxels) and scatter the chunk's
//                        entries, fence, arrive; three teams, chunks in turn;
//   MMA (1 thread)       tcgen05.mma kind::f16 M128 N256 K16, 4 per chunk
//                        and tile (hi, lo), into one of two TMEM accumulators
//                        (2 x 256 columns), tcgen05.commit frees the stage;
//   epilogue (4 warps)   thread t = TMEM lane t = voxel t of the group: reads
//                        its 256 hours with tcgen05.ld, sums them and adds them
//                        to the voxel's own sum of the block (k_own_blocks),
//                        while the MMAs of the next group fill the other
//                        accumulator.
// k_mma_accumulate then adds up each voxel's hour blocks (FP64, Kahan or plain).
//
// Bound: the MMAs, and FP32 issue in k_light.  A chunk's eight MMAs take 1024 cycles
// of the tensor pipe (measured alone, B MN-major or K-major alike), reading 96 KB of
// shared memory that the staging writes as much to; with all cells in the unions
// a chunk took 1630 to 1800 here, and 2300 to 2500 with one launch an hour block, one
// builder team, the own terms in the epilogue and each chunk published after the
// wait for the stage of the chunk two ahead.  Without the light cells a chunk has 2.5
// times the entries and takes about 2200: three builder teams take 21.1 ms at 1024^2
// where two took 22.9 (light cells of up to 6 entries).
// Reflection of the 1024^2 city 78.5 ms at first, 58.6 with all cells in the
// unions, 30.8 with light cells; 512^2 20.1, 13.0 and 7.3; 160^2 2.38, 1.13 and 0.73.
//
// fp16 I values (RN, unbiased) and split fp16 weights keep the annual error
// far below 1e-4 (the rounding errors of I are independent across hours).
// Every mbarrier wait is bounded (1 s); on expiry the kernel flags
// kErrWaitTimeout, stops issuing, lets its copies and MMAs finish (bounded)
// and frees TMEM before it exits.
#include "solar_pair.cuh"

#include <algorithm>
#include <atomic>
#include <cstdlib>

#include <cuda_fp16.h>

namespace sgb {
namespace {

constexpr int kGroup = 128;                 // voxels per group = MMA M = TMEM lanes
constexpr int kHours = 256;                 // hours per block = MMA N
constexpr int kChunk = 64;                  // union rows per stage = MMA K per stage
constexpr int kBStages = 4;                 // slab-row stages (gathered: latency to hide)
constexpr int kAStages = 3;                 // weight-tile stages (built from registers)
constexpr int kCopyLag = kBStages - 2;      // a producer publishes chunk k - kCopyLag after issuing chunk k
constexpr int kUnionCap = 16384;            // distinct cells of a group the build handles
constexpr int kHashSlots = 2 * kUnionCap;
constexpr int kSmallCap = 8192;             // first pass: unions up to this many cells
constexpr int kBuildThreads = 1024;
constexpr int kLayoutThreads = 512;
constexpr int kMaxChunks = kUnionCap / kChunk;
constexpr int kLight = 8;                   // entries of a light cell of a group at most
constexpr int kLightShift = 3;              // a union takes at most an entry in kLight + 1, so one in 8
static_assert((1 << kLightShift) <= kLight + 1, "room of a union");
constexpr unsigned short kLightSlot = 0xFFFF;
constexpr int kNoSlot = -1;
constexpr unsigned long long kWaitNs = 1000000000ull;   // 1 s
constexpr int kMaxDevices = 64;

// warp roles of the hour-block kernel
constexpr int kProducerWarps = 4;           // warps 0-3
constexpr int kEpilogueWarp0 = 4;           // warps 4-7 (TMEM lane quarters 0-3)
constexpr int kMmaWarp = 8;
constexpr int kBuilderWarp0 = 9;            // warps 9-11, 12-14 and 15-17: three teams, chunks in turn
constexpr int kBuilderWarps = 3;
constexpr int kTeams = 3;
static_assert(kTeams <= kAStages, "a team that is a stage's second next user would mistake its phase");
constexpr int kThreads = (kBuilderWarp0 + kTeams * kBuilderWarps) * 32;

// shared memory: 3 x (W hi tile | W lo tile), 4 x slab rows (the hour table
// is read through L1: every epilogue lane reads the same entry)
constexpr int kTileA = kGroup * kChunk * 2;        // 16 KB, fp16 [128][64], K-major, 128B swizzle
constexpr int kTileB = kChunk * kHours * 2;        // 32 KB, fp16 [64 rows][256 hours], MN-major, 128B swizzle
constexpr int kAStageBytes = 2 * kTileA;           // 32 KB: hi and lo tiles
constexpr int kBRegion = kAStages * kAStageBytes;  // slab stages start here
constexpr int kSmemBytes = kBRegion + kBStages * kTileB + 1024;   // 225 KB + 1024-byte alignment slack
static_assert(kSmemBytes <= 227 * 1024 - 512, "dynamic + static shared memory of one CTA");

// Instruction descriptor, kind::f16: f32 accumulator, fp16 A and B, A
// K-major, B MN-major, N = 256, M = 128.
constexpr unsigned kIdesc = (1u << 4) | (1u << 16) | ((unsigned)(kHours >> 3) << 17) | ((unsigned)(kGroup >> 4) << 24);

// ---- union of each group ------------------------------------------------------

__device__ __forceinline__ void block_sort_desc(uint32_t* keys, int n2)
{
    for (int size = 2; size <= n2; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int t = threadIdx.x; t < (n2 >> 1); t += blockDim.x) {
                const int i = 2 * t - (t & (stride - 1));
                const int j = i + stride;
                const bool desc = (i & size) == 0;
                const uint32_t a = keys[i], b = keys[j];
                if ((a < b) == desc) {
                    keys[i] = b;
                    keys[j] = a;
                }
            }
            __syncthreads();
        }
    }
}

// The union of group q, in one CTA: the distinct cells of its weighted entries
// (cells[e], 0-based), descending, from ucells[woff[p0]] on (ucells = cells:
// they are written over the entries' cells); slots[e] = index of the entry's
// cell in it.  LIGHT: cells with at most kLight entries stay out of the union,
// which starts at ucells[woff[p0] >> kLightShift]; their entries get the slot
// kLightSlot and are counted per cell in light.  Returns false, writing
// nothing, when the group has more than CAP distinct cells.
template <int CAP, bool LIGHT>
__device__ bool union_group(int q, int N, const long long* __restrict__ woff, const int* cells, int* ucells,
                            unsigned short* __restrict__ slots, int* __restrict__ unions, int* __restrict__ nch,
                            int* __restrict__ light, uint32_t* sm, int* s_count)
{
    constexpr int kSlots = 2 * CAP;
    constexpr int kBits = CAP == 16384 ? 15 : CAP == 8192 ? 14 : 0;
    static_assert(kBits > 0, "union cap of 8192 or 16384 cells");
    uint32_t* table = sm;                 // [kSlots], key = cell + 1, 0 = empty
    uint32_t* uni = sm + kSlots;          // [CAP]
    uint32_t* many = uni + CAP;           // LIGHT: [kSlots] bytes, entries of the cell, up to kLight + 1
    const int p0 = q * kGroup, p1 = min(N, p0 + kGroup);
    const long long e0 = woff[p0], e1 = woff[p1];
    for (int i = threadIdx.x; i < kSlots; i += blockDim.x) table[i] = 0u;
    if (LIGHT)
        for (int i = threadIdx.x; i < kSlots / 4; i += blockDim.x) many[i] = 0u;
    if (threadIdx.x == 0) *s_count = 0;
    __syncthreads();
    for (long long e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
        const uint32_t key = (uint32_t)cells[e] + 1u;
        uint32_t h = (key * 2654435761u) >> (32 - kBits);
        for (int probe = 0; probe < kSlots; ++probe) {
            const uint32_t prev = atomicCAS(&table[h], 0u, key);
            if (prev == 0u) {
                const int at = atomicAdd(s_count, 1);
                if (!LIGHT && at < CAP) uni[at] = key;
            }
            if (prev == 0u || prev == key) {
                if (LIGHT) {   // saturating: a caller's list may name a cell any number of times
                    const int sh = 8 * (int)(h & 3u);
                    uint32_t old = *reinterpret_cast<volatile uint32_t*>(many + (h >> 2));
                    while (((old >> sh) & 0xFFu) <= (uint32_t)kLight) {
                        const uint32_t was = atomicCAS(many + (h >> 2), old, old + (1u << sh));
                        if (was == old) break;
                        old = was;
                    }
                }
                break;
            }
            h = (h + 1u) & (kSlots - 1);
        }
    }
    __syncthreads();
    int u = *s_count;
    if (u > CAP) return false;   // uniform: every thread read the same count
    const auto is_light = [&](uint32_t h) { return ((many[h >> 2] >> (8 * (h & 3u))) & 0xFFu) <= (uint32_t)kLight; };
    if (LIGHT) {   // the cells that stay in the union
        __syncthreads();
        if (threadIdx.x == 0) *s_count = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < kSlots; i += blockDim.x) {
            const bool in = table[i] != 0u && !is_light((uint32_t)i);
            const unsigned bal = __ballot_sync(0xFFFFFFFFu, in);
            int at = 0;
            if ((threadIdx.x & 31) == 0 && bal) at = atomicAdd(s_count, __popc(bal));
            at = __shfl_sync(0xFFFFFFFFu, at, 0);
            if (in) uni[at + __popc(bal & ((1u << (threadIdx.x & 31)) - 1u))] = table[i];
        }
        __syncthreads();
        u = *s_count;
    }
    int u2 = 64;
    while (u2 < u) u2 <<= 1;
    for (int i = u + threadIdx.x; i < u2; i += blockDim.x) uni[i] = 0u;
    __syncthreads();
    block_sort_desc(uni, u2);
    int* ucell = reinterpret_cast<int*>(uni);
    for (int i = threadIdx.x; i < u; i += blockDim.x) ucell[i] = (int)uni[i] - 1;
    __syncthreads();
    for (long long e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
        const int cell = cells[e];
        if (LIGHT) {
            const uint32_t key = (uint32_t)cell + 1u;
            uint32_t h = (key * 2654435761u) >> (32 - kBits);
            while (table[h] != key) h = (h + 1u) & (kSlots - 1);   // every entry's key is in the table
            if (is_light(h)) {
                slots[e] = kLightSlot;
                atomicAdd(light + cell, 1);
                continue;
            }
        }
        int lo = 0, hi = u - 1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (ucell[mid] > cell) lo = mid + 1; else hi = mid;
        }
        slots[e] = (unsigned short)lo;
    }
    __syncthreads();
    int* dst = ucells + (LIGHT ? e0 >> kLightShift : e0);
    for (int i = threadIdx.x; i < u; i += blockDim.x) dst[i] = ucell[i];
    if (threadIdx.x == 0) {
        unions[q] = u;
        nch[q] = (u + kChunk - 1) / kChunk;
    }
    return true;
}

// First pass, one CTA per group with room for kSmallCap cells (96 KB of
// shared memory: two CTAs a SM); a group with a larger union is listed in
// retry[1 ..] (count in retry[0]) and left untouched.
template <bool LIGHT>
__global__ void __launch_bounds__(kBuildThreads)
k_mma_union_small(int N, const long long* __restrict__ woff, const int* cells, int* ucells,
                  unsigned short* __restrict__ slots, int* __restrict__ unions, int* __restrict__ nch,
                  int* __restrict__ light, int* __restrict__ retry, int hand_on_all)
{
    extern __shared__ __align__(16) uint32_t sm[];
    __shared__ int s_count;
    const int q = blockIdx.x;
    if ((hand_on_all ||
         !union_group<kSmallCap, LIGHT>(q, N, woff, cells, ucells, slots, unions, nch, light, sm, &s_count)) &&
        threadIdx.x == 0)
        retry[1 + atomicAdd(retry, 1)] = q;
}

// Second pass over the listed groups with room for kUnionCap cells; a union
// above that leaves the group untouched and counts it in *over.
template <bool LIGHT>
__global__ void __launch_bounds__(kBuildThreads)
k_mma_union_large(int N, const long long* __restrict__ woff, const int* cells, int* ucells,
                  unsigned short* __restrict__ slots, int* __restrict__ unions, int* __restrict__ nch,
                  int* __restrict__ light, const int* __restrict__ retry, int* __restrict__ over)
{
    extern __shared__ __align__(16) uint32_t sm[];
    __shared__ int s_count;
    const int n = retry[0];
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        const int q = retry[1 + i];
        if (!union_group<kUnionCap, LIGHT>(q, N, woff, cells, ucells, slots, unions, nch, light, sm, &s_count) &&
            threadIdx.x == 0) {
            atomicAdd(over, 1);
            unions[q] = 0;
            nch[q] = 0;
        }
        __syncthreads();
    }
}

// Byte offset of W element (voxel t, row k of the chunk) in the K-major,
// 128-byte-swizzled tile: 8-voxel atoms of 1024 bytes, 128 bytes (64 fp16)
// a voxel, 16-byte pieces XOR-ed with the voxel's row in the atom.
__device__ __forceinline__ unsigned a_offset(int t, int k)
{
    const int r = t & 7;
    return (unsigned)((t >> 3) * 1024 + r * 128 + (((k >> 3) ^ r) << 4) + ((k & 7) << 1));
}

// One CTA per group.  PASS 0: entries per chunk (ccnt at cbase[q]) and the
// per-position scale 2^e; PASS 1: the entries at coff (ent must not be
// read before).  Groups that overflowed the union cap have no chunks.
template <int PASS, bool LIGHT>
__global__ void __launch_bounds__(kLayoutThreads)
k_mma_layout(int N, const long long* __restrict__ woff, const unsigned short* __restrict__ slots,
             const float* __restrict__ wts, const int* __restrict__ nch, const long long* __restrict__ cbase,
             int* __restrict__ ccnt, const long long* __restrict__ coff, uint2* __restrict__ ent,
             float* __restrict__ scale, LightLists ll)
{
    __shared__ int s_cnt[kMaxChunks];
    __shared__ int s_exp[kGroup];
    const int q = blockIdx.x;
    const int p0 = q * kGroup, p1 = min(N, p0 + kGroup);
    const int nc = nch[q];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int c = threadIdx.x; c < nc; c += blockDim.x) s_cnt[c] = 0;
    // exponent of each voxel's largest weight (weights are > 0)
    for (int t = warp; t < kGroup; t += kLayoutThreads / 32) {
        const int p = p0 + t;
        float m = 0.0f;
        if (p < p1)
            for (long long e = woff[p] + lane; e < woff[p + 1]; e += 32) m = fmaxf(m, wts[e]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
        int ex = 0;
        if (m > 0.0f) frexpf(m, &ex);   // m in [2^(ex-1), 2^ex)
        if (lane == 0) {
            s_exp[t] = ex;
            if (PASS == 0 && p < p1) scale[p] = ldexpf(1.0f, ex);
        }
    }
    __syncthreads();
    if (nc == 0 && !LIGHT) return;
    const long long cb = cbase[q];
    // voxel t owns entries [woff[p0 + t], woff[p0 + t + 1])
    for (int t = warp; t < p1 - p0; t += kLayoutThreads / 32) {
        const int p = p0 + t;
        const float sc = ldexpf(1.0f, -s_exp[t]);
        int nl = 0;   // light entries of the voxel so far
        const long long eb = woff[p], ee = woff[p + 1];
        for (long long e0 = eb; e0 < ee; e0 += 32) {
            const long long e = e0 + lane;
            const int sl = e < ee ? slots[e] : kNoSlot;
            if (LIGHT) {
                const bool is = sl == kLightSlot;
                const unsigned bal = __ballot_sync(0xFFFFFFFFu, is);
                if (PASS == 1 && is) {   // to its cell's list, in any order: each product stands for itself
                    const int cell = ll.cells[e];
                    const long long at = ll.off[cell] + (atomicSub(ll.cnt + cell, 1) - 1);
                    ll.ent[at] = make_uint2((uint32_t)(eb + nl + __popc(bal & ((1u << lane) - 1u))),
                                            __float_as_uint(wts[e]));
                }
                nl += __popc(bal);
                if (is) continue;
            }
            if (sl == kNoSlot) continue;
            const int c = sl / kChunk;
            const int at = atomicAdd(&s_cnt[c], 1);
            if (PASS == 1) {
                const float w = wts[e] * sc;   // exact: a power-of-two scale
                const __half hi = __float2half_rn(w);
                const __half lo = __float2half_rn(w - __half2float(hi));
                const __half2 hl = __halves2half2(hi, lo);
                ent[coff[cb + c] + at] = make_uint2(a_offset(t, sl - c * kChunk), *reinterpret_cast<const unsigned*>(&hl));
            }
        }
        if (LIGHT && PASS == 1 && lane == 0) ll.many[p] = nl;
    }
    if (PASS == 0) {
        __syncthreads();
        for (int c = threadIdx.x; c < nc; c += blockDim.x) ccnt[cb + c] = s_cnt[c];
    }
}

// slab[hour block][top cell][256 hours]: I in fp16, from hour j0 of the table on.
// A lane owns 4 consecutive hours (their table entries stay in registers, two
// packed pairs), a warp 128; the 8 warps of a CTA sweep the same run of cells,
// whose normals (each component twice, as the packed pairs want them) and
// shadow words are in shared memory.  One 256-byte store a cell and warp.  The
// hours' entries are a cost per CTA, so large scenes take long runs (512^2,
// 4352 hours: 64 cells 1.10 ms, 128 0.88), and small ones short runs that fill
// the GPU.
constexpr int kSlabWarps = 8;

__global__ void __launch_bounds__(kSlabWarps * 32)
k_solar_slab16(const float4* __restrict__ geo_n, int T, const uint32_t* __restrict__ shadow, int words32,
               const HourEntry* __restrict__ table, int j0, int nb, int run, uint2* __restrict__ slab)
{
    extern __shared__ __align__(16) unsigned char s_run[];
    NormalPair* s_n = reinterpret_cast<NormalPair*>(s_run);
    uint32_t* s_shadow = reinterpret_cast<uint32_t*>(s_n + run);   // [run][words32]
    const int lane = threadIdx.x & 31, hc = blockIdx.y * kSlabWarps + (threadIdx.x >> 5);
    const int g0 = blockIdx.x * run, cells = min(run, T - g0);
    for (int i = threadIdx.x; i < cells; i += kSlabWarps * 32) s_n[i] = NormalPair(__ldg(geo_n + g0 + i));
    for (int i = threadIdx.x; i < cells * words32; i += kSlabWarps * 32)
        s_shadow[i] = __ldg(shadow + (size_t)g0 * words32 + i);
    __syncthreads();
    if (hc >= nb * (kHours / 128)) return;
    const int b = hc * 128 + 4 * lane;
    const HourPair e = make_pair2(table[j0 + b], table[j0 + b + 1]), f = make_pair2(table[j0 + b + 2], table[j0 + b + 3]);
    const uint32_t *e0 = s_shadow + e.word[0], *e1 = s_shadow + e.word[1], *f0 = s_shadow + f.word[0],
                   *f1 = s_shadow + f.word[1];
    uint2* dst = slab + (((size_t)(b / kHours) * T + g0) * kHours + b % kHours) / 4;
#pragma unroll 4
    for (int g = 0; g < cells; ++g) {
        const NormalPair n = s_n[g];
        const int w = g * words32;
        const float2 i0 = unpack2(solar_I2(n, e, e0[w], e1[w]));
        const float2 i1 = unpack2(solar_I2(n, f, f0[w], f1[w]));
        const __half2 h0 = __float22half2_rn(i0), h1 = __float22half2_rn(i1);
        dst[(size_t)g * (kHours / 4)] =
            make_uint2(*reinterpret_cast<const unsigned*>(&h0), *reinterpret_cast<const unsigned*>(&h1));
    }
}

// ---- light cells ------------------------------------------------------------------

// One block of the cell's row (8 hours a lane) times the weights of E entries.
template <int E>
__device__ __forceinline__ void light_row(const uint4& r, const f32x2 (&w)[E / 2], f32x2 (&acc)[E / 2])
{
    const unsigned x[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&x[i]));
        const f32x2 a = pack2(h.x, h.x), b = pack2(h.y, h.y);
#pragma unroll
        for (int j = 0; j < E / 2; ++j) acc[j] = fma2(w[j], a, acc[j]);
#pragma unroll
        for (int j = 0; j < E / 2; ++j) acc[j] = fma2(w[j], b, acc[j]);
    }
}

// n (at most E) entries of one cell over nb hour blocks; row: this lane's piece
// of the cell's row in the first block, `stride` pieces to the next one's.
template <int E>
__device__ __forceinline__ void light_cell(const uint4* __restrict__ row, size_t stride, int nb,
                                           const uint2* __restrict__ ent, int n, float* __restrict__ val, int lane)
{
    constexpr int kAhead = 2;   // rows in flight (4: +6%, 6: +14%, for the registers they take)
    const uint2 en = lane < n ? __ldg(ent + lane) : make_uint2(0u, 0u);
    uint4 r[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i) r[i] = i < nb ? __ldg(row + i * stride) : make_uint4(0u, 0u, 0u, 0u);
    f32x2 w[E / 2], acc[E / 2];
#pragma unroll
    for (int j = 0; j < E / 2; ++j) {
        w[j] = pack2(__uint_as_float(__shfl_sync(0xFFFFFFFFu, en.y, 2 * j)),
                     __uint_as_float(__shfl_sync(0xFFFFFFFFu, en.y, 2 * j + 1)));
        acc[j] = 0ull;
    }
    for (int b = 0; b < nb; b += kAhead) {
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            if (b + i >= nb) break;
            const uint4 x = r[i];
            if (b + i + kAhead < nb) r[i] = __ldg(row + (size_t)(b + i + kAhead) * stride);
            light_row<E>(x, w, acc);
        }
    }
    // the lanes' sums of every entry: lane l ends with entry l / (32 / E)
    float a[E];
#pragma unroll
    for (int j = 0; j < E / 2; ++j) {
        const float2 v = unpack2(acc[j]);
        a[2 * j] = v.x;
        a[2 * j + 1] = v.y;
    }
#pragma unroll
    for (int k = E / 2, o = 16; o > 0; k >>= 1, o >>= 1) {
        if (k >= 1) {
#pragma unroll
            for (int j = 0; j < k; ++j) {
                const float keep = (lane & o) ? a[j + k] : a[j], give = (lane & o) ? a[j] : a[j + k];
                a[j] = keep + __shfl_xor_sync(0xFFFFFFFFu, give, o);
            }
        } else {
            a[0] += __shfl_xor_sync(0xFFFFFFFFu, a[0], o);
        }
    }
    const int i = lane / (32 / E);
    const uint32_t at = __shfl_sync(0xFFFFFFFFu, en.x, i);
    if (lane % (32 / E) == 0 && i < n) val[at] = a[0];
}

constexpr int kLightWarps = 8;
constexpr int kLightWindow = 128;   // entries of a warp (64: +2% in a run, 32: +20%)

// Products of the light entries with the rows of their cells, hour by hour,
// summed over the nb hour blocks of the slab: val[entry].
__global__ void __launch_bounds__(kLightWarps * 32, 4)
k_light(const uint4* __restrict__ slab, int T, int nb, int window, const long long* __restrict__ off,
        const uint2* __restrict__ ent, float* __restrict__ val)
{
    const int lane = threadIdx.x & 31;
    const long long total = __ldg(off + T);
    long long at = ((long long)blockIdx.x * kLightWarps + (threadIdx.x >> 5)) * window;
    const long long end = min(total, at + window);
    if (at >= end) return;
    int lo = 0, hi = T - 1;   // the last cell that starts at or before the first entry
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(off + mid) <= at) lo = mid; else hi = mid - 1;
    }
    int cell = lo;
    const size_t stride = (size_t)T * (kHours / 8);
    while (at < end) {
        // the cell of entry `at`: the first one that ends after it
        long long stop = 0;
        for (;;) {
            const int c = cell + lane;
            const long long e = c < T ? __ldg(off + c + 1) : total;
            const unsigned past = __ballot_sync(0xFFFFFFFFu, e > at);
            if (past) {
                const int i = __ffs(past) - 1;
                cell += i;
                stop = __shfl_sync(0xFFFFFFFFu, e, i);
                break;
            }
            cell += 32;
        }
        int n = (int)(min(stop, end) - at);
        const uint4* row = slab + (size_t)cell * (kHours / 8) + lane;
        while (n > 0) {
            int k;
            if (n > 8) light_cell<16>(row, stride, nb, ent + at, k = min(n, 16), val, lane);
            else if (n > 4) light_cell<8>(row, stride, nb, ent + at, k = n, val, lane);
            else light_cell<4>(row, stride, nb, ent + at, k = n, val, lane);
            at += k;
            n -= k;
        }
    }
}

// ---- hour-block kernel ----------------------------------------------------------

__device__ __forceinline__ unsigned su32(const void* p)
{
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long gtime()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits for the phase of the given parity; false on expiry or when another
// role gave up.
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity, const volatile int* fail,
                                         unsigned long long limit = kWaitNs)
{
    unsigned long long t0 = 0;
    for (unsigned i = 0;; ++i) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if ((i & 63u) == 63u) {
            if (fail && *fail) return false;
            const unsigned long long t = gtime();
            if (t0 == 0) t0 = t;
            else if (t - t0 > limit) return false;
        }
    }
}

__device__ __forceinline__ void bar_arrive(unsigned bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// K-major, 128-byte swizzle (layout 2, sm_100 version 1): 8-row atoms 1024
// bytes apart (SBO), leading offset unused.
__device__ __forceinline__ unsigned long long desc_k_sw128(unsigned addr)
{
    return (unsigned long long)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((unsigned long long)(1024 >> 4) << 32) |
           (1ull << 46) | (2ull << 61);
}

// MN-major, 128-byte swizzle: atoms of 8 K-rows x 64 fp16 (1024 bytes); the
// next 64 hours (MN) are 8 KB further (LBO), the next 8 rows (K) 1 KB (SBO).
__device__ __forceinline__ unsigned long long desc_mn_sw128(unsigned addr)
{
    return (unsigned long long)((addr >> 4) & 0x3FFFu) | ((unsigned long long)(8192 >> 4) << 16) |
           ((unsigned long long)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void mma_f16(unsigned d, unsigned long long a, unsigned long long b, unsigned acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(kIdesc), "r"(acc), "r"(0), "r"(0), "r"(0), "r"(0));
}

__device__ __forceinline__ void mma_commit(unsigned bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// Items of a launch: (hour block, group), hour block by hour block, handed to
// the CTAs in turn, so that the CTAs work on neighbouring groups of one or two
// hour blocks at a time (their union rows meet in L2) and a CTA's share of the
// uneven groups averages out over the hour blocks.  One launch for all hour
// blocks has one ragged end instead of 17, and small scenes (45 groups at 64^2)
// fill the GPU with several hour blocks at once.
struct MmaTiles {
    int N, T, NG, items, rot;  // item n: hour block n / NG, group (n + rot * (n / NG)) % NG
    const long long* woff;     // [N + 1]; the union of group q starts at woff[128 q] >> shift
    int shift;
    const int* cells;          // union cells (descending) per group
    const int* unions;         // [NG] union size
    const long long* cbase;    // [NG + 1] first chunk of each group
    const long long* coff;     // [C + 1] first entry of each chunk
    const uint2* ent;          // entries: x = byte offset in the W tile, y = half2 (hi, lo)
    const float* scale;        // [N] 2^e per visiting position
    __device__ int block_of(int n) const { return n / NG; }
    __device__ int group_of(int n) const
    {
        const int hb = n / NG;
        return (int)((unsigned)(n - hb * NG + rot * hb) % (unsigned)NG);
    }
};

// Walks the (item, chunk) sequence of one CTA: the CTA's items, chunks of 64
// union rows inside each group (groups with an empty union have none) -- the
// order every role follows.
struct Cursor {
    int n, q, c, u;
    long long ub;   // first union cell of group q
    long long cb;   // first chunk of group q
    long long row0; // slab row of cell 0 in the item's hour block
    __device__ Cursor(const MmaTiles& mt, int cta) : n(cta), q(0), c(0), u(0), ub(0), cb(0), row0(0) { settle(mt); }
    __device__ bool valid(const MmaTiles& mt) const { return n < mt.items; }
    __device__ void settle(const MmaTiles& mt)
    {
        for (; n < mt.items; n += gridDim.x, c = 0) {
            q = mt.group_of(n);
            u = __ldg(mt.unions + q);
            if (c * kChunk < u) break;
        }
        if (n < mt.items) {
            ub = __ldg(mt.woff + (long long)q * kGroup) >> mt.shift;
            cb = __ldg(mt.cbase + q);
            row0 = (long long)mt.block_of(n) * mt.T;
        }
    }
    __device__ void advance(const MmaTiles& mt)
    {
        ++c;
        if (c * kChunk >= u) {
            n += gridDim.x;
            c = 0;
            if (n < mt.items) settle(mt);
        }
    }
    // cell of row r of the current chunk (padding rows repeat row 0: their weights are 0)
    __device__ int row_cell(const MmaTiles& mt, int r, bool want) const
    {
        if (!want || !valid(mt)) return 0;
        const int rows = min(kChunk, u - c * kChunk);
        return __ldg(mt.cells + ub + (long long)c * kChunk + (r < rows ? r : 0));
    }
};

__global__ void __launch_bounds__(kThreads, 1)
k_reflect_mma(const __half* __restrict__ slab, MmaTiles mt, float* __restrict__ sums, int* __restrict__ err)
{
    extern __shared__ __align__(1024) unsigned char dsm[];
    __shared__ __align__(8) unsigned long long full[kBStages], emptyB[kBStages], aready[kAStages], emptyA[kAStages],
        dfull[2], dempty[2], drain;
    __shared__ unsigned s_tmem;
    __shared__ volatile int s_fail;
    __shared__ volatile int s_bok[kTeams];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned base = (su32(dsm) + 1023u) & ~1023u;               // stages, 1024-byte aligned
    unsigned char* gbase = dsm + (base - su32(dsm));

    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&s_tmem)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < kBStages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(&full[s])), "r"(kProducerWarps));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(&emptyB[s])), "r"(1));
        }
        for (int s = 0; s < kAStages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(&aready[s])), "r"(1));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(&emptyA[s])), "r"(1));
        }
        for (int b = 0; b < 2; ++b) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(&dfull[b])), "r"(1));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(&dempty[b])), "r"(4));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(&drain)), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_fail = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = s_tmem;
    bool ok = true;

    if (warp < kProducerWarps) {
        // ---- producers: 16 rows a warp, one 16-byte piece a lane per row
        long long k = 0;
        const int r0 = warp * 16;
        Cursor cur(mt, blockIdx.x);
        auto publish = [&](long long j) {   // chunk j's copies of this warp have landed
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(su32(&full[j % kBStages]));
        };
        // Cells of the next two chunks, in registers of their own (a move would wait
        // for the load): a chunk's ids load while the chunk before it is copied.
        int cell_a = cur.row_cell(mt, r0 + lane, lane < 16), cell_b = 0;
        long long row_a = cur.row0, row_b = 0;
        bool more_a = cur.valid(mt), more_b = false;
        if (more_a) {
            cur.advance(mt);
            more_b = cur.valid(mt);
            cell_b = cur.row_cell(mt, r0 + lane, lane < 16);
            row_b = cur.row0;
        }
        // Copies chunk k (cells `cell`) and loads the cells of chunk k + 2.  Chunk
        // k - 2 is published before the stage of chunk k is waited for: after it,
        // the MMAs waited for two things in turn, the stage and the copies.
        auto copy = [&](int& cell, long long& row0, bool& more) {
            static_assert(kCopyLag == 2, "wait_group count below");
            if (k >= kCopyLag) {
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                publish(k - kCopyLag);
            }
            const int s = (int)(k % kBStages);
            const bool w_ok = k < kBStages || bar_wait(su32(&emptyB[s]), (unsigned)(((k / kBStages) - 1) & 1), &s_fail);
            if (!__all_sync(0xFFFFFFFFu, w_ok)) {   // the warp decides as one
                ok = false;
                return;
            }
            const __half* chunk = slab + row0 * kHours + lane * 8;
            const int na = lane >> 3, cc = lane & 7;
            const unsigned bst = base + (unsigned)(kBRegion + s * kTileB) + (unsigned)(na * 8192 + (r0 >> 3) * 1024);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int r8 = i & 7;
                const __half* src = chunk + (long long)__shfl_sync(0xFFFFFFFFu, cell, i) * kHours;
                const unsigned dst = bst + (unsigned)((i >> 3) * 1024 + r8 * 128 + ((cc ^ r8) << 4));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            ++k;
            more = false;
            if (cur.valid(mt)) {
                cur.advance(mt);
                more = cur.valid(mt);
                cell = cur.row_cell(mt, r0 + lane, lane < 16);
                row0 = cur.row0;
            }
        };
        while (more_a && ok) {
            copy(cell_a, row_a, more_a);
            if (!more_b || !ok) break;
            copy(cell_b, row_b, more_b);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        for (long long j = k >= kCopyLag ? k - kCopyLag : 0; j < k; ++j) publish(j);
        if (!ok) {
            if (lane == 0) atomicOr(err, kErrWaitTimeout);
            s_fail = 1;
        }
    } else if (warp == kMmaWarp) {
        // ---- one thread issues the MMAs
        if (lane == 0) {
            long long k = 0;
            int gi = 0;
            for (int n = blockIdx.x; n < mt.items && ok; n += gridDim.x, ++gi) {
                const int q = mt.group_of(n);
                const int b = gi & 1;
                if (gi >= 2 && !bar_wait(su32(&dempty[b]), (unsigned)(((gi >> 1) - 1) & 1), &s_fail)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int u = mt.unions[q];
                const unsigned d = tmem + (unsigned)(b * kHours);
                for (int c = 0; c * kChunk < u; ++c, ++k) {
                    const int s = (int)(k % kBStages), t = (int)(k % kAStages);
                    if (!bar_wait(su32(&full[s]), (unsigned)((k / kBStages) & 1), &s_fail) ||
                        !bar_wait(su32(&aready[t]), (unsigned)((k / kAStages) & 1), &s_fail)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned sa = base + (unsigned)(t * kAStageBytes);
                    const unsigned sb = base + (unsigned)(kBRegion + s * kTileB);
                    const int ks = (min(kChunk, u - c * kChunk) + 15) >> 4;
                    for (int j = 0; j < ks; ++j) {
                        const unsigned long long db = desc_mn_sw128(sb + 2048u * j);
                        mma_f16(d, desc_k_sw128(sa + 32u * j), db, (c > 0 || j > 0) ? 1u : 0u);
                        mma_f16(d, desc_k_sw128(sa + kTileA + 32u * j), db, 1u);
                    }
                    // both stages are free once these MMAs have read them
                    mma_commit(su32(&emptyB[s]));
                    mma_commit(su32(&emptyA[t]));
                }
                if (!ok) break;
                mma_commit(su32(&dfull[b]));       // the group's accumulator is complete
            }
            if (!ok) {
                atomicOr(err, kErrWaitTimeout);
                s_fail = 1;
            }
        }
        __syncwarp();
    } else if (warp >= kBuilderWarp0) {
        // ---- builders: zero the W tiles, scatter the chunk's weights.  The teams
        // take the chunks in turn, and a team loads the entries of its next chunk
        // into registers while the others build: one team's chunk takes 1300
        // cycles and more, the chunk's MMAs 1024
        const int team = (warp - kBuilderWarp0) / kBuilderWarps;
        const int bt = threadIdx.x - (kBuilderWarp0 + team * kBuilderWarps) * 32;
        constexpr int kBuilders = kBuilderWarps * 32;
        constexpr int kPref = 16;   // entries a thread holds ahead (8: +11%, 12: +1.6%, 20: +2%); more load at scatter
        Cursor cur(mt, blockIdx.x);
        for (int i = 0; i < team && cur.valid(mt); ++i) cur.advance(mt);
        uint2 pre[kPref];
        long long pe0 = 0, pe1 = 0;
        auto prefetch = [&]() {
            pe0 = pe1 = 0;
            if (cur.valid(mt)) {
                const long long ci = cur.cb + cur.c;
                pe0 = __ldg(mt.coff + ci);
                pe1 = __ldg(mt.coff + ci + 1);
            }
#pragma unroll
            for (int i = 0; i < kPref; ++i) {
                const long long e = pe0 + bt + (long long)i * kBuilders;
                pre[i] = e < pe1 ? __ldg(mt.ent + e) : make_uint2(0xFFFFFFFFu, 0u);
            }
        };
        prefetch();
        long long k = team;
        while (cur.valid(mt) && ok) {
            const int s = (int)(k % kAStages);
            // one thread waits for the stage; every builder of the team takes its decision
            if (bt == 0)
                s_bok[team] = (k < kAStages || bar_wait(su32(&emptyA[s]), (unsigned)(((k / kAStages) - 1) & 1), &s_fail))
                                  ? 1 : 0;
            asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(kBuilders) : "memory");
            ok = s_bok[team] != 0;
            if (!ok) break;
            unsigned char* sa = gbase + (size_t)s * kAStageBytes;
            uint4* z = reinterpret_cast<uint4*>(sa);
            for (int i = bt; i < 2 * kTileA / 16; i += kBuilders) z[i] = make_uint4(0u, 0u, 0u, 0u);
            asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(kBuilders) : "memory");
#pragma unroll
            for (int i = 0; i < kPref; ++i) {
                if (pre[i].x != 0xFFFFFFFFu) {
                    *reinterpret_cast<unsigned short*>(sa + pre[i].x) = (unsigned short)(pre[i].y & 0xFFFFu);
                    *reinterpret_cast<unsigned short*>(sa + kTileA + pre[i].x) = (unsigned short)(pre[i].y >> 16);
                }
            }
            for (long long e = pe0 + bt + (long long)kPref * kBuilders; e < pe1; e += kBuilders) {
                const uint2 en = __ldg(mt.ent + e);
                *reinterpret_cast<unsigned short*>(sa + en.x) = (unsigned short)(en.y & 0xFFFFu);
                *reinterpret_cast<unsigned short*>(sa + kTileA + en.x) = (unsigned short)(en.y >> 16);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(kBuilders) : "memory");
            if (bt == 0) bar_arrive(su32(&aready[s]));
            // the team's next chunk's entries (after the arrive: their latency stays
            // off the MMA's path)
            for (int i = 0; i < kTeams && cur.valid(mt); ++i) cur.advance(mt);
            prefetch();
            k += kTeams;
        }
        if (!ok) {
            if (bt == 0) atomicOr(err, kErrWaitTimeout);
            s_fail = 1;
        }
    } else {
        // ---- epilogue: thread t = TMEM lane t = voxel t of the group: adds the sum
        // of its 256 hours to the voxel's own (k_own_blocks; computing that here
        // took most of the epilogue's time, which nothing hides when a CTA has few
        // groups)
        const int t = threadIdx.x - kEpilogueWarp0 * 32;
        const unsigned lane_base = (unsigned)((warp & 3) * 32) << 16;
        int gi = 0;
        for (int n = blockIdx.x; n < mt.items && ok; n += gridDim.x, ++gi) {
            const int q = mt.group_of(n);
            const int b = gi & 1;
            const int p = q * kGroup + t;
            const bool valid = p < mt.N;
            const float sc = valid ? __ldg(mt.scale + p) : 0.0f;
            const bool any = __ldg(mt.unions + q) > 0;
            const bool w_ok = bar_wait(su32(&dfull[b]), (unsigned)((gi >> 1) & 1), &s_fail, 2 * kWaitNs);
            if (!__all_sync(0xFFFFFFFFu, w_ok)) {   // tcgen05.ld below needs the whole warp
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 2
            for (int c0 = 0; c0 < kHours; c0 += 32) {
                unsigned r[32];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                    "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                      "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
                      "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
                      "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                    : "r"(tmem + lane_base + (unsigned)(b * kHours + c0)));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int i = 0; i < 32; ++i) sum[i & 3] += __uint_as_float(r[i]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(su32(&dempty[b]));
            if (valid && any) sums[(size_t)mt.block_of(n) * mt.N + p] += ((sum[0] + sum[1]) + (sum[2] + sum[3])) * sc;
        }
        if (!ok) {
            if (lane == 0) atomicOr(err, kErrWaitTimeout);
            s_fail = 1;
        }
    }

    // Drain: every MMA this CTA issued completes before TMEM is freed
    // (tcgen05.commit tracks all of the issuing thread's earlier MMAs).
    __syncthreads();
    if (warp == kMmaWarp) {
        if (lane == 0) {
            mma_commit(su32(&drain));
            if (!bar_wait(su32(&drain), 0u, nullptr, 2 * kWaitNs)) atomicOr(err, kErrWaitTimeout);
        }
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
}

// Accumulates the hour blocks' sums (sums [nb][N] by visiting position) of every
// voxel; first / last: the launch's blocks begin / end the year (else the
// accumulators are read / kept).
template <int MODE>
__global__ void __launch_bounds__(256)
k_mma_accumulate(const int* __restrict__ order, int N, int nb, const float* __restrict__ sums, LightLists ll,
                 const long long* __restrict__ woff, Accum acc, bool first, bool last, float* __restrict__ out)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= N) return;
    const int v = __ldg(order + p);
    double a64 = 0.0;
    float a32 = 0.0f, comp = 0.0f;
    if (!first) {
        if (MODE == 0) a64 = acc.f64[v];
        else a32 = acc.f32[v];
        if (MODE == 1) comp = acc.comp[v];
    }
    const auto add = [&](float x) {
        if (MODE == 0) {
            a64 += (double)x;
        } else if (MODE == 1) {
            const float y = __fsub_rn(x, comp);
            const float s = __fadd_rn(a32, y);
            comp = __fsub_rn(__fsub_rn(s, a32), y);
            a32 = s;
        } else {
            a32 = __fadd_rn(a32, x);
        }
    };
#pragma unroll 4
    for (int hb = 0; hb < nb; ++hb) add(__ldg(sums + (size_t)hb * N + p));
    if (ll.many) {   // the voxel's light entries, as one more block
        const float* val = ll.val + woff[p];
        float x = 0.0f;
        for (int i = 0, n = __ldg(ll.many + p); i < n; ++i) x += __ldg(val + i);
        add(x);
    }
    if (last) {
        out[v] = MODE == 0 ? (float)a64 : a32;
    } else if (MODE == 0) {
        acc.f64[v] = a64;
    } else {
        acc.f32[v] = a32;
        if (MODE == 1) acc.comp[v] = comp;
    }
}

int mma_sms()
{
    static std::atomic<int> cached{0};
    int sms = cached.load(std::memory_order_relaxed);
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
        cached.store(sms, std::memory_order_relaxed);
    }
    return sms;
}

template <typename K>
cudaError_t allow_smem(K kernel, size_t bytes, std::atomic<bool> (&done)[kMaxDevices])
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    if (!done[dev].load(std::memory_order_acquire)) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return e;
        done[dev].store(true, std::memory_order_release);
    }
    return cudaSuccess;
}

}  // namespace

int mma_group_count(int N) { return (N + kGroup - 1) / kGroup; }

// Light cells from 20,000 voxels on: below, the launches for them and their lists
// cost more than the MMAs they save (runs of 112^2, 17,500 voxels: 1.94 ms with them,
// 1.88 without; 128^2, 23,000: 2.26 and 2.36; 64^2 1.14 and 1.07).  Entries are
// numbered with 32 bits.
bool mma_light_ok(int N, long long entries) { return N >= 20000 && entries < 0xFFFFFFFFll; }
long long mma_union_room(long long entries) { return (entries >> kLightShift) + 1; }

cudaError_t launch_mma_union(int N, const long long* woff, int* cells, int* ucells, unsigned short* slots, int* unions,
                             int* nch, int* light, int* over, int* retry, cudaStream_t st)
{
    const int NG = mma_group_count(N);
    if (NG <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(retry, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    // with the light cells' byte a slot: 112 KB (two CTAs a SM) and 224 KB
    const size_t small = sizeof(uint32_t) * (size_t)(3 * kSmallCap) + (light ? 2 * kSmallCap : 0);
    const size_t large = sizeof(uint32_t) * (size_t)(kHashSlots + kUnionCap) + (light ? kHashSlots : 0);
    static std::atomic<bool> attr_s[2][kMaxDevices], attr_l[2][kMaxDevices];
    const auto ks = light ? k_mma_union_small<true> : k_mma_union_small<false>;
    const auto kl = light ? k_mma_union_large<true> : k_mma_union_large<false>;
    if ((e = allow_smem(ks, small, attr_s[light ? 1 : 0])) != cudaSuccess) return e;
    if ((e = allow_smem(kl, large, attr_l[light ? 1 : 0])) != cudaSuccess) return e;
    // SGB_UNION_SECOND_PASS=1 hands every group to the second pass (tests use
    // it to check that pass; the unions are the same either way)
    const char* env = std::getenv("SGB_UNION_SECOND_PASS");
    const int all = (env && env[0] == '1') ? 1 : 0;
    ks<<<NG, kBuildThreads, small, st>>>(N, woff, cells, ucells, slots, unions, nch, light, retry, all);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    // the groups the first pass listed (usually few; the grid exits at once when none)
    kl<<<mma_sms(), kBuildThreads, large, st>>>(N, woff, cells, ucells, slots, unions, nch, light, retry, over);
    return cudaGetLastError();
}

cudaError_t launch_mma_layout(int pass, int N, const long long* woff, const unsigned short* slots, const float* wts,
                              const int* nch, const long long* cbase, int* ccnt, const long long* coff, uint2* ent,
                              float* scale, const LightLists& ll, cudaStream_t st)
{
    const int NG = mma_group_count(N);
    if (NG <= 0) return cudaSuccess;
    const auto k = ll.many ? (pass == 0 ? k_mma_layout<0, true> : k_mma_layout<1, true>)
                           : (pass == 0 ? k_mma_layout<0, false> : k_mma_layout<1, false>);
    k<<<NG, kLayoutThreads, 0, st>>>(N, woff, slots, wts, nch, cbase, ccnt, coff, ent, scale, ll);
    return cudaGetLastError();
}

cudaError_t launch_light(const void* slab16, int T, int nb, const LightLists& ll, cudaStream_t st)
{
    if (!ll.many || ll.total <= 0 || nb <= 0) return cudaSuccess;
    // entries of a warp: enough to share the rows, fewer where the GPU would not be full
    const int window = (int)std::max<long long>(16, std::min<long long>(kLightWindow, ll.total / (24 * mma_sms())) & ~15ll);
    const long long warps = (ll.total + window - 1) / window;
    k_light<<<(unsigned)((warps + kLightWarps - 1) / kLightWarps), kLightWarps * 32, 0, st>>>(
        static_cast<const uint4*>(slab16), T, nb, window, ll.off, ll.ent, ll.val);
    return cudaGetLastError();
}

cudaError_t launch_solar_slab16(const DevGeom& g, int T, const uint32_t* shadow, int words32, const HourEntry* table,
                                int j0, int nb, void* slab16, cudaStream_t st)
{
    if (T <= 0 || nb <= 0) return cudaSuccess;
    const int run = T >= 1 << 17 ? 256 : T >= 1 << 15 ? 128 : 64;
    const size_t smem = (size_t)run * (sizeof(NormalPair) + sizeof(uint32_t) * words32);
    if (smem > 48 * 1024) {   // up to 41 words: 54 KB
        const cudaError_t e = cudaFuncSetAttribute(k_solar_slab16, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    const dim3 grid((T + run - 1) / run, (nb * (kHours / 128) + kSlabWarps - 1) / kSlabWarps);
    k_solar_slab16<<<grid, kSlabWarps * 32, smem, st>>>(g.geo_n, T, shadow, words32, table, j0, nb, run,
                                                        static_cast<uint2*>(slab16));
    return cudaGetLastError();
}

cudaError_t launch_reflect_mma(const void* slab16, int T, const MmaLists& ml, int nb, float* sums, int* err,
                               cudaStream_t st)
{
    const int NG = mma_group_count(ml.N);
    if (NG <= 0 || nb <= 0) return cudaSuccess;
    static std::atomic<bool> attr[kMaxDevices];
    cudaError_t e = allow_smem(k_reflect_mma, (size_t)kSmemBytes, attr);
    if (e != cudaSuccess) return e;
    if ((long long)NG * nb > 0x7FFFFFFFLL - 4096) return cudaErrorInvalidValue;
    const int items = NG * nb, grid = items < mma_sms() ? items : mma_sms();
    // with a multiple of the grid's size a CTA would meet the same groups in every hour block
    MmaTiles mt{ml.N, T, NG, items, NG % grid == 0 ? 1 : 0, ml.woff, ml.light.many ? kLightShift : 0, ml.cells, ml.unions, ml.cbase, ml.coff,
                reinterpret_cast<const uint2*>(ml.ent), ml.scale};
    k_reflect_mma<<<grid, kThreads, kSmemBytes, st>>>(static_cast<const __half*>(slab16), mt, sums, err);
    return cudaGetLastError();
}

cudaError_t launch_mma_accumulate(const int* order, int nb, const float* sums, const MmaLists& ml, const Accum& acc,
                                  bool first, bool last, float* out, cudaStream_t st)
{
    const int N = ml.N;
    if (N <= 0) return cudaSuccess;
    const unsigned grid = (unsigned)((N + 255) / 256);
    if (acc.mode == 0) k_mma_accumulate<0><<<grid, 256, 0, st>>>(order, N, nb, sums, ml.light, ml.woff, acc, first, last, out);
    else if (acc.mode == 1) k_mma_accumulate<1><<<grid, 256, 0, st>>>(order, N, nb, sums, ml.light, ml.woff, acc, first, last, out);
    else k_mma_accumulate<2><<<grid, 256, 0, st>>>(order, N, nb, sums, ml.light, ml.woff, acc, first, last, out);
    return cudaGetLastError();
}

}  // namespace sgb
