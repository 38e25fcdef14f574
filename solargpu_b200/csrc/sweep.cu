// Stage 1 tracer by azimuth sweeps.
//
// All 36 elevations of an azimuth leave a voxel along one line on the ground:
// the origin of a ray is gx + 2 cx, gy + 2 cy with (cx, cy) = cos(elevation)
// times the azimuth's vector, so its cells are those of the line from the
// corner (gx, gy), from the distance 2 cos(elevation) on.  Over the same cell a
// steeper ray is higher.  So instead of one walk per direction (trace.cu) one
// sweep along the line serves all 36: at each cell only the lowest ray still
// alive is tested; if the cell is above it, that ray is resolved (its hit) and
// the next one is tested on the same cell; if not, no higher ray hits it
// either.  The results are the per-direction walk's, bit for bit, because
// every test is the reference's own float expression for that ray, and
// because of two facts about its float arithmetic:
//
//   1. A ray's crossing times t_k and its cells relative to (gx, gy) do not
//      depend on the voxel.  gx is an integer, so inside one binade
//      [2^e, 2^(e+1)) of the rounded origin the rounding adds the same amount to
//      every gx (the spacing of floats there divides every integer, and ties
//      go by the same parity); the fraction of the origin, the first crossing
//      times and so the whole sequence are one per direction and pair of
//      classes on x and y.  A class is the binade of the origin from 4 on,
//      and below 4 the cell itself (0 to 5).  The crossing times are
//      tabulated per (azimuth, class pair) once per context.
//   2. The rays of an azimuth visit the same cells from the first cell of the
//      lowest upper ray on, whatever their classes.  Rounding can break this
//      where the line passes near a lattice point, so k_sweep_match counts, for
//      every azimuth, the cells over which all sequences (36 rays, all pairs of
//      classes) agree: 353 or more up to 4096^2, and the sweep ends there.  The
//      one or two cells before the common ones belong to the steep rays alone
//      (which of them is the same for all classes, k_sweep_match checks it).
//
// Order of heights: at a common cell two neighbouring rays differ by at least
// 2 tan 5 deg = 0.17 m (the cells lie 2 cells or more from the corner) and by
// a sixth of their rise, the float errors of both by less than 0.02 m for base
// heights below 65536 m; voxels beyond that, or not finite, are walked
// direction by direction.
//
// A warp sweeps one azimuth of 32 voxels in lockstep.  Groups of 8 cells are
// skipped: k_box_max takes, per call and quadrant, the
// maximum of the heights over the cells (i, j), i + j < 8, away from each cell
// along the quadrant's signs (+inf where they leave the grid), which holds the
// group's cells; a group is walked only if that is above the lowest height of
// the lowest ray in it for some lane.  Both sides are monotone, so no cell of a skipped group
// is hit.  Range tests: a ray's height is monotone along it, so testing it
// where the ray is next looked at, and where it stops, gives the reference's
// result.  The sweep ends when the lowest ray left is an upper one above the
// early-exit bound of its cell (cone.cu): all others are above it.
//
// A ray that is the lowest one at the end of its tabulated times is walked on
// by the general code (dda.cuh) from its state there.
//
// Bound: instructions.  On the 1024^2 city (1.47 M voxels) a warp's azimuth
// takes 21 groups, 65 tested cells and 57 changes of its lanes' lowest ray,
// about 9,000 instructions, where 36 walks took 18,000; L1 hits 75%, 75% of the
// issue slots are used.  Trace stage, tables and box maxima included, against
// one walk a direction (trace.cu): 79.2 -> 44.9 ms on the 1024^2 city, 18.4 ->
// 10.8 ms at 512^2, 0.42 -> 0.24 ms at 64^2.  Also tried: the heights of a tile
// in shared memory, walked direction by direction along the tabulated paths
// (111 ms), and skipping groups direction by direction (92 ms): both keep a
// walk per direction.  Lanes on their own groups instead of lockstep took 107
// ms, 32-bit hits in the stage (18 KB a block, less L1) 4 ms more.
#include "dda.cuh"

#include <algorithm>
#include <climits>
#include <vector>

namespace sgb {
namespace {

constexpr int kRanks = 36;             // rays of an azimuth, by elevation: -87.5 ... 87.5 degrees
constexpr int kUp = 18;                // first upper rank; its cells are the common ones
constexpr int kGroup = 8;              // cells of a group
constexpr int kSweep = 768;            // common cells of a block at most
constexpr int kCellClasses = 6;        // classes of origins below 4: the cells 0 to 5
constexpr int kBlockVox = 128;

__host__ __device__ constexpr int dir_of_rank(int r) { return r < kUp ? kRanks - 1 - r : r - kUp; }
__host__ __device__ constexpr int rank_of_dir(int j) { return j < kRanks - kUp ? j + kUp : kRanks - 1 - j; }

// Tabulated times of a rank: the flat rays run long, the steep ones are
// resolved or above a 30 m scene within 64 cells.
constexpr int rank_steps(int r)
{
    constexpr int lower[6] = {80, 96, 128, 128, 256, 0}, upper[7] = {kSweep, 320, 192, 192, 128, 104, 80};
    return r >= kUp + 7 || r < kUp - 5 ? 64 : r >= kUp ? upper[r - kUp] : lower[r - (kUp - 5)];
}
struct RankTable {
    int first[kRanks + 1] = {};   // first time of a rank in a block's times, and their end
    int steps[kRanks] = {};
    constexpr RankTable()
    {
        for (int r = 0; r < kRanks; ++r) {
            steps[r] = rank_steps(r);
            first[r + 1] = first[r] + 2 + steps[r] + kGroup;   // two near times, the times, the next group's
        }
    }
};
constexpr RankTable kRankTable;
__constant__ RankTable c_ranks = kRankTable;

// A table block (azimuth, class pair): per rank the next crossing times after
// its last time, then the ranks' times (kNear before the common cells' ones).
constexpr int kNear = 2;
constexpr int kAtTimes = 2 * kRanks;
constexpr int kBlockWords = kAtTimes + kRankTable.first[kRanks];
// An azimuth's words: common cells, start masks (lower and upper ranks that
// visit near cell -2, then -1), the ranks' cz, the cells from -2 on.
constexpr int kAtMasks = 1;
constexpr int kAtCz = 8;
constexpr int kAtCells = kAtCz + kRanks + kNear;   // cell 0
constexpr int kLineWords = kAtCells + kSweep + kGroup;

// Cell dx, dy away, packed so that dy = v >> 16.
__host__ __device__ __forceinline__ int pack_cell(int dx, int dy) { return dy * 65536 + (dx + 32768); }

__device__ __forceinline__ int origin_class(float o, int g)
{
    return o >= 4.0f ? (int)(__float_as_uint(o) >> 23) - (127 + 2) + kCellClasses : g;
}

// The path of direction e for a class pair, a step at a time.
struct Path {
    Ray r;
    int dx, dy;
    __device__ Path(const DirEntry& e, int pair, int ne)
    {
        // the cell itself, or one whose origin lies in the binade for every direction (|2 c| < 2)
        const int cx = pair % ne, cy = pair / ne;
        const int gx = cx < kCellClasses ? cx : (4 << (cx - kCellClasses)) + 2;
        const int gy = cy < kCellClasses ? cy : (4 << (cy - kCellClasses)) + 2;
        const float ox = __fadd_rn((float)gx, __fmul_rn(e.cx, 2.0f));
        const float oy = __fadd_rn((float)gy, __fmul_rn(e.cy, 2.0f));
        const int ix = __float2int_rd(ox), iy = __float2int_rd(oy);
        const bool px = e.cx >= 0.0f, py = e.cy >= 0.0f;
        r.tMaxX = __fdiv_rn(px ? __fsub_rn(__fadd_rn((float)ix, 1.0f), ox) : __fsub_rn(ox, (float)ix), e.ax);
        r.tMaxY = __fdiv_rn(py ? __fsub_rn(__fadd_rn((float)iy, 1.0f), oy) : __fsub_rn(oy, (float)iy), e.ay);
        r.cell = 0;
        dx = ix - gx;
        dy = iy - gy;
    }
    __device__ void step(const DirEntry& e)
    {
        const bool xs = r.tMaxX < r.tMaxY;
        dda_step(r, 0, 0, e.dX, e.dY);
        if (xs) dx += e.cx >= 0.0f ? 1 : -1; else dy += e.cy >= 0.0f ? 1 : -1;
    }
};

// Steps p to cell (dx0, dy0), storing the times on the cells before it from
// t on (nullptr: none) and the cells (cell, may be nullptr); the number of
// those cells, -1 when it is not within kNear.
__device__ int path_to_common(const DirEntry& e, Path& p, int dx0, int dy0, float* t, int* cell)
{
    for (int k = 0; k <= kNear; ++k) {
        p.step(e);
        if (p.dx == dx0 && p.dy == dy0) return k;
        if (t && k < kNear) t[k] = p.r.t;
        if (cell && k < kNear) cell[k] = pack_cell(p.dx, p.dy);
    }
    return -1;
}

// line[a][0] (kSweep before the launch): the cells over which every rank and
// class pair has the sequence of the first upper rank in the last class pair;
// 0 where a rank's cells before them depend on the class, or are not the last
// ones of the steepest ray's.
__global__ void k_sweep_match(const DirEntry* __restrict__ dirs, int ne, int* __restrict__ line)
{
    const int a = blockIdx.x, pair = blockIdx.y, rank = threadIdx.x, ref = ne * ne - 1;
    if (rank >= kRanks) return;
    const DirEntry e0 = dirs[a * kRanks + dir_of_rank(kUp)], e = dirs[a * kRanks + dir_of_rank(rank)];
    const DirEntry e1 = dirs[a * kRanks + dir_of_rank(kRanks - 1)];
    Path c(e0, ref, ne), p(e, pair, ne), q(e, ref, ne), steep(e1, ref, ne);
    c.step(e0);
    int near_p[kNear] = {}, near_s[kNear] = {};
    const int kp = path_to_common(e, p, c.dx, c.dy, nullptr, near_p), kq = path_to_common(e, q, c.dx, c.dy, nullptr, nullptr);
    const int ks = path_to_common(e1, steep, c.dx, c.dy, nullptr, near_s);
    bool ok = kp >= 0 && kp == kq && ks >= kp;
    for (int k = 0; ok && k < kp; ++k) ok = near_p[k] == near_s[ks - kp + k];
    int n = 0;
    while (ok && n < kSweep && c.dx == p.dx && c.dy == p.dy) {
        ++n;
        c.step(e0);
        p.step(e);
    }
    atomicMin(line + a * kLineWords, n & ~(kGroup - 1));
}

__global__ void k_sweep_tables(const DirEntry* __restrict__ dirs, int ne, int* __restrict__ line,
                               float* __restrict__ blocks)
{
    const int a = blockIdx.x, pair = blockIdx.y, rank = threadIdx.x, ref = ne * ne - 1;
    if (rank >= kRanks) return;
    float* blk = blocks + ((size_t)pair * gridDim.x + a) * kBlockWords;
    int* ln = line + a * kLineWords;
    const DirEntry e0 = dirs[a * kRanks + dir_of_rank(kUp)], e = dirs[a * kRanks + dir_of_rank(rank)];
    Path c(e0, ref, ne), p(e, pair, ne);
    c.step(e0);
    float near_t[kNear] = {};
    int near_c[kNear] = {};
    const int k0 = path_to_common(e, p, c.dx, c.dy, near_t, near_c);
    const int n = min(c_ranks.steps[rank], ln[0]);
    float* t = blk + kAtTimes + c_ranks.first[rank] + kNear;
    for (int k = 0; k < k0; ++k) t[k - k0] = near_t[k];
    if (pair == ref) {
        ln[kAtCz + rank] = __float_as_int(e.cz);
        for (int k = 0; k < k0; ++k) {   // mask of near cell -(k + 1)
            atomicOr(ln + kAtMasks + 2 * (kNear - 1 - k) + (rank < kUp ? 0 : 1), 1 << (rank < kUp ? rank : rank - kUp));
            if (rank == kRanks - 1) ln[kAtCells - 1 - k] = near_c[k0 - 1 - k];
        }
    }
    for (int k = 0; k < c_ranks.steps[rank] + kGroup; ++k) {
        t[k] = p.r.t;   // the time after the last group bounds that group's heights
        if (rank == kUp && pair == ref) ln[kAtCells + k] = pack_cell(p.dx, p.dy);
        if (k + 1 == n) {
            blk[2 * rank] = p.r.tMaxX;
            blk[2 * rank + 1] = p.r.tMaxY;
        }
        p.step(e);
    }
}

constexpr int kBoxX = 32, kBoxY = 16;   // cells of a block (512 threads)

// box[q][cell of the bordered grid], q = (x step > 0) + 2 (y step > 0).
__global__ void __launch_bounds__(kBoxX * kBoxY)
k_box_max(const float* __restrict__ gpad, int W, int H, float* __restrict__ box, size_t stride)
{
    constexpr int R = kGroup - 1;
    __shared__ float tile[kBoxY + R][kBoxX + R + 1];
    const int Wp = W + 2, Hp = H + 2;
    const int q = blockIdx.z, sx = (q & 1) ? 1 : -1, sy = (q & 2) ? 1 : -1;
    const int x0 = blockIdx.x * kBoxX, y0 = blockIdx.y * kBoxY;
    const int tx = threadIdx.x % kBoxX, ty = threadIdx.x / kBoxX;
    // the tile's first column and row, R cells before the block where the steps are negative
    const int bx = x0 - (sx < 0 ? R : 0), by = y0 - (sy < 0 ? R : 0);
    for (int i = threadIdx.x; i < (kBoxY + R) * (kBoxX + R); i += kBoxX * kBoxY) {
        const int x = bx + i % (kBoxX + R), y = by + i / (kBoxX + R);
        const float h = __ldg(gpad + (size_t)min(max(y, 0), Hp - 1) * Wp + min(max(x, 0), Wp - 1));
        tile[i / (kBoxX + R)][i % (kBoxX + R)] = (x >= 0 && x < Wp && y >= 0 && y < Hp) ? h : __int_as_float(0x7f800000);
    }
    __syncthreads();
    const int x = x0 + tx, y = y0 + ty;
    if (x >= Wp || y >= Hp) return;
    const int cx = x - bx, cy = y - by;
    float m = -__int_as_float(0x7f800000);
#pragma unroll
    for (int j = 0; j < kGroup; ++j)
#pragma unroll
        for (int i = 0; i + j < kGroup; ++i) m = fmaxf(m, tile[cy + sy * j][cx + sx * i]);
    box[stride * q + (size_t)y * Wp + x] = m;
}

// ---- the sweep -----------------------------------------------------------------

// A lane's sweep of one azimuth.
template <bool CONE>
struct Sweep {
    int W, H, ne;
    float maxz;
    const float* blocks;
    const int4* ranks;            // the warp's ranks (shared memory): time 0 in a block, tabulated times, cz
    unsigned short* hits;         // this lane's hits by rank, kBlockVox apart: number of the cell on the line + 1 + kNear
    int gx, gy, a, na;
    float base_z;
    const DirEntry* da;           // the azimuth's directions
    const int* line;
    const float* blk;             // table block of ray E
    const float* bound;           // early-exit table: one, all rays of an azimuth are in one cone
    bool mixed;                   // the rays' origins are of several classes
    int common;
    // rays alive: the lowest ones, of ranks `base` on, and the upper ones while those are lower;
    // rays left to the general walk
    unsigned low, up, far_lo, far_up;
    int base;
    int E, nt, row;               // the lowest ray alive, its tabulated times, its time 0 in the block
    float cz, oz;
    bool live;

    __device__ __forceinline__ const float* block_of(const DirEntry& d) const
    {
        const int kx = origin_class(__fadd_rn((float)gx, __fmul_rn(d.cx, 2.0f)), gx);
        const int ky = origin_class(__fadd_rn((float)gy, __fmul_rn(d.cy, 2.0f)), gy);
        return blocks + ((size_t)(ky * ne + kx) * na + a) * kBlockWords;
    }
    // cell of the bordered grid of a packed cell of the line
    __device__ __forceinline__ unsigned cell_of(int c) const
    {
        const int Wp = W + 2;
        const unsigned last = (unsigned)Wp * (unsigned)(H + 2) - 1u;
        return min((unsigned)((gx + 1) + (gy + 1) * Wp - 32768 + c + (c >> 16) * (Wp - 65536)), last);
    }
    __device__ __forceinline__ bool inside(int c) const
    {
        return (unsigned)(gx + (c & 0xFFFF) - 32768) < (unsigned)W && (unsigned)(gy + (c >> 16)) < (unsigned)H;
    }
    __device__ __forceinline__ int id_of(int c) const { return gx + (c & 0xFFFF) - 32768 + (gy + (c >> 16)) * W + 1; }
    __device__ __forceinline__ void load_rank(int r)
    {
        E = r;
        const int4 rk = ranks[r];
        row = rk.x;
        nt = rk.y;
        cz = __int_as_float(rk.z);
        oz = __fmaf_rn(cz, 2.0f, base_z);   // 2 cz is exact
        if (mixed) blk = block_of(da[r < kUp ? kRanks - 1 - r : r - kUp]);
    }
    __device__ __forceinline__ float height(int k) const { return __fmaf_rn(cz, __ldg(blk + row + k), oz); }
    __device__ __forceinline__ float limit(int c) const { return CONE ? __ldg(bound + cell_of(c)) : maxz; }
    __device__ __forceinline__ void store(int k) { hits[E * kBlockVox] = (unsigned short)(k + 1 + kNear); }
    // the lowest ray alive for cell k; rays past their times are left to the general walk, unless
    // they are out of range by their last tabulated height (not above the one here)
    __device__ __forceinline__ void settle(int k, int c)
    {
        for (;;) {
            if (low == 0u) {
                low = up;
                up = 0u;
                base = kUp;
            }
            live = low != 0u;
            if (!live) return;
            load_rank(base + __ffs(low) - 1);
            if (k < nt) return;
            const float z = height(nt);
            if (base != 0 && z > limit(c)) {
                low = 0u;
            } else {
                if (base != 0) far_up |= low & (0u - low);
                else if (!(z < 0.0f)) far_lo |= low & (0u - low);
                low &= low - 1u;
            }
        }
    }
    // resolves the rays that end on cell k of the line (packed c, height h): the lowest one alive as
    // long as the cell is above it
    __device__ __forceinline__ void resolve(int k, int c, float h)
    {
        float z = height(k);
        if (!(__fsub_rn(h, z) > 0.01f)) return;
        if (h == __int_as_float(0x7f800000) && !inside(c)) {   // off the grid: so are the others
            low = up = 0u;
            live = false;
            return;
        }
        do {
            const bool out = base != 0 ? z > maxz : z < 0.0f;
            if (!out) store(k);
            low = out && base != 0 ? 0u : low & (low - 1u);   // above the scene: so are the others
            settle(k, c);
            if (!live) return;
            z = height(k);
        } while (__fsub_rn(h, z) > 0.01f);
    }
};

// 11 blocks a SM, 40 registers: 44.9 ms; 9 or 10 (56, 48 registers, fewer spills): 48.3, 48.6
template <bool CONE>
__global__ void __launch_bounds__(kBlockVox, 11)
k_trace_sweep(DevScene s, const DirEntry* __restrict__ dirs, int D, int words32, int voxel_offset, int chunk_count,
              int* __restrict__ raw, uint32_t* __restrict__ shadow, const int* __restrict__ perm, SweepTables tabs,
              int* __restrict__ err)
{
    constexpr unsigned kAll = 0xFFFFFFFFu, kHalf = (1u << kUp) - 1u;
    __shared__ __align__(4) unsigned short stage[kRanks][kBlockVox];
    __shared__ int4 s_rank[kBlockVox / 32][kRanks];
    const int tid = threadIdx.x, lane = tid & 31;
    const int lv = blockIdx.x * kBlockVox + tid;
    const bool active = lv < chunk_count;
    const int v = voxel_offset + (perm ? __ldg(perm + (active ? lv : 0)) : (active ? lv : 0));
    const int top = __ldg(s.pix_parent + v);
    Sweep<CONE> w;
    w.W = s.W;
    w.H = s.H;
    w.ne = tabs.ne;
    w.maxz = s.maxz;
    w.blocks = tabs.blocks;
    int4* ranks = s_rank[tid >> 5];
    w.ranks = ranks;
    w.hits = &stage[0][tid];
    w.gy = top / s.W;
    w.gx = top - w.gy * s.W;
    w.base_z = (v < s.T) ? __ldg(s.grid + top) : __ldg(s.wall_z + (v - s.T));
    const int na = D / kRanks;
    w.na = na;
    const int a0 = (int)((long long)na * blockIdx.y / gridDim.y), a1 = (int)((long long)na * (blockIdx.y + 1) / gridDim.y);
    uint32_t acc = 0;
    int cur_word = -1;

    for (int a = a0; a < a1; ++a) {
        const DirEntry* da = dirs + a * kRanks;
        const int* line = tabs.line + a * kLineWords;
        w.a = a;
        w.da = da;
        w.line = line;
        w.common = __ldg(line);
        // the warp's columns of the stage, two hits a word
#pragma unroll
        for (int q = 0; q < kRanks / 2; ++q)
            reinterpret_cast<uint32_t*>(&stage[2 * q + (lane >> 4)][tid & ~31])[lane & 15] = 0u;
        for (int r = lane; r < kRanks; r += 32)
            ranks[r] = make_int4(kAtTimes + c_ranks.first[r] + kNear, min(c_ranks.steps[r], w.common),
                                 __ldg(line + kAtCz + r), 0);
        __syncwarp(kAll);
        const float* box = tabs.box + tabs.box_stride * ((da[0].cx >= 0.0f ? 1 : 0) + (da[0].cy >= 0.0f ? 2 : 0));
        w.bound = CONE ? s.cone + s.cone_stride * ((da[0].meta >> 17) & (kMaxConeTables - 1)) : nullptr;
        // the origins move monotonically with the elevation's cosine, so the flattest and the
        // steepest ray's classes tell whether all rays of the azimuth are of one
        w.blk = w.block_of(da[0]);
        w.mixed = w.blk != w.block_of(da[kUp - 1]);
        const bool swept = active && fabsf(w.base_z) < 65536.0f && w.common >= kGroup;   // false for NaN
        w.low = w.up = swept ? kHalf : 0u;
        w.base = 0;
        w.far_lo = w.far_up = active && !swept ? kHalf : 0u;

        // ---- the cells before the common ones, for the ranks that visit them
        for (int g = 0; g < kNear; ++g) {
            const unsigned mlo = __ldg(line + kAtMasks + 2 * g), mup = __ldg(line + kAtMasks + 2 * g + 1);
            if ((mlo | mup) == 0u) continue;
            const int c = __ldg(line + kAtCells - kNear + g);
            if (!w.inside(c)) {
                w.low &= ~mlo;
                w.up &= ~mup;
            }
            const float h = __ldg(s.gpad + w.cell_of(c));
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                for (;;) {
                    unsigned& alive = half ? w.up : w.low;
                    const unsigned m = alive & (half ? mup : mlo);
                    if (m == 0u) break;
                    w.load_rank((half ? kUp : 0) + __ffs(m) - 1);
                    const float z = w.height(g - kNear);
                    const bool out = half ? z > s.maxz : z < 0.0f;
                    if (!out && !(__fsub_rn(h, z) > 0.01f)) break;
                    if (!out) w.store(g - kNear);
                    alive &= out && half ? ~m : ~(m & (0u - m));   // above the scene: so are those above it
                }
            }
            __syncwarp(kAll);
        }

        // ---- the common cells, in groups
        {
            const int c = __ldg(line + kAtCells);
            if (!w.inside(c)) w.low = w.up = 0u;   // the rays leave the grid
            w.settle(0, c);
        }
        for (int i = 0; __any_sync(kAll, w.live); i += kGroup) {
            bool walk = false;
            const int c = __ldg(line + kAtCells + i);
            const unsigned cell = w.cell_of(c);
            if (w.live && i >= w.nt) w.settle(i, c);
            while (w.live) {
                const float z = w.height(i);
                float lowest = z;
                if (w.base != 0) {
                    if (z > w.limit(c)) {
                        w.live = false;   // so are the rays above it
                        break;
                    }
                } else {
                    if (z < 0.0f) {
                        w.low &= w.low - 1u;
                        w.settle(i, c);
                        continue;
                    }
                    lowest = w.height(i + kGroup);
                }
                walk = __fsub_rn(__ldg(box + cell), lowest) > 0.01f;
                break;
            }
            if (!__any_sync(kAll, walk)) continue;
            int cn = c;
            float hn = __ldg(s.gpad + cell);
#pragma unroll 1
            for (int k = i; k < i + kGroup; ++k) {
                const int ck = cn;
                const float h = hn;
                cn = __ldg(line + kAtCells + k + 1);   // the next cell's loads fly during this one's tests
                hn = __ldg(s.gpad + w.cell_of(cn));
                if (walk && w.live) w.resolve(k, ck, h);
                __syncwarp(kAll);
            }
        }

        // ---- the azimuth's hits: 144 bytes of the row, and the shadow bits
        if (active) {
            int4* dst = reinterpret_cast<int4*>(raw + (size_t)lv * D + a * kRanks);
            auto id_at = [&](int j) {
                const int h = stage[rank_of_dir(j)][tid];
                return h ? w.id_of(__ldg(line + kAtCells - 1 - kNear + h)) : 0;
            };
#pragma unroll
            for (int q = 0; q < kRanks / 4; ++q)
                dst[q] = make_int4(id_at(4 * q), id_at(4 * q + 1), id_at(4 * q + 2), id_at(4 * q + 3));
            for (int j = 0; j < kRanks - kUp; ++j) {
                const int dense = (da[j].meta & 0xFFFF) - 1;   // warp-uniform
                if (dense < 0) continue;
                if ((dense >> 5) != cur_word) {
                    // a word may be shared with the neighbouring part of the azimuths
                    if (acc) atomicOr(shadow + (size_t)v * words32 + cur_word, acc);
                    acc = 0;
                    cur_word = dense >> 5;
                }
                if (stage[kUp + j][tid]) acc |= 1u << (dense & 31);
            }
        }

        // ---- the rays past their times, and all rays of the voxels that are not swept
        while (__any_sync(kAll, (w.far_lo | w.far_up) != 0u)) {
            if ((w.far_lo | w.far_up) != 0u) {
                const int r = w.far_lo ? __ffs(w.far_lo) - 1 : kUp + __ffs(w.far_up) - 1;
                if (w.far_lo) w.far_lo &= w.far_lo - 1u; else w.far_up &= w.far_up - 1u;
                const int j = r < kUp ? kRanks - 1 - r : r - kUp;
                const DirEntry d = da[j];
                Ray ray;
                bool go = true;
                if (swept) {
                    const float* b = w.mixed ? w.block_of(d) : w.blk;
                    const int n = ranks[r].y;
                    ray.tMaxX = __ldg(b + 2 * r);
                    ray.tMaxY = __ldg(b + 2 * r + 1);
                    ray.oz = __fmaf_rn(d.cz, 2.0f, w.base_z);
                    ray.cell = (int)w.cell_of(__ldg(line + kAtCells + n - 1));
                    dda_step(ray, d.cx >= 0.0f ? 1 : -1, d.cy >= 0.0f ? s.W + 2 : -(s.W + 2), d.dX, d.dY);
                } else {
                    go = ray_start(s.W, s.H, w.gx, w.gy, w.base_z, d, ray);
                }
                int hit = 0;
                if (go) {
                    if (r < kUp) hit = ray_walk<false, false>(s.gpad, nullptr, s.W, s.H, s.maxz, ray, d);
                    else hit = ray_walk<true, CONE>(s.gpad, w.bound, s.W, s.H, s.maxz, ray, d);
                }
                if (hit < 0) {
                    atomicOr(err, kErrTraceBounds);
                    hit = 0;
                }
                if (hit) {   // over the 0 of the row piece above
                    raw[(size_t)lv * D + a * kRanks + j] = hit;
                    const int dense = (d.meta & 0xFFFF) - 1;
                    if (dense >= 0) atomicOr(shadow + (size_t)v * words32 + (dense >> 5), 1u << (dense & 31));
                }
            }
            __syncwarp(kAll);
        }
        __syncwarp(kAll);
    }
    if (active && acc) atomicOr(shadow + (size_t)v * words32 + cur_word, acc);
}

}  // namespace

int sweep_classes(int W, int H)
{
    const int m = W > H ? W : H;
    if (m > 32767) return 0;   // cells are packed in 16 bits an axis; the tables grow with the square of the classes
    int e = 2;
    while ((2 << e) <= m + 1) ++e;   // up to the binade of the last cell's origin, below m + 1
    return kCellClasses + e - 2 + 1;
}

size_t sweep_block_bytes(int D, int ne) { return sizeof(float) * kBlockWords * (size_t)(D / kRanks) * ne * ne; }
size_t sweep_line_bytes(int D) { return sizeof(int) * kLineWords * (size_t)(D / kRanks); }

cudaError_t launch_sweep_tables(const DirEntry* dirs, int D, const SweepTables& t, cudaStream_t st)
{
    const int na = D / kRanks;
    int* line = const_cast<int*>(t.line);
    std::vector<int> init((size_t)na * kLineWords, 0);
    for (int a = 0; a < na; ++a) init[(size_t)a * kLineWords] = kSweep;
    cudaError_t e = cudaMemcpyAsync(line, init.data(), sizeof(int) * init.size(), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    const dim3 grid(na, t.ne * t.ne);
    k_sweep_match<<<grid, 64, 0, st>>>(dirs, t.ne, line);
    k_sweep_tables<<<grid, 64, 0, st>>>(dirs, t.ne, line, const_cast<float*>(t.blocks));
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return cudaStreamSynchronize(st);   // `init` is read, and later calls may run on other streams
}

cudaError_t launch_box_max(const float* gpad, int W, int H, float* box, size_t stride, cudaStream_t st)
{
    if (W <= 0 || H <= 0) return cudaSuccess;
    const dim3 grid((W + 2 + kBoxX - 1) / kBoxX, (H + 2 + kBoxY - 1) / kBoxY, 4);
    k_box_max<<<grid, kBoxX * kBoxY, 0, st>>>(gpad, W, H, box, stride);
    return cudaGetLastError();
}

cudaError_t launch_trace_sweep(const DevScene& s, const DirEntry* dirs, int D, int words32, int voxel_offset,
                               int chunk_count, int* raw, uint32_t* shadow, const int* perm, const SweepTables& tabs,
                               int* err, cudaStream_t st)
{
    if (chunk_count <= 0) return cudaSuccess;
    if (!s.gpad || D % kRanks != 0) return cudaErrorInvalidValue;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int na = D / kRanks, runs = (chunk_count + kBlockVox - 1) / kBlockVox;
    // about 32 blocks for each of the 8 that a SM holds, so that the last wave is short
    const int parts = std::max(1, std::min(na, (32 * 8 * sms + runs - 1) / runs));
    const dim3 grid(runs, parts);
    if (s.cone)
        k_trace_sweep<true><<<grid, kBlockVox, 0, st>>>(s, dirs, D, words32, voxel_offset, chunk_count, raw, shadow,
                                                        perm, tabs, err);
    else
        k_trace_sweep<false><<<grid, kBlockVox, 0, st>>>(s, dirs, D, words32, voxel_offset, chunk_count, raw, shadow,
                                                         perm, tabs, err);
    return cudaGetLastError();
}

}  // namespace sgb
