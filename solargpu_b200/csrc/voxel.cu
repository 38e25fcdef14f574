// Voxelization on the GPU: the column-drop wall voxels and the top slope /
// aspect of a heightmap, packed as the reference CLI packs them for the
// irradiance entry points (src/main.cpp:112-127).
//
// The reference computes these on the host (src/voxelization.cpp:10-97,
// detect_wall_voxels and compute_top_slope_aspect), one cell after the other.
// Here a count pass sums the wall voxels of every run of 1024 cells, a scan turns
// the sums into offsets, and a write pass (one block a run, which counts and
// scans its cells again) fills the voxel arrays:
//   voxels [0, T)        top voxel i = cell i (pixel_parent i), its slope
//                        and aspect from central differences;
//   voxels [T, T + walls) walls in raster order of their cell, from the top of
//                        the drop downwards (the order the reference appends
//                        them), at z0 - (v + 0.5) voxel_size, slope pi / 2,
//                        aspect from the openness of the four sides.
// Float operations are written out (no contraction) in the reference's order,
// so wall counts and heights are identical; angles come from CUDA's atan2f
// and may differ from the host library's in the last bits.
//
// Bound: the launches' latency and the bytes written (a block's walls are one stretch
// of the arrays, a thread a wall, its cell found in the block's scan).  With a thread
// a cell writing its walls one by one, and counts and 64-bit offsets of every cell
// in memory, 2000^2 (4 M cells, 1.6 M walls) took 212 us a call; now 111.
#include "sgb_internal.cuh"

namespace sgb {
namespace {

constexpr float kOpenOutside = -1e30f;   // voxelization.cpp:16
constexpr int kVoxRun = 1024;   // cells of a run
constexpr float kPiF = 3.14159265358979323846f;

__device__ __forceinline__ float height_at(const float* g, int W, int H, int x, int y)
{
    // clamped load: in bounds however the select is compiled
    const float h = g[(size_t)min(max(y, 0), H - 1) * W + min(max(x, 0), W - 1)];
    return (x >= 0 && x < W && y >= 0 && y < H) ? h : kOpenOutside;
}

// A cell's height and its sides' (kOpenOutside off the grid).
struct Cell {
    float z0, hE, hW, hN, hS;
    bool inner;   // all sides are on the grid
    __device__ Cell(const float* g, int W, int H, int i)
    {
        const int gy = i / W, gx = i - gy * W;
        inner = gx > 0 && gx < W - 1 && gy > 0 && gy < H - 1;
        z0 = g[i];
        if (inner) {
            hE = g[i + 1];
            hW = g[i - 1];
            hN = g[i - W];
            hS = g[(long long)i + W];
        } else {
            hE = height_at(g, W, H, gx + 1, gy);
            hW = height_at(g, W, H, gx - 1, gy);
            hN = height_at(g, W, H, gx, gy - 1);
            hS = height_at(g, W, H, gx, gy + 1);
        }
    }
};

// Its wall voxels.
__device__ __forceinline__ int wall_count(const Cell& c, float vs)
{
    const float z0 = c.z0, hE = c.hE, hW = c.hW, hN = c.hN, hS = c.hS;
    const float half = kOpenOutside * 0.5f;
    const float cE = (hE <= half) ? z0 : hE;
    const float cW = (hW <= half) ? z0 : hW;
    const float cN = (hN <= half) ? z0 : hN;
    const float cS = (hS <= half) ? z0 : hS;
    const float mn = fminf(fminf(cE, cW), fminf(cN, cS));
    const float drop = __fsub_rn(z0, mn);
    if (!(drop > vs)) return 0;
    return (int)__fdiv_rn(drop, vs);
}

constexpr int kVoxThreads = 256;
constexpr int kVoxPer = kVoxRun / kVoxThreads;   // cells of a thread

// sums[b] = wall voxels of the cells of run b.
__global__ void __launch_bounds__(kVoxThreads)
k_vox_count(const float* __restrict__ g, int W, int H, float vs, long long* __restrict__ sums)
{
    __shared__ long long part[kVoxThreads / 32];
    const int T = W * H, i0 = blockIdx.x * kVoxRun;
    long long n = 0;
#pragma unroll
    for (int j = 0; j < kVoxPer; ++j) {
        const long long i = (long long)i0 + j * kVoxThreads + threadIdx.x;
        if (i < T) n += wall_count(Cell(g, W, H, (int)i), vs);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xFFFFFFFFu, n, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = n;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kVoxThreads / 32; ++k) n += part[k];
        sums[blockIdx.x] = n;
    }
}

// off: the scan of the runs' sums.  All voxels fit an int, so a run's walls do.
__global__ void __launch_bounds__(kVoxThreads)
k_vox_write(const float* __restrict__ g, int W, int H, float vs, float scale, const long long* __restrict__ off,
            int* __restrict__ parent, float* __restrict__ wall_z, float* __restrict__ slopes,
            float* __restrict__ aspects)
{
    __shared__ int first[kVoxRun + 1];   // first wall of each cell of the run, then its walls
    __shared__ int part[kVoxThreads / 32];
    const int T = W * H, i0 = blockIdx.x * kVoxRun;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int j = 0; j < kVoxPer; ++j) {
        const int q = j * kVoxThreads + tid;
        int n = 0;
        if ((long long)i0 + q < T) {
            const int i = i0 + q;
            const Cell c(g, W, H, i);
            // top voxel: central differences, clamped at the border (voxelization.cpp:66-97)
            float zl = c.hW, zr = c.hE, zu = c.hN, zd = c.hS, nx = 2.0f, ny = 2.0f;
            if (!c.inner) {
                const int gy = i / W, gx = i - gy * W;
                if (gx == 0) { zl = c.z0; nx -= 1.0f; }
                if (gx == W - 1) { zr = c.z0; nx -= 1.0f; }
                if (gy == 0) { zu = c.z0; ny -= 1.0f; }
                if (gy == H - 1) { zd = c.z0; ny -= 1.0f; }
            }
            const float dx = __fdiv_rn(__fsub_rn(zr, zl), __fmul_rn(nx, scale));
            const float dy = __fdiv_rn(__fsub_rn(zd, zu), __fmul_rn(ny, scale));
            const float mag = __fsqrt_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)));
            parent[i] = i;
            slopes[i] = atan2f(mag, 1.0f);
            float a = atan2f(-dx, dy);
            if (a < 0.0f) a = __fadd_rn(a, 2.0f * kPiF);
            aspects[i] = a;
            n = wall_count(c, vs);
        }
        first[q] = n;
    }
    __syncthreads();
    int c[kVoxPer], sum = 0;   // this thread's cells are side by side from here on
#pragma unroll
    for (int j = 0; j < kVoxPer; ++j) {
        c[j] = sum;
        sum += first[tid * kVoxPer + j];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) part[warp] = incl;
    __syncthreads();
    int before = incl - sum;
    for (int k = 0; k < warp; ++k) before += part[k];
#pragma unroll
    for (int j = 0; j < kVoxPer; ++j) first[tid * kVoxPer + j] = before + c[j];
    if (tid == kVoxThreads - 1) first[kVoxRun] = before + sum;
    __syncthreads();
    const int walls = first[kVoxRun];
    const long long w0 = off[blockIdx.x], base = (long long)T + w0;
    for (int k = tid; k < walls; k += kVoxThreads) {
        int lo = 0, hi = kVoxRun - 1;   // the last cell that starts at or before wall k: the one it belongs to
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (first[mid] <= k) lo = mid; else hi = mid - 1;
        }
        const int i = i0 + lo, v = k - first[lo];
        const Cell c(g, W, H, i);
        const float zz = __fsub_rn(c.z0, __fmul_rn(__fadd_rn((float)v, 0.5f), vs));
        const float oE = fmaxf(0.0f, __fsub_rn(zz, c.hE));
        const float oW = fmaxf(0.0f, __fsub_rn(zz, c.hW));
        const float oN = fmaxf(0.0f, __fsub_rn(zz, c.hN));
        const float oS = fmaxf(0.0f, __fsub_rn(zz, c.hS));
        float a = atan2f(__fsub_rn(oE, oW), __fsub_rn(oN, oS));
        if (a < 0.0f) a = __fadd_rn(a, 2.0f * kPiF);
        parent[base + k] = i;
        wall_z[w0 + k] = zz;
        slopes[base + k] = kPiF * 0.5f;
        aspects[base + k] = a;
    }
}

}  // namespace

int vox_runs(int T) { return (int)(((long long)T + kVoxRun - 1) / kVoxRun); }

cudaError_t launch_vox_count(const float* grid, int W, int H, float voxel_size, long long* sums, cudaStream_t st)
{
    const int T = W * H;
    if (T <= 0) return cudaSuccess;
    k_vox_count<<<vox_runs(T), kVoxThreads, 0, st>>>(grid, W, H, voxel_size, sums);
    const cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? e : launch_scan_sums(sums, vox_runs(T), st);
}

cudaError_t launch_vox_write(const float* grid, int W, int H, float voxel_size, float scale, const long long* off,
                             int* parent, float* wall_z, float* slopes, float* aspects, cudaStream_t st)
{
    const int T = W * H;
    if (T <= 0) return cudaSuccess;
    k_vox_write<<<vox_runs(T), kVoxThreads, 0, st>>>(grid, W, H, voxel_size, scale, off, parent, wall_z, slopes, aspects);
    return cudaGetLastError();
}

}  // namespace sgb
