// Early-exit bounds for upward rays of the tracer.
//
// The reference ends an upward ray when its height passes the scene maximum
// (viewshed_kernels.cu:42).  A ray that is already above every cell it can
// still reach cannot hit anything either, so it may end there with the same
// result.  For each group of directions this file builds one table over the
// bordered grid,
//
//     bound[cell] = min(maxz, max of the heights of every block of 2 x 2 cells a ray
//                   of the group can visit from a cell of `cell`'s block on),
//
// and the tracer ends an upward ray with no hit when its height exceeds the
// bound of a cell it has reached (it loads the bound of the cell a group of
// steps starts on and compares it with the height at the group's end, every
// cell after that being reachable from the first).  The result is the
// reference's, bit for bit:
//   * upward rays only rise (t never decreases, cz > 0, and the fused
//     multiply-add is monotone in t), so every later height test compares a
//     cell height <= bound with a ray height > bound and fails;
//   * bound <= maxz, so a ray the reference ends on the range test ends here
//     too, and the tracer checks the range test first after the loop.
//
// Which cells a ray can still visit.  Work in the quadrant's unsigned
// coordinates (X grows along the ray's x step, Y along its y step).  The DDA
// adds dX and dY (floats) to its crossing times; without rounding its cells
// are exactly the cells a straight line of direction (1/dX, 1/dY) passes
// through.  After i additions a crossing time is off by at most i * 2^-24 of
// itself, i.e. the crossing moves by at most eps = L(L + 1) 2^-24 cells for
// L crossings, so every visited cell lies within eps of that line at the same
// time.  The cells from the current cell c on therefore lie in
// c + (-1 - 2 eps, 1 + 2 eps]^2 + K, where K is any closed cone containing
// (1/dX, 1/dY).  Divided by 2, with c at any place f in [0, 1)^2 of its block and
// a cell anywhere in its own, the blocks from c's block B on lie in
// B + (-1 - q, 1 + q)^2 + K, q = (1 + 2 eps) / 2: the same cone (it has no scale) and
// a box that replaces 1 + 2 eps by 1 + q.
//
// K is taken between two consecutive primitive vectors a, b of the Farey set of order 4 (all primitive (p, q) with p, q <= 4, sorted by
// angle), so det(a, b) = 1 and the lattice points of K are exactly the
// non-negative combinations of a and b.  Then
//   M(c)     = max(h(c), M(c + a), M(c + b))      (max over c + K)
// is two suffix maxima along lattice lines (first along a, then along b), and
// any lattice point of p + K with p in the box above is in e + K for the
// lattice point e = p - frac_ab(p), frac_ab(p) in {s a + t b : s, t in [0,1)};
// so the bound is the maximum of M over the window
//   e_X in [-(r + a_X + b_X), r],  e_Y in [-(r + a_Y + b_Y), r],
//   r = 1 + ceil(q),
// taken as two one-dimensional passes.  All of it runs over the blocks with a
// margin of r + 8 on every side (heights -inf), so that every apex of a block's
// window has its M.  A ray off the grid hits nothing more, so the bound there may
// be anything; the tables have +inf on the border.  Non-finite heights: NaN never
// hits and fmaxf skips it; +inf enters the maximum as itself.
//
// Bound: latency of the lines (a thread follows one line of blocks), launches, and
// the bytes of the tables per cell (0.3 GB at 1024^2, which the tracer reads with the
// index it has anyway; reading them by block cost it 4 ms there).  Built per cell,
// with cones of order 8, they took 2.9 ms of a 1024^2 run and 64 us of a 64^2 one.
// Trace stage then, with blocks of 4 x 4 and order 8, 4 x 4 and order 4, 2 x 2 and order 4: 1024^2
// 44.6, 44.5, 44.2, 43.9 ms; 512^2 10.75, 10.60, 10.52, 10.44; 160^2 0.99, 0.91, 0.90, 0.90; 64^2
// 0.248, 0.229, 0.215, 0.220.
#include "sgb_internal.cuh"

#include <climits>
#include <cmath>

namespace sgb {
namespace {

// W and H below are those of the blocks with their margins.
__device__ __forceinline__ size_t block_index(int x, int y, int W) { return (size_t)y * W + x; }

__device__ __forceinline__ void to_grid(const ConeSpec& c, int X, int Y, int W, int H, int& x, int& y)
{
    x = c.sx > 0 ? X : W - 1 - X;
    y = c.sy > 0 ? Y : H - 1 - Y;
}

// Heights of the blocks, -inf in the margins.
__global__ void k_cone_blocks(const float* __restrict__ grid, int gw, int gh, int margin, int W, int H,
                              float* __restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * H) return;
    const int y = i / W, x = i - y * W;
    const int cx = (x - margin) << kConeShift, cy = (y - margin) << kConeShift;
    float m = -__int_as_float(0x7f800000);
    for (int v = max(cy, 0); v < min(cy + (1 << kConeShift), gh); ++v)
        for (int u = max(cx, 0); u < min(cx + (1 << kConeShift), gw); ++u) m = fmaxf(m, __ldg(grid + (size_t)v * gw + u));
    out[i] = m;
}

// Suffix maxima along the lattice lines of one cone vector (u, v) (unsigned
// coordinates): dst(c) = max(src(c), dst(c + (u, v))).  One thread a line,
// started at the line's last cell inside the grid (c + (u, v) outside).
// PASS 0: src = the blocks' heights;  PASS 1: src = a table.
template <int PASS>
__global__ void k_cone_lines(const float* __restrict__ src, int W, int H, const ConeSpec* __restrict__ specs,
                             float* __restrict__ dst, size_t stride)
{
    const ConeSpec c = specs[blockIdx.y];
    const int u = PASS == 0 ? c.ax : c.bx, v = PASS == 0 ? c.ay : c.by;
    const int uu = min(u, W), vv = min(v, H);
    const long long n1 = (long long)uu * H, n2 = (long long)(W - uu) * vv;
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n1 + n2) return;
    int X, Y;
    if (k < n1) { X = W - uu + (int)(k % uu); Y = (int)(k / uu); }
    else        { const long long k2 = k - n1; X = (int)(k2 % (W - uu)); Y = H - vv + (int)(k2 / (W - uu)); }
    const float* in = PASS == 0 ? src : src + stride * blockIdx.y;
    float* out = dst + stride * blockIdx.y;
    // a known trip count lets the loads of an unrolled stretch issue together
    const int n = min(u > 0 ? X / u : INT_MAX, v > 0 ? Y / v : INT_MAX) + 1;
    float m = -__int_as_float(0x7f800000);
#pragma unroll 8
    for (int i = 0; i < n; ++i, X -= u, Y -= v) {
        int x, y;
        to_grid(c, X, Y, W, H, x, y);
        const size_t p = block_index(x, y, W);
        m = fmaxf(m, in[p]);
        out[p] = m;
    }
}

// Window maxima of M: PASS 0 over X offsets, PASS 1 over Y offsets (then
// min with maxz); both read src and write dst (tables).  A block
// stages the stretch of its rows (PASS 0: 256 cells of one row; PASS 1: 64
// rows of 32 columns) plus the window's reach in shared memory, cells past
// the grid as -inf (a window clipped at the grid's edge), and each cell
// takes the maximum of its window from there.
constexpr int kWinRow = 256;          // PASS 0: cells of a row per block
constexpr int kWinCols = 32, kWinRows = 64, kWinRowsPerThread = 8;   // PASS 1 (256 threads)

template <int PASS>
__global__ void __launch_bounds__(256)
k_cone_window(int W, int H, float maxz, int r, const ConeSpec* __restrict__ specs,
              const float* __restrict__ src, float* __restrict__ dst, size_t stride)
{
    extern __shared__ float span[];
    const ConeSpec c = specs[blockIdx.y];
    const float* in = src + stride * blockIdx.y;
    float* out = dst + stride * blockIdx.y;
    // window in unsigned offsets [-(r + a + b), r], mirrored into grid offsets
    const int back = r + (PASS == 0 ? c.ax + c.bx : c.ay + c.by);
    const int s = PASS == 0 ? c.sx : c.sy;
    const int lo = s > 0 ? -back : -r, hi = s > 0 ? r : back;
    const int width = hi - lo + 1;
    const float ninf = -__int_as_float(0x7f800000);
    if (PASS == 0) {
        const int segs = (W + kWinRow - 1) / kWinRow;
        const int y = (int)(blockIdx.x / segs), x0 = (int)(blockIdx.x % segs) * kWinRow;
        const int n = kWinRow + width - 1;
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            const int q = x0 + lo + j;
            span[j] = (q >= 0 && q < W) ? in[block_index(q, y, W)] : ninf;
        }
        __syncthreads();
        const int x = x0 + (int)threadIdx.x;
        if (x >= W) return;
        float m = ninf;
        for (int j = 0; j < width; ++j) m = fmaxf(m, span[threadIdx.x + j]);
        out[block_index(x, y, W)] = m;
    } else {
        const int cols = (W + kWinCols - 1) / kWinCols;
        const int x0 = (int)(blockIdx.x % cols) * kWinCols, y0 = (int)(blockIdx.x / cols) * kWinRows;
        const int tx = threadIdx.x % kWinCols, ty = threadIdx.x / kWinCols;
        const int x = x0 + tx;
        const int rows = kWinRows + width - 1;
        for (int j = ty; j < rows; j += blockDim.x / kWinCols) {
            const int q = y0 + lo + j;
            span[j * kWinCols + tx] = (x < W && q >= 0 && q < H) ? in[block_index(x, q, W)] : ninf;
        }
        __syncthreads();
        if (x >= W) return;
        for (int k = 0; k < kWinRowsPerThread; ++k) {
            const int yl = ty * kWinRowsPerThread + k, y = y0 + yl;
            if (y >= H) break;
            float m = ninf;
            for (int j = 0; j < width; ++j) m = fmaxf(m, span[(yl + j) * kWinCols + tx]);
            out[block_index(x, y, W)] = fminf(maxz, m);
        }
    }
}

// The blocks' bounds to the cells of the bordered tables, kExpand tables a block.
constexpr int kExpand = 8;

__global__ void __launch_bounds__(256)
k_cone_cells(const float* __restrict__ src, size_t blocks, int W, int margin, int gw, int gh, int n_specs,
             float* __restrict__ tabs, size_t stride)
{
    const int Wp = gw + 2;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)Wp * (gh + 2)) return;
    const int y = (int)(i / Wp), x = (int)(i - (long long)y * Wp);
    const bool in = x > 0 && x <= gw && y > 0 && y <= gh;
    // a border cell's block may be the margin's first one
    const size_t from = block_index(((x - 1) >> kConeShift) + margin, ((y - 1) >> kConeShift) + margin, W);
    const int t0 = blockIdx.y * kExpand, n = min(kExpand, n_specs - t0);
    float v[kExpand];
#pragma unroll
    for (int t = 0; t < kExpand; ++t) v[t] = t < n ? __ldg(src + blocks * (t0 + t) + from) : 0.0f;
#pragma unroll
    for (int t = 0; t < kExpand; ++t)
        if (t < n) tabs[stride * (t0 + t) + i] = in ? v[t] : __int_as_float(0x7f800000);
}

}  // namespace

static int cone_window_radius(int W, int H)
{
    const double L = (double)(W > H ? W : H) + 4.0;
    const double eps2 = 2.0 * L * (L + 1.0) / 16777216.0;
    return 1 + (int)std::ceil((1.0 + eps2) / (1 << kConeShift));
}

static int cone_margin(int W, int H) { return cone_window_radius(W, H) + 2 * kConeOrder; }
static int cone_blocks(int cells, int margin) { return ((cells + (1 << kConeShift) - 1) >> kConeShift) + 2 * margin; }

size_t cone_scratch(int W, int H, int n_specs)
{
    const int margin = cone_margin(W, H);
    return (size_t)cone_blocks(W, margin) * cone_blocks(H, margin) * (2 * (size_t)n_specs + 1);
}

cudaError_t launch_cone_tables(const float* grid, int gw, int gh, float maxz, const ConeSpec* specs, int n_specs,
                               float* tabs, float* tmp, size_t stride, cudaStream_t st)
{
    if (gw <= 0 || gh <= 0 || n_specs <= 0) return cudaSuccess;
    const int r = cone_window_radius(gw, gh), margin = cone_margin(gw, gh);
    const int W = cone_blocks(gw, margin), H = cone_blocks(gh, margin);
    const size_t blocks = (size_t)W * H;
    float *base = tmp, *a = base + blocks, *b = a + blocks * n_specs;
    // start blocks of a line family: at most kConeOrder (W + H)
    const unsigned lines = (unsigned)(((long long)kConeOrder * (W + H) + 255) / 256);
    k_cone_blocks<<<(unsigned)((blocks + 255) / 256), 256, 0, st>>>(grid, gw, gh, margin, W, H, base);
    k_cone_lines<0><<<dim3(lines, n_specs), 256, 0, st>>>(base, W, H, specs, a, blocks);
    k_cone_lines<1><<<dim3(lines, n_specs), 256, 0, st>>>(a, W, H, specs, b, blocks);
    // the widest window: r on one side, r + a + b (components <= kConeOrder each) on the other
    const int wmax = 2 * r + 2 * kConeOrder + 1;
    const unsigned win0 = (unsigned)(((long long)W + kWinRow - 1) / kWinRow * H);
    const unsigned win1 = (unsigned)(((long long)W + kWinCols - 1) / kWinCols * ((H + kWinRows - 1) / kWinRows));
    k_cone_window<0><<<dim3(win0, n_specs), 256, sizeof(float) * (kWinRow + wmax), st>>>(W, H, maxz, r, specs, b, a,
                                                                                       blocks);
    k_cone_window<1><<<dim3(win1, n_specs), 256, sizeof(float) * kWinCols * (kWinRows + wmax), st>>>(W, H, maxz, r,
                                                                                                 specs, a, b, blocks);
    const size_t cells = (size_t)(gw + 2) * (gh + 2);
    k_cone_cells<<<dim3((unsigned)((cells + 255) / 256), (n_specs + kExpand - 1) / kExpand), 256, 0, st>>>(
        b, blocks, W, margin, gw, gh, n_specs, tabs, stride);
    return cudaGetLastError();
}

}  // namespace sgb
