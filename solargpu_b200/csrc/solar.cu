// Solar pass: FP64 per-hour geometry table, per-voxel geometry, and the
// direct + Perez diffuse kernels (src/cuda/kernels/solar_kernel.cu:8-85).
//
// The reference recomputes the sun geometry and every Perez term
// (acosf/powf/cosf per voxel and hour, solar_kernel.cu:8-50, 66-74) for every
// voxel.  Those terms depend only on the hour, so here one FP64 kernel
// evaluates them once per daylight hour (k_hour_table); the per voxel-hour
// work is a dot product, a shadow-bit test and three FMAs (solar_I).
#include "solar_pair.cuh"

namespace sgb {
namespace {

// Reference constants at their float values (solar_kernel.cu:8-50,
// src/cuda/device_globals.cu:50-57, include/pipeline_math_constants.h:15).
#define FC(x) ((double)(float)(x))
__constant__ double c_F[6][8] = {
    { FC(-0.0083117), FC(0.1299457), FC(0.3296958), FC(0.5682053), FC(0.8730280), FC(1.1326077), FC(1.0601591), FC(0.6777470) },
    { FC(0.5877285), FC(0.6825954), FC(0.4868735), FC(0.1874525), FC(-0.3920403), FC(-1.2367284), FC(-1.5999137), FC(-0.3272588) },
    { FC(-0.0620636), FC(-0.1513752), FC(-0.2210958), FC(-0.2951290), FC(-0.3616149), FC(-0.4118494), FC(-0.3589221), FC(-0.2504286) },
    { FC(-0.0596012), FC(-0.0189325), FC(0.0554140), FC(0.1088631), FC(0.2255647), FC(0.2877813), FC(0.2642124), FC(0.1561313) },
    { FC(0.0721249), FC(0.0659650), FC(-0.0639588), FC(-0.1519229), FC(-0.4620442), FC(-0.8230357), FC(-1.1272340), FC(-1.3765031) },
    { FC(-0.0220216), FC(-0.0288748), FC(-0.0260542), FC(-0.0139754), FC(0.0012448), FC(0.0558651), FC(0.1310694), FC(0.2506212) },
};

__global__ void k_hour_table(const float* __restrict__ nudged, const float* __restrict__ dni,
                             const float* __restrict__ dhi, const int* __restrict__ sun_dense,
                             const int* __restrict__ hour_index, int n_hours, int n_padded,
                             HourEntry* __restrict__ table)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_padded) return;
    HourEntry e;
    e.sx = e.sy = e.sz = e.dni_eff = e.c0 = e.c1 = e.c2 = 0.0f;
    e.dense = -1;
    if (j < n_hours) {
        const int k = hour_index[j];
        const double kDeg = FC(0.0174532925);
        const double pi_f = FC(3.14159265358979323846);
        const double alt = nudged[2 * k + 1];
        const double az = nudged[2 * k];
        const double cz = cos((90.0 - alt) * kDeg);
        const double z = acos(cz);
        const double sz = sin(z);
        const double dn = dni[k], df = dhi[k];
        // Perez sky model, solar_kernel.cu:8-50
        const double z_deg = z * (180.0 / pi_f);
        const double AM = 1.0 / (cz + FC(0.50572) * pow(FC(96.07995) - z_deg, FC(-1.6364)));
        const double b = fmax(FC(0.08715574), cz);
        const double z3 = z * z * z;
        double eps = ((df + dn / cos(z)) / df + FC(1.041) * z3) / (1.0 + FC(1.041) * z3);
        const double day = (double)(k / 24);
        const double B = 2.0 * pi_f * (day / 365.0);
        const double E0 = 1367.0 * (FC(1.00011) + FC(0.034221) * cos(B) + FC(0.00128) * sin(B)
                                    + FC(0.000719) * cos(2.0 * B) + FC(0.000077) * sin(2.0 * B));
        const double delta = (AM * df) / E0;
        eps = fmax(1.0, eps);   // NaN (DHI = DNI = 0) -> 1, as fmaxf does in the reference
        int bin = 7;
        if (eps < FC(1.065)) bin = 0;
        else if (eps < FC(1.230)) bin = 1;
        else if (eps < FC(1.500)) bin = 2;
        else if (eps < FC(1.950)) bin = 3;
        else if (eps < FC(2.800)) bin = 4;
        else if (eps < FC(4.500)) bin = 5;
        else if (eps < FC(6.200)) bin = 6;
        const double F1 = fmax(0.0, c_F[0][bin] + c_F[1][bin] * delta + c_F[2][bin] * z);
        const double F2 = c_F[3][bin] + c_F[4][bin] * delta + c_F[5][bin] * z;
        e.sx = (float)(sz * sin(az * kDeg));
        e.sy = (float)(-sz * cos(az * kDeg));
        e.sz = (float)cz;
        e.dni_eff = (float)fmax(dn, FC(1e-3));
        e.c0 = (float)(df * (1.0 - F1) * 0.5);
        e.c1 = (float)(df * F1 / b);
        e.c2 = (float)(df * F2);
        e.dense = sun_dense[k];
    }
    table[j] = e;
}

__global__ void k_voxel_geom(DevScene s, float4* __restrict__ geo_n, float4* __restrict__ geo_p)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= s.N) return;
    const int top = s.pix_parent[v];
    const int gx = top % s.W, gy = top / s.W;
    const float z = (v < s.T) ? s.grid[top] : s.wall_z[v - s.T];
    const float sl = s.slopes[v], as = s.aspects[v];
    const float ss = sinf(sl);
    geo_n[v] = make_float4(ss * sinf(as), -ss * cosf(as), cosf(sl), ss);
    geo_p[v] = make_float4((float)gx, (float)gy, z, 0.0f);
}

// slab[g * B + b] = I(g, j0 + b) for every top cell g.  A warp owns 32
// consecutive hours of the block (their table entries stay in registers)
// and sweeps a run of cells, writing one coalesced 128-byte row piece per
// cell; the voxel normal is a broadcast load.
constexpr int kSlabCellsPerWarp = 64;

__global__ void __launch_bounds__(256)
k_solar_slab(const float4* __restrict__ geo_n, int T, const uint32_t* __restrict__ shadow, int words32,
             const HourEntry* __restrict__ table, int j0, int B, float* __restrict__ slab)
{
    const int lane = threadIdx.x & 31;
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int hchunks = B >> 5;
    const int hc = (int)(wid % hchunks);
    const long long g0 = (wid / hchunks) * kSlabCellsPerWarp;
    if (g0 >= T) return;
    const int b = hc * 32 + lane;
    const HourEntry e = table[j0 + b];
    const int word = e.dense >= 0 ? (e.dense >> 5) : 0;
    const uint32_t mask = e.dense >= 0 ? (1u << (e.dense & 31)) : 0u;
    const long long g1 = min((long long)T, g0 + kSlabCellsPerWarp);
#pragma unroll 4
    for (long long g = g0; g < g1; ++g) {
        const float4 n4 = __ldg(geo_n + g);
        const uint32_t bit = (__ldg(shadow + g * words32 + word) & mask) ? 1u : 0u;
        slab[g * B + b] = solar_I(n4, e, bit);
    }
}

__global__ void __launch_bounds__(256)
k_solar_hour(const float4* __restrict__ geo_n, int N, const uint32_t* __restrict__ shadow, int words32,
             const HourEntry* __restrict__ table, int j, float* __restrict__ hourly)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= N) return;
    const HourEntry e = table[j];
    hourly[v] = solar_I(__ldg(geo_n + v), e, shadow_bit(shadow, words32, v, e.dense));
}

// ---- sums over hours ---------------------------------------------------------
//
// A thread sums the hours of two voxels, two hours at a time (solar_I2), with
// the hours' pairs and the voxels' shadow words in shared memory: 11
// instructions a voxel-hour, where a thread per voxel reading the table and its
// shadow words through L1 took 34.

constexpr int kPairs = 128;          // pairs of hours staged at a time (256 hours)

__device__ __forceinline__ void stage_pairs(const HourEntry* __restrict__ table, HourPair* s_pair, int tid, int threads)
{
    for (int i = tid; i < kPairs; i += threads) s_pair[i] = make_pair2(table[2 * i], table[2 * i + 1]);
}

// own[hb][p] = sum of I over hour block hb (256 hours), for the voxel at
// visiting position p.
constexpr int kOwnThreads = 128;     // and 256 voxels

__global__ void __launch_bounds__(kOwnThreads)
k_own_blocks(const float4* __restrict__ geo_n, const int* __restrict__ order, int N, const uint32_t* __restrict__ shadow,
             int words32, const HourEntry* __restrict__ table, float* __restrict__ own)
{
    extern __shared__ __align__(16) unsigned char sm[];
    HourPair* s_pair = reinterpret_cast<HourPair*>(sm);
    uint32_t* s_shadow = reinterpret_cast<uint32_t*>(s_pair + kPairs);   // [words32][2 kOwnThreads]
    const int tid = threadIdx.x;
    const int p0 = blockIdx.x * 2 * kOwnThreads + tid, p1 = p0 + kOwnThreads;
    const int v0 = __ldg(order + min(p0, N - 1)), v1 = __ldg(order + min(p1, N - 1));
    stage_pairs(table + (size_t)blockIdx.y * 2 * kPairs, s_pair, tid, kOwnThreads);
    for (int w = 0; w < words32; ++w) {
        s_shadow[w * 2 * kOwnThreads + tid] = __ldg(shadow + (size_t)v0 * words32 + w);
        s_shadow[w * 2 * kOwnThreads + kOwnThreads + tid] = __ldg(shadow + (size_t)v1 * words32 + w);
    }
    __syncthreads();
    const NormalPair n0(__ldg(geo_n + v0)), n1(__ldg(geo_n + v1));
    f32x2 a0 = 0ull, b0 = 0ull, a1 = 0ull, b1 = 0ull;
    const uint32_t* sh = s_shadow + tid;
#pragma unroll 2
    for (int i = 0; i < kPairs; i += 2) {
        const HourPair e = s_pair[i], f = s_pair[i + 1];
        const uint32_t *e0 = sh + e.word[0] * 2 * kOwnThreads, *e1 = sh + e.word[1] * 2 * kOwnThreads;
        const uint32_t *f0 = sh + f.word[0] * 2 * kOwnThreads, *f1 = sh + f.word[1] * 2 * kOwnThreads;
        a0 = add2(a0, solar_I2(n0, e, e0[0], e1[0]));
        a1 = add2(a1, solar_I2(n1, e, e0[kOwnThreads], e1[kOwnThreads]));
        b0 = add2(b0, solar_I2(n0, f, f0[0], f1[0]));
        b1 = add2(b1, solar_I2(n1, f, f0[kOwnThreads], f1[kOwnThreads]));
    }
    const float2 s0 = unpack2(add2(a0, b0)), s1 = unpack2(add2(a1, b1));
    float* dst = own + (size_t)blockIdx.y * N;
    if (p0 < N) dst[p0] = s0.x + s0.y;
    if (p1 < N) dst[p1] = s1.x + s1.y;
}

// sums[v] = sum over all daylight hours of I(v, h): FP32 over 32 hours, FP64
// over those.  A CTA takes 64 voxels; its 4 warps take the staged hours in turn
// (32 at a time) and their sums are added at the end, so that small scenes
// fill the GPU.
constexpr int kSumWarps = 4;

__global__ void __launch_bounds__(kSumWarps * 32)
k_solar_sum(const float4* __restrict__ geo_n, int N, const uint32_t* __restrict__ shadow, int words32,
            const HourEntry* __restrict__ table, int n_hours, double* __restrict__ sums)
{
    extern __shared__ __align__(16) unsigned char sm[];
    HourPair* s_pair = reinterpret_cast<HourPair*>(sm);
    uint32_t* s_shadow = reinterpret_cast<uint32_t*>(s_pair + kPairs);   // [words32][64]
    __shared__ double s_sum[kSumWarps][64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int v = blockIdx.x * 64;
    for (int i = threadIdx.x; i < 64 * words32; i += kSumWarps * 32)
        s_shadow[(i % words32) * 64 + i / words32] =
            v + i / words32 < N ? __ldg(shadow + (size_t)v * words32 + i) : 0u;
    const NormalPair n0(__ldg(geo_n + min(v + lane, N - 1))), n1(__ldg(geo_n + min(v + 32 + lane, N - 1)));
    const uint32_t* sh = s_shadow + lane;
    double a0 = 0.0, a1 = 0.0;
    for (int j = 0; j < n_hours; j += 2 * kPairs) {   // the table is padded with hours of no light
        __syncthreads();
        stage_pairs(table + j, s_pair, threadIdx.x, kSumWarps * 32);
        __syncthreads();
        for (int i = warp * 16; i < kPairs; i += kSumWarps * 16) {
            f32x2 t0 = 0ull, t1 = 0ull;
#pragma unroll 4
            for (int k = 0; k < 16; ++k) {
                const HourPair e = s_pair[i + k];
                const uint32_t *w0 = sh + e.word[0] * 64, *w1 = sh + e.word[1] * 64;
                t0 = add2(t0, solar_I2(n0, e, w0[0], w1[0]));
                t1 = add2(t1, solar_I2(n1, e, w0[32], w1[32]));
            }
            const float2 s0 = unpack2(t0), s1 = unpack2(t1);
            a0 += (double)s0.x + (double)s0.y;
            a1 += (double)s1.x + (double)s1.y;
        }
    }
    s_sum[warp][lane] = a0;
    s_sum[warp][32 + lane] = a1;
    __syncthreads();
    if (threadIdx.x < 64 && v + (int)threadIdx.x < N) {
        double a = 0.0;
        for (int w = 0; w < kSumWarps; ++w) a += s_sum[w][threadIdx.x];
        sums[v + threadIdx.x] = a;
    }
}

}  // namespace

cudaError_t launch_hour_table(const float* nudged, const float* dni, const float* dhi,
                              const int* sun_dense, const int* hour_index, int n_hours,
                              int n_padded, HourEntry* table, cudaStream_t st)
{
    k_hour_table<<<(n_padded + 127) / 128, 128, 0, st>>>(nudged, dni, dhi, sun_dense, hour_index,
                                                          n_hours, n_padded, table);
    return cudaGetLastError();
}

cudaError_t launch_voxel_geom(const DevScene& s, DevGeom g, cudaStream_t st)
{
    if (s.N <= 0) return cudaSuccess;
    k_voxel_geom<<<(s.N + 255) / 256, 256, 0, st>>>(s, g.geo_n, g.geo_p);
    return cudaGetLastError();
}

cudaError_t launch_solar_slab(const DevGeom& g, int T, const uint32_t* shadow, int words32,
                              const HourEntry* table, int j0, int B, float* slab, cudaStream_t st)
{
    if (B < 32 || (B & 31)) return cudaErrorInvalidValue;
    const long long warps = ((long long)T + kSlabCellsPerWarp - 1) / kSlabCellsPerWarp * (B / 32);
    k_solar_slab<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, st>>>(g.geo_n, T, shadow, words32, table,
                                                                        j0, B, slab);
    return cudaGetLastError();
}

cudaError_t launch_solar_hour(const DevGeom& g, int N, const uint32_t* shadow, int words32,
                              const HourEntry* table, int j, float* hourly, cudaStream_t st)
{
    k_solar_hour<<<(N + 255) / 256, 256, 0, st>>>(g.geo_n, N, shadow, words32, table, j, hourly);
    return cudaGetLastError();
}

cudaError_t launch_solar_sum(const DevGeom& g, int N, const uint32_t* shadow, int words32,
                             const HourEntry* table, int n_hours, double* sums, cudaStream_t st)
{
    const size_t smem = sizeof(HourPair) * kPairs + sizeof(uint32_t) * 64 * (size_t)words32;
    k_solar_sum<<<(N + 63) / 64, kSumWarps * 32, smem, st>>>(g.geo_n, N, shadow, words32, table, n_hours, sums);
    return cudaGetLastError();
}

cudaError_t launch_own_blocks(const DevGeom& g, const int* order, int N, const uint32_t* shadow, int words32,
                              const HourEntry* table, int j0, int nb, float* own, cudaStream_t st)
{
    if (N <= 0 || nb <= 0) return cudaSuccess;
    const size_t smem = sizeof(HourPair) * kPairs + sizeof(uint32_t) * 2 * kOwnThreads * (size_t)words32;
    if (smem > 48 * 1024) {   // up to 41 words: 52 KB
        const cudaError_t e = cudaFuncSetAttribute(k_own_blocks, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    const dim3 grid((unsigned)((N + 2 * kOwnThreads - 1) / (2 * kOwnThreads)), nb);
    k_own_blocks<<<grid, kOwnThreads, smem, st>>>(g.geo_n, order, N, shadow, words32, table + j0, own);
    return cudaGetLastError();
}

}  // namespace sgb
