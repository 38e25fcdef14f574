// Direct + Perez diffuse of a voxel for two hours at a time, on packed FP32
// pairs (fma.rn.f32x2 and the like: one issue slot for both hours).  The same
// terms as solar_I (solar_math.cuh), with the direct part fused into the sum.
#pragma once

#include "solar_math.cuh"

namespace sgb {

using f32x2 = unsigned long long;

__device__ __forceinline__ f32x2 pack2(float lo, float hi)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 a)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 max2(f32x2 a)   // max(0, a)
{
    const float2 v = unpack2(a);
    return pack2(fmaxf(0.0f, v.x), fmaxf(0.0f, v.y));
}

// Two hours of the table: DNI is 0 and the mask empty where the hour has no sun
// bin, so that no test of the bin is left.
struct HourPair {
    f32x2 sx, sy, sz, dni, c0, c1, c2;
    int word[2];      // shadow word of the hour
    unsigned bit[2];  // its bit in it
    int pad[2];
};
static_assert(sizeof(HourPair) == 80, "five 16-byte loads");

__device__ __forceinline__ HourPair make_pair2(const HourEntry& a, const HourEntry& b)
{
    HourPair p;
    p.sx = pack2(a.sx, b.sx);
    p.sy = pack2(a.sy, b.sy);
    p.sz = pack2(a.sz, b.sz);
    p.dni = pack2(a.dense >= 0 ? a.dni_eff : 0.0f, b.dense >= 0 ? b.dni_eff : 0.0f);
    p.c0 = pack2(a.c0, b.c0);
    p.c1 = pack2(a.c1, b.c1);
    p.c2 = pack2(a.c2, b.c2);
    p.word[0] = a.dense >= 0 ? a.dense >> 5 : 0;
    p.word[1] = b.dense >= 0 ? b.dense >> 5 : 0;
    p.bit[0] = a.dense >= 0 ? 1u << (a.dense & 31) : 0u;
    p.bit[1] = b.dense >= 0 ? 1u << (b.dense & 31) : 0u;
    p.pad[0] = p.pad[1] = 0;
    return p;
}

// A voxel's normal, each component twice.
struct NormalPair {
    f32x2 x, y, z, z1, s, pad;   // z1 = 1 + z, s = sin slope; three 16-byte loads
    NormalPair() = default;
    __device__ __forceinline__ explicit NormalPair(const float4& n)
        : x(pack2(n.x, n.x)), y(pack2(n.y, n.y)), z(pack2(n.z, n.z)), z1(pack2(1.0f + n.z, 1.0f + n.z)),
          s(pack2(n.w, n.w)), pad(0ull)
    {
    }
};

// The two hours' I; w0, w1: the shadow words the pair names.
__device__ __forceinline__ f32x2 solar_I2(const NormalPair& n, const HourPair& e, uint32_t w0, uint32_t w1)
{
    const f32x2 p = max2(fma2(n.x, e.sx, fma2(n.y, e.sy, mul2(n.z, e.sz))));
    const f32x2 dif = max2(fma2(e.c0, n.z1, fma2(e.c1, p, mul2(e.c2, n.s))));
    const float2 d = unpack2(e.dni), q = unpack2(p);
    // q > 0: an infinite DNI is nothing on a voxel that faces away
    return fma2(pack2(!(w0 & e.bit[0]) && q.x > 0.0f ? d.x : 0.0f, !(w1 & e.bit[1]) && q.y > 0.0f ? d.y : 0.0f), p, dif);
}

}  // namespace sgb
