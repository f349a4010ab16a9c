// hydro_pair.cuh - the hydraulic cell in packed form, two cells at a time (pair.cuh), shared by the tile
// and the marching kernel: the arithmetic of flux_ieee and flow_cell_general (erosion.cuh), operation for
// operation.
#pragma once

#include "erosion.cuh"
#include "pair.cuh"

namespace tecto {

namespace {

// The packed path's constants, both halves equal, in the kernel's parameters: the packed instructions
// take them from the constant bank, where immediates would occupy register pairs through the march.
struct PairConst {
    f2 dt, G, nL, rL, dtA, Kc, Ks, Kd, evap;
    f2 Z, M, one, mone, half, tiny;  // Z: (-0, -0), see mul2_z; M: 1.5 x 2^23; tiny: 1e-6
    f2 top, C1, C2, C3, C4;          // 2 / pi and the split of pi / 2
    f2 S3, S5, S7, S9, S11, K2, K4, K6, K8, K10;
};

inline PairConst pair_const(const HydroParams &p)
{
    auto d = [](float v) { return pk_host(v); };
    PairConst c{};
    c.dt = d(p.dt);
    c.G = d(p.G);
    c.nL = d(-p.L);
    c.rL = d(p.rL);
    c.dtA = d(p.dt * p.A);
    c.Kc = d(p.Kc);
    c.Ks = d(p.Ks);
    c.Kd = d(p.Kd);
    c.evap = d(p.evap);
    c.Z = d(-0.0f);
    c.M = d(12582912.0f);
    c.one = d(1.0f);
    c.mone = d(-1.0f);
    c.half = d(0.5f);
    c.tiny = d(1e-6f);
    c.top = d(TECTO_TWO_OVER_PI);
    c.C1 = d(TECTO_PIO2_C1);
    c.C2 = d(TECTO_PIO2_C2);
    c.C3 = d(TECTO_PIO2_C3);
    c.C4 = d(TECTO_PIO2_C4);
    c.S3 = d(TECTO_SIN_S3);
    c.S5 = d(TECTO_SIN_S5);
    c.S7 = d(TECTO_SIN_S7);
    c.S9 = d(TECTO_SIN_S9);
    c.S11 = d(TECTO_SIN_S11);
    c.K2 = d(TECTO_COS_K2);
    c.K4 = d(TECTO_COS_K4);
    c.K6 = d(TECTO_COS_K6);
    c.K8 = d(TECTO_COS_K8);
    c.K10 = d(TECTO_COS_K10);
    return c;
}

constexpr uint32_t kNz90 = 0x24ffffffu, kNz100 = 0x1affffffu;  // nz_bits of 2^-90 and 2^-100

// The flux of one cell (:2439-2485) in scalar IEEE form.
__device__ __forceinline__ float4 flux_ieee(const HydroParams &p, float4 f, float h, float w, float hl, float wl,
                                            float hu, float wu, float hr, float wr, float hd, float wd)
{
    const float dt = p.dt, dtA = dt * p.A, G = p.G, L = p.L;
    const float hw = h + w;
    const float o0 = fmaxf(0.0f, f.x + dtA * ((G * ((hw - hl) - wl)) / L));
    const float o1 = fmaxf(0.0f, f.y + dtA * ((G * ((hw - hu) - wu)) / L));
    const float o2 = fmaxf(0.0f, f.z + dtA * ((G * ((hw - hr) - wr)) / L));
    const float o3 = fmaxf(0.0f, f.w + dtA * ((G * ((hw - hd) - wd)) / L));
    const float total = (((o0 + o1) + o2) + o3) + 1e-6f;
    float K = fminf(1.0f, w / (total * dt + 1e-6f));
    K = fmaxf(K, 0.01f);
    return make_float4(o0 * K, o1 * K, o2 * K, o3 * K);
}

// sin(x) of both halves for 0.03 <= x < 2^21: tecto_sinf's reduction and series.  The rounding to the
// nearest integer is the addition of 1.5 x 2^23 (ties to even, as rintf), whose low bits are the
// quadrant.
__device__ __forceinline__ f2 sin2(f2 x, const PairConst &c)
{
    const f2 t = add2(mul2_z(x, c.top, c.Z), c.M);
    const f2 nk = sub2(c.M, t);  // -k
    f2 r = fma2(nk, c.C1, x);
    r = fma2(nk, c.C2, r);
    r = fma2(nk, c.C3, r);
    r = fma2(nk, c.C4, r);
    const f2 r2 = mul2(r, r);
    f2 ps = fma2(r2, c.S11, c.S9);
    ps = fma2(r2, ps, c.S7);
    ps = fma2(r2, ps, c.S5);
    ps = fma2(r2, ps, c.S3);
    const f2 sn = fma2(mul2(r, r2), ps, r);
    f2 pc = fma2(r2, c.K10, c.K8);
    pc = fma2(r2, pc, c.K6);
    pc = fma2(r2, pc, c.K4);
    pc = fma2(r2, pc, c.K2);
    const f2 cs = fma2(r2, pc, c.one);
    const uint32_t q0 = __float_as_uint(lo(t)), q1 = __float_as_uint(hi(t));
    const float v0 = (q0 & 1u) ? lo(cs) : lo(sn), v1 = (q1 & 1u) ? hi(cs) : hi(sn);
    return pk(__uint_as_float(__float_as_uint(v0) ^ ((q0 & 2u) << 30)),
              __uint_as_float(__float_as_uint(v1) ^ ((q1 & 2u) << 30)));
}

// base + i elements, in one multiply-add
template <typename T>
__device__ __forceinline__ unsigned long long gaddr64(const T *base, uint32_t i)
{
    unsigned long long a;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(a) : "r"(i), "n"((int)sizeof(T)), "l"(base));
    return a;
}
// Predicated stores: two cells of one row where s0, s1 (VEC: s0 for both), and one cell's flux.
template <bool VEC>
__device__ __forceinline__ void gst2(float *base, uint32_t i, f2 v, bool s0, bool s1)
{
    const unsigned long long a = gaddr64(base, i);
    if (VEC) {
        if (s0) asm volatile("st.global.b64 [%0], %1;" ::"l"(a), "l"(v) : "memory");
    } else {
        if (s0) asm volatile("st.global.f32 [%0], %1;" ::"l"(a), "f"(lo(v)) : "memory");
        if (s1) asm volatile("st.global.f32 [%0+4], %1;" ::"l"(a), "f"(hi(v)) : "memory");
    }
}

template <bool VEC>
__device__ __forceinline__ void gst_flux(float4 *base, uint32_t i, f2 x, f2 y, f2 z, f2 w, bool s0, bool s1)
{
    const unsigned long long a = gaddr64(base, i);
    if (VEC) {
        if (s0)
            asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(a), "f"(lo(x)), "f"(lo(y)),
                         "f"(lo(z)), "f"(lo(w)), "f"(hi(x)), "f"(hi(y)), "f"(hi(z)), "f"(hi(w))
                         : "memory");
        return;
    }
    if (s0)
        asm volatile("st.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(a), "f"(lo(x)), "f"(lo(y)), "f"(lo(z)), "f"(lo(w))
                     : "memory");
    if (s1)
        asm volatile("st.global.v4.f32 [%0+16], {%1, %2, %3, %4};" ::"l"(a), "f"(hi(x)), "f"(hi(y)), "f"(hi(z)),
                     "f"(hi(w))
                     : "memory");
}

struct Flux2 {
    f2 x, y, z, w;  // left, +y, right, -y of two adjacent cells
};

// The flux of two adjacent cells (:2439-2485): their heights h and water w (rain added), those left of
// the first (hl, wl), right of the second (hr, wr), at +y (hu, wu) and -y (hd, wd), their old fluxes fa and
// fb.  True where `mine` holds and an operand is outside the packed path's ranges.
__device__ __forceinline__ bool flux_pair(const PairConst &c, f2 h, f2 w, float hl, float hr, float wl, float wr, f2 hu,
                                          f2 wu, f2 hd, f2 wd, float4 fa, float4 fb, bool mine, Flux2 &o)
{
    const f2 hw = add2(h, w);
    // (left of cell 0, right of cell 1), (right of cell 0, left of cell 1), +y, -y
    f2 gA = sub2(sub2(hw, pk(hl, hr)), pk(wl, wr));
    f2 gB = pk((lo(hw) - hi(h)) - hi(w), (hi(hw) - lo(h)) - lo(w));
    f2 gU = sub2(sub2(hw, hu), wu);
    f2 gD = sub2(sub2(hw, hd), wd);
    const f2 G = c.G;
    gA = mul2(G, gA);
    gB = mul2(G, gB);
    gU = mul2(G, gU);
    gD = mul2(G, gD);
    const f2 nL = c.nL, rL = c.rL, dtA = c.dtA;
    const f2 tA = mul2_z(dtA, div2(gA, nL, rL), c.Z), tB = mul2_z(dtA, div2(gB, nL, rL), c.Z);
    const f2 tU = mul2_z(dtA, div2(gU, nL, rL), c.Z), tD = mul2_z(dtA, div2(gD, nL, rL), c.Z);
    // the sign of a zero quotient does not survive the sums and clamps below
    const f2 ox = pk(fmaxf(0.0f, fa.x + lo(tA)), fmaxf(0.0f, fb.x + hi(tB)));
    const f2 oy = pk(fmaxf(0.0f, fa.y + lo(tU)), fmaxf(0.0f, fb.y + hi(tU)));
    const f2 oz = pk(fmaxf(0.0f, fa.z + lo(tB)), fmaxf(0.0f, fb.z + hi(tA)));
    const f2 ow = pk(fmaxf(0.0f, fa.w + lo(tD)), fmaxf(0.0f, fb.w + hi(tD)));
    const f2 total = add2(add2(add2(add2(ox, oy), oz), ow), c.tiny);
    const f2 den = add2(mul2_z(total, c.dt, c.Z), c.tiny);
    const f2 nden = mul2(den, c.mone);
    const f2 qK = div2(w, nden, rcp2(den, nden, c.one));
    const f2 Kf = max2(min2(qK, 1.0f), 0.01f);
    // every dividend a zero or in [2^-90, 2^64), the denominators (>= 1e-6) at most 2^32; a water
    // below 2^-90 has a quotient far below 0.01, whatever its last bits.  A dividend below 2^-90
    // is looked at again: it may be a zero.
    const float mx = max3_nan(max3_nan(max3_nan(max3_nan(lo(gA), hi(gA), lo(gB)), hi(gB), lo(gU)), hi(gU),
                                       lo(gD)), hi(gD), max3_nan(lo(w), hi(w), 0.0f));
    const float mn = min3(min3(min3(lo(gA), hi(gA), lo(gB)), hi(gB), lo(gU)), min3(hi(gU), lo(gD), hi(gD)), 1.0f);
    bool bad = false;
    if (mine && (!(mx < 0x1p64f) || mn < 0x1p-90f || !(fmaxf(lo(den), hi(den)) <= 0x1p32f))) {
        const uint32_t z = min(
            min(min(nz_bits(lo(gA)), nz_bits(hi(gA))), min(nz_bits(lo(gB)), nz_bits(hi(gB)))),
            min(min(nz_bits(lo(gU)), nz_bits(hi(gU))), min(nz_bits(lo(gD)), nz_bits(hi(gD)))));
        bad = !(mx < 0x1p64f) || z < kNz90 || !(fmaxf(lo(den), hi(den)) <= 0x1p32f);
    }
    o.x = mul2(ox, Kf);
    o.y = mul2(oy, Kf);
    o.z = mul2(oz, Kf);
    o.w = mul2(ow, Kf);
    return bad;
}

struct Flow2 {
    f2 hn, wn, s1, ux, uy;  // new height, water before evaporation, eroded sediment, velocity
};

// Flow (:2487-2533) and the sediment exchange (:2535-2570) of two adjacent cells: their fluxes b, the left
// cell's .z and the right cell's .x, the +y cells' .w, the -y cells' .y and .w, their water w, height hc and
// sediment sd, the heights left, right, +y and -y.  True as in flux_pair.  All lanes of the warp.
__device__ __forceinline__ bool flow_pair(const PairConst &c, const Flux2 &b, float lz, float rx, f2 uw, f2 dy, f2 dw,
                                          f2 w, f2 hc, float hl, float hr, f2 hu, f2 hd, f2 sd, bool mine, Flow2 &o)
{
    // flow (:2487-2533); a flux is never -0, so the reference's sum from zero starts at its first term
    const f2 in = add2(pk((lz + lo(uw)) + hi(b.x), (lo(b.z) + hi(uw)) + rx), dy);
    const f2 out = add2(add2(add2(b.x, b.y), b.z), b.w);
    const f2 wn = max2(add2(w, mul2_z(c.dt, sub2(in, out), c.Z)), 0.0f);
    const f2 nx = add2(pk(lz - lo(b.x), lo(b.z) - hi(b.x)), b.z);
    const f2 nfx = mul2(pk(lo(nx) - hi(b.x), hi(nx) - rx), c.half);
    const f2 nfy = mul2(sub2(add2(sub2(uw, b.y), b.y), dw), c.half);
    const f2 hh = max2(wn, 0.01f);
    const f2 nhh = mul2(hh, c.mone);
    const f2 rh = rcp2(hh, nhh, c.one);
    f2 ux = div2(nfx, nhh, rh), uy = div2(nfy, nhh, rh);
    f2 m2 = add2(mul2_z(ux, ux, c.Z), mul2_z(uy, uy, c.Z));
    f2 mag = sqrt2(m2, c.half, c.mone);
    const bool over = !(lo(m2) <= 0x1p64f) || !(hi(m2) <= 0x1p64f);
    const float m0 = lo(mag), m1 = hi(mag);
    if (__any_sync(0xffffffffu, m0 > 50.0f || m1 > 50.0f)) {  // the velocity clamp (:2524-2528)
        const f2 mc = pk(m0 > 50.0f ? m0 : 50.0f, m1 > 50.0f ? m1 : 50.0f);
        const f2 nm = mul2(mc, c.mone);
        const f2 sc = div2(dup2(50.0f), nm, rcp2(mc, nm, c.one));  // 1 where there is no clamp
        ux = mul2(ux, sc);
        uy = mul2(uy, sc);
        const f2 mm = add2(mul2_z(ux, ux, c.Z), mul2_z(uy, uy, c.Z));
        const f2 mr = sqrt2(mm, c.half, c.mone);
        mag = pk(m0 > 50.0f ? lo(mr) : m0, m1 > 50.0f ? hi(mr) : m1);
    }
    // sediment (:2535-2570); the slope reads the pre-erosion height (:351-358)
    const f2 dzx = mul2(pk(hi(hc) - hl, hr - lo(hc)), c.half);
    const f2 dzy = mul2(sub2(hu, hd), c.half);
    const f2 s2 = add2(mul2_z(dzx, dzx, c.Z), mul2_z(dzy, dzy, c.Z));
    const f2 sx = max2(sqrt2(s2, c.half, c.mone), 0.03f);
    const f2 C = min2(mul2(mul2(c.Kc, sin2(sx, c)), mag), 5.0f);
    const f2 ce = mul2(mul2(c.Ks, sub2(C, sd)), c.dt);
    const f2 cd = mul2(mul2(c.Kd, sub2(sd, C)), c.dt);
    // what leaves the bed: eroded where the capacity exceeds the sediment, else minus the deposit
    const f2 de = pk(lo(C) > lo(sd) ? fminf(lo(ce), lo(hc)) : -fminf(lo(cd), lo(sd)),
                     hi(C) > hi(sd) ? fminf(hi(ce), hi(hc)) : -fminf(hi(cd), hi(sd)));
    o.hn = sub2(hc, de);
    o.s1 = add2(sd, de);
    o.wn = wn;
    o.ux = ux;
    o.uy = uy;
    // quotients: dividends a zero or at least 2^-90 (one above 2^64 fails the test on m2), depth at
    // most 2^32; roots: arguments a zero or at least 2^-100; sine argument below 2^21
    const bool big = !(max3_nan(lo(s2), hi(s2), 0.0f) <= 0x1p42f) || !(fmaxf(lo(hh), hi(hh)) <= 0x1p32f);
    const float mq = fminf(min3(lo(nfx), hi(nfx), lo(nfy)), fabsf(hi(nfy)));
    const float ms = fminf(min3(lo(m2), hi(m2), lo(s2)), fabsf(hi(s2)));
    bool bad = false;
    if (mine && (over || big || mq < 0x1p-90f || ms < 0x1p-100f)) {
        const uint32_t zq = min(min(nz_bits(lo(nfx)), nz_bits(hi(nfx))), min(nz_bits(lo(nfy)), nz_bits(hi(nfy))));
        const uint32_t zs = min(min(nz_bits(lo(m2)), nz_bits(hi(m2))), min(nz_bits(lo(s2)), nz_bits(hi(s2))));
        bad = over || big || zq < kNz90 || zs < kNz100;
    }
    return bad;
}

// evaporate (:2587-2593)
__device__ __forceinline__ f2 evaporate2(const PairConst &c, f2 wn)
{
    return max2(sub2(wn, mul2_z(mul2(min2(wn, 20.0f), c.evap), c.dt, c.Z)), 0.0f);
}

}  // namespace

}  // namespace tecto
