// k_hydro_tile.cu - the hydraulic sub-iteration on tiles, two cells per lane, and the rain field and the
// transport pass of the split path.
// Reference: rain/flux/flow/sediment/transport/evaporate,
// src/cuda_compute/plate_tectonics_kernel.cu:2430-2593; driver plate_tectonic_sim.cu:331-373.
//
// One sub-iteration of applyHydraulicErosion in one pass over HBM.  A block owns a tile of 56 x TY cells and
// its halo of 4 in shared memory; a warp works on one row at a time, 64 columns, two adjacent cells a lane
// (a row of the tile with its halo is a warp wide, so no index is divided).  Three phases with a block
// barrier between them: the new flux on a halo of 3; the flow (water, velocity), the sediment exchange and
// the evaporation on a halo of 2; the semi-Lagrangian sediment transport on the tile.  Transport's
// back-trace reaches |v| dt <= 50 dt cells (velocity clamp at :2524-2528), inside the halo when 50 dt < 1.5;
// larger steps take the split path (FUSED false: velocity and eroded sediment go to HBM and k_transport
// gathers from there), which needs a halo of 2 alone: 60 x TY cells of 64 x (TY + 4) instead of 56 x TY of
// 64 x (TY + 8), the reference's 1024^2 step 25.5 -> 21.5 us a launch.
//
// All loads are asynchronous copies to where a phase reads them (the old flux of a pair to the pair's own
// four flux slots), so that a tile's loads are in flight together without registers.  The velocity
// replaces the water and the eroded sediment the sediment, which only their own cell reads in the flow phase.
// The arithmetic is packed (hydro_pair.cuh); a block with an operand outside its ranges runs that phase once
// more in scalar IEEE form.
//
// Before (one cell a thread, 64 columns, 1024 threads) and now, us per sub-iteration: 256^2 12.7 -> 5.7,
// 1024^2 31.2 -> 23, 2048^2 103 -> 78, 8192^2 1444 -> 1150.  Bound by the latency of the three phases at
// small sizes, where k_hydro_two takes two sub-iterations at once (256^2 3.5), and by issue at large ones,
// where the march (k_hydro_march.cu) computes less halo.
#include "hydro_pair.cuh"
#include "noise.cuh"

namespace tecto {

namespace {

constexpr int HTX = 56;                   // interior columns of a tile
constexpr int HTXS = 60;                  // on the split path
constexpr uint32_t kRow = 64 * 4;         // bytes of a shared-memory row: 64 columns with the halo
constexpr uint32_t kGuard = 16;           // an edge lane reads one cell past a row's end

// Byte layout: guard, height, water (+ rain, then velocity x), sediment (then eroded), flux left, +y, right,
// -y, velocity y (before: rain), guard.
// HX: the halo, 4 cells where the transport follows, 2 on the split path.
template <int TY, int HX>
struct TileMem {
    static constexpr uint32_t A = (TY + 2 * HX) * kRow;  // bytes of an array
    static constexpr uint32_t H = kGuard, W = H + A, S = W + A, X = S + A, Y = X + A, Z = Y + A, F = Z + A, V = F + A;
    static constexpr uint32_t bytes = V + A + kGuard;
};

struct TileParams {
    HydroParams p;
    PairConst c;
    int ieee;  // the flux phase in scalar form: a pipe length outside [2^-32, 2^32] or dt < 0
};

__device__ __forceinline__ void cp8(uint32_t dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src));
}
__device__ __forceinline__ void cp4(uint32_t dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src));
}
template <bool VEC>
__device__ __forceinline__ void cp_pair(uint32_t dst, const float *row, uint32_t c0, uint32_t c1)
{
    if (VEC) {
        cp8(dst, row + c0);
    } else {
        cp4(dst, row + c0);
        cp4(dst + 4, row + c1);
    }
}

// The flux phase in scalar form.  FIRST: nothing has run on the tile, and the old fluxes lie where the loads put
// them; else the packed run replaced them, and they come from HBM again.
template <int TY, int NW, int HX, bool FIRST>
__device__ __noinline__ void flux_rows_ieee(const HydroParams &p, const HydroWorld &q, char *S, int x0, int y0)
{
    using M = TileMem<TY, HX>;
    const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5, lx = 2 * lane, gx = x0 - HX + lx;
    for (int ly = warp + 1; ly < TY + 2 * HX - 1; ly += NW) {
        const int gy = y0 - HX + ly;
        const uint32_t o = (uint32_t)ly * kRow + (uint32_t)lx * 4u;
        float4 f[2], v[2];
        if (FIRST) {
            const f2 a = ld2(S, o + M::X), b = ld2(S, o + M::Y), d = ld2(S, o + M::Z), e = ld2(S, o + M::F);
            f[0] = make_float4(lo(a), hi(a), lo(b), hi(b));
            f[1] = make_float4(lo(d), hi(d), lo(e), hi(e));
        } else {
            f[0] = q.f_in[cidx(gx, gy, q.W, q.H)];
            f[1] = q.f_in[cidx(gx + 1, gy, q.W, q.H)];
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint32_t c = o + 4u * j;
            v[j] = flux_ieee(p, f[j], mld(S, c + M::H), mld(S, c + M::W), mld(S, c + M::H - 4), mld(S, c + M::W - 4),
                             mld(S, c + M::H + kRow), mld(S, c + M::W + kRow), mld(S, c + M::H + 4),
                             mld(S, c + M::W + 4), mld(S, c + M::H - kRow), mld(S, c + M::W - kRow));
            if (lx + j >= HX && lx + j < 64 - HX && ly >= HX && ly < TY + HX && gx + j < q.W && gy < q.H)
                q.f_out[(uint32_t)gy * (uint32_t)q.W + (uint32_t)(gx + j)] = v[j];
        }
        st2(S, o + M::X, pk(v[0].x, v[1].x));
        st2(S, o + M::Y, pk(v[0].y, v[1].y));
        st2(S, o + M::Z, pk(v[0].z, v[1].z));
        st2(S, o + M::F, pk(v[0].w, v[1].w));
    }
}

// The flow phase in scalar form: water and sediment come from HBM again, as the packed run replaced them.
template <int TY, int NW, bool FUSED>
__device__ __noinline__ void flow_rows_ieee(const HydroParams &p, const HydroWorld &q, char *S, int x0, int y0)
{
    constexpr int HX = FUSED ? 4 : 2;
    using M = TileMem<TY, HX>;
    const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5;
    for (int ly = warp + 2; ly < TY + 2 * HX - 2; ly += NW) {
#pragma unroll 1
        for (int j = 0; j < 2; ++j) {
            const int lx = 2 * lane + j, gx = x0 - HX + lx, gy = y0 - HX + ly;
            const uint32_t o = (uint32_t)ly * kRow + (uint32_t)lx * 4u, i = cidx(gx, gy, q.W, q.H);
            const float4 fC = make_float4(mld(S, o + M::X), mld(S, o + M::Y), mld(S, o + M::Z), mld(S, o + M::F));
            const FlowOut v = flow_cell_general(
                p, fC, mld(S, o + M::Z - 4), mld(S, o + M::F + kRow), mld(S, o + M::X + 4), mld(S, o + M::Y - kRow),
                mld(S, o + M::F - kRow), q.w_in[i] + q.rain[i], mld(S, o + M::H), q.s_in[i], mld(S, o + M::H - 4),
                mld(S, o + M::H + 4), mld(S, o + M::H + kRow), mld(S, o + M::H - kRow));
            mst(S, o + M::W, v.ux);
            mst(S, o + M::V, v.uy);
            mst(S, o + M::S, v.s1);
            if (lx >= HX && lx < 64 - HX && ly >= HX && ly < TY + HX && gx < q.W && gy < q.H) {
                const uint32_t g = (uint32_t)gy * (uint32_t)q.W + (uint32_t)gx;
                q.h_out[g] = v.hn;
                q.w_out[g] = fmaxf(0.0f, v.wn - (fminf(v.wn, 20.0f) * p.evap) * p.dt);
                if (!FUSED) {
                    q.s1_out[g] = v.s1;
                    q.vel_out[g] = make_float2(v.ux, v.uy);
                }
            }
        }
    }
}

template <int TY, int NW, bool FUSED, bool VEC>
__device__ __forceinline__ void tile_body(const TileParams &tp, const HydroWorld &q, char *S, int x0, int y0)
{
    constexpr int HX = FUSED ? 4 : 2;
    using M = TileMem<TY, HX>;
    const PairConst &c = tp.c;
    const int W = q.W, H = q.H;
    const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5, col = 2 * lane;
    const uint32_t Sa = (uint32_t)__cvta_generic_to_shared(S);
    const uint32_t c0 = (uint32_t)wrapc(x0 - HX + col, W), c1 = VEC ? c0 + 1 : (uint32_t)wrapc(x0 - HX + 1 + col, W);
    const int iw = min(64 - 2 * HX, W - x0), ih = min(TY, H - y0);
    const bool in0 = col >= HX && col < iw + HX, in1 = col >= HX && col + 1 < iw + HX;
    const bool live_f = col < iw + 2 * HX - 1, live_w = col >= 2 && col < iw + 2 * HX - 2;
    const uint32_t L = (uint32_t)lane * 8u;
    const uint32_t B = (uint32_t)y0 * (uint32_t)W + (uint32_t)(x0 - HX + col);  // global offset of row y0, this pair

    // every load of the tile
#pragma unroll 2
    for (int ly = warp; ly < TY + 2 * HX; ly += NW) {
        const uint32_t g = (uint32_t)wrapc(y0 - HX + ly, H) * (uint32_t)W, d = Sa + (uint32_t)ly * kRow + L;
        cp_pair<VEC>(d + M::H, q.h_in + g, c0, c1);
        cp_pair<VEC>(d + M::W, q.w_in + g, c0, c1);
        cp_pair<VEC>(d + M::V, q.rain + g, c0, c1);
        if (ly >= 2 && ly < TY + 2 * HX - 2) cp_pair<VEC>(d + M::S, q.s_in + g, c0, c1);
        if (ly >= 1 && ly < TY + 2 * HX - 1) {
            const char *f0 = reinterpret_cast<const char *>(q.f_in + g + c0), *f1 = reinterpret_cast<const char *>(q.f_in + g + c1);
            cp8(d + M::X, f0);
            cp8(d + M::Y, f0 + 8);
            cp8(d + M::Z, f1);
            cp8(d + M::F, f1 + 8);
        }
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    for (int ly = warp; ly < TY + 2 * HX; ly += NW) {
        const uint32_t o = (uint32_t)ly * kRow + L;
        st2(S, o + M::W, add2(ld2(S, o + M::W), ld2(S, o + M::V)));
    }
    __syncthreads();

    // flux on all rows but the first and the last
    bool bad = false;
    if (tp.ieee) {
        flux_rows_ieee<TY, NW, HX, true>(tp.p, q, S, x0, y0);
        __syncthreads();
    } else {
#pragma unroll 1
        for (int ly = warp + 1; ly < TY + 2 * HX - 1; ly += NW) {
            const uint32_t o = (uint32_t)ly * kRow + L;
            const f2 f0 = ld2(S, o + M::X), f1 = ld2(S, o + M::Y), f2_ = ld2(S, o + M::Z), f3 = ld2(S, o + M::F);
            Flux2 v;
            const bool b = flux_pair(c, ld2(S, o + M::H), ld2(S, o + M::W), mld(S, o + M::H - 4), mld(S, o + M::H + 8),
                                     mld(S, o + M::W - 4), mld(S, o + M::W + 8), ld2(S, o + M::H + kRow),
                                     ld2(S, o + M::W + kRow), ld2(S, o + M::H - kRow), ld2(S, o + M::W - kRow),
                                     make_float4(lo(f0), hi(f0), lo(f1), hi(f1)), make_float4(lo(f2_), hi(f2_), lo(f3), hi(f3)),
                                     live_f, v);
            bad = bad || b;
            st2(S, o + M::X, v.x);
            st2(S, o + M::Y, v.y);
            st2(S, o + M::Z, v.z);
            st2(S, o + M::F, v.w);
            const bool row = (unsigned)(ly - HX) < (unsigned)ih;
            gst_flux<VEC>(q.f_out, B + (uint32_t)(ly - HX) * (uint32_t)W, v.x, v.y, v.z, v.w, row && in0, row && in1);
        }
        if (__syncthreads_or(bad)) {
            flux_rows_ieee<TY, NW, HX, false>(tp.p, q, S, x0, y0);
            __syncthreads();
        }
    }

    // flow, sediment exchange and evaporation on all but two at either end
    bad = false;
#pragma unroll 1
    for (int ly = warp + 2; ly < TY + 2 * HX - 2; ly += NW) {
        const uint32_t o = (uint32_t)ly * kRow + L;
        const Flux2 b{ld2(S, o + M::X), ld2(S, o + M::Y), ld2(S, o + M::Z), ld2(S, o + M::F)};
        Flow2 v;
        const bool x = flow_pair(c, b, mld(S, o + M::Z - 4), mld(S, o + M::X + 8), ld2(S, o + M::F + kRow),
                                 ld2(S, o + M::Y - kRow), ld2(S, o + M::F - kRow), ld2(S, o + M::W), ld2(S, o + M::H),
                                 mld(S, o + M::H - 4), mld(S, o + M::H + 8), ld2(S, o + M::H + kRow),
                                 ld2(S, o + M::H - kRow), ld2(S, o + M::S), live_w, v);
        bad = bad || x;
        if (FUSED) {
            st2(S, o + M::W, v.ux);
            st2(S, o + M::V, v.uy);
            st2(S, o + M::S, v.s1);
        }
        const bool row = (unsigned)(ly - HX) < (unsigned)ih, s0 = row && in0, s1 = row && in1;
        const uint32_t g = B + (uint32_t)(ly - HX) * (uint32_t)W;
        gst2<VEC>(q.h_out, g, v.hn, s0, s1);
        gst2<VEC>(q.w_out, g, evaporate2(c, v.wn), s0, s1);
        if (!FUSED) {
            gst2<VEC>(q.s1_out, g, v.s1, s0, s1);
            if (s0) q.vel_out[g] = make_float2(lo(v.ux), lo(v.uy));
            if (s1) q.vel_out[g + 1] = make_float2(hi(v.ux), hi(v.uy));
        }
    }
    if (__syncthreads_or(bad)) {
        flow_rows_ieee<TY, NW, FUSED>(tp.p, q, S, x0, y0);
        __syncthreads();
    }
    kernel_release();
    if (!FUSED) return;

    // transport (:2572-2585, bilinear with wrap, cuda_helper.cuh:48-65) on rows 4 .. TY + 3.  The byte offset
    // of a tap's cell is its floored row * 256 + column * 4 from the tile's corner; the floors come as the
    // bits of 1.5 x 2^23 + floor.  A tap offset is in [-2, 1] by the velocity clamp; the minimum keeps any
    // other inside the array.
    const f2 gx = pk((float)(x0 - 4 + col), (float)(x0 - 3 + col));
    const uint32_t tap_c = 0u - ((0x4B400000u + (uint32_t)(y0 - 4)) << 8) - ((0x4B400000u + (uint32_t)(x0 - 4)) << 2);
    constexpr uint32_t kLast = M::A - kRow - 8;
#pragma unroll 1
    for (int ly = warp + 4; ly < ih + 4; ly += NW) {
        const uint32_t o = (uint32_t)ly * kRow + L;
        const f2 px = sub2(gx, mul2_z(ld2(S, o + M::W), c.dt, c.Z));
        const f2 py = sub2(dup2((float)(y0 - 4 + ly)), mul2_z(ld2(S, o + M::V), c.dt, c.Z));
        const f2 tx = add2_rm(px, c.M), ty = add2_rm(py, c.M);
        const f2 wx = sub2(px, sub2(tx, c.M)), wy = sub2(py, sub2(ty, c.M));
        const f2 vx = sub2(c.one, wx), vy = sub2(c.one, wy);
        const uint32_t t0 = min(tap_c + (__float_as_uint(lo(ty)) << 8) + (__float_as_uint(lo(tx)) << 2), kLast);
        const uint32_t t1 = min(tap_c + (__float_as_uint(hi(ty)) << 8) + (__float_as_uint(hi(tx)) << 2), kLast);
        const char *u = S + M::S + t0, *v = S + M::S + t1;
        const f2 I0 = add2(mul2_z(vx, pk(mld(u, 0), mld(v, 0)), c.Z), mul2_z(wx, pk(mld(u, 4), mld(v, 4)), c.Z));
        const f2 I1 = add2(mul2_z(vx, pk(mld(u, kRow), mld(v, kRow)), c.Z),
                           mul2_z(wx, pk(mld(u, kRow + 4), mld(v, kRow + 4)), c.Z));
        gst2<VEC>(q.s_out, B + (uint32_t)(ly - HX) * (uint32_t)W, add2(mul2_z(vy, I0, c.Z), mul2_z(wy, I1, c.Z)), in0, in1);
    }
}

template <int TY, int NW, int MINB, bool FUSED>
__global__ __launch_bounds__(NW * 32, MINB) void k_hydro(const __grid_constant__ TileParams tp)
{
    extern __shared__ float4 tile_smem[];
    __shared__ HydroWorld s_q;
    __shared__ int s_xy[2];
    char *S = reinterpret_cast<char *>(tile_smem);
    if (threadIdx.x == 0) {
        int wi, tx, ty;
        tile_of(tp.p.tiles[blockIdx.x], &wi, &tx, &ty);
        s_q = hydro_world(tp.p, tp.p.worlds[wi]);
        s_xy[0] = tx * (FUSED ? HTX : HTXS);
        s_xy[1] = ty * TY;
    }
    __syncthreads();
    kernel_wait();
    if (s_q.W & 1) tile_body<TY, NW, FUSED, false>(tp, s_q, S, s_xy[0], s_xy[1]);
    else tile_body<TY, NW, FUSED, true>(tp, s_q, S, s_xy[0], s_xy[1]);
}

// ---- two sub-iterations on one tile ------------------------------------------------------------------
//
// Where the launches and the latency of the phases are the time (small worlds), a tile of 64 columns takes two
// sub-iterations at once: a halo of 6 instead of 4, 52 columns inside, and nothing but the second's results
// leaves the block.  Four phases between barriers: the first's flux; its flow; its transport together with the
// second's flux; the second's flow; then the second's transport.
// One sub-iteration as the two of a launch, us: 256^2 5.7 -> 3.5, 512^2 9.6 -> 7.4, 1001x613 17 -> 14.8; the
// launch and the loads come once for two, against 1.7 to 2.3 times the cells inside (1.5 to 2.1 with a halo of
// 4).  The shapes differ in rows, warps and tiles an SM holds; default_hydro_variant chooses by the waves.
constexpr int HTX2 = 52;

// Byte layout as TileMem's, with 12 rows of halo; rain of its own (the second adds it too), and the height
// and water the second starts from.  The first's transported sediment takes the place of its height.
template <int TY>
struct TwoMem {
    static constexpr int rows = TY + 12;
    static constexpr uint32_t A = rows * kRow;
    static constexpr uint32_t H = kGuard, W = H + A, S = W + A, X = S + A, Y = X + A, Z = Y + A, F = Z + A, V = F + A,
                              R = V + A, H2 = R + A, W2 = H2 + A;
    static constexpr uint32_t bytes = W2 + A + kGuard;
};

// The flux of the pair at byte o from heights at h and water at w, fluxes from o + x0 .. on.
template <bool IEEE>
__device__ __forceinline__ bool two_flux(const TileParams &tp, const char *S, uint32_t h, uint32_t w, float4 fa,
                                         float4 fb, bool mine, Flux2 &v)
{
    if constexpr (IEEE) {
        float4 u[2];
#pragma unroll
        for (uint32_t c = 0; c < 8; c += 4)
            u[c >> 2] = flux_ieee(tp.p, c ? fb : fa, mld(S, h + c), mld(S, w + c), mld(S, h + c - 4), mld(S, w + c - 4),
                                  mld(S, h + c + kRow), mld(S, w + c + kRow), mld(S, h + c + 4), mld(S, w + c + 4),
                                  mld(S, h + c - kRow), mld(S, w + c - kRow));
        v = Flux2{pk(u[0].x, u[1].x), pk(u[0].y, u[1].y), pk(u[0].z, u[1].z), pk(u[0].w, u[1].w)};
        return false;
    }
    return flux_pair(tp.c, ld2(S, h), ld2(S, w), mld(S, h - 4), mld(S, h + 8), mld(S, w - 4), mld(S, w + 8),
                     ld2(S, h + kRow), ld2(S, w + kRow), ld2(S, h - kRow), ld2(S, w - kRow), fa, fb, mine, v);
}

// The flow of the pair whose fluxes lie at x, y, z, f, with the height at h, water at w and sediment sd.
template <bool IEEE>
__device__ __forceinline__ bool two_flow(const TileParams &tp, const char *S, uint32_t x, uint32_t y, uint32_t z,
                                         uint32_t f, uint32_t h, uint32_t w, f2 sd, bool mine, Flow2 &v)
{
    if constexpr (IEEE) {
        FlowOut u[2];
#pragma unroll
        for (uint32_t c = 0; c < 8; c += 4)
            u[c >> 2] = flow_cell_general(
                tp.p, make_float4(mld(S, x + c), mld(S, y + c), mld(S, z + c), mld(S, f + c)), mld(S, z + c - 4),
                mld(S, f + c + kRow), mld(S, x + c + 4), mld(S, y + c - kRow), mld(S, f + c - kRow), mld(S, w + c),
                mld(S, h + c), c ? hi(sd) : lo(sd), mld(S, h + c - 4), mld(S, h + c + 4), mld(S, h + c + kRow),
                mld(S, h + c - kRow));
        v = Flow2{pk(u[0].hn, u[1].hn), pk(u[0].wn, u[1].wn), pk(u[0].s1, u[1].s1), pk(u[0].ux, u[1].ux),
                  pk(u[0].uy, u[1].uy)};
        return false;
    }
    const Flux2 b{ld2(S, x), ld2(S, y), ld2(S, z), ld2(S, f)};
    return flow_pair(tp.c, b, mld(S, z - 4), mld(S, x + 8), ld2(S, f + kRow), ld2(S, y - kRow), ld2(S, f - kRow),
                     ld2(S, w), ld2(S, h), mld(S, h - 4), mld(S, h + 8), ld2(S, h + kRow), ld2(S, h - kRow), sd, mine, v);
}

// The sediment that reaches the pair with velocity (ux, uy) at the columns gx and the row gy: taps around the
// bytes t0, t1 that the floored position 0 stands for, in the array of `size` bytes at S.
__device__ __forceinline__ f2 two_transport(const PairConst &c, const char *S, uint32_t size, f2 ux, f2 uy, f2 gx, float gy,
                                            uint32_t t0, uint32_t t1)
{
    const f2 px = sub2(gx, mul2_z(ux, c.dt, c.Z)), py = sub2(dup2(gy), mul2_z(uy, c.dt, c.Z));
    const f2 tx = add2_rm(px, c.M), ty = add2_rm(py, c.M);
    const f2 wx = sub2(px, sub2(tx, c.M)), wy = sub2(py, sub2(ty, c.M));
    const f2 vx = sub2(c.one, wx), vy = sub2(c.one, wy);
    // a tap offset is in [-2, 1] by the velocity clamp; the minimum keeps any other inside the array
    const uint32_t last = size - kRow - 8;
    const char *u = S + min(t0 + (__float_as_uint(lo(ty)) << 8) + (__float_as_uint(lo(tx)) << 2), last);
    const char *v = S + min(t1 + (__float_as_uint(hi(ty)) << 8) + (__float_as_uint(hi(tx)) << 2), last);
    const f2 I0 = add2(mul2_z(vx, pk(mld(u, 0), mld(v, 0)), c.Z), mul2_z(wx, pk(mld(u, 4), mld(v, 4)), c.Z));
    const f2 I1 = add2(mul2_z(vx, pk(mld(u, kRow), mld(v, kRow)), c.Z), mul2_z(wx, pk(mld(u, kRow + 4), mld(v, kRow + 4)), c.Z));
    return add2(mul2_z(vy, I0, c.Z), mul2_z(wy, I1, c.Z));
}

// True where an operand of this thread left the packed ranges (IEEE: never).
template <int TY, int NW, bool VEC, bool IEEE>
__device__ __forceinline__ bool two_body(const TileParams &tp, const HydroWorld &q, char *S, int x0, int y0)
{
    using M = TwoMem<TY>;
    const PairConst &c = tp.c;
    const int W = q.W, H = q.H;
    const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5, col = 2 * lane;
    const uint32_t Sa = (uint32_t)__cvta_generic_to_shared(S);
    const uint32_t c0 = (uint32_t)wrapc(x0 - 6 + col, W), c1 = VEC ? c0 + 1 : (uint32_t)wrapc(x0 - 5 + col, W);
    const int iw = min(HTX2, W - x0), ih = min(TY, H - y0);
    const bool in0 = col >= 6 && col < iw + 6, in1 = col >= 6 && col + 1 < iw + 6;
    const uint32_t L = (uint32_t)lane * 8u;
    const uint32_t B = (uint32_t)y0 * (uint32_t)W + (uint32_t)(x0 - 6 + col);  // global offset of row y0, this pair

#pragma unroll 2
    for (int ly = warp; ly < M::rows; ly += NW) {
        const uint32_t g = (uint32_t)wrapc(y0 - 6 + ly, H) * (uint32_t)W, d = Sa + (uint32_t)ly * kRow + L;
        cp_pair<VEC>(d + M::H, q.h_in + g, c0, c1);
        cp_pair<VEC>(d + M::W, q.w_in + g, c0, c1);
        cp_pair<VEC>(d + M::R, q.rain + g, c0, c1);
        if (ly >= 2 && ly < M::rows - 2) cp_pair<VEC>(d + M::S, q.s_in + g, c0, c1);
        if (ly >= 1 && ly < M::rows - 1) {
            const char *f0 = reinterpret_cast<const char *>(q.f_in + g + c0), *f1 = reinterpret_cast<const char *>(q.f_in + g + c1);
            cp8(d + M::X, f0);
            cp8(d + M::Y, f0 + 8);
            cp8(d + M::Z, f1);
            cp8(d + M::F, f1 + 8);
        }
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    for (int ly = warp; ly < M::rows; ly += NW) {
        const uint32_t o = (uint32_t)ly * kRow + L;
        st2(S, o + M::W, add2(ld2(S, o + M::W), ld2(S, o + M::R)));
    }
    __syncthreads();

    // the first's flux
    bool bad = false;
#pragma unroll 1
    for (int ly = warp + 1; ly < M::rows - 1; ly += NW) {
        const uint32_t o = (uint32_t)ly * kRow + L;
        const f2 a = ld2(S, o + M::X), b = ld2(S, o + M::Y), d = ld2(S, o + M::Z), e = ld2(S, o + M::F);
        Flux2 v;
        const bool x = two_flux<IEEE>(tp, S, o + M::H, o + M::W, make_float4(lo(a), hi(a), lo(b), hi(b)),
                                      make_float4(lo(d), hi(d), lo(e), hi(e)), col < iw + 11, v);
        bad = bad || x;
        st2(S, o + M::X, v.x);
        st2(S, o + M::Y, v.y);
        st2(S, o + M::Z, v.z);
        st2(S, o + M::F, v.w);
    }
    __syncthreads();

    // the first's flow, sediment exchange and evaporation, and the second's rain
#pragma unroll 1
    for (int ly = warp + 2; ly < M::rows - 2; ly += NW) {
        const uint32_t o = (uint32_t)ly * kRow + L;
        Flow2 v;
        const bool x = two_flow<IEEE>(tp, S, o + M::X, o + M::Y, o + M::Z, o + M::F, o + M::H, o + M::W,
                                      ld2(S, o + M::S), col >= 2 && col < iw + 10, v);
        bad = bad || x;
        st2(S, o + M::W, v.ux);
        st2(S, o + M::V, v.uy);
        st2(S, o + M::S, v.s1);
        st2(S, o + M::H2, v.hn);
        st2(S, o + M::W2, add2(evaporate2(c, v.wn), ld2(S, o + M::R)));
    }
    __syncthreads();

    // the first's transport, at the positions of the world's own rows and columns, and the second's flux
    const f2 gx = pk((float)(int)c0, (float)(int)c1);
    const uint32_t zero = 0u - (0x4B400000u << 8) - (0x4B400000u << 2);
#pragma unroll 1
    for (int ly = warp + 3; ly < M::rows - 3; ly += NW) {
        const uint32_t o = (uint32_t)ly * kRow + L;
        if (ly >= 4 && ly < M::rows - 4) {
            const int gy = wrapc(y0 - 6 + ly, H);
            const uint32_t t = zero + ((uint32_t)(ly - gy) << 8) + ((uint32_t)col << 2);
            st2(S, o + M::H, two_transport(c, S + M::S, M::A, ld2(S, o + M::W), ld2(S, o + M::V), gx, (float)gy, t - (c0 << 2),
                                           t + 4u - (c1 << 2)));
        }
        const f2 a = ld2(S, o + M::X), b = ld2(S, o + M::Y), d = ld2(S, o + M::Z), e = ld2(S, o + M::F);
        Flux2 v;
        const bool x = two_flux<IEEE>(tp, S, o + M::H2, o + M::W2, make_float4(lo(a), lo(b), lo(d), lo(e)),
                                      make_float4(hi(a), hi(b), hi(d), hi(e)), col >= 2 && col < iw + 9, v);
        bad = bad || x;
        st2(S, o + M::X, v.x);
        st2(S, o + M::Y, v.y);
        st2(S, o + M::Z, v.z);
        st2(S, o + M::F, v.w);
        const bool row = (unsigned)(ly - 6) < (unsigned)ih;
        gst_flux<VEC>(q.f_out, B + (uint32_t)(ly - 6) * (uint32_t)W, v.x, v.y, v.z, v.w, row && in0, row && in1);
    }
    __syncthreads();

    // the second's flow, sediment exchange and evaporation
#pragma unroll 1
    for (int ly = warp + 4; ly < M::rows - 4; ly += NW) {
        const uint32_t o = (uint32_t)ly * kRow + L;
        Flow2 v;
        const bool x = two_flow<IEEE>(tp, S, o + M::X, o + M::Y, o + M::Z, o + M::F, o + M::H2, o + M::W2,
                                      ld2(S, o + M::H), col >= 4 && col < iw + 8, v);
        bad = bad || x;
        st2(S, o + M::W, v.ux);
        st2(S, o + M::V, v.uy);
        st2(S, o + M::S, v.s1);
        const bool row = (unsigned)(ly - 6) < (unsigned)ih, s0 = row && in0, s1 = row && in1;
        const uint32_t g = B + (uint32_t)(ly - 6) * (uint32_t)W;
        gst2<VEC>(q.h_out, g, v.hn, s0, s1);
        gst2<VEC>(q.w_out, g, evaporate2(c, v.wn), s0, s1);
    }
    __syncthreads();
    kernel_release();

    // the second's transport
    const f2 hx = pk((float)(x0 - 6 + col), (float)(x0 - 5 + col));
    const uint32_t t = zero - ((uint32_t)(y0 - 6) << 8) - ((uint32_t)(x0 - 6) << 2);
#pragma unroll 1
    for (int ly = warp + 6; ly < ih + 6; ly += NW) {
        const uint32_t o = (uint32_t)ly * kRow + L;
        const f2 v = two_transport(c, S + M::S, M::A, ld2(S, o + M::W), ld2(S, o + M::V), hx, (float)(y0 - 6 + ly), t, t);
        gst2<VEC>(q.s_out, B + (uint32_t)(ly - 6) * (uint32_t)W, v, in0, in1);
    }
    return bad;
}

template <int TY, int NW>
__device__ __noinline__ void two_ieee(const TileParams &tp, const HydroWorld &q, char *S, int x0, int y0)
{
    two_body<TY, NW, false, true>(tp, q, S, x0, y0);
}

template <int TY, int NW, int MINB>
__global__ __launch_bounds__(NW * 32, MINB) void k_hydro_two(const __grid_constant__ TileParams tp)
{
    extern __shared__ float4 tile_smem[];
    __shared__ HydroWorld s_q;
    __shared__ int s_xy[2];
    char *S = reinterpret_cast<char *>(tile_smem);
    if (threadIdx.x == 0) {
        int wi, tx, ty;
        tile_of(tp.p.tiles[blockIdx.x], &wi, &tx, &ty);
        s_q = hydro_world(tp.p, tp.p.worlds[wi]);
        s_xy[0] = tx * HTX2;
        s_xy[1] = ty * TY;
    }
    __syncthreads();
    kernel_wait();
    const bool bad = s_q.W & 1 ? two_body<TY, NW, false, false>(tp, s_q, S, s_xy[0], s_xy[1])
                               : two_body<TY, NW, true, false>(tp, s_q, S, s_xy[0], s_xy[1]);
    // an operand outside the packed ranges: the tile once more in scalar form, from the same inputs
    if (__syncthreads_or(bad)) two_ieee<TY, NW>(tp, s_q, S, s_xy[0], s_xy[1]);
}

// The step's rain increment (:2430-2437 with the seed of plate_tectonic_sim.cu:338), over the
// hydraulic work list (tiles of 64 x ty cells).
__global__ void k_rain(const WorldDev *worlds, const uint2 *tiles, int ty_cells, float dt, float rainfall)
{
    kernel_wait();
    int wi, tx, ty;
    tile_of(tiles[blockIdx.x], &wi, &tx, &ty);
    const WorldDev &wd = worlds[wi];
    const int seed = (int)(wd.ctl->seed + wd.ctl->iteration);
    for (int e = threadIdx.x; e < HTX * ty_cells; e += blockDim.x) {
        const int oy = e / HTX, ox = e - oy * HTX;
        const int x = tx * HTX + ox, y = ty * ty_cells + oy;
        if (x < wd.W && y < wd.H)
            wd.rain[(size_t)y * wd.W + x] = (fmaxf(0.0f, rain_noise(x, y, seed)) * dt) * rainfall;
    }
}

// Split path: transport as a gather from global memory (any dt), over the hydraulic work list.
__global__ __launch_bounds__(256) void k_transport(const WorldDev *worlds, const uint2 *tiles, int ty_cells,
                                                   int cur_wsf, float dt)
{
    kernel_wait();
    int wi, tx, ty;
    tile_of(tiles[blockIdx.x], &wi, &tx, &ty);
    const WorldDev &wd = worlds[wi];
    const int W = wd.W, H = wd.H;
    const float *s1 = wd.s1;
    float *s_out = wd.s[cur_wsf ^ 1];
    for (int e = threadIdx.x; e < HTX * ty_cells; e += blockDim.x) {
        const int oy = e / HTX, ox = e - oy * HTX;
        const int x = tx * HTX + ox, y = ty * ty_cells + oy;
        if (x >= W || y >= H) continue;
        const size_t i = (size_t)y * W + x;
        const float2 v = wd.vel[i];
        const float px = (float)x - v.x * dt, py = (float)y - v.y * dt;
        const int ix0 = (int)floorf(px), iy0 = (int)floorf(py);
        const float wx = px - (float)ix0, wy = py - (float)iy0;
        const int xa = wrap_fast(ix0, W), xb = wrap_fast(ix0 + 1, W);
        const float *ra = s1 + (uint32_t)(wrap_fast(iy0, H) * W), *rb = s1 + (uint32_t)(wrap_fast(iy0 + 1, H) * W);
        const float I0 = (1.0f - wx) * ra[xa] + wx * ra[xb];
        const float I1 = (1.0f - wx) * rb[xa] + wx * rb[xb];
        s_out[i] = (1.0f - wy) * I0 + wy * I1;
    }
}

// Tile variants (tecto_step_settings::hydraulicTile 1 .. 7): 56 x TY cells, NW warps, MINB blocks per SM.
struct HydroVariant {
    int ty, nt;
    size_t smem, smem_split;
    void (*fused)(TileParams);
    void (*split)(TileParams);
    int ty2, nt2;  // two sub-iterations at once, 52 x ty2 cells (0: never)
    size_t smem2;
    void (*two)(TileParams);
};
#define TECTO_HYDRO_VARIANT(TY, NW, MINB) \
    TY, NW * 32, TileMem<TY, 4>::bytes, TileMem<TY, 2>::bytes, k_hydro<TY, NW, MINB, true>, k_hydro<TY, NW, MINB, false>
#define TECTO_HYDRO_TWO(TY, NW, MINB) TY, NW * 32, TwoMem<TY>::bytes, k_hydro_two<TY, NW, MINB>
const HydroVariant kHydroVariants[7] = {
    {TECTO_HYDRO_VARIANT(8, 16, 2), TECTO_HYDRO_TWO(9, 20, 1)},
    {TECTO_HYDRO_VARIANT(8, 8, 4), TECTO_HYDRO_TWO(12, 8, 3)},
    {TECTO_HYDRO_VARIANT(16, 8, 4), TECTO_HYDRO_TWO(24, 16, 2)},
    {TECTO_HYDRO_VARIANT(24, 8, 3), TECTO_HYDRO_TWO(28, 12, 2)},
    {TECTO_HYDRO_VARIANT(32, 10, 2), TECTO_HYDRO_TWO(20, 12, 2)},
    {TECTO_HYDRO_VARIANT(16, 6, 4), 0, 0, 0, nullptr},
    {TECTO_HYDRO_VARIANT(4, 12, 2), 0, 0, 0, nullptr},
};
#undef TECTO_HYDRO_VARIANT
#undef TECTO_HYDRO_TWO
// The rain field and the split path of the marching variants run on the tiles of variant 4.
const HydroVariant &variant_of(int v) { return kHydroVariants[(v > 7 ? 4 : v) - 1]; }
}  // namespace

int hydro_tile_attributes()
{
    for (const HydroVariant &v : kHydroVariants) {
        TECTO_CUDA(cudaFuncSetAttribute(v.fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v.smem));
        TECTO_CUDA(cudaFuncSetAttribute(v.split, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v.smem_split));
        if (v.ty2) TECTO_CUDA(cudaFuncSetAttribute(v.two, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v.smem2));
    }
    return TECTO_OK;
}

void hydro_split_extent(int variant, int *tx, int *ty)
{
    *tx = HTXS;
    *ty = variant_of(variant).ty;
}

void hydro_tile_extent(int variant, bool two, int *tx, int *ty)
{
    const HydroVariant &v = variant_of(variant);
    two = two && v.ty2;
    *tx = two ? HTX2 : HTX;
    *ty = two ? v.ty2 : v.ty;
}

bool hydro_tile_two(const Batch &b, const HydroParams &p)
{
    return b.hydro_variant < kHydroStripVariant && variant_of(b.hydro_variant).ty2 && hydro_packed(p);
}

void launch_rain(const Batch &b, float dt, float rainfall, cudaStream_t st)
{
    launch_chained(k_rain, (unsigned)b.ntiles[TK_HYDRO], 256, 0, st, b.d_worlds, b.d_tiles[TK_HYDRO],
                   variant_of(b.hydro_variant).ty, dt, rainfall);
}

void launch_transport(const Batch &b, float dt, cudaStream_t st)
{
    launch_chained(k_transport, (unsigned)b.ntiles[TK_HYDRO], 256, 0, st, b.d_worlds, b.d_tiles[TK_HYDRO],
                   variant_of(b.hydro_variant).ty, b.cur_wsf, dt);
}

void launch_hydro_tile(const Batch &b, const HydroParams &p, bool fused, bool two, cudaStream_t st)
{
    const HydroVariant &v = variant_of(b.hydro_variant);
    TileParams tp{};
    tp.p = p;
    tp.c = pair_const(p);
    tp.ieee = !hydro_packed(p);
    if (two) {
        tp.p.tiles = b.d_tiles[TK_HYDRO_TWO];
        launch_chained(v.two, (unsigned)b.ntiles[TK_HYDRO_TWO], v.nt2, v.smem2, st, tp);
        return;
    }
    if (!fused) tp.p.tiles = b.d_tiles[TK_HYDRO_SPLIT];
    launch_chained(fused ? v.fused : v.split, (unsigned)b.ntiles[fused ? TK_HYDRO : TK_HYDRO_SPLIT], v.nt,
                   fused ? v.smem : v.smem_split, st, tp);
}

}  // namespace tecto
