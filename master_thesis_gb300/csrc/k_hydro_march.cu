// k_hydro_march.cu - the hydraulic sub-iteration as a persistent march down column strips, two cells
// per thread.
// Reference: rain/flux/flow/sediment/transport/evaporate,
// src/cuda_compute/plate_tectonics_kernel.cu:2430-2593; driver plate_tectonic_sim.cu:331-373.
//
// The same sub-iteration as k_hydro (k_hydro_tile.cu), with no row of the vertical halo computed twice.
// A block of 256 threads owns a column strip of a world (up to kMarchInner = 120 interior columns, 128
// with the halo of 4 on each side) and marches down its rows, 4 rows per chunk; a thread owns two
// adjacent cells of one row (64 pairs a row, a warp is half a row).  With r its first row, a chunk
// computes
//   the flux of rows r+7 .. r+10,
//   the flow, the sediment exchange and the evaporation of rows r+2 .. r+5,
//   the transport of rows r-4 .. r-1,
// each from what earlier chunks left in shared memory, so the three are independent of each other (one
// block barrier per chunk, and the latencies of one hidden by the others).  The height, water and rain
// of rows r+12 .. r+15 are loaded into registers at the chunk's start and go to shared memory at its
// end; the old flux and the sediment of the next chunk are loaded where the current ones were used up.
// Two cells a thread and packed arithmetic take 523 warp-instructions per 64 cells where one cell a
// thread took 1036; two blocks of up to 128 registers per SM (three blocks of 80 wait on the shared-memory
// pipe: 990 against 762 us).  One sub-iteration, before and after, us: 2048^2 93.9 -> 72, 4096^2
// 303 -> 232, 8192^2 1120 -> 852 (4.8 TB/s of DRAM traffic), the 49.7 M cell batch 966 -> 759; with the
// global accesses taken out 58 / 635 / 566 at 2048^2 / 8192^2 / the batch, so it is bound by issue and
// shared-memory latency with DRAM close behind.  Two at once: 52 / 703 / 647 (k_hydro_march_pair).
// Rows live in rings of 16 rows indexed by the march's own row number (a chunk touches at most 15
// consecutive rows of a ring).  A piece of a strip starts with three chunks of warm-up; every chunk
// runs all three stages, and only the stores are limited to the piece's rows.  All strip-rows of the
// batch are laid end to end and each block takes one contiguous range of them.
// Two sub-iterations go through one march where an even number is left (k_hydro_march_pair).
//
// The per-cell arithmetic is k_hydro's, operation for operation, two cells at a time in packed
// instructions (pair.cuh).  The packed path holds for operands inside the ranges of the engine's own
// quotients and roots.  A thread with an operand outside them flags its chunk, and when the piece is
// done the block runs the rows that the flagged chunks reach once more in the scalar IEEE form, whose
// results are the same bits wherever the packed form holds (inputs and outputs are different buffers,
// so a second run of a row starts from the same inputs).  Of two sub-iterations in a world of even width a piece's
// chunks are flagged by up to 64 segments, so that two far apart do not send the rows between them too.  A flag costs
// its block some 30 rows in scalar form and a warm-up: two sub-iterations with no / 1 / 40 / 1000 such cells spread over
// the world, us: 2048^2 115 / 181 / 240 / 343, 8192^2 1525 / 1583 / 1732 / 2769 (one range from the first flag to the
// last: 313 and 2417 with 40; the tiles of variant 4, which repeat a tile: 165 / 165 / 187 / 302 and 2413 / 2413 / 2437 /
// 2603).
//
// Addressing.  A thread keeps one running value P = row * 512 + column * 4 (unsigned, wrapping); the
// byte offset of a ring cell is P & (ring bytes - 1) plus the ring's base and a constant column step.
// Lanes read their pair's neighbours without clamping: the edge lanes of a phase compute values that no
// later phase reads, and the guards around the rings keep every read inside the block's shared memory.
#include "hydro_pair.cuh"

namespace tecto {

namespace {

struct PairParams {
    StripParams sp;
    PairConst c;
};

constexpr int kPairThreads = 256;
constexpr int kPairRows = 4;       // rows per chunk
constexpr uint32_t kRing = 16;     // rows of a ring
constexpr uint32_t kRBytes = kRing * kMRow, kRMask = kRBytes - 1;
constexpr uint32_t kOH = kMGuard;          // height
constexpr uint32_t kOW = kOH + kRBytes;    // water + rain
constexpr uint32_t kOS = kOW + kRBytes;    // eroded sediment
constexpr uint32_t kOX = kOS + kRBytes;    // flux left, +y, right, -y
constexpr uint32_t kOY = kOX + kRBytes;
constexpr uint32_t kOZ = kOY + kRBytes;
constexpr uint32_t kOF = kOZ + kRBytes;
constexpr uint32_t kOVX = kOF + kRBytes;   // velocity
constexpr uint32_t kOVY = kOVX + kRBytes;
constexpr uint32_t kHydroMarchSmem = kOVY + kRBytes + kMGuard;
// two sub-iterations at once: a tenth ring to each set, the rain of the first and the sediment that the
// second takes from it; the second's set after the first's, its rows kLag behind
constexpr uint32_t kOE = kOVY + kRBytes;
constexpr uint32_t kSet = 10 * kRBytes;
constexpr uint32_t kHydroPairSmem = kOE + kRBytes + kSet + kMGuard;
constexpr int kLag = 10;
// What a piece costs beside its rows, in rows: its warm-up, of two also the second's lag, and its first loads.
// Of two, 16 / 26 / 36 / 48: 1024^2 20.9 / 19.1 / 18.9 / 19.1 us, the batch 672 / 655 / 648 / 657.
constexpr unsigned kWarmAlone = 24, kWarmRows = 36;
enum Role { kAlone = 0, kFirstOfTwo, kSecondOfTwo };
static_assert(kPairThreads / 64 == kPairRows && kHydroMarchSmem % 16 == 0, "march: one pair per thread and phase");

// Loads that stay where they are written (the march's prefetches): two cells of one row; VEC, adjacent
// and 8-byte aligned (even world width), else `step` apart; and one cell's flux.  Not the read-only path: a march
// is resident while the kernel ahead of it still writes these fields, and kernel_wait() makes them visible to
// ordinary loads.
template <bool VEC>
__device__ __forceinline__ f2 gld2(const float *base, uint32_t i, uint32_t step)
{
    if (VEC) {
        f2 v;
        asm volatile("ld.global.b64 %0, [%1];" : "=l"(v) : "l"(gaddr64(base, i)));
        return v;
    }
    float x, y;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(x) : "l"(gaddr64(base, i)));
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(y) : "l"(gaddr64(base, i + step)));
    return pk(x, y);
}
// the fluxes of two cells: VEC, one 32-byte access (a whole sector: two 16-byte halves of it, loaded or
// stored one after the other, cost twice the L1 and L2 requests)
template <bool VEC>
__device__ __forceinline__ void gld_flux(const float4 *base, uint32_t i, uint32_t step, float4 &a, float4 &b)
{
    if (VEC) {
        asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                     : "l"(gaddr64(base, i)));
        return;
    }
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w)
                 : "l"(gaddr64(base, i)));
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(gaddr64(base, i + step)));
}
// The flags of a piece, two shared words.  Two sub-iterations of an even width: the segments of its chunks kFirst ..
// K with an operand outside the packed ranges; chunk k is in segment (k - kFirst) >> shift, of 64 at most.  Odd widths,
// and a single sub-iteration: the first and the last such chunk, as the segment's arithmetic, in a branch that is
// hardly ever taken, changes how the loop compiles (20 sub-iterations, 2047x2048 1113 -> 1147 us, the 49.7 M cell batch
// 13.1 -> 13.9 ms; even widths 1052 -> 1042; one sub-iteration at 8192^2 978 -> 986).
struct Chunks {
    int first, last, shift;
};
__device__ __forceinline__ Chunks chunks_of(int nrows)
{
    const int first = -4, last = (nrows + kLag + kPairRows - 1) / kPairRows;
    return Chunks{first, last, max(0, 26 - __clz(last - first))};
}

__device__ __forceinline__ void clear_flags(unsigned *flagged, bool range)
{
    flagged[0] = range ? 0x7fffffffu : 0u;
    flagged[1] = range ? 0x80000000u : 0u;
}

// Runs the rows that the flagged chunks reach once more: `run(lo, hi)` for each range of rows.  A cell of a chunk
// whose first row is r reaches outputs r - back .. r + ahead - 1.
template <typename F>
__device__ __forceinline__ void rerun_range(const unsigned *flagged, int r0, int r1, int back, int ahead, F &&run)
{
    const int k0 = (int)flagged[0], k1 = (int)flagged[1];
    if (k1 >= k0) run(max(r0, r0 + kPairRows * k0 - back), min(r1, r0 + kPairRows * k1 + ahead));
}
// The same by segments; ranges closer than a run's warm-up are one.
template <typename F>
__device__ __forceinline__ void rerun_segments(const unsigned *flagged, int r0, int r1, int back, int ahead, F &&run)
{
    const Chunks c = chunks_of(r1 - r0);
    int lo = 0, hi = 0;
    for (unsigned long long m = (unsigned long long)flagged[1] << 32 | flagged[0]; m; m &= m - 1ull) {
        const int s = __ffsll((long long)m) - 1;
        const int a = max(r0, r0 + kPairRows * ((s << c.shift) + c.first) - back);
        const int b = min(r1, r0 + kPairRows * (((s + 1) << c.shift) - 1 + c.first) + ahead);
        if (a >= b) continue;
        if (hi > lo && a > hi + (int)kWarmRows) {
            run(lo, hi);
            lo = a;
        } else if (hi == lo) {
            lo = a;
        }
        hi = max(hi, b);
    }
    if (hi > lo) run(lo, hi);
}

// Rows [r0, r1) of the strip with interior columns [x0, x0 + iw) of world q.  VEC: the world's width is
// even.  IEEE: the scalar form, for any operands; else the packed form, which needs p.fastL, dt >= 0 and
// H >= 4, and flags in flagged[0], flagged[1] the chunks with an operand outside its ranges.  ROLE: a sub-iteration by itself, or the first or the second of two (k_hydro_march_pair).
template <bool VEC, bool IEEE, int ROLE>
__device__ __forceinline__ void march_piece(const HydroParams &p, const PairConst &c, const HydroWorld &q, char *S,
                                            int x0, int iw, int r0, int r1, unsigned *flagged)
{
    const int W = q.W, H = q.H;
    const uint32_t Wu = (uint32_t)W, N = Wu * (uint32_t)H, W4 = 4u * Wu;
    const f2 Z = c.Z;
    constexpr int HALO = ROLE ? 6 : 4, LAG = ROLE == kSecondOfTwo ? kLag : 0;
    constexpr uint32_t D = ROLE == kSecondOfTwo ? kSet : 0;
    constexpr uint32_t OH = kOH + D, OW = kOW + D, OS = kOS + D, OX = kOX + D, OY = kOY + D, OZ = kOZ + D, OF = kOF + D,
                       OVX = kOVX + D, OVY = kOVY + D;
    const int col = 2 * ((int)threadIdx.x & 63), rr = (int)threadIdx.x >> 6 & (kPairRows - 1);
    const uint32_t gcol = (uint32_t)wrapc(x0 - HALO + col, W);
    const uint32_t gstep = VEC ? 1u : (uint32_t)wrapc(x0 - HALO + 1 + col, W) - gcol;
    const int gxi = x0 + col - HALO;  // global column of the pair's first cell, interior columns
    // columns each stage covers: loads [0, iw+8), flux [1, iw+7), flow [2, iw+6), interior [4, iw+4).  Of two, the first
    // loads [0, iw+12): its flux covers [1, iw+11), its flow, whose height and water the second's flux needs,
    // [2, iw+10), its transport [4, iw+8); the second's flux [3, iw+9), flow [4, iw+8), interior [6, iw+6).
    // A warp with no such column only keeps the barriers; the others run all 32 lanes.
    const bool in0 = col >= HALO && col < iw + HALO, in1 = col >= HALO && col + 1 < iw + HALO;
    const bool live_f = ROLE == kFirstOfTwo ? col < iw + 11 : col >= HALO - 4 && col < iw + HALO + 3;
    const bool live_w = ROLE == kFirstOfTwo ? col >= 2 && col < iw + 10 : col >= HALO - 2 && col < iw + HALO + 2;
    const bool active = __any_sync(0xffffffffu, (col & ~63) < iw + 2 * HALO);
    const int K = (r1 - r0 + (ROLE ? kLag : 0) + kPairRows - 1) / kPairRows;
    const uint32_t nrows = (uint32_t)(r1 - r0);
    // rows the first of two gives to the second on each side
    constexpr int MORE = ROLE == kFirstOfTwo ? 2 : 0;
    // g + 4 rows, and g - 1 row, wrapped (g < N; the packed forms run where 4 rows are at most N)
    auto adv = [&](uint32_t g) -> uint32_t {
        if (IEEE) return (uint32_t)(((unsigned long long)g + 4ull * Wu) % N);
        const uint32_t v = g + W4;  // < 2N <= 2^31
        return min(v, v - N);
    };
    // Whether a stage's operands are loaded before the stage ahead stores its results.  Of two at once: 8192^2
    // 728 -> 712 us, 2048^2 54.1 -> 52.6, 1500x1100 25.5 -> 24.8; for odd widths it is the other way round (the
    // batch, half of its worlds odd, 653 without and 664 with it).
    constexpr bool EARLY = VEC && ROLE != kAlone;
    // Per chunk k (first row rk = r0 + 4k) this thread's base row is t = rk + rr and its items are rows
    // t + c: flux c = 7, flow c = 2, transport c = -4, and the loads c = 12 (height, water and rain),
    // c = 11 (old flux) and c = 6 (sediment).
    constexpr int kFirst = ROLE ? -4 : -3;  // of two as in chunks_of
    uint32_t P = (uint32_t)(r0 + kFirst * kPairRows - LAG + rr) * kMRow + (uint32_t)col * 4u;  // ring value of row t
    int tr = rr + kFirst * kPairRows - LAG;                                                    // t - r0
    uint32_t B = (uint32_t)(r0 + kFirst * kPairRows - LAG + rr) * Wu + (uint32_t)gxi;          // global offset of row t
    // Row t - 4 and the pair's columns as positions.  The first of two transports cells of the halo too, whose
    // positions are those of the world's own rows and columns: their taps are shifted back by what wrapping
    // took off.
    int yw = wrapc(r0 + (kFirst - 1) * kPairRows + rr, H);
    float fy = ROLE == kFirstOfTwo ? (float)yw : (float)(r0 + (kFirst - 1) * kPairRows - LAG + rr);
    const int gx0 = ROLE == kFirstOfTwo ? (int)gcol : gxi, gx1 = ROLE == kFirstOfTwo ? wrapc(gxi + 1, W) : gxi + 1;
    const f2 fgx = pk((float)gx0, (float)gx1);
    // ring value of the sediment tap of a floored position (fx, fy) is fy * 512 + (fx - x0 + halo) * 4;
    // the floors come as the bits of 1.5 x 2^23 + floor
    const uint32_t tap_c = 0u - (0x4B400000u << 9) - ((0x4B400000u + (uint32_t)(x0 - HALO)) << 2);
    uint32_t g = (uint32_t)wrapc(r0 + kFirst * kPairRows + 8 + rr, H) * Wu + gcol;    // height row t + 8, then t + 12 ahead
    uint32_t gs = (uint32_t)wrapc(r0 + kFirst * kPairRows - 2 + rr, H) * Wu + gcol;  // sediment row t - 2, then t + 2 ahead
    uint32_t gf = (uint32_t)wrapc(r0 + kFirst * kPairRows + 7 + rr, H) * Wu + gcol;   // flux row t + 7
    if (ROLE != kSecondOfTwo && active) {
        const uint32_t a = (P + 8 * kMRow) & kRMask;
        const f2 rain = gld2<VEC>(q.rain, g, gstep);
        st2(S, a + OH, gld2<VEC>(q.h_in, g, gstep));
        st2(S, a + OW, add2(gld2<VEC>(q.w_in, g, gstep), rain));
        if (ROLE == kFirstOfTwo) st2(S, a + kOE, rain);
        g = adv(g);
        gs = adv(gs);
    }
    f2 lh = 0, lw = 0, lr = 0, ns = 0;
    float4 fa, fb;  // old flux of this thread's two cells
    // the loads of the next chunk: its old flux (row t + 7), its sediment (t + 2), and the height, water
    // and rain that it puts into the rings at its end (t + 12)
    auto prefetch = [&]() {
        lh = gld2<VEC>(q.h_in, g, gstep);
        lw = gld2<VEC>(q.w_in, g, gstep);
        lr = gld2<VEC>(q.rain, g, gstep);
        ns = gld2<VEC>(q.s_in, gs, gstep);
        gld_flux<VEC>(q.f_in, gf, gstep, fa, fb);
        g = adv(g);
        gs = adv(gs);
        gf = adv(gf);
    };
    const auto barrier = [&]() {
        if constexpr (ROLE == kAlone) __syncthreads();
        else asm volatile("bar.sync 1, %0;" ::"n"(2 * kPairThreads) : "memory");  // both halves of the block
    };
    if (ROLE != kSecondOfTwo && active) prefetch();
    barrier();

#pragma unroll 1
    for (int k = kFirst; k <= K; ++k) {
        bool bad = false;  // an operand of this thread outside the packed path's ranges
        if (active && (ROLE != kSecondOfTwo || k >= 0)) {
            // ---- transport (:2572-2585): bilinear taps within two cells ----
            f2 sn;
            {
                const uint32_t pv = (P - 4 * kMRow) & kRMask;
                const f2 px = sub2(fgx, mul2_z(ld2(S, pv + OVX), c.dt, Z));
                const f2 py = sub2(dup2(fy), mul2_z(ld2(S, pv + OVY), c.dt, Z));
                const f2 tx = add2_rm(px, c.M), ty = add2_rm(py, c.M);
                const f2 wx = sub2(px, sub2(tx, c.M)), wy = sub2(py, sub2(ty, c.M));
                const f2 vx = sub2(c.one, wx), vy = sub2(c.one, wy);
                // a tap offset is in [-2, 1] by the velocity clamp; the mask keeps any other inside the ring
                uint32_t c0 = tap_c, c1 = tap_c;
                if (ROLE == kFirstOfTwo) {
                    const uint32_t row = P - 4 * kMRow - (uint32_t)col * 4u - ((uint32_t)yw << 9);
                    c0 += row + ((uint32_t)(gxi - gx0) << 2);
                    c1 += row + ((uint32_t)(gxi + 1 - gx1) << 2);
                }
                const uint32_t o0 = c0 + (__float_as_uint(lo(ty)) << 9) + (__float_as_uint(lo(tx)) << 2);
                const uint32_t o1 = c1 + (__float_as_uint(hi(ty)) << 9) + (__float_as_uint(hi(tx)) << 2);
                const uint32_t u0 = (o0 & kRMask) + OS, d0 = ((o0 + kMRow) & kRMask) + OS;
                const uint32_t u1 = (o1 & kRMask) + OS, d1 = ((o1 + kMRow) & kRMask) + OS;
                const f2 I0 = add2(mul2_z(vx, pk(mld(S, u0), mld(S, u1)), Z), mul2_z(wx, pk(mld(S, u0 + 4), mld(S, u1 + 4)), Z));
                const f2 I1 = add2(mul2_z(vx, pk(mld(S, d0), mld(S, d1)), Z), mul2_z(wx, pk(mld(S, d0 + 4), mld(S, d1 + 4)), Z));
                sn = add2(mul2_z(vy, I0, Z), mul2_z(wy, I1, Z));
            }
            // ---- flow, sediment exchange, evaporation ----
            uint32_t fa0, fau, fad;
            f2 sd;
            Flux2 fc;
            f2 fuw, fdy, fdw, fw, fh, fhu, fhd;
            float flz, frx, fhl, fhr;
            const auto load_flow = [&]() {
                fa0 = (P + 2 * kMRow) & kRMask, fau = (P + 3 * kMRow) & kRMask, fad = (P + kMRow) & kRMask;
                sd = ROLE == kSecondOfTwo ? ld2(S, fa0 + kOE + kSet) : ns;
                fc = Flux2{ld2(S, fa0 + OX), ld2(S, fa0 + OY), ld2(S, fa0 + OZ), ld2(S, fa0 + OF)};
                fuw = ld2(S, fau + OF), fdy = ld2(S, fad + OY), fdw = ld2(S, fad + OF);
                fw = ld2(S, fa0 + OW), fh = ld2(S, fa0 + OH), fhu = ld2(S, fau + OH), fhd = ld2(S, fad + OH);
                flz = mld(S, fa0 + OZ - 4), frx = mld(S, fa0 + OX + 8);
                fhl = mld(S, fa0 + OH - 4), fhr = mld(S, fa0 + OH + 8);
            };
            if (EARLY) load_flow();
            {
                const uint32_t pv = (P - 4 * kMRow) & kRMask;
                if (ROLE == kFirstOfTwo) {
                    st2(S, pv + kOE + kSet, sn);
                } else {
                    const bool row = (uint32_t)(tr - 4) < nrows;
                    gst2<VEC>(q.s_out, B - W4, sn, row && in0, row && in1);
                }
            }
            if (!EARLY) load_flow();
            f2 hn, wn, s_new, ux, uy;
            {
                if constexpr (IEEE) {
                    FlowOut v[2];
#pragma unroll
                    for (uint32_t c4 = 0; c4 < 8; c4 += 4) {
                        const float4 fC = make_float4(mld(S, fa0 + c4 + OX), mld(S, fa0 + c4 + OY), mld(S, fa0 + c4 + OZ),
                                                      mld(S, fa0 + c4 + OF));
                        v[c4 >> 2] = flow_cell_general(
                            p, fC, mld(S, fa0 + c4 + OZ - 4), mld(S, fau + c4 + OF), mld(S, fa0 + c4 + OX + 4),
                            mld(S, fad + c4 + OY), mld(S, fad + c4 + OF), mld(S, fa0 + c4 + OW), mld(S, fa0 + c4 + OH),
                            c4 ? hi(sd) : lo(sd), mld(S, fa0 + c4 + OH - 4), mld(S, fa0 + c4 + OH + 4),
                            mld(S, fau + c4 + OH), mld(S, fad + c4 + OH));
                    }
                    hn = pk(v[0].hn, v[1].hn);
                    wn = pk(v[0].wn, v[1].wn);
                    s_new = pk(v[0].s1, v[1].s1);
                    ux = pk(v[0].ux, v[1].ux);
                    uy = pk(v[0].uy, v[1].uy);
                } else {
                    Flow2 o;
                    const bool mine = live_w && (uint32_t)(tr + 4 + MORE) < nrows + 4u + 2u * MORE;
                    bad = flow_pair(c, fc, flz, frx, fuw, fdy, fdw, fw, fh, fhl, fhr, fhu, fhd, sd, mine, o) || bad;
                    hn = o.hn, wn = o.wn, s_new = o.s1, ux = o.ux, uy = o.uy;
                }
            }
            // ---- flux (:2439-2485) ----
            uint32_t xa0, xau, xad;
            f2 xh, xw, xhu, xwu, xhd, xwd;
            float xhl, xhr, xwl, xwr;
            const auto load_flux = [&]() {
                xa0 = (P + 7 * kMRow) & kRMask, xau = (P + 8 * kMRow) & kRMask, xad = (P + 6 * kMRow) & kRMask;
                if (ROLE == kSecondOfTwo) {
                    const f2 x = ld2(S, xa0 + kOX), y = ld2(S, xa0 + kOY), z = ld2(S, xa0 + kOZ), f = ld2(S, xa0 + kOF);
                    fa = make_float4(lo(x), lo(y), lo(z), lo(f));
                    fb = make_float4(hi(x), hi(y), hi(z), hi(f));
                }
                xh = ld2(S, xa0 + OH), xw = ld2(S, xa0 + OW), xhu = ld2(S, xau + OH), xwu = ld2(S, xau + OW);
                xhd = ld2(S, xad + OH), xwd = ld2(S, xad + OW);
                xhl = mld(S, xa0 + OH - 4), xhr = mld(S, xa0 + OH + 8);
                xwl = mld(S, xa0 + OW - 4), xwr = mld(S, xa0 + OW + 8);
            };
            if (EARLY) load_flux();
            {
                st2(S, fa0 + OS, s_new);
                st2(S, fa0 + OVX, ux);
                st2(S, fa0 + OVY, uy);
                // evaporate (:2587-2593)
                const f2 wo = evaporate2(c, wn);
                if (ROLE == kFirstOfTwo) {
                    st2(S, fa0 + kSet + kOH, hn);
                    st2(S, fa0 + kSet + kOW, add2(wo, ld2(S, fa0 + kOE)));
                } else {
                    const bool row = (uint32_t)(tr + 2) < nrows, s0 = row && in0, s1 = row && in1;
                    gst2<VEC>(q.h_out, B + 2u * Wu, hn, s0, s1);
                    gst2<VEC>(q.w_out, B + 2u * Wu, wo, s0, s1);
                }
            }
            if (!EARLY) load_flux();
            f2 ox, oy, oz, ow;
            {
                if constexpr (IEEE) {
                    float4 v[2];
#pragma unroll
                    for (uint32_t c4 = 0; c4 < 8; c4 += 4)
                        v[c4 >> 2] = flux_ieee(p, c4 ? fb : fa, mld(S, xa0 + c4 + OH), mld(S, xa0 + c4 + OW),
                                               mld(S, xa0 + c4 + OH - 4), mld(S, xa0 + c4 + OW - 4),
                                               mld(S, xau + c4 + OH), mld(S, xau + c4 + OW), mld(S, xa0 + c4 + OH + 4),
                                               mld(S, xa0 + c4 + OW + 4), mld(S, xad + c4 + OH), mld(S, xad + c4 + OW));
                    ox = pk(v[0].x, v[1].x);
                    oy = pk(v[0].y, v[1].y);
                    oz = pk(v[0].z, v[1].z);
                    ow = pk(v[0].w, v[1].w);
                } else {
                    Flux2 o;
                    const bool mine = live_f && (uint32_t)(tr + 10 + MORE) < nrows + 6u + 2u * MORE;
                    bad = flux_pair(c, xh, xw, xhl, xhr, xwl, xwr, xhu, xwu, xhd, xwd, fa, fb, mine, o) || bad;
                    ox = o.x, oy = o.y, oz = o.z, ow = o.w;
                }
            }
            {
                st2(S, xa0 + OX, ox);
                st2(S, xa0 + OY, oy);
                st2(S, xa0 + OZ, oz);
                st2(S, xa0 + OF, ow);
                if (ROLE != kFirstOfTwo) {
                    const bool row = (uint32_t)(tr + 7) < nrows, s0 = row && in0, s1 = row && in1;
                    gst_flux<VEC>(q.f_out, B + 7u * Wu, ox, oy, oz, ow, s0, s1);
                }
            }
            // ---- the loaded rows ----
            if (ROLE != kSecondOfTwo) {
                const uint32_t a = (P + 12 * kMRow) & kRMask;
                st2(S, a + OH, lh);
                st2(S, a + OW, add2(lw, lr));
                if (ROLE == kFirstOfTwo) st2(S, a + kOE, lr);
                prefetch();
            }
        }
        if (!IEEE && bad) {
            if constexpr (VEC && ROLE != kAlone) {
                const uint32_t seg = (uint32_t)(k - kFirst) >> max(0, 26 - __clz(K - kFirst));
                atomicOr(flagged + (seg >> 5), 1u << (seg & 31u));
            } else {
                atomicMin(reinterpret_cast<int *>(flagged), k);
                atomicMax(reinterpret_cast<int *>(flagged) + 1, k);
            }
        }
        barrier();
        P += kPairRows * kMRow;
        tr += kPairRows;
        B += W4;
        if (ROLE == kFirstOfTwo) {
            yw = IEEE ? (yw + kPairRows) % H : yw + kPairRows < H ? yw + kPairRows : yw + kPairRows - H;
            fy = (float)yw;
        } else {
            fy = fy + (float)kPairRows;
        }
    }
}

__device__ __noinline__ void march_ieee(const PairParams &pp, const HydroWorld &q, char *S, int x0, int iw, int r0,
                                        int r1)
{
    march_piece<false, true, kAlone>(pp.sp.p, pp.c, q, S, x0, iw, r0, r1, nullptr);
}

__global__ __launch_bounds__(kPairThreads, 2) void k_hydro_march(const __grid_constant__ PairParams pp)
{
    kernel_release();
    const StripParams &sp = pp.sp;
    extern __shared__ float4 march_smem[];
    char *S = reinterpret_cast<char *>(march_smem);
    __shared__ HydroWorld s_q;
    __shared__ unsigned s_flag[2];
    // the edge lanes read ring cells before anything writes them: start from zeros
    for (uint32_t i = threadIdx.x; i < kHydroMarchSmem / 16; i += kPairThreads)
        march_smem[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    // this block's strip-rows [a0, b0), with kWarmAlone more to each strip (see k_hydro_march_pair)
    const unsigned long long nb = gridDim.x, all = sp.rows + (unsigned long long)sp.nstrips * kWarmAlone;
    const unsigned long long a0 = all * (unsigned long long)blockIdx.x / nb;
    const unsigned long long b0 = all * (unsigned long long)(blockIdx.x + 1) / nb;
    int lo_s = 0, hi_s = sp.nstrips - 1;
    while (lo_s < hi_s) {
        const int mid = (lo_s + hi_s + 1) >> 1;
        if ((unsigned long long)sp.strips[mid].w + (unsigned long long)mid * kWarmAlone <= a0) lo_s = mid;
        else hi_s = mid - 1;
    }
    kernel_wait();
    unsigned long long a = a0;
    for (int s = lo_s; a < b0 && s < sp.nstrips; ++s) {
        const uint4 d = sp.strips[s];
        __syncthreads();  // the previous piece is done with s_q and the rings
        if (threadIdx.x == 0) {
            s_q = hydro_world(sp.p, sp.p.worlds[d.x]);
            clear_flags(s_flag, true);
        }
        __syncthreads();
        const unsigned long long first = d.w + (unsigned long long)(s + 1) * kWarmAlone,
                                 last = first + (unsigned long long)s_q.H;
        if (a >= last) continue;
        if (b0 <= first) break;
        const int r0 = a > first ? (int)(a - first) : 0, r1 = (int)((b0 < last ? b0 : last) - first);
        const int x0 = (int)d.y, iw = (int)d.z;
        if (s_q.H < kPairRows) {
            march_ieee(pp, s_q, S, x0, iw, r0, r1);
        } else {
            if (s_q.W & 1) march_piece<false, false, kAlone>(sp.p, pp.c, s_q, S, x0, iw, r0, r1, s_flag);
            else march_piece<true, false, kAlone>(sp.p, pp.c, s_q, S, x0, iw, r0, r1, s_flag);
            // The piece's last barrier has passed since the last flag.  A cell of chunk k (flux rows r+7 .. r+10, flow
            // rows r+2 .. r+5) reaches outputs three rows away.
            rerun_range(s_flag, r0, r1, 0, 14, [&](int lo, int hi) {
                __syncthreads();
                march_ieee(pp, s_q, S, x0, iw, lo, hi);
            });
        }
        a = first + (unsigned long long)r1;
    }
}

// Both roles of two sub-iterations: the block's first half is the first of the two.
template <bool VEC, bool IEEE>
__device__ __forceinline__ void march_two(const HydroParams &p, const PairConst &c, const HydroWorld &q, char *S, int x0,
                                          int iw, int r0, int r1, unsigned *flagged)
{
    if (threadIdx.x < kPairThreads) march_piece<VEC, IEEE, kFirstOfTwo>(p, c, q, S, x0, iw, r0, r1, flagged);
    else march_piece<VEC, IEEE, kSecondOfTwo>(p, c, q, S, x0, iw, r0, r1, flagged);
}

__device__ __noinline__ void march_two_ieee(const PairParams &pp, const HydroWorld &q, char *S, int x0, int iw, int r0,
                                            int r1)
{
    march_two<false, true>(pp.sp.p, pp.c, q, S, x0, iw, r0, r1, nullptr);
}

// Two sub-iterations in one march.  The block's first 256 threads run the first on 128 columns, leaving what
// it would store in shared memory; the other 256 run the second on the 116 columns inside, ten rows behind,
// which is as close as the first's height and as far as the rings allow.
// A sub-iteration moves 35 bytes a cell instead of 60 (DRAM 37% busy), and its instructions are as many as
// alone (530 a 64 cells, issue 56%, the shared-memory pipe 59%); one sub-iteration, alone and of two, us:
// 2048^2 72 -> 52, 4096^2 232 -> 187, 8192^2 852 -> 703, the 49.7 M cell batch 759 -> 647.  Leaving out, by a
// test a chunk, the stages that a piece's first and last chunks do not need gains where pieces are short (1024^2
// 24.6 -> 22) and loses elsewhere (8192^2 747 -> 805: the branches keep the compiler from overlapping stages).
__global__ __launch_bounds__(2 * kPairThreads, 1) void k_hydro_march_pair(const __grid_constant__ PairParams pp)
{
    kernel_release();
    const StripParams &sp = pp.sp;
    extern __shared__ float4 march_smem[];
    char *S = reinterpret_cast<char *>(march_smem);
    __shared__ HydroWorld s_q;
    __shared__ unsigned s_flag[2];
    for (uint32_t i = threadIdx.x; i < kHydroPairSmem / 16; i += 2 * kPairThreads)
        march_smem[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    // Each strip counts kWarmRows more than it has, before its first: a block that starts another strip pays a
    // second warm-up, and takes that many rows less.
    const unsigned long long nb = gridDim.x, all = sp.rows + (unsigned long long)sp.nstrips * kWarmRows;
    const unsigned long long a0 = all * (unsigned long long)blockIdx.x / nb;
    const unsigned long long b0 = all * (unsigned long long)(blockIdx.x + 1) / nb;
    int lo_s = 0, hi_s = sp.nstrips - 1;
    while (lo_s < hi_s) {
        const int mid = (lo_s + hi_s + 1) >> 1;
        if ((unsigned long long)sp.strips[mid].w + (unsigned long long)mid * kWarmRows <= a0) lo_s = mid;
        else hi_s = mid - 1;
    }
    kernel_wait();
    unsigned long long a = a0;
    for (int s = lo_s; a < b0 && s < sp.nstrips; ++s) {
        const uint4 d = sp.strips[s];
        __syncthreads();  // the previous piece is done with s_q and the rings
        if (threadIdx.x == 0) {
            s_q = hydro_world(sp.p, sp.p.worlds[d.x]);
            clear_flags(s_flag, s_q.W & 1);
        }
        __syncthreads();
        const unsigned long long first = d.w + (unsigned long long)(s + 1) * kWarmRows,
                                 last = first + (unsigned long long)s_q.H;
        if (a >= last) continue;
        if (b0 <= first) break;
        const int r0 = a > first ? (int)(a - first) : 0, r1 = (int)((b0 < last ? b0 : last) - first);
        const int x0 = (int)d.y, iw = (int)d.z;
        if (s_q.H < kPairRows) {
            march_two_ieee(pp, s_q, S, x0, iw, r0, r1);
        } else {
            if (s_q.W & 1) march_two<false, false>(sp.p, pp.c, s_q, S, x0, iw, r0, r1, s_flag);
            else march_two<true, false>(sp.p, pp.c, s_q, S, x0, iw, r0, r1, s_flag);
            // a cell of the first's chunk k (flux rows r+7 .. r+10, flow rows r+2 .. r+5) reaches outputs
            // r-2 .. r+15, one of the second's, ten rows behind, outputs r-10 .. r+3
            const auto run = [&](int lo, int hi) {
                __syncthreads();
                march_two_ieee(pp, s_q, S, x0, iw, lo, hi);
            };
            if (s_q.W & 1) rerun_range(s_flag, r0, r1, kLag, 16, run);
            else rerun_segments(s_flag, r0, r1, kLag, 16, run);
        }
        a = first + (unsigned long long)r1;
    }
}

constexpr int kHydroMarchMinRows = 16;

}  // namespace

int hydro_march_attributes()
{
    TECTO_CUDA(cudaFuncSetAttribute(k_hydro_march, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kHydroMarchSmem));
    TECTO_CUDA(cudaFuncSetAttribute(k_hydro_march_pair, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kHydroPairSmem));
    return TECTO_OK;
}

// Parameters that hydro_packed takes.  `two`: two sub-iterations at once, with the strips of ST_HYDRO_TWO.
void launch_hydro_march(const Batch &b, StripParams sp, bool two, cudaStream_t st)
{
    const void *kern = two ? (const void *)k_hydro_march_pair : (const void *)k_hydro_march;
    const int threads = two ? 2 * kPairThreads : kPairThreads;
    const size_t smem = two ? kHydroPairSmem : kHydroMarchSmem;
    sp.nwarps = march_blocks(b, sp.rows, kern, threads, smem, kHydroMarchMinRows);
    PairParams pp{};
    pp.sp = sp;
    pp.c = pair_const(sp.p);
    launch_chained(two ? k_hydro_march_pair : k_hydro_march, (unsigned)sp.nwarps, threads, smem, st, pp);
}

}  // namespace tecto
