// k_thermal_march.cu - the thermal iteration as a march of independent warps down column strips.
// Reference: thermalErosionKernel, src/cuda_compute/plate_tectonics_kernel.cu:2735-2786; driver
// plate_tectonic_sim.cu:73.
//
// One iteration per launch, the same as k_thermal's (k_erosion.cu): every cell's outflows from the heights
// at the start, a cell loses its own outflows and gains its neighbours' flows towards it, both in
// direction order.  A warp owns a column strip of a world, 64 columns (kThermalInner = 60 interior ones and
// a halo of 2 on each side), two adjacent cells per lane, and marches down its rows.  Step t computes the
// outflows of row t and completes the new heights of row t - 1.  Flows never leave registers: those towards
// the same lane's cells are there, those towards the adjacent lane's come by shuffle (six per row), and
// what a row sends to the row above waits one step.  Only the heights go through shared memory: a ring of
// 16 rows per warp that asynchronous copies fill 12 rows ahead, so that a warp's own loads cover the
// DRAM latency without registers.  Steps come in groups of three without branches between them, one wait
// and one warp barrier a group, so that the rows' dependent chains overlap.  All strip-rows of the batch are laid end to end and each warp takes
// one contiguous range of them.
//
// 179 warp-instructions per 64 cells; the form before it (one cell a thread, flows in shared-memory rings,
// two block barriers per 8 rows) took 390.  20 warps per SM (96 registers).  One iteration, before and
// after, us: 2048^2 38.0 -> 19.2, 8192^2 416 -> 224, a 49.7 M cell batch 361 -> 189; the tiles of variant 4
// take 37.4, 570 and 463.  Bound by the floating-point and the compare-select pipes (48 % and 49 % busy)
// and the dependent sums of 20 warps; DRAM is at 40 % of its rate at 8192^2.
//
// MODE 2 (threshold at least 2^-32, strength 1, amplitude a power of two): the packed form (pair.cuh) with
// the amplitude folded into the quotient, MODE 1 the packed form for other amplitudes and strengths that
// are finite and not negative, MODE 0 the scalar form for any parameters.  The packed forms hold for slope
// sums up to 2^32 (a sum that is not zero is above the threshold); a warp that met a larger one runs its
// piece once more in MODE 0 (inputs and outputs are different buffers).
#include <cmath>

#include "erosion.cuh"
#include "pair.cuh"

namespace tecto {

namespace {

constexpr int kTWarps = 4;              // warps per block (independent)
constexpr uint32_t kTRow = 64 * 4;      // bytes of a ring row
constexpr uint32_t kTRows = 16;         // rows of a ring
constexpr int kTGroup = 3;              // steps between two waits
constexpr int kTAhead = 4;              // groups copied ahead of the march
constexpr uint32_t kTMask = kTRows * kTRow - 1;
constexpr uint32_t kTGuard = 16;        // an edge lane reads one cell past a row's end
constexpr uint32_t kTWarpSmem = kTGuard + kTRows * kTRow + kTGuard;
static_assert(kTWarpSmem % 16 == 0, "zeroed by 16 bytes");
static_assert(kThermalInner == 64 - 4, "strips: interior plus a halo of 2 each side");
static_assert(kTGroup * (kTAhead + 1) <= (int)kTRows, "no row is overwritten before its last reader is done");

struct TMarchParams {
    ThermalParams p;
    const uint4 *strips;
    int nstrips;
    unsigned long long rows;
    int nwarps;
    // packed constants: (-0, -0) (mul2_z), 1, -1, A and S, and with MODE 2 -1 / A
    f2 Z, one, mone, A, S, nrA;
};

__device__ __forceinline__ float from_left(float v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ float from_right(float v) { return __shfl_down_sync(0xffffffffu, v, 1); }

// Asynchronous copy of a strip row's 64 cells where left > 0: two adjacent cells a lane (VEC: even world width), else
// two cells 32 columns apart.
template <bool VEC>
__device__ __forceinline__ void copy_row(uint32_t dst, const float *row, uint32_t c0, uint32_t c1, int lane, int left)
{
    if (VEC) {
        asm volatile(
            "{.reg .pred p; setp.gt.s32 p, %2, 0; @p cp.async.ca.shared.global [%0], [%1], 8;}" ::"r"(dst + lane * 8u),
            "l"(row + c0), "r"(left));
    } else {
        asm volatile(
            "{.reg .pred p; setp.gt.s32 p, %3, 0; @p cp.async.ca.shared.global [%0], [%1], 4;\n\t"
            "@p cp.async.ca.shared.global [%0+128], [%2], 4;}" ::"r"(dst + lane * 4u),
            "l"(row + c0), "l"(row + c1), "r"(left));
    }
}

// Rows [r0, r1) of the strip with interior columns [x0, x0 + iw).  S: the warp's ring, its guard before it.
// Returns the lane's largest slope sum (MODE > 0).
template <bool VEC, int MODE>
__device__ __forceinline__ float tmarch_piece(const TMarchParams &tp, const float *hin, float *hout, int W, int H,
                                             char *S, int x0, int iw, int r0, int r1)
{
    const uint32_t Wu = (uint32_t)W, N = Wu * (uint32_t)H;
    const int lane = (int)threadIdx.x & 31, col = 2 * lane;
    const uint32_t c0 = (uint32_t)wrapc(x0 - 2 + (VEC ? col : lane), W), c1 = (uint32_t)wrapc(x0 + 30 + lane, W);
    const bool in0 = col >= 2 && col < iw + 2, in1 = col >= 2 && col + 1 < iw + 2;
    const bool live = col < iw + 3;
    float smax = 0.0f;
    const float thr = tp.p.thr;
    const int nrows = r1 - r0, steps = nrows + 2;  // steps t = r0 - 1 .. r1
    const uint32_t Sa = (uint32_t)__cvta_generic_to_shared(S);
    const char *L = S + lane * 8;  // this lane's pair of a ring row
    uint32_t g = (uint32_t)wrapc(r0 - 2, H) * Wu;  // first cell of the row to copy next
    uint32_t w = 0;                                // its ring offset
    int left = nrows + 4;                          // rows still to copy: r0 - 2 .. r1 + 1
    auto copy = [&](int rows) {
#pragma unroll
        for (int i = 0; i < rows; ++i) {
            copy_row<VEC>(Sa + w, hin + g, c0, c1, lane, left);
            const uint32_t v = g + Wu;
            g = min(v, v - N);
            w = (w + kTRow) & kTMask;
            left -= 1;
        }
        asm volatile("cp.async.commit_group;");
    };
    copy(2);
#pragma unroll
    for (int i = 0; i < kTAhead; ++i) copy(kTGroup);
    asm volatile("cp.async.wait_group %0;" ::"n"(kTAhead) : "memory");
    __syncwarp();
    // heights of rows t - 1, t: the pair and the cells left and right of it
    f2 hA = ld2(L, 0), hB = ld2(L, kTRow);
    f2 oA = pk(mld(L, 0u - 4u), mld(L, 8)), oB = pk(mld(L, kTRow - 4), mld(L, kTRow + 8));
    // row t - 1: its heights less outflows (v), plus the first three inflows (acc); the flows of row t - 2
    // towards it from below left and right (q4, q6).  Flows of row t - 1 towards row t: p2, p4, p6.
    f2 v1 = 0, acc = 0, q4 = 0, q6 = 0, p2 = 0, p4 = 0, p6 = 0;
    uint32_t r = 2 * kTRow;                                               // ring offset of row t + 1
    uint32_t B = (uint32_t)(r0 - 2) * Wu + (uint32_t)(x0 - 2 + col);      // row t - 1, unwrapped
    auto step = [&](int k) {
        const char *R = L + r;
        const f2 hC = ld2(R, 0), oC = pk(mld(R, 0u - 4u), mld(R, 8));
        r = (r + kTRow) & kTMask;
        // outflows of row t, by direction: left, right, down (y - 1), up, and the diagonals
        f2 fL, fR, fD, fU, fLD, fLU, fRD, fRU, v;
        if constexpr (MODE == 0) {
            const float n0[8] = {lo(oB), hi(hB), lo(hA), lo(hC), lo(oA), lo(oC), hi(hA), hi(hC)};
            const float n1[8] = {lo(hB), hi(oB), hi(hA), hi(hC), lo(hA), lo(hC), hi(oA), hi(oC)};
            float f0[8], f1[8];
            const float v0 = thermal_flow(lo(hB), n0, tp.p, 0xffffffffu, f0);
            v = pk(v0, thermal_flow(hi(hB), n1, tp.p, 0xffffffffu, f1));
            fL = pk(f0[0], f1[0]), fR = pk(f0[1], f1[1]), fD = pk(f0[2], f1[2]), fU = pk(f0[3], f1[3]);
            fLD = pk(f0[4], f1[4]), fLU = pk(f0[5], f1[5]), fRD = pk(f0[6], f1[6]), fRU = pk(f0[7], f1[7]);
        } else {
            // differences: outer ones packed (left of cell 0, right of cell 1), inner ones scalar
            const f2 dB = sub2(hB, oB), dA = sub2(hB, oA), dC = sub2(hB, oC), dD = sub2(hB, hA), dU = sub2(hB, hC);
            const float i = lo(hB) - hi(hB);
            auto sel = [&](float d) { return d > thr ? d : 0.0f; };
            const f2 sL = pk(sel(lo(dB)), sel(-i)), sR = pk(sel(i), sel(hi(dB)));
            const f2 sD = pk(sel(lo(dD)), sel(hi(dD))), sU = pk(sel(lo(dU)), sel(hi(dU)));
            const f2 sLD = pk(sel(lo(dA)), sel(hi(hB) - lo(hA))), sLU = pk(sel(lo(dC)), sel(hi(hB) - lo(hC)));
            const f2 sRD = pk(sel(lo(hB) - hi(hA)), sel(hi(dA))), sRU = pk(sel(lo(hB) - hi(hC)), sel(hi(dC)));
            // a direction that does not flow adds +0
            const f2 s = add2(add2(add2(add2(add2(add2(add2(sL, sR), sD), sU), sLD), sLU), sRD), sRU);
            const f2 sc = max2(s, 0x1p-33f);  // a sum of zero has only zero dividends, any other is above thr >= 2^-32
            const f2 y = rcp2(sc, mul2(sc, tp.mone), tp.one);
            if constexpr (MODE == 2) {
                // A a power of two, S = 1: (A (d / s)) S is the quotient by s / A with the same roundings (d is a
                // zero or above 2^-32, so no step of it underflows)
                const f2 ns = mul2(sc, tp.nrA), yA = mul2(y, tp.A);
                fL = div2(sL, ns, yA), fR = div2(sR, ns, yA), fD = div2(sD, ns, yA), fU = div2(sU, ns, yA);
                fLD = div2(sLD, ns, yA), fLU = div2(sLU, ns, yA), fRD = div2(sRD, ns, yA), fRU = div2(sRU, ns, yA);
            } else {
                const f2 ns = mul2(sc, tp.mone);
                auto fl = [&](f2 d) { return mul2_z(mul2(tp.A, div2(d, ns, y)), tp.S, tp.Z); };
                fL = fl(sL), fR = fl(sR), fD = fl(sD), fU = fl(sU), fLD = fl(sLD), fLU = fl(sLU), fRD = fl(sRD),
                fRU = fl(sRU);
            }
            v = sub2(sub2(sub2(sub2(sub2(sub2(sub2(sub2(hB, fL), fR), fD), fU), fLD), fLU), fRD), fRU);
            if (k < steps) smax = fmaxf(fmaxf(smax, lo(s)), hi(s));  // not the steps that fill the last group
        }
        // inflows of row t - 1 from row t, after those from its own row and from row t - 2
        const f2 d5 = pk(from_left(hi(fRD)), lo(fRD)), d7 = pk(hi(fLD), from_right(lo(fLD)));
        f2 n;
        if constexpr (MODE == 0) {
            auto gain = [](f2 a, f2 f) {  // adding +0 would turn -0 into +0
                return pk(lo(f) != 0.0f ? lo(a) + lo(f) : lo(a), hi(f) != 0.0f ? hi(a) + hi(f) : hi(a));
            };
            n = gain(gain(gain(gain(gain(acc, fD), q4), d5), q6), d7);
            const f2 d0 = pk(from_left(hi(fR)), lo(fR)), d1 = pk(hi(fL), from_right(lo(fL)));
            acc = gain(gain(gain(v, d0), d1), p2);
        } else {
            n = add2(add2(add2(add2(add2(acc, fD), q4), d5), q6), d7);
            // every flow is +0 or positive: adding the +0s changes nothing but a -0 that received nothing
            n = pk(lo(n) == 0.0f && lo(v1) == 0.0f ? lo(v1) : lo(n), hi(n) == 0.0f && hi(v1) == 0.0f ? hi(v1) : hi(n));
            const f2 d0 = pk(from_left(hi(fR)), lo(fR)), d1 = pk(hi(fL), from_right(lo(fL)));
            acc = add2(add2(add2(v, d0), d1), p2);
            v1 = v;
        }
        const bool row = (unsigned)(k - 2) < (unsigned)nrows;  // t - 1 = r0 + k - 2
        const float *o = hout + B;
        if (VEC) {
            if (row && in0) asm volatile("st.global.b64 [%0], %1;" ::"l"(o), "l"(n));
        } else {
            if (row && in0) asm volatile("st.global.f32 [%0], %1;" ::"l"(o), "f"(lo(n)));
            if (row && in1) asm volatile("st.global.f32 [%0+4], %1;" ::"l"(o), "f"(hi(n)));
        }
        q4 = p4, q6 = p6;
        p2 = fU;
        p4 = pk(from_left(hi(fRU)), lo(fRU));
        p6 = pk(hi(fLU), from_right(lo(fLU)));
        hA = hB, oA = oB, hB = hC, oB = oC;
        B += Wu;
    };
#pragma unroll 1
    for (int k = 0; k < steps; k += kTGroup) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kTAhead - 1) : "memory");
        __syncwarp();  // the group's rows have arrived, and every lane is done with those of the group before
        copy(kTGroup);
#pragma unroll
        for (int i = 0; i < kTGroup; ++i) step(k + i);
    }
    return live ? smax : 0.0f;
}

__device__ __noinline__ void tmarch_scalar(const TMarchParams &tp, const float *hin, float *hout, int W, int H, char *S,
                                           int x0, int iw, int r0, int r1)
{
    tmarch_piece<false, 0>(tp, hin, hout, W, H, S, x0, iw, r0, r1);
}

// What a piece costs beside its rows (its first loads, three rows, a last group), in rows.  0 / 4 / 8 / 12:
// 1024^2 9.7 / 8.4 / 8.4 / 8.4 us, 1500x1100 11.4 / 10.6 / 10.1 / 10.2, 2048^2 20.4 / 19.6 / 19.2 / 19.3.
constexpr unsigned kTWarmRows = 8;

template <int MODE>
__global__ __launch_bounds__(kTWarps * 32, 5) void k_thermal_march(const __grid_constant__ TMarchParams tp)
{
    __shared__ __align__(16) char s_ring[kTWarps][kTWarpSmem];
    kernel_release();
    const int lane = (int)threadIdx.x & 31, wib = (int)threadIdx.x >> 5;
    const int gw = (int)blockIdx.x * kTWarps + wib;
    char *S = s_ring[wib] + kTGuard;
    // Columns 0 and 63, which no stored height needs, read past their row: their sums count for the piece's largest
    // and would send it through the scalar form by what an earlier kernel left there.
    for (uint32_t i = lane; i < kTWarpSmem / 16; i += 32)
        reinterpret_cast<float4 *>(s_ring[wib])[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();
    // this warp's strip-rows [a, b); each strip counts kTWarmRows more before its first, which a warp that
    // starts another strip spends on it
    const unsigned long long all = tp.rows + (unsigned long long)tp.nstrips * kTWarmRows;
    unsigned long long a = all * (unsigned long long)gw / (unsigned long long)tp.nwarps;
    const unsigned long long b = all * (unsigned long long)(gw + 1) / (unsigned long long)tp.nwarps;
    int lo_s = 0, hi_s = tp.nstrips - 1;  // the strip holding a: the last whose first strip-row is <= a
    while (lo_s < hi_s) {
        const int mid = (lo_s + hi_s + 1) >> 1;
        if ((unsigned long long)tp.strips[mid].w + (unsigned long long)mid * kTWarmRows <= a) lo_s = mid;
        else hi_s = mid - 1;
    }
    kernel_wait();
    if (gw >= tp.nwarps) return;
    for (int s = lo_s; a < b && s < tp.nstrips; ++s) {
        const uint4 d = tp.strips[s];
        const WorldDev &wd = tp.p.worlds[d.x];
        const int W = wd.W, H = wd.H, x0 = (int)d.y, iw = (int)d.z;
        const float *hin = wd.h[tp.p.cur_h];
        float *hout = wd.h[tp.p.cur_h ^ 1];
        const unsigned long long first = d.w + (unsigned long long)(s + 1) * kTWarmRows, last = first + (unsigned long long)H;
        if (a >= last) continue;
        if (b <= first) break;
        const int r0 = a > first ? (int)(a - first) : 0, r1 = (int)((b < last ? b : last) - first);
        __syncwarp();  // the previous piece is done with the ring
        if constexpr (MODE == 0) {
            tmarch_scalar(tp, hin, hout, W, H, S, x0, iw, r0, r1);
        } else {
            const float smax = W & 1 ? tmarch_piece<false, MODE>(tp, hin, hout, W, H, S, x0, iw, r0, r1)
                                     : tmarch_piece<true, MODE>(tp, hin, hout, W, H, S, x0, iw, r0, r1);
            if (__any_sync(0xffffffffu, smax > 0x1p32f)) tmarch_scalar(tp, hin, hout, W, H, S, x0, iw, r0, r1);
        }
        a = first + (unsigned long long)r1;
    }
}

constexpr int kTMinRows = 6;  // fewest strip-rows per warp

template <int MODE>
void launch_mode(const Batch &b, TMarchParams &tp, cudaStream_t st)
{
    const int nb = march_blocks(b, tp.rows, (const void *)k_thermal_march<MODE>, kTWarps * 32, 0, kTWarps * kTMinRows);
    tp.nwarps = nb * kTWarps;
    launch_chained(k_thermal_march<MODE>, (unsigned)nb, kTWarps * 32, 0, st, tp);
}

}  // namespace

int thermal_march_attributes() { return TECTO_OK; }

void launch_thermal_march(const Batch &b, const ThermalParams &p, cudaStream_t st)
{
    const StripTable &t = b.strips[ST_THERMAL];
    TMarchParams tp{};
    tp.p = p;
    tp.strips = t.d;
    tp.nstrips = t.n;
    tp.rows = t.rows;
    tp.Z = pk_host(-0.0f);
    tp.one = pk_host(1.0f);
    tp.mone = pk_host(-1.0f);
    tp.A = pk_host(p.A);
    tp.S = pk_host(p.S);
    int e = 0;
    const bool pow2 = p.A > 0.0f && std::frexp(p.A, &e) == 0.5f && e >= -16 && e <= 16;
    tp.nrA = pk_host(pow2 ? -1.0f / p.A : 0.0f);
    if (!p.packed) launch_mode<0>(b, tp, st);
    else if (pow2 && p.S == 1.0f) launch_mode<2>(b, tp, st);
    else launch_mode<1>(b, tp, st);
}

}  // namespace tecto
