// k_sort.cu - stable LSD radix sort of (destination cell, source cell) pairs.
//
// Replaces registerPlateCollisions' atomic slotting (src/cuda_compute/plate_tectonics_kernel.cu:
// 273-298): arrivals are grouped by sorting on the destination key; the sort is stable, so
// within one destination the sources stay in ascending order, which is the engine's canonical
// arrival-slot order.
//
// Onesweep structure: one kernel builds the digit histograms of every pass in a single read;
// then each pass is one kernel that ranks a tile of 4096 keys with warp ballots, publishes the
// tile's digit counts, walks back over earlier tiles (decoupled look-back, bounded spin) and
// scatters through shared memory so that runs of equal digits leave as contiguous stores.
// The keys can be generated from plate ids (advection fused into the sort: the key of cell i is
// getPixelMovements' wrapped destination, plate_tectonics_kernel.cu:248-265): the histogram
// kernel generates them once, counts them and stores them for the first pass, whose values are
// then the cell indices themselves.
//
// The digit width RB is a template parameter (8..11 bits): wider digits mean fewer passes over
// the keys but larger per-tile histograms and look-back tables; the autotuner picks per size.
#include "tecto_internal.cuh"

namespace tecto {

namespace {

constexpr int kWarps = kSortThreads / 32;
constexpr int kLookAhead = 8;  // predecessor tiles read per look-back round

template <int RB>
struct Digits {
    static constexpr int R = 1 << RB;               // digit values per pass
    static constexpr int DPT = R / kSortThreads;     // digits owned by each thread of the scan
    static constexpr uint32_t MASK = (uint32_t)R - 1u;
    static constexpr int MAX_PASSES = (32 + RB - 1) / RB;
    static_assert(RB >= 8 && RB <= kMaxRadixBits, "digit width out of range");
};

// Whether a pass ranks with lane masks: a warp's masks share its part of the staging area (R words in
// 2 * 32 * kSortItems).
template <int RB>
constexpr bool kMaskRank = (1 << RB) <= 2 * 32 * kSortItems;

// Dynamic shared memory of one pass: per-warp digit counts, the digits' offsets, the staged keys and values.
template <int RB>
constexpr size_t pass_smem()
{
    return ((size_t)(kWarps + 1) * Digits<RB>::R + 2 * (size_t)kSortTile) * sizeof(uint32_t);
}

// Batch-virtual destination of virtual cell i: the owning world's getPixelMovements destination
// (plate_tectonics_kernel.cu:248-265) offset by the world's virtual base.
struct GenArgs {
    const WorldDev *worlds;
    const uint32_t *vbase;
    int nworlds;
    int cur_id;
};

// The keys of the `count` (1 .. 4) cells from virtual cell v on: the world and the row are found once and
// advanced.
__device__ __forceinline__ void gen_keys(uint32_t v, int count, const GenArgs &g, const uint32_t *s_vbase, uint32_t *key)
{
    int wi = find_world(s_vbase, g.nworlds, v);
    const WorldDev *wd = g.worlds + wi;
    uint32_t local = v - wd->vbase;
    int W = wd->W, H = wd->H;
    int y = (int)(local / (uint32_t)W), x = (int)(local - (uint32_t)y * (uint32_t)W);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (q >= count) break;
        const int2 o = wd->off[wd->id[g.cur_id][local]];
        key[q] = wd->vbase + cidx(x + o.x, y + o.y, W, H);
        ++local;
        if (++x == W) {
            x = 0;
            if (++y == H && q + 1 < count) {  // the next world's first cell
                wd = g.worlds + ++wi;
                W = wd->W, H = wd->H;
                y = 0;
                local = 0;
            }
        }
    }
}

__device__ __forceinline__ void load_vbase(const GenArgs &g, uint32_t *s_vbase)
{
    for (int i = threadIdx.x; i < g.nworlds; i += blockDim.x) s_vbase[i] = g.vbase[i];
}

__device__ __forceinline__ uint32_t ld_volatile(const uint32_t *p)
{
    return *(const volatile uint32_t *)p;
}

__device__ __forceinline__ void st_volatile(uint32_t *p, uint32_t v)
{
    *(volatile uint32_t *)p = v;
}

// Block-wide exclusive scan of one value per thread (W warps); returns the exclusive prefix and the block
// total.  s_w holds W words; the call ends with a barrier.
template <int W>
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t *s_w, uint32_t *total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) s_w[warp] = inc;
    __syncthreads();
    uint32_t wb = 0, all = 0;
#pragma unroll
    for (int k = 0; k < W; ++k) {
        const uint32_t x = s_w[k];
        wb += k < warp ? x : 0u;
        all += x;
    }
    __syncthreads();
    *total = all;
    return wb + inc - v;
}

// Digit histograms of all passes in one read of the keys; generated keys are stored to keys_gen.  The block
// that finishes last turns each pass's counts into exclusive digit starts, in place (thread t owns digits
// t, t + 256, ...; the chunks of 256 digits are scanned in order).  With generated keys the blocks first
// clear the decoded accretion marks of the step before (the worlds' lists, split over the blocks).
template <bool GEN, int RB>
__global__ __launch_bounds__(256) void k_sort_hist(GenArgs g, const uint32_t *keys_in, size_t n,
                                                   int passes, uint32_t *hist, uint32_t *keys_gen, uint32_t *done)
{
    using D = Digits<RB>;
    kernel_wait();
    if (GEN) {
        const int parts = max(1, (int)gridDim.x / g.nworlds);
        for (int it = (int)blockIdx.x; it < g.nworlds * parts; it += (int)gridDim.x) {
            const int wi = it / parts, part = it - wi * parts;
            const WorldDev &wd = g.worlds[wi];
            const uint32_t count = wd.ctl->acc_count;
            for (uint32_t i = (uint32_t)part * 256u + threadIdx.x; i < count; i += (uint32_t)parts * 256u)
                wd.acc_u8[wd.acc_list[i]] = 0;
        }
    }
    __shared__ uint32_t s_hist[D::MAX_PASSES][D::R];
    __shared__ uint32_t s_vbase[GEN ? kMaxBatchWorlds : 1];
    for (int i = threadIdx.x; i < D::MAX_PASSES * D::R; i += blockDim.x) (&s_hist[0][0])[i] = 0;
    if (GEN) load_vbase(g, s_vbase);
    __syncthreads();
    // four consecutive keys a thread; every lane runs the same number of rounds for the votes below
    const unsigned lane = threadIdx.x & 31u;
    const size_t stride = (size_t)gridDim.x * 1024u;
    const bool vec = !GEN && (reinterpret_cast<uintptr_t>(keys_in) & 15u) == 0;  // the caller's alignment
    for (size_t b0 = (size_t)blockIdx.x * 1024u; b0 < n; b0 += stride) {
        const size_t i = b0 + 4u * threadIdx.x;
        const int count = i >= n ? 0 : n - i < 4 ? (int)(n - i) : 4;
        uint32_t key[4] = {0u, 0u, 0u, 0u};
        if (GEN) {
            if (count) gen_keys((uint32_t)i, count, g, s_vbase, key);
            if (count == 4) *reinterpret_cast<uint4 *>(keys_gen + i) = make_uint4(key[0], key[1], key[2], key[3]);
            else
                for (int q = 0; q < count; ++q) keys_gen[i + q] = key[q];
        } else {
            if (vec && count == 4) {
                const uint4 k4 = *reinterpret_cast<const uint4 *>(keys_in + i);
                key[0] = k4.x, key[1] = k4.y, key[2] = k4.z, key[3] = k4.w;
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (q < count) key[q] = keys_in[i + q];
            }
        }
        for (int p = 0; p < passes; ++p) {
            uint32_t d[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) d[q] = (key[q] >> (RB * p)) & D::MASK;
            const bool four = count == 4 && d[0] == d[1] && d[0] == d[2] && d[0] == d[3];
            const uint32_t d0 = __shfl_sync(0xffffffffu, d[0], 0);
            if (__all_sync(0xffffffffu, four && d[0] == d0)) {  // the warp's 128 keys share the digit
                if (lane == 0) atomicAdd(&s_hist[p][d0], 128u);
            } else if (four) {
                atomicAdd(&s_hist[p][d[0]], 4u);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (q < count) atomicAdd(&s_hist[p][d[q]], 1u);
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * D::R; i += blockDim.x) {
        const uint32_t v = (&s_hist[0][0])[i];
        if (v) atomicAdd(&hist[i], v);
    }
    __shared__ uint32_t s_w[kWarps];
    __shared__ bool s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int t = threadIdx.x;
    for (int p = 0; p < passes; ++p) {
        uint32_t carry = 0;
        for (int c = 0; c < D::DPT; ++c) {
            uint32_t *h = hist + (size_t)p * D::R + c * kSortThreads + t;
            const uint32_t v = ld_volatile(h);
            uint32_t tot = 0;
            const uint32_t ex = block_scan<kWarps>(v, s_w, &tot);
            *h = carry + ex;
            carry += tot;
        }
    }
}

// One tile of a onesweep pass.  vals_in == nullptr: the value of position i is i.
// FULL: every position of the tile is below n.
template <int RB, bool FULL>
__device__ __forceinline__ void sort_tile(const uint32_t *keys_in, const uint32_t *vals_in, uint32_t *keys_out,
                                          uint32_t *vals_out, uint32_t n, int shift, const uint32_t *digit_start,
                                          uint32_t *status, uint32_t tile, uint32_t *error, uint32_t *sm, uint32_t *s_w)
{
    using D = Digits<RB>;
    constexpr int R = D::R, W = kWarps, DPT = D::DPT, NT = kSortThreads;
    constexpr uint32_t T = kSortTile;
    uint32_t *s_cnt = sm;               // [W][R] per-warp counts, then the tile position of the warp's first key
    uint32_t *s_off = s_cnt + W * R;    // output position of a digit's run less its position in the tile
    uint32_t *s_keys = s_off + R;
    uint32_t *s_vals = s_keys + T;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t base = tile * T, wbase = base + (uint32_t)warp * (32 * kSortItems) + (uint32_t)lane;

    uint32_t k[kSortItems], rank[kSortItems];
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) k[it] = FULL || wbase + it * 32 < n ? keys_in[wbase + it * 32] : 0u;

    // Warp-level ranking: items are visited in element order (item, lane), so the rank of an
    // item among equal digits of its warp preserves input order (stability).  The lanes with an item's digit
    // come from a vote where the whole warp has one digit (the upper digits of keys that are nearly in
    // order), else from a lane mask per digit that the lanes set with shared atomics and the first of them
    // clears again.  The widest digits, whose masks do not fit the staging area, take a ballot per bit.
    const unsigned lt = (1u << lane) - 1u;
    uint32_t *my_cnt = s_cnt + warp * R;
    uint32_t *my_mask = s_keys + warp * R;  // the staging area is not in use yet
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
        const bool valid = FULL || wbase + it * 32 < n;
        const uint32_t d = (k[it] >> shift) & D::MASK;
        const uint32_t d0 = __shfl_sync(0xffffffffu, d, 0);
        if (__all_sync(0xffffffffu, valid && d == d0)) {
            const uint32_t before = my_cnt[d0];
            __syncwarp();
            if (lane == 0) my_cnt[d0] = before + 32u;
            __syncwarp();
            rank[it] = before + (uint32_t)lane;
            continue;
        }
        unsigned peers;
        if constexpr (kMaskRank<RB>) {
            if (valid) atomicOr(my_mask + d, 1u << lane);
            __syncwarp();
            peers = valid ? my_mask[d] : 0u;
        } else {
            peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
            for (int b = 0; b < RB; ++b) {
                const bool bit = (d >> b) & 1u;
                const unsigned bb = __ballot_sync(0xffffffffu, bit);
                peers &= bit ? bb : ~bb;
            }
        }
        const uint32_t before = my_cnt[d];
        __syncwarp();
        if (valid && (peers & lt) == 0) {
            my_cnt[d] = before + (uint32_t)__popc(peers);
            if constexpr (kMaskRank<RB>) my_mask[d] = 0u;
        }
        __syncwarp();
        rank[it] = before + (uint32_t)__popc(peers & lt);
    }
    __syncthreads();

    // Per owned digit: the tile's count of it, published at once so that later tiles can start their
    // look-back; then its tile-local start (chunks of 256 digits in order) and the position of each warp's
    // first key of it.
    uint32_t run[DPT];
    uint32_t *my_status = status + (size_t)tile * R;
#pragma unroll
    for (int c = 0; c < DPT; ++c) {
        const int d = t + c * NT;
        uint32_t r = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) r += s_cnt[w * R + d];
        st_volatile(my_status + d, (tile == 0 ? kFlagPrefix : kFlagAggregate) | r);
        run[c] = r;
    }
    uint32_t carry = 0, start[DPT];
#pragma unroll
    for (int c = 0; c < DPT; ++c) {
        const int d = t + c * NT;
        uint32_t tot = 0;
        start[c] = carry + block_scan<W>(run[c], s_w, &tot);
        carry += tot;
        uint32_t r = start[c];
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const uint32_t x = s_cnt[w * R + d];
            s_cnt[w * R + d] = r;
            r += x;
        }
    }
    __syncthreads();

    // Scatter the keys into shared memory in digit order.
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
        if (FULL || wbase + it * 32 < n) {
            rank[it] += my_cnt[(k[it] >> shift) & D::MASK];
            s_keys[rank[it]] = k[it];
        }
    }

    // Decoupled look-back for the owned digits.  Each round reads the status words of up to kLookAhead
    // predecessors at once (independent loads in flight together) and consumes them newest first until one
    // is not yet published or carries an inclusive prefix.
    uint32_t prefix[DPT];
#pragma unroll
    for (int c = 0; c < DPT; ++c) prefix[c] = 0;
    if (tile > 0) {
        uint32_t spins = 0;
#pragma unroll
        for (int c = 0; c < DPT; ++c) {
            const int d = t + c * NT;
            int j = (int)tile - 1;
            while (j >= 0) {
                const uint32_t *col = status + (size_t)j * R + d;
                uint32_t sv[kLookAhead];
#pragma unroll
                for (int q = 0; q < kLookAhead; ++q) sv[q] = j >= q ? ld_volatile(col - q * R) : kFlagPrefix;
                bool go = true;
                int used = 0;
#pragma unroll
                for (int q = 0; q < kLookAhead; ++q) {
                    go = go && (sv[q] & ~kValueMask) != 0;  // not yet published: read it again next round
                    if (go) {
                        prefix[c] += sv[q] & kValueMask;
                        used = q + 1;
                        if (sv[q] & kFlagPrefix) {
                            used = j + 1;
                            go = false;
                        }
                    }
                }
                j -= used;
                if (used == 0 && ++spins > kSpinLimit) {  // a predecessor never published
                    atomicOr(error, kErrLookbackTimeout);
                    break;
                }
            }
            st_volatile(my_status + d, kFlagPrefix | ((prefix[c] + run[c]) & kValueMask));
        }
    }
#pragma unroll
    for (int c = 0; c < DPT; ++c) {
        const int d = t + c * NT;
        s_off[d] = digit_start[d] + prefix[c] - start[c];
    }
    // the values are read only now, so that they occupy no registers while the keys are ranked
#pragma unroll
    for (int it = 0; it < kSortItems; ++it)
        if (FULL || wbase + it * 32 < n) s_vals[rank[it]] = vals_in ? vals_in[wbase + it * 32] : wbase + it * 32;
    __syncthreads();
    const uint32_t tile_n = FULL ? T : n - base;
#pragma unroll 4
    for (uint32_t jj = t; jj < tile_n; jj += NT) {
        const uint32_t key = s_keys[jj];
        const uint32_t out = s_off[(key >> shift) & D::MASK] + jj;
        keys_out[out] = key;
        vals_out[out] = s_vals[jj];
    }
}

// A sort of 3 M pairs 193 -> 103 us, of 43.6 M 1.91 -> 1.01 ms, against ranking by eight ballots a key with
// the values held in registers at two and three blocks per SM.
// Four blocks per SM (64 registers, some of the ranks spilled): a tile waits on its loads and its look-back
// most of the time.  Shared memory admits three of 10-bit digits (70 KB each) and two of 11 (106 KB), which take the
// registers that leaves.  Tiles of 8192 keys by 512 threads were no faster (8192^2: 3.99 against 3.60 ms for a
// step's phases other than erosion).
template <int RB>
__global__ __launch_bounds__(kSortThreads, RB <= 9 ? 4 : RB == 10 ? 3 : 2) void k_sort_pass(
    const uint32_t *keys_in, const uint32_t *vals_in, uint32_t *keys_out, uint32_t *vals_out, uint32_t n,
    int shift, const uint32_t *digit_start, uint32_t *status, uint32_t *tile_counter, uint32_t *error)
{
    using D = Digits<RB>;
    extern __shared__ __align__(16) uint32_t sm_sort[];
    __shared__ uint32_t s_w[kWarps];
    __shared__ uint32_t s_tile;
    kernel_wait();
    if (threadIdx.x == 0) s_tile = atomicAdd(tile_counter, 1u);
    for (int i = threadIdx.x; i < kWarps * D::R; i += kSortThreads) {
        sm_sort[i] = 0;
        if constexpr (kMaskRank<RB>) sm_sort[(kWarps + 1) * D::R + i] = 0;
    }
    __syncthreads();
    const uint32_t tile = s_tile;
    if ((tile + 1) * kSortTile <= n)
        sort_tile<RB, true>(keys_in, vals_in, keys_out, vals_out, n, shift, digit_start, status, tile, error, sm_sort, s_w);
    else
        sort_tile<RB, false>(keys_in, vals_in, keys_out, vals_out, n, shift, digit_start, status, tile, error, sm_sort, s_w);
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

template <int RB>
int set_sort_attributes()
{
    TECTO_CUDA(cudaFuncSetAttribute(k_sort_pass<RB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pass_smem<RB>()));
    return TECTO_OK;
}

bool g_sort_attr_done = false;

template <int RB>
int run_sort_rb(const SortArgs &a, const SortScratch &scr, cudaStream_t st, int *result_half)
{
    const int passes = scr.passes;
    const size_t tiles = (a.n + kSortTile - 1) / kSortTile;
    constexpr int R = Digits<RB>::R;
    const bool gen = a.worlds != nullptr;
    const GenArgs g{a.worlds, a.vbase, a.nworlds, a.cur_id};
    int hist_blocks = (int)((a.n + 1023) / 1024);
    if (hist_blocks > 152 * 8) hist_blocks = 152 * 8;
    // generated keys go to the second key half, which the first pass reads and does not write
    const uint32_t *kin = a.keys_in, *vin = a.vals_in;
    if (gen) {
        launch_chained(k_sort_hist<true, RB>, hist_blocks, 256, 0, st, g, nullptr, a.n, passes, scr.hist, a.keys[1],
                       scr.counters + kSortDoneCounter);
        kin = a.keys[1];
        vin = nullptr;
    } else {
        launch_chained(k_sort_hist<false, RB>, hist_blocks, 256, 0, st, g, a.keys_in, a.n, passes, scr.hist, nullptr,
                       scr.counters + kSortDoneCounter);
    }
    int half = 0;
    for (int p = 0; p < passes; ++p) {
        const bool direct = a.keys_final && p > 0 && p == passes - 1;
        uint32_t *kout = direct ? a.keys_final : a.keys[half], *vout = direct ? a.vals_final : a.vals[half];
        uint32_t *status = scr.status + (size_t)p * tiles * R;
        launch_chained(k_sort_pass<RB>, (unsigned)tiles, kSortThreads, pass_smem<RB>(), st, kin, vin, kout, vout,
                       (uint32_t)a.n, RB * p, scr.hist + (size_t)p * R, status, scr.counters + p, scr.error);
        kin = kout;
        vin = vout;
        half ^= 1;
    }
    TECTO_CUDA(cudaGetLastError());
    *result_half = half ^ 1;
    return TECTO_OK;
}

}  // namespace

int sort_kernel_attributes()
{
    if (g_sort_attr_done) return TECTO_OK;
    int rc;
    if ((rc = set_sort_attributes<8>()) != TECTO_OK || (rc = set_sort_attributes<9>()) != TECTO_OK ||
        (rc = set_sort_attributes<10>()) != TECTO_OK || (rc = set_sort_attributes<11>()) != TECTO_OK)
        return rc;
    g_sort_attr_done = true;
    return TECTO_OK;
}

int key_bits_for(size_t n)
{
    int b = 1;
    while (b < 32 && ((size_t)1 << b) < n) ++b;
    return b;
}

bool valid_radix_bits(int rb) { return rb >= 8 && rb <= kMaxRadixBits; }

int sort_passes_for(int key_bits, int rb) { return (key_bits + rb - 1) / rb; }

size_t sort_scratch_bytes(size_t n, int key_bits, int rb)
{
    const size_t passes = (size_t)sort_passes_for(key_bits, rb);
    const size_t tiles = (n + kSortTile - 1) / kSortTile;
    const size_t R = (size_t)1 << rb;
    return align256(passes * R * 4) + align256(passes * tiles * R * 4) + align256(kSortCounters * 4) +
           align256(4);
}

void sort_scratch_carve(void *base, size_t n, int key_bits, int rb, SortScratch *out)
{
    const int passes = sort_passes_for(key_bits, rb);
    const size_t tiles = (n + kSortTile - 1) / kSortTile;
    const size_t R = (size_t)1 << rb;
    char *p = (char *)base;
    out->passes = passes;
    out->tiles = (int)tiles;
    out->radix_bits = rb;
    out->hist = (uint32_t *)p;
    p += align256((size_t)passes * R * 4);
    out->status = (uint32_t *)p;
    p += align256((size_t)passes * tiles * R * 4);
    out->counters = (uint32_t *)p;
    p += align256(kSortCounters * 4);
    out->error = (uint32_t *)p;
}

// hist, status and counters, contiguous in the scratch layout
size_t sort_clear_bytes(const SortScratch &scr, size_t n)
{
    const size_t R = (size_t)1 << scr.radix_bits, tiles = (n + kSortTile - 1) / kSortTile;
    return align256((size_t)scr.passes * R * 4) + align256((size_t)scr.passes * tiles * R * 4) +
           align256(kSortCounters * 4);
}

int run_sort_clear(const SortScratch &scr, size_t n, cudaStream_t st)
{
    TECTO_CUDA(cudaMemsetAsync(scr.hist, 0, sort_clear_bytes(scr, n), st));
    return TECTO_OK;
}

int run_sort(const SortArgs &a, const SortScratch &scr, cudaStream_t st, int *result_half)
{
    const int rb = scr.radix_bits;
    if (!valid_radix_bits(rb) || sort_passes_for(a.key_bits, rb) != scr.passes || a.n == 0 ||
        a.n > (size_t)kValueMask || (a.n + kSortTile - 1) / kSortTile > (size_t)scr.tiles) {
        set_error("run_sort: scratch does not match the problem size");
        return TECTO_ERR_INVALID;
    }
    if (a.worlds != nullptr && (a.nworlds < 1 || a.nworlds > kMaxBatchWorlds)) {
        set_error("run_sort: batch world count out of range");
        return TECTO_ERR_INVALID;
    }
    if (rb > 8 && !g_sort_attr_done) {  // wide digits need the opt-in shared memory size
        set_error("run_sort: sort kernel attributes not set");
        return TECTO_ERR_INVALID;
    }
    switch (rb) {
        case 8: return run_sort_rb<8>(a, scr, st, result_half);
        case 9: return run_sort_rb<9>(a, scr, st, result_half);
        case 10: return run_sort_rb<10>(a, scr, st, result_half);
        default: return run_sort_rb<11>(a, scr, st, result_half);
    }
}

}  // namespace tecto

// ---- C ABI: standalone sort -------------------------------------------------------------------

extern "C" size_t tecto_sort_scratch_bytes_radix(size_t n, int key_bits, int radix_bits)
{
    if (key_bits < 1 || key_bits > 32) return 0;
    if (radix_bits == 0) radix_bits = 8;
    if (!tecto::valid_radix_bits(radix_bits)) return 0;
    // two ping-pong halves for keys and values are carved after the sort's own scratch
    return tecto::sort_scratch_bytes(n, key_bits, radix_bits) + 4 * tecto::align256(n * sizeof(uint32_t));
}

extern "C" size_t tecto_sort_scratch_bytes(size_t n, int key_bits)
{
    return tecto_sort_scratch_bytes_radix(n, key_bits, 8);
}

extern "C" int tecto_sort_wide_pass(size_t n)
{
    return n > ((size_t)1 << 24) - (size_t)tecto::kSortTile ? 1 : 0;
}

extern "C" int tecto_sort_pairs_radix(const uint32_t *keys_in, const uint32_t *vals_in, uint32_t *keys_out,
                                      uint32_t *vals_out, size_t n, int key_bits, int radix_bits, void *scratch,
                                      size_t scratch_bytes, tecto_stream_t stream)
{
    using namespace tecto;
    if (n == 0) return TECTO_OK;
    if (radix_bits == 0) radix_bits = 8;
    if (!keys_in || !vals_in || !keys_out || !vals_out || !scratch || key_bits < 1 ||
        key_bits > 32 || n > (size_t)kValueMask || !valid_radix_bits(radix_bits)) {
        set_error("tecto_sort_pairs: invalid argument");
        return TECTO_ERR_INVALID;
    }
    if (scratch_bytes < tecto_sort_scratch_bytes_radix(n, key_bits, radix_bits)) {
        set_error("tecto_sort_pairs: scratch too small");
        return TECTO_ERR_INVALID;
    }
    int rc;
    if (radix_bits > 8 && (rc = sort_kernel_attributes()) != TECTO_OK) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    SortScratch scr{};
    sort_scratch_carve(scratch, n, key_bits, radix_bits, &scr);
    char *p = (char *)scratch + sort_scratch_bytes(n, key_bits, radix_bits);
    const size_t arr = align256(n * sizeof(uint32_t));
    SortArgs a{};
    a.keys_in = keys_in;
    a.vals_in = vals_in;
    a.keys[0] = (uint32_t *)p;
    a.vals[0] = (uint32_t *)(p + arr);
    a.keys[1] = (uint32_t *)(p + 2 * arr);
    a.vals[1] = (uint32_t *)(p + 3 * arr);
    a.n = n;
    a.key_bits = key_bits;
    a.keys_final = keys_out;
    a.vals_final = vals_out;
    TECTO_CUDA(cudaMemsetAsync(scr.error, 0, 4, st));
    int half = 0;
    rc = run_sort_clear(scr, n, st);
    if (rc == TECTO_OK) rc = run_sort(a, scr, st, &half);
    if (rc != TECTO_OK) return rc;
    if (scr.passes == 1) {  // the one pass reads the inputs, which the outputs may overlap
        TECTO_CUDA(cudaMemcpyAsync(keys_out, a.keys[half], n * 4, cudaMemcpyDeviceToDevice, st));
        TECTO_CUDA(cudaMemcpyAsync(vals_out, a.vals[half], n * 4, cudaMemcpyDeviceToDevice, st));
    }
    uint32_t err = 0;
    TECTO_CUDA(cudaMemcpyAsync(&err, scr.error, 4, cudaMemcpyDeviceToHost, st));
    TECTO_CUDA(cudaStreamSynchronize(st));
    if (err) {
        set_error("tecto_sort_pairs: look-back wait gave up");
        return TECTO_ERR_DEVICE_TIMEOUT;
    }
    return TECTO_OK;
}

extern "C" int tecto_sort_pairs(const uint32_t *keys_in, const uint32_t *vals_in, uint32_t *keys_out,
                                uint32_t *vals_out, size_t n, int key_bits, void *scratch,
                                size_t scratch_bytes, tecto_stream_t stream)
{
    return tecto_sort_pairs_radix(keys_in, vals_in, keys_out, vals_out, n, key_bits, 8, scratch, scratch_bytes,
                                  stream);
}
