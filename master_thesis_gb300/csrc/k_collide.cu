// k_collide.cu - plate displacement, collision words from the sorted arrivals, collision-type
// evidence and the plate-pair type bitmap.  Reference: src/cuda_compute/plate_tectonics_kernel.cu.
#include <algorithm>

#include "tecto_internal.cuh"

namespace tecto {

namespace {

// Per-plate integer displacement (getPixelMovements, :248-257) and the sub-cell centre update
// of applyPlateMovementChanges (:1871-1878), one block per world; the record before the update is
// kept in plates_prev for the kernels of the same step.  The blocks after those of the worlds clear the
// sort's scratch (clear_words 16-byte words).  With plate dynamics it first turns the sums k_plate_stats left into each
// plate's mass, size and geometric centre (mergeAndCountSizeMass, calculatePlateCenters
// :2191-2226: the angular means back to cells through atan2), and clears them.  The reference
// computes no centre before its first iteration ends, so iteration 0 keeps the stored one.
__global__ void k_plates(const WorldDev *worlds, int nworlds, int dynamics, uint4 *clear, size_t clear_words)
{
    kernel_wait();
    if ((int)blockIdx.x >= nworlds) {
        const size_t step = (size_t)(gridDim.x - nworlds) * blockDim.x;
        for (size_t i = (size_t)(blockIdx.x - nworlds) * blockDim.x + threadIdx.x; i < clear_words; i += step)
            clear[i] = make_uint4(0u, 0u, 0u, 0u);
        return;
    }
    const WorldDev &wd = worlds[blockIdx.x];
    const int k = threadIdx.x;
    if (dynamics && k < kPlates) {
        PlateAcc &a = wd.pacc[k];
        tecto_plate_dynamics dd = wd.dyn[k];
        dd.mass = tecto_unfix((long long)a.mass, 1.0 / (double)kMassScale);
        dd.size = a.size;
        if (a.samples > 0 && wd.ctl->iteration > 0) {
            const float n = (float)a.samples;
            const float sx = tecto_unfix((long long)a.ang[0], 1.0 / (double)kAngScale) / n;
            const float cx = tecto_unfix((long long)a.ang[1], 1.0 / (double)kAngScale) / n;
            const float sy = tecto_unfix((long long)a.ang[2], 1.0 / (double)kAngScale) / n;
            const float cy = tecto_unfix((long long)a.ang[3], 1.0 / (double)kAngScale) / n;
            float gx = tecto_atan2f(sx, cx) * (float)wd.W / kTwoPiF;
            float gy = tecto_atan2f(sy, cy) * (float)wd.H / kTwoPiF;
            if (gx < 0.0f) gx += (float)wd.W;
            if (gy < 0.0f) gy += (float)wd.H;
            dd.geometricCenter_x = gx;
            dd.geometricCenter_y = gy;
        }
        wd.dyn[k] = dd;
        a.mass = 0ull;
        a.ang[0] = a.ang[1] = a.ang[2] = a.ang[3] = 0ull;
        a.size = 0;
        a.samples = 0;
    }
    if (k < kPlates) {
        tecto_plate p = wd.plates[k];
        wd.plates_prev[k] = p;  // the record the rest of the step sees in the reference
        const float mx = p.direction_x * p.velocity;
        const float my = p.direction_y * p.velocity;
        const float cx = p.pixelCenter_x + mx;
        const float cy = p.pixelCenter_y + my;
        const float fx = floorf(cx), fy = floorf(cy);
        wd.off[k] = make_int2((int)fx, (int)fy);
        p.pixelCenter_x = cx - fx;
        p.pixelCenter_y = cy - fy;
        wd.plates[k] = p;
    } else if (k == kPlates) {
        wd.off[k] = make_int2(0, 0);
    }
}

// writeCollision's classification (:794-836): returns category 0..4 or -1 to skip.  The early
// exit is the as-compiled `(packed & 1) && ((packed >> 4) & (15 < cooldown))` (:813).
__device__ __forceinline__ int evidence_category(const uint8_t *bm, uint8_t A, uint8_t B, float hA,
                                                 float hB, float thr, int cooldown, uint32_t *pair)
{
    const bool cond = A < B;
    const uint8_t mn = cond ? A : B, mx = cond ? B : A;
    const float mnH = cond ? hA : hB, mxH = cond ? hB : hA;
    const uint32_t idx = tri_index(mn, mx);
    *pair = idx;
    const uint32_t packed = bm[idx];
    if ((packed & 1u) && ((packed >> 4) & (uint32_t)(0x0F < cooldown))) return -1;
    const bool minCont = mnH >= thr, maxCont = mxH >= thr;
    if (minCont && maxCont) return 4;
    if (minCont) return 2;
    if (maxCont) return 0;
    if (mnH <= mxH) return 1;
    return 3;
}

// Segmented winner pick over the sorted (destination, source) pairs of the whole batch: the
// first position of each destination's run builds the packed arrival word of
// registerPlateCollisions (:273-298) from its first four sources (ascending source order),
// writes zero words into the gap of destinations nobody moved into, and for convergent cells
// adds the collision-type evidence of the determineCollisionType kernel (:838-888) with
// warp-aggregated atomics.
//
// The bytes (13 a cell) take 100 us for a batch of 49.7 M cells; instructions and the chain of gathers
// (key, source, plate, height) bound it: 248 us there, 260 us for 67 M cells in one world.  With one position
// a thread and runs, gaps and evidence worked off in place it took 629 and 508 us (230 warp instructions per
// 32 positions, now 104), since nearly every warp held some lane with each of them.  So a block takes
// EACH x 256 positions: the worlds of its first and last key bound every search (most blocks lie in one
// world), keys and plate ids are staged in shared memory, runs of two and more are collected and worked off
// densely, and a warp fills a gap with all its lanes.
template <int EACH>
__global__ __launch_bounds__(256) void k_words(const uint32_t *keys, const uint32_t *vals, uint32_t n,
                                               const WorldDev *worlds, const uint32_t *vbase, int nworlds,
                                               int cur_id, int cur_h, float thr, int cooldown)
{
    kernel_wait();
    constexpr int kSpan = EACH * 256;
    constexpr uint32_t kNone = 0xffffffffu;   // no key: the batch has fewer cells
    __shared__ uint32_t s_vbase[kMaxBatchWorlds + 1];
    __shared__ uint32_t s_key[kSpan + 4];  // [1 + p]: position p of the block; one before and three after
    __shared__ uint8_t s_id[kSpan + 3];    // plate of position p's source
    __shared__ uint16_t s_run[kSpan / 2];  // first positions of the runs of two and more
    __shared__ int s_w[2], s_runs;
    const int t = threadIdx.x;
    const unsigned lane = t & 31u;
    const uint32_t j0 = blockIdx.x * (uint32_t)kSpan;
    const int m = (int)min((uint32_t)kSpan, n - j0);
    const uint32_t last = keys[j0 + m - 1], before = j0 > 0 ? keys[j0 - 1] : kNone;
    uint32_t key[EACH], val[EACH];
#pragma unroll
    for (int i = 0; i < EACH; ++i) {
        const int p = i * 256 + t;
        key[i] = p < m ? keys[j0 + p] : kNone;
        val[i] = p < m ? vals[j0 + p] : 0u;
    }
    if (nworlds > 1)
        for (int i = t; i <= nworlds; i += 256) s_vbase[i] = vbase[i];
    if (t < 2) s_w[t] = 0;
    if (t == 2) s_runs = 0;
    __syncthreads();
    if (nworlds > 1) {
        // of the first cell the block writes and of the last (a gap may begin in an earlier world)
        if (t == 0) s_w[0] = find_world(s_vbase, nworlds, min(before + 1u, key[0]));
        if (t == 32) s_w[1] = find_world(s_vbase, nworlds, last);
        __syncthreads();
    }
    const int w0 = s_w[0], nw = s_w[1] - w0 + 1;
    const auto world_of = [&](uint32_t c) -> const WorldDev & {
        return worlds[nw == 1 ? w0 : w0 + find_world(s_vbase + w0, nw, c)];
    };
#pragma unroll
    for (int i = 0; i < EACH; ++i) {
        const int p = i * 256 + t;
        s_key[1 + p] = key[i];
        if (p < m) {
            const WorldDev &wd = world_of(key[i]);
            s_id[p] = wd.id[cur_id][val[i] - wd.vbase];
        }
    }
    if (t < 3) {  // the run at the block's end may go on
        const uint64_t j = (uint64_t)j0 + kSpan + t;
        const uint32_t k = j < n ? keys[j] : kNone;
        s_key[1 + kSpan + t] = k;
        if (j < n && k == last) {
            const WorldDev &wd = world_of(k);
            s_id[kSpan + t] = wd.id[cur_id][vals[j] - wd.vbase];
        }
    } else if (t == 3) {
        s_key[0] = before;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < EACH; ++i) {
        const int p = i * 256 + t;
        const uint32_t prev = s_key[p];
        const bool leader = p < m && prev != key[i];
        const bool run = leader && s_key[p + 2] == key[i];
        if (leader && !run) {
            const WorldDev &wd = world_of(key[i]);
            wd.word[key[i] - wd.vbase] = 255u - s_id[p];
        }
        const unsigned runs = __ballot_sync(0xffffffffu, run);
        if (runs) {
            int at = 0;
            if (lane == 0) at = atomicAdd(&s_runs, __popc(runs));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(runs & ((1u << lane) - 1u));
            if (run) s_run[at] = (uint16_t)p;
        }
        // destinations without arrivals before this one (from 0 at the first position: kNone + 1)
        const uint32_t gap = leader ? key[i] - (prev + 1u) : 0u;
        for (unsigned g = __ballot_sync(0xffffffffu, gap > 0u); g; g &= g - 1u) {
            const int from = __ffs(g) - 1;
            const uint32_t c0 = __shfl_sync(0xffffffffu, prev, from) + 1u, len = __shfl_sync(0xffffffffu, gap, from);
            for (uint32_t c = lane; c < len; c += 32) {
                const WorldDev &wd = world_of(c0 + c);
                wd.word[c0 + c - wd.vbase] = 0u;
            }
        }
    }
    if (j0 + m == n) {
        const uint32_t total = nworlds > 1 ? s_vbase[nworlds] : vbase[nworlds];  // the batch's cell count
        for (uint32_t c = last + 1u + t; c < total; c += 256) {
            const WorldDev &wd = worlds[nworlds > 1 ? find_world(s_vbase, nworlds, c) : 0];
            wd.word[c - wd.vbase] = 0u;
        }
    }
    __syncthreads();
    // Convergent cells.  Evidence: pairs in determineCollisionType's order for 2, 3 and 4 arrivals (counts
    // are sums, so the order only has to cover the same pairs).
    const int nruns = s_runs;
    for (int r = t; r - (int)lane < nruns; r += 256) {
        uint8_t ids[4] = {0, 0, 0, 0};
        float hs[4] = {0, 0, 0, 0};
        int cnt = 0, wi = 0;
        const uint8_t *bm = nullptr;
        if (r < nruns) {
            const int p = s_run[r];
            const uint32_t k = s_key[1 + p];
            cnt = 2 + (s_key[p + 3] == k);
            cnt += s_key[p + 4] == k;
            const WorldDev &wd = world_of(k);
            wi = (int)(&wd - worlds);
            const float *h = wd.h[cur_h];
            uint32_t wv = 0;
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                if (a >= cnt) break;
                ids[a] = s_id[p + a];
                hs[a] = h[vals[j0 + p + a] - wd.vbase];  // determineCollisionHeight: height at the arrival's source
                wv |= (uint32_t)(255u - ids[a]) << (8 * a);
            }
            wd.word[k - wd.vbase] = wv;
            bm = wd.type_bitmap;
        }
        const int npairs = cnt >= 4 ? 6 : cnt == 3 ? 3 : cnt == 2 ? 1 : 0;
        const uint8_t PA[6] = {0, 0, 0, 1, 1, 2};
        const uint8_t PB[6] = {1, 2, 3, 2, 3, 3};
        const uint8_t PA3[3] = {0, 0, 1};
        const uint8_t PB3[3] = {1, 2, 2};
#pragma unroll
        for (int slot = 0; slot < 6; ++slot) {
            uint32_t keyv = kNone;
            uint32_t pair = 0;
            int cat = -1;
            if (slot < npairs) {
                const int a = PA[slot], b = PB[slot], a3 = PA3[slot < 3 ? slot : 0], b3 = PB3[slot < 3 ? slot : 0];
                const bool three = cnt == 3;
                cat = evidence_category(bm, three ? ids[a3] : ids[a], three ? ids[b3] : ids[b], three ? hs[a3] : hs[a],
                                        three ? hs[b3] : hs[b], thr, cooldown, &pair);
                // aggregation key: world, pair and category (worlds differ within a warp rarely)
                if (cat >= 0) keyv = ((uint32_t)wi * (uint32_t)kPairs + pair) * 5u + (uint32_t)cat;
            }
            const unsigned any = __ballot_sync(0xffffffffu, keyv != kNone);
            if (any == 0) continue;
            const unsigned peers = __match_any_sync(0xffffffffu, keyv);
            if (keyv != kNone && (peers & ((1u << lane) - 1u)) == 0)
                atomicAdd(&worlds[wi].counts[pair].c[cat], __popc(peers));
        }
    }
}

// createCollisionTypeMatrix (:890-972) for every world of the batch; also clears the evidence and resets
// the world's accretion list (k_sort_hist has cleared the cells of the step before's).
__global__ void k_type_matrix(const WorldDev *worlds, int cooldown, int minSize)
{
    kernel_wait();
    const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (uint32_t)kPairs) return;
    const WorldDev &wd = worlds[blockIdx.y];
    if (idx == 0) wd.ctl->acc_count = 0;
    PairCounts *counts = wd.counts;
    uint8_t *bm = wd.type_bitmap;
    const PairCounts pc = counts[idx];
    const int *c = pc.c;
    const uint32_t total = (uint32_t)(c[0] + c[1] + c[2] + c[3] + c[4]);
    if (total == 0) return;  // no evidence: the counts are zero already
    int *cp = counts[idx].c;
    cp[0] = cp[1] = cp[2] = cp[3] = cp[4] = 0;
    const uint32_t packed = bm[idx];
    const bool hasType = packed & 1u;
    const int count = (int)((packed >> 4) & 0x0Fu);
    if (hasType && count < cooldown) {
        bm[idx] = (uint8_t)((packed & 0x0Fu) | (((uint32_t)(count + 1) & 0x0Fu) << 4));
        return;
    }
    if (total < (uint32_t)minSize) return;
    uint32_t out = packed & 0x0Fu;
    const bool hasPol = (packed >> 2) & 1u;
    const bool polA = (packed >> 3) & 1u;
    const int oppA = c[2] + c[4], oppB = c[0] + c[4];
    const int subA = c[0] + c[1] - oppA, subB = c[2] + c[3] - oppB;
    if (c[4] >= c[0] + c[1] && c[4] >= c[2] + c[3]) out |= 3u;
    else if (subA > 0 && subA > subB && (!hasPol || polA)) out = (out & ~2u) | 13u;
    else if (subB > 0 && subB > subA && (!hasPol || !polA)) out = (out & ~10u) | 5u;
    bm[idx] = (uint8_t)out;
}

}  // namespace

int launch_plates(Batch &b, cudaStream_t st)
{
    const int dyn = b.settings.step.plateDynamics;
    if (dyn != TECTO_PLATE_DYNAMICS_OFF && dyn != TECTO_PLATE_DYNAMICS_REFERENCE) {
        set_error("plateDynamics must be TECTO_PLATE_DYNAMICS_OFF or TECTO_PLATE_DYNAMICS_REFERENCE");
        return TECTO_ERR_UNSUPPORTED;
    }
    int rc;
    // plate dynamics and the plate policy read the per-plate mass, size and centre of the step
    const int stats = dyn != TECTO_PLATE_DYNAMICS_OFF || b.settings.step.platePolicy != 0;
    if (stats && (rc = launch_plate_stats(b, st)) != TECTO_OK) return rc;
    // the clear is spread over up to two blocks per SM, 16 KB each at least
    const size_t bytes = sort_clear_bytes(b.sort, b.total);
    const unsigned nw = (unsigned)b.members.size(), nclear = (unsigned)std::min<size_t>((bytes + 16383) / 16384, 304);
    launch_chained(k_plates, nw + nclear, 256, 0, st, b.d_worlds, (int)nw, stats, reinterpret_cast<uint4 *>(b.sort.hist),
                   bytes / 16);
    TECTO_CUDA(cudaGetLastError());
    b.launches += 1;
    return TECTO_OK;
}

int launch_sort_keys(Batch &b, cudaStream_t st)
{
    SortArgs a{};
    a.worlds = b.d_worlds;
    a.vbase = b.d_vbase;
    a.nworlds = (int)b.members.size();
    a.cur_id = b.cur_id;
    a.keys[0] = b.keys[0];
    a.keys[1] = b.keys[1];
    a.vals[0] = b.vals[0];
    a.vals[1] = b.vals[1];
    a.n = b.total;
    a.key_bits = key_bits_for(b.total);
    int half = 0;
    const int rc = run_sort(a, b.sort, st, &half);
    if (rc != TECTO_OK) return rc;
    b.sort_final = half;
    b.launches += 1 + (uint64_t)b.sort.passes;
    return TECTO_OK;
}

int launch_words(Batch &b, cudaStream_t st)
{
    const uint32_t n = (uint32_t)b.total;
    const tecto_kernel_settings &ks = b.settings.kernel;
    // Four positions a thread halve the time where the chip is full; below that one a thread leaves more
    // blocks (steps without erosion, one against four a thread: 256^2 44.3 / 46.2 us, 512^2 51.6 / 53.4,
    // 1001x613 65.7 / 64.5, 1024^2 86.8 / 83.4, 2048^2 224 / 215).
    const int each = n >= (1u << 19) ? 4 : 1;
    launch_chained(each == 4 ? k_words<4> : k_words<1>, (n + each * 256u - 1) / (each * 256u), 256, 0, st, b.keys[b.sort_final],
                   b.vals[b.sort_final], n, b.d_worlds, b.d_vbase, (int)b.members.size(), b.cur_id, b.cur_h,
                   ks.continentalCrustThreshold, ks.collisionTypeUpdateCooldown);
    TECTO_CUDA(cudaGetLastError());
    b.launches += 1;
    return TECTO_OK;
}

int launch_type_matrix(Batch &b, cudaStream_t st)
{
    const tecto_kernel_settings &ks = b.settings.kernel;
    const dim3 grid((kPairs + 255) / 256, (unsigned)b.members.size());
    launch_chained(k_type_matrix, grid, 256, 0, st, b.d_worlds, ks.collisionTypeUpdateCooldown, ks.minCollisionSize);
    TECTO_CUDA(cudaGetLastError());
    b.launches += 1;
    return TECTO_OK;
}

}  // namespace tecto
