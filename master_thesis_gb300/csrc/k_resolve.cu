// k_resolve.cu - per-destination-cell resolve (divergence / movement / convergence), the
// Gaussian uplift fused into the same tile, the divergence-bitmap flip, and accretion.
// Reference: processCollisions and helpers, src/cuda_compute/plate_tectonics_kernel.cu:301-780.
#include "noise.cuh"
#include "tecto_internal.cuh"

namespace tecto {

namespace {

constexpr int RX = 64;   // resolve tile width (cells)
constexpr int RY = 16;   // resolve tile height
constexpr int kMaxBlurRadius = 8;

struct ResolveParams {
    const WorldDev *worlds;
    const uint2 *tiles;
    int cur_h, cur_id;
    float thr;
    float tmin, tmax, tfac;
    float amount;
    float wts[2 * kMaxBlurRadius + 1];
    float tap0;        // what a tap without a convergent cell adds: +0, or NaN with weights that are NaN
    int centre;        // Gaussian uplift of radius 0: the centre tap alone, centre_up[0] on a cell that is not
    float centre_up[2];  // convergent and centre_up[1] on one that is
    float *upl_h;      // reference uplift: processConvergence's records by virtual cell, or null
    uint8_t *upl_t;
    float fricC, fricA, fricS;  // frictionCoefficientContinental / Accretion / Subduction
};

// Plate dynamics' view inside the resolve: velocity and mass per plate, and the block's friction
// sums (fixed point, see PlateAcc).
struct ResolveDyn {
    const float *vel;
    const float *mass;
    unsigned long long *fric;
};

// One world's view inside the resolve kernel.
struct ResolveWorld {
    int W, H;
    uint32_t vbase;
    const uint32_t *word;
    const uint8_t *id_old;
    const float *h_old;
    const uint8_t *bm;
    const uint32_t *div_bitmap;
    uint32_t *has_div;
    unsigned long long *acc;
    uint32_t *acc_list;
    uint32_t *acc_count;
};

// determineCollisionType device function (:611-649)
__device__ __forceinline__ uint32_t pair_type(const uint8_t *bm, uint8_t A, uint8_t B, float hA,
                                              float hB, float thr)
{
    const bool cond = A < B;
    const uint8_t mn = cond ? A : B, mx = cond ? B : A;
    const float mnH = cond ? hA : hB, mxH = cond ? hB : hA;
    const uint32_t packed = bm[tri_index(mn, mx)];
    const uint32_t hasType = packed & 1u, type = (packed >> 1) & 1u, pol = (packed >> 3) & 1u;
    uint32_t out = 0;
    if (hasType && type == 0) {
        if (pol == 1) out = (mnH >= thr) ? (mn == A ? 3u : 4u) : (mn == A ? 1u : 2u);
        if (pol == 0) out = (mxH >= thr) ? (mx == A ? 3u : 4u) : (mx == A ? 1u : 2u);
    }
    return out;
}

__device__ __forceinline__ void mark_accretion(const ResolveParams &p, const ResolveWorld &w,
                                               uint32_t target, uint32_t d, uint8_t owner)
{
    // last writer in cell order wins (the reference writes the byte plainly, :531-555)
    const unsigned long long v = ((unsigned long long)(d + 1u) << 8) | (unsigned long long)(255u - owner);
    const unsigned long long old = atomicMax(w.acc + target, v);
    if (old == 0ull) {
        const uint32_t slot = atomicAdd(w.acc_count, 1u);
        w.acc_list[slot] = target;
    }
}

// processDivergence (:301-362) of cell d = (x, y) without arrivals; returns its new height (before uplift).
__device__ __forceinline__ float diverge_cell(const ResolveParams &p, const ResolveWorld &w, const int2 *s_off, int x,
                                              int y, uint32_t d, uint32_t seed, uint32_t iteration, uint8_t *id_out)
{
    const uint8_t prev = w.id_old[d];
    const int2 o = s_off[prev];
    const uint32_t cvo = w.word[cidx(x - o.x, y - o.y, w.W, w.H)];
    const uint8_t oppId = (uint8_t)((255u - cvo) & 0xFFu);
    uint8_t nid = prev;
    if (cvo != 0u && cvo <= 0xFFu && oppId != prev) {
        const uint8_t mn = prev < oppId ? prev : oppId;
        const uint8_t mx = prev < oppId ? oppId : prev;
        const uint32_t bit = tri_index(mn, mx);
        nid = (w.div_bitmap[bit / 32u] & (1u << (bit % 32u))) ? mn : mx;
        atomicOr(w.has_div + bit / 32u, 1u << (bit % 32u));
    }
    const float noise = simplex3((float)x, (float)y, (float)iteration, 0.01f, (int)seed);
    const float target = p.tmin + noise * (p.tmax - p.tmin);
    *id_out = nid;
    return lerp_p0811(w.h_old[d], target, p.tfac);
}

// processConvergence (:469-584) of cell d = (x, y) with the arrivals cv; returns its new height (before
// uplift).  Leaves its UpliftData (:501-582) for the reference uplift when it is on: heightAddition, the
// sum of each owner pair's lower height, and typeByte.
template <bool DYN>
__device__ __forceinline__ float converge_cell(const ResolveParams &p, const ResolveWorld &w, const int2 *s_off, int x,
                                               int y, uint32_t d, uint32_t cv, uint8_t *id_out, const ResolveDyn &dyn)
{
    const int W = w.W, H = w.H;
    uint8_t ids[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) ids[k] = (uint8_t)(255u - ((cv >> (8 * k)) & 0xFFu));
    const int n = ids[3] != 255 ? 4 : ids[2] != 255 ? 3 : 2;
    const int pairLen = n == 4 ? 6 : n == 3 ? 3 : 1;
    const int PA[6] = {0, 0, 1, 0, 1, 2};
    const int PB[6] = {1, 2, 2, 3, 3, 3};
    float heights[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int k = 0; k < n; ++k) {
        const int2 o = s_off[ids[k]];
        heights[k] = w.h_old[cidx(x - o.x, y - o.y, W, H)];
    }
    uint32_t types[6];
    bool sub[4] = {false, false, false, false};
    for (int a = 0; a < pairLen; ++a) {
        types[a] = pair_type(w.bm, ids[PA[a]], ids[PB[a]], heights[PA[a]], heights[PB[a]], p.thr);
        if (types[a] == 1u || types[a] == 3u) sub[PA[a]] = true;
        else if (types[a] == 2u || types[a] == 4u) sub[PB[a]] = true;
    }
    if (DYN) {
        // applyInelasticCollision's friction (:397-466 with applyElasticVelocityChange :371-394):
        // per arrival, velocity x coefficient x (source height / plate mass); the coefficient is the
        // continental one when a pair with this arrival has type 0, else the accretion one when a
        // pair has type 3 or 4, else the subduction one
        for (int k = 0; k < n; ++k) {
            bool cont = false, accr = false;
            for (int a = 0; a < pairLen; ++a) {
                if (PA[a] != k && PB[a] != k) continue;
                cont = cont || types[a] == 0u;
                accr = accr || types[a] == 3u || types[a] == 4u;
            }
            const float coef = cont ? p.fricC : (accr ? p.fricA : p.fricS);
            const float f = (dyn.vel[ids[k]] * coef) * (heights[k] / dyn.mass[ids[k]]);
            atomicAdd(dyn.fric + ids[k], (unsigned long long)tecto_fix(f, kFricScale, kFricLimit));
        }
    }
    int owner = 0;
    for (int i = 0; i < n; ++i)
        if (!sub[i]) owner = i;
    const uint8_t ownerId = ids[owner];
    float writeH = heights[owner];
    float hadd = 0.0f;
    uint32_t tbyte = 0;
    for (int a = 0; a < pairLen; ++a) {
        const int ia = PA[a], ib = PB[a];
        float hh;
        if (ia == owner) hh = heights[ib];
        else if (ib == owner) hh = heights[ia];
        else continue;
        if (hh > writeH) {  // writeHeight keeps the larger of the pair, the sum the smaller
            const float tmp = hh;
            hh = writeH;
            writeH = tmp;
        }
        hadd = hadd + hh;
        if (ia == owner)
            tbyte |= (types[a] == 2u ? 0u : 1u) | ((uint32_t)(ia & 3) << 1) | ((uint32_t)(ib & 3) << 3);
        else
            tbyte |= (types[a] == 1u ? 0u : 1u) | ((uint32_t)(ib & 3) << 1) | ((uint32_t)(ia & 3) << 3);
        int other = -1;
        if (ia == owner && types[a] == 4u) other = ib;
        else if (ib == owner && types[a] == 3u) other = ia;
        if (other >= 0) {
            const int2 oo = s_off[ids[other]];
            uint32_t target;
            if (oo.x != 0 || oo.y != 0) {
                target = cidx(x - oo.x, y - oo.y, W, H);
            } else {
                const int2 ow = s_off[ownerId];
                target = cidx(x + ow.x, y + ow.y, W, H);
            }
            mark_accretion(p, w, target, d, ownerId);
        }
    }
    if (p.upl_h) {
        p.upl_h[w.vbase + d] = hadd;
        p.upl_t[w.vbase + d] = (uint8_t)tbyte;
    }
    *id_out = ownerId;
    return writeH;
}

// A tile in two parts.  First every thread takes its four cells of a column: cells with one arrival, nearly
// all, are moved at once, the others are listed by class.  Then the lists are worked off densely, the
// divergent cells (their noise is 250 instructions) before the convergent ones (pairs), a warp in one class;
// in place, nearly every warp of a small world held lanes of all three.  The blur reads the convergent cells
// as bits: a row's window of 2R+1 taps is a funnel shift, a tap that is not set adds nothing, and rows and
// warps without any skip their pass (an uplift of +0).
// A batch of 49.7 M cells (100 us at its 13 bytes a cell) 645 -> 395 us, 8192^2 680 -> 400, 2048^2 54 -> 35;
// it waits on its chain of gathers (word, offset, height) and issues in 62% of the cycles.  Eight blocks per
// SM (32 registers) hide more of that than six or five: the batch 395, 500 and 560 us.
template <int R, bool DYN>
__global__ __launch_bounds__(256, 8) void k_resolve(ResolveParams p)
{
    kernel_wait();
    constexpr int SX = RX + 2 * R, SY = RY + 2 * R, kRows = RX * RY / 256;
    constexpr int kTaps = 2 * R + 1;
    static_assert(SX <= 96, "k_resolve: a row's bits and the word after them in four");
    static_assert(256 % RX == 0 && RX * RY == 256 * kRows, "k_resolve: whole rows of threads");
    __shared__ uint32_t s_word[SY * SX];
    __shared__ uint32_t s_bits[R > 0 ? SY : 1][4];  // convergent cells of a row
    __shared__ float s_tmp[(R > 0) ? SY * RX : 1];
    __shared__ int2 s_off[kPlates + 1];
    __shared__ uint16_t s_list[RX * RY];  // divergent cells from the front, convergent ones from the back
    __shared__ int s_ndiv, s_nconv;
    __shared__ uint32_t s_seed, s_iteration;
    // one entry more than plates: an arrival from a cell without a plate (id 255) has no velocity, its friction is 0
    __shared__ float s_vel[DYN ? kPlates + 1 : 1], s_mass[DYN ? kPlates + 1 : 1];
    __shared__ unsigned long long s_fric[DYN ? kPlates + 1 : 1];
    int wi, tx, ty;
    tile_of(p.tiles[blockIdx.x], &wi, &tx, &ty);
    const WorldDev &wd = p.worlds[wi];
    ResolveWorld w;
    w.W = wd.W;
    w.H = wd.H;
    w.vbase = wd.vbase;
    w.word = wd.word;
    w.id_old = wd.id[p.cur_id];
    w.h_old = wd.h[p.cur_h];
    w.bm = wd.type_bitmap;
    w.div_bitmap = wd.div_bitmap;
    w.has_div = wd.has_div;
    w.acc = wd.acc;
    w.acc_list = wd.acc_list;
    w.acc_count = &wd.ctl->acc_count;
    float *h_new = wd.h[p.cur_h ^ 1];
    uint8_t *id_new = wd.id[p.cur_id ^ 1];
    const int t = threadIdx.x;
    const unsigned lane = t & 31u;
    const int x0 = tx * RX, y0 = ty * RY;
    for (int i = t; i < kPlates + 1; i += 256) s_off[i] = wd.off[i];
    if (DYN) {
        for (int i = t; i < kPlates + 1; i += 256) {
            s_vel[i] = i < kPlates ? wd.plates[i].velocity : 0.0f;
            s_mass[i] = i < kPlates ? wd.dyn[i].mass : 1.0f;
            s_fric[i] = 0ull;
        }
    }
    const ResolveDyn dyn{s_vel, s_mass, s_fric};
    if (t == 0) s_ndiv = s_nconv = 0;
    if (t == 32) {
        s_seed = wd.ctl->seed;
        s_iteration = wd.ctl->iteration;
    }
    int conv = R > 0 && p.tap0 != 0.0f;
    int gx[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) gx[k] = wrap_fast(x0 + (int)lane + 32 * k - R, w.W);
    for (int ly = t / 32; ly < SY; ly += 8) {
        const uint32_t *row = w.word + (size_t)wrap_fast(y0 + ly - R, w.H) * w.W;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int c = (int)lane + 32 * k;
            if (32 * k >= SX) continue;
            uint32_t v = 0u;
            if (c < SX) {
                v = row[gx[k]];
                s_word[ly * SX + c] = v;
            }
            if (R > 0) {
                const unsigned m = __ballot_sync(0xffffffffu, v > 0xFFu);
                if (lane == 0) s_bits[ly][k] = m;
                conv |= (int)m;
            }
        }
    }
    const bool blur = R > 0 ? __syncthreads_or(conv) != 0 : (__syncthreads(), false);
    const int lx = t % RX, half = lx / 32;
    // the taps of the warp's half of row ly
    const auto taps = [&](int ly, uint32_t *lo) {
        const uint32_t w0 = s_bits[ly][half], w1 = s_bits[ly][half + 1] & ((1u << (2 * R)) - 1u);
        *lo = __funnelshift_r(w0, w1, lane);
        return (w0 | w1) != 0u || p.tap0 != 0.0f;
    };
    if (blur) {
        // horizontal pass of the separable blur over the convergent-cell field
        for (int ly = t / RX; ly < SY; ly += 256 / RX) {
            uint32_t m;
            float a = p.tap0;
            if (taps(ly, &m)) {
#pragma unroll
                for (int k = 0; k < kTaps; ++k)
                    if (m >> k & 1u) a = a + p.wts[k] * p.amount;
            }
            s_tmp[ly * RX + lx] = a;
        }
        __syncthreads();
    }
    const auto uplift = [&](int lx, int ly) {
        float a = 0.0f;
#pragma unroll
        for (int k = 0; k < kTaps; ++k) a = a + p.wts[k] * s_tmp[(ly + k) * RX + lx];
        return a;
    };
    bool raised = false;  // some tap of the warp's rows is set
    if (blur) {
        uint32_t m;
        static_assert(kRows + 2 * R <= 32, "k_resolve: a lane a row");
        raised = __any_sync(0xffffffffu, (int)lane < kRows + 2 * R && taps(t / RX * kRows + min((int)lane, kRows + 2 * R - 1), &m));
    }
    const int x = x0 + lx;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
        const int ly = t / RX * kRows + i, y = y0 + ly;
        const bool in = x < w.W && y < w.H;
        const uint32_t cv = s_word[(ly + R) * SX + lx + R];
        const uint8_t id0 = (uint8_t)(255u - (cv & 0xFFu)), id1 = (uint8_t)(255u - (cv >> 8 & 0xFFu));
        const bool div = in && cv == 0u, con = in && cv != 0u && id1 != 255;
        if (in && cv != 0u && id1 == 255) {
            // processMovement (:586-609)
            const int2 o = s_off[id0];
            const uint32_t d = (uint32_t)y * (uint32_t)w.W + (uint32_t)x;
            float hn = w.h_old[cidx(x - o.x, y - o.y, w.W, w.H)];
            if (R > 0) hn = hn + (raised ? uplift(lx, ly) : 0.0f);
            else if (p.centre) hn = hn + p.centre_up[cv > 0xFFu];
            h_new[d] = hn;
            id_new[d] = id0;
        }
        const unsigned md = __ballot_sync(0xffffffffu, div), mc = __ballot_sync(0xffffffffu, con);
        if (md | mc) {
            int at = 0;
            if (lane == 0 && md) at = atomicAdd(&s_ndiv, __popc(md));
            if (lane == 1 && mc) at = atomicAdd(&s_nconv, __popc(mc));
            const int ad = __shfl_sync(0xffffffffu, at, 0), ac = __shfl_sync(0xffffffffu, at, 1);
            const unsigned below = (1u << lane) - 1u;
            if (div) s_list[ad + __popc(md & below)] = (uint16_t)(ly * RX + lx);
            if (con) s_list[RX * RY - 1 - ac - __popc(mc & below)] = (uint16_t)(ly * RX + lx);
        }
    }
    __syncthreads();
    const int ndiv = s_ndiv, split = (ndiv + 31) / 32 * 32, end = split + s_nconv;
#pragma unroll 1
    for (int e = t; e < end; e += 256) {
        if (e >= ndiv && e < split) continue;
        const int c = s_list[e < ndiv ? e : RX * RY - 1 - (e - split)];
        const int cy = c / RX, cx = c - cy * RX;
        const int cellx = x0 + cx, celly = y0 + cy;
        const uint32_t d = (uint32_t)celly * (uint32_t)w.W + (uint32_t)cellx;
        uint8_t nid;
        float hn = e < ndiv ? diverge_cell(p, w, s_off, cellx, celly, d, s_seed, s_iteration, &nid)
                            : converge_cell<DYN>(p, w, s_off, cellx, celly, d, s_word[(cy + R) * SX + cx + R], &nid, dyn);
        if (R > 0) hn = hn + (blur ? uplift(cx, cy) : 0.0f);
        else if (p.centre) hn = hn + p.centre_up[s_word[(cy + R) * SX + cx + R] > 0xFFu];
        h_new[d] = hn;
        id_new[d] = nid;
    }
    if (DYN) {
        __syncthreads();
        for (int i = t; i < kPlates; i += 256)
            if (s_fric[i] != 0ull) atomicAdd(&wd.pacc[i].fric, s_fric[i]);
    }
}

// flipDivergedBitmap (:772-780) for one world; clears the per-step bits for the next step
__device__ __forceinline__ void flip_word(const WorldDev &wd, int i)
{
    if (i < kDivWords) {
        wd.div_bitmap[i] ^= wd.has_div[i];
        wd.has_div[i] = 0u;
    }
}

__global__ void k_flip(const WorldDev *worlds)
{
    kernel_wait();
    flip_word(worlds[blockIdx.y], blockIdx.x * blockDim.x + threadIdx.x);
}

// applyAccretion (:747-770) over the cells that received a mark this step; clears the marks.  With flip the
// divergence bitmap, with bump the iteration counter (nothing after it in the step reads it).
// Grid: (blocks, worlds), at least kDivWords threads per world.
__global__ void k_finish(const WorldDev *worlds, int cur_h, int cur_id, float thr, int flip, int bump)
{
    kernel_wait();
    const WorldDev &wd = worlds[blockIdx.y];
    const uint32_t count = wd.ctl->acc_count;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t i = t; i < count; i += gridDim.x * blockDim.x) {
        const uint32_t c = wd.acc_list[i];
        const unsigned long long m = wd.acc[c];
        wd.acc[c] = 0ull;
        const uint8_t value = (uint8_t)(m & 0xFFu);
        wd.acc_u8[c] = value;
        const uint8_t accId = (uint8_t)(255u - value);
        if (accId != 255 && wd.h[cur_h][c] >= thr) wd.id[cur_id][c] = accId;
    }
    if (flip) flip_word(wd, (int)t);
    if (bump && t == 0) wd.ctl->iteration += 1u;
}

__global__ void k_bump_iteration(const WorldDev *worlds, int nworlds)
{
    kernel_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nworlds) worlds[i].ctl->iteration += 1u;
}

}  // namespace

void gaussian_weights(float sigma, int radius, float *out)
{
    double tmp[2 * kMaxBlurRadius + 1];
    double sum = 0.0;
    for (int k = -radius; k <= radius; ++k) {
        tmp[k + radius] = exp(-(double)(k * k) / (2.0 * (double)sigma * (double)sigma));
        sum += tmp[k + radius];
    }
    for (int k = 0; k <= 2 * radius; ++k) out[k] = (float)(tmp[k] / sum);
}

int launch_resolve(Batch &b, bool flip, cudaStream_t st)
{
    const tecto_settings &s = b.settings;
    ResolveParams p{};
    p.worlds = b.d_worlds;
    p.tiles = b.d_tiles[TK_RESOLVE];
    p.cur_h = b.cur_h;
    p.cur_id = b.cur_id;
    p.thr = s.kernel.continentalCrustThreshold;
    p.tmin = s.kernel.divergence_height_target_min;
    p.tmax = s.kernel.divergence_height_target_max;
    p.tfac = s.kernel.divergence_interpolation_factor;
    p.amount = s.step.upliftAmount;
    p.fricC = s.kernel.frictionCoefficientContinental;
    p.fricA = s.kernel.frictionCoefficientAccretion;
    p.fricS = s.kernel.frictionCoefficientSubduction;
    if (s.step.upliftMode == TECTO_UPLIFT_REFERENCE) {
        p.upl_h = b.upref.upl_h;
        p.upl_t = b.upref.upl_t;
        if (!p.upl_h) {
            set_error("reference uplift scratch not prepared");
            return TECTO_ERR_INVALID;
        }
    }
    int R = 0;
    if (s.step.upliftMode == TECTO_UPLIFT_GAUSSIAN) {
        R = s.step.upliftRadius;
        if (R < 0 || R > kMaxBlurRadius) {
            set_error("upliftRadius must be in 0..8");
            return TECTO_ERR_UNSUPPORTED;
        }
        gaussian_weights(s.step.upliftSigma, R, p.wts);
        p.tap0 = p.wts[0] * 0.0f;  // the weights are finite or all NaN
        p.centre = R == 0;
        p.centre_up[0] = 0.0f + p.wts[0] * (0.0f + p.wts[0] * 0.0f);
        p.centre_up[1] = 0.0f + p.wts[0] * (0.0f + p.wts[0] * p.amount);
    }
    static constexpr void (*kern[2][kMaxBlurRadius + 1])(ResolveParams) = {
        {k_resolve<0, false>, k_resolve<1, false>, k_resolve<2, false>, k_resolve<3, false>, k_resolve<4, false>,
         k_resolve<5, false>, k_resolve<6, false>, k_resolve<7, false>, k_resolve<8, false>},
        {k_resolve<0, true>, k_resolve<1, true>, k_resolve<2, true>, k_resolve<3, true>, k_resolve<4, true>,
         k_resolve<5, true>, k_resolve<6, true>, k_resolve<7, true>, k_resolve<8, true>}};
    const int dyn = s.step.plateDynamics == TECTO_PLATE_DYNAMICS_REFERENCE ? 1 : 0;
    launch_chained(kern[dyn][R], (unsigned)b.ntiles[TK_RESOLVE], 256, 0, st, p);
    if (flip) launch_chained(k_flip, dim3((kDivWords + 255) / 256, (unsigned)b.members.size()), 256, 0, st, b.d_worlds);
    TECTO_CUDA(cudaGetLastError());
    b.launches += flip ? 2 : 1;
    b.cur_h ^= 1;
    b.cur_id ^= 1;
    return TECTO_OK;
}

int launch_finish(Batch &b, bool flip, bool bump, cudaStream_t st)
{
    if (b.settings.step.plateDynamics == TECTO_PLATE_DYNAMICS_REFERENCE) {
        const int rc = launch_plate_motion(b, st);  // executeIteration: before applyAccretion
        if (rc != TECTO_OK) return rc;
    }
    static_assert(4 * 256 >= kDivWords, "k_finish: one thread per divergence word");
    launch_chained(k_finish, dim3(4, (unsigned)b.members.size()), 256, 0, st, b.d_worlds, b.cur_h, b.cur_id,
                   b.settings.kernel.continentalCrustThreshold, (int)flip, (int)bump);
    TECTO_CUDA(cudaGetLastError());
    b.launches += 1;
    return TECTO_OK;
}

int launch_bump_iteration(Batch &b, cudaStream_t st)
{
    const int n = (int)b.members.size();
    launch_chained(k_bump_iteration, (n + 255) / 256, 256, 0, st, b.d_worlds, n);
    TECTO_CUDA(cudaGetLastError());
    b.launches += 1;
    return TECTO_OK;
}

}  // namespace tecto
