// tecto_batch.cu - batches of worlds: device tables, per-phase (world, tile) work lists,
// batch-level buffers, ping-pong alignment of members, and the step driver with CUDA-graph
// replay.  A world stepped on its own uses a private batch of one.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "tecto_internal.cuh"

namespace tecto {

namespace {

size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }

void drop_graphs(Batch &b)
{
    for (int i = 0; i < 16; ++i) {
        if (b.graph_valid[i]) cudaGraphExecDestroy(b.graphs[i]);
        b.graph_valid[i] = false;
    }
}

// the tiles of a W x H world, row by row
void add_tiles(int world, int W, int H, int tx, int ty, std::vector<uint2> &out)
{
    const int nx = (W + tx - 1) / tx, ny = (H + ty - 1) / ty;
    for (int y = 0; y < ny; ++y)
        for (int x = 0; x < nx; ++x) out.push_back(tile_pack(world, x, y));
}

void build_tiles(const Batch &b, int kind, std::vector<uint2> &out)
{
    int tx = 0, ty = 0;
    tile_extent(kind, kind == TK_THERMAL ? b.thermal_variant : b.hydro_variant, &tx, &ty);
    out.clear();
    for (size_t wi = 0; wi < b.members.size(); ++wi)
        add_tiles((int)wi, b.members[wi]->W, b.members[wi]->H, tx, ty, out);
}

// every member's columns cut into strips of `inner`
std::vector<uint4> build_strips(const Batch &b, int inner, unsigned long long *rows)
{
    std::vector<uint4> out;
    unsigned long long r = 0;
    for (size_t wi = 0; wi < b.members.size(); ++wi) {
        const tecto_world *w = b.members[wi];
        for (int x0 = 0; x0 < w->W; x0 += inner) {
            const int iw = std::min(inner, w->W - x0);
            out.push_back(make_uint4((unsigned)wi, (unsigned)x0, (unsigned)iw, (unsigned)r));
            r += (unsigned long long)w->H;
        }
    }
    *rows = r;
    return out;
}

// Copy the state of group `g` (0 height, 1 water/sediment/flux, 2 plate ids) of world w into
// ping-pong half `to`.
int move_half(tecto_world *w, int g, int to, cudaStream_t st)
{
    const size_t N = w->N;
    const int from = to ^ 1;
    if (g == 0) {
        TECTO_CUDA(cudaMemcpyAsync(w->dev.h[to], w->dev.h[from], N * 4, cudaMemcpyDeviceToDevice, st));
    } else if (g == 1) {
        TECTO_CUDA(cudaMemcpyAsync(w->dev.w[to], w->dev.w[from], N * 4, cudaMemcpyDeviceToDevice, st));
        TECTO_CUDA(cudaMemcpyAsync(w->dev.s[to], w->dev.s[from], N * 4, cudaMemcpyDeviceToDevice, st));
        TECTO_CUDA(cudaMemcpyAsync(w->dev.flux[to], w->dev.flux[from], N * 16, cudaMemcpyDeviceToDevice, st));
    } else {
        TECTO_CUDA(cudaMemcpyAsync(w->dev.id[to], w->dev.id[from], N, cudaMemcpyDeviceToDevice, st));
    }
    return TECTO_OK;
}

// Whether two worlds step alike: every parameter a step reads (the kernel and step settings and the
// CCL period).  The rest of SimulationSettings (plate count, seed, Voronoi generations) is read by
// the initialisation only, so worlds initialised differently may share a batch.
bool same_step_settings(const tecto_settings &a, const tecto_settings &b)
{
    return std::memcmp(&a.kernel, &b.kernel, sizeof(a.kernel)) == 0 &&
           std::memcmp(&a.step, &b.step, sizeof(a.step)) == 0 && a.sim.iterationsForCCL == b.sim.iterationsForCCL;
}

}  // namespace

int batch_join(Batch &b, tecto_world *w, cudaStream_t st)
{
    if (std::find(b.members.begin(), b.members.end(), w) != b.members.end()) return TECTO_OK;
    if ((int)b.members.size() >= kMaxBatchWorlds) {
        set_error("batch is full (1024 worlds)");
        return TECTO_ERR_INVALID;
    }
    if (b.members.empty()) {
        b.settings = w->settings;
        b.has_settings = true;
        b.device = w->device;
        b.cur_h = w->cur_h;
        b.cur_wsf = w->cur_wsf;
        b.cur_id = w->cur_id;
    } else {
        if (!same_step_settings(b.settings, w->settings)) {
            set_error("all worlds of a batch must share the same step settings");
            return TECTO_ERR_INVALID;
        }
        if (w->device != b.device) {
            set_error("all worlds of a batch must live on the same device");
            return TECTO_ERR_INVALID;
        }
        int rc;
        if (w->cur_h != b.cur_h && (rc = move_half(w, 0, b.cur_h, st)) != TECTO_OK) return rc;
        if (w->cur_wsf != b.cur_wsf && (rc = move_half(w, 1, b.cur_wsf, st)) != TECTO_OK) return rc;
        if (w->cur_id != b.cur_id && (rc = move_half(w, 2, b.cur_id, st)) != TECTO_OK) return rc;
        w->cur_h = b.cur_h;
        w->cur_wsf = b.cur_wsf;
        w->cur_id = b.cur_id;
    }
    b.members.push_back(w);
    b.dirty = true;
    return TECTO_OK;
}

int batch_leave(Batch &b, tecto_world *w)
{
    auto it = std::find(b.members.begin(), b.members.end(), w);
    if (it == b.members.end()) {
        set_error("world is not a member of this batch");
        return TECTO_ERR_INVALID;
    }
    b.members.erase(it);
    b.dirty = true;
    if (b.members.empty()) b.has_settings = false;
    return TECTO_OK;
}

void batch_release(Batch &b)
{
    drop_graphs(b);
    uplift_ref_release(b);
    if (b.table_arena) cudaFree(b.table_arena);
    if (b.arena) cudaFree(b.arena);
    if (b.stage) cudaFree(b.stage);
    for (int f = 0; f < 6; ++f) {
        for (int k = 0; k < 2; ++k) {
            if (b.up_stage[f][k]) cudaFree(b.up_stage[f][k]);
            if (b.down_stage[f][k]) cudaFree(b.down_stage[f][k]);
            b.up_stage[f][k] = b.down_stage[f][k] = nullptr;
            cudaEvent_t *evs[4] = {&b.ev_up_ready[f][k], &b.ev_up_free[f][k], &b.ev_down_ready[f][k],
                                   &b.ev_down_free[f][k]};
            for (cudaEvent_t *e : evs) {
                if (*e) cudaEventDestroy(*e);
                *e = nullptr;
            }
        }
        b.up_bytes[f] = b.down_bytes[f] = 0;
        b.n_staged[f] = b.n_committed[f] = b.n_gathered[f] = b.n_fetched[f] = 0;
    }
    b.table_arena = nullptr;
    b.arena = nullptr;
    b.stage = nullptr;
    b.stage_bytes = 0;
    b.capacity = 0;
    b.arena_bytes = 0;
    b.table_bytes = 0;
    b.members.clear();
}

// Tile variant and digit width: explicit settings first, then the autotuner's choice for this
// batch (or its cached choice for the shape class), then the defaults.
// The default digit width: 9 bits where they save a pass.  A step's phases other than erosion, us, with 8 and 9
// bits: 512^2 57.6 / 53.4 (18-bit keys), 2048^2 234 / 238 (22), 8192^2 3258 / 3049 (26).
static int default_radix_bits(size_t cells)
{
    const int kb = key_bits_for(cells);
    return sort_passes_for(kb, 9) < sort_passes_for(kb, 8) ? 9 : kDefaultRadixBits;
}

// The default thermal variant: one iteration with tiles (variant 4, two iterations a launch) against the
// march (5), us: 512^2 5.3 / 6.5, 1024^2 11.6 / 8.4, 2048^2 37.4 / 19.2, 8192^2 570 / 224; whole steps at 1001x613
// 430 / 435, 900x800 444 / 443, 40 worlds of 1.1 M cells 783 / 746.  Variant 3 (three iterations a launch, more
// warps a tile) against 4 in whole steps: 64^2 112.6 / 115.9, 256^2 126.4 / 129.0, 384^2 162.2 / 165.0, 512^2
// 220.3 / 220.2, 600^2 259 / 254.
// Parameters that the march's packed forms do not take (a threshold below 2^-32, a negative amplitude): ten
// iterations with tiles / the march, threshold 0 and 1e-12, us: 1024^2 115 / 156 and 104 / 139, 1500x1100 174 / 194
// and 157 / 171, 2048^2 407 / 402 and 363 / 348, 4096^2 1616 / 1347 and 1458 / 1162.
// The default hydraulic variant: the one whose two sub-iterations a model of the measured shapes puts lowest.  The
// times are one chip's, and so is its number of SMs here, which belongs to them.
// Tiles run in waves of 152 SMs x the tiles an SM holds, and a wave's time depends on how many it holds; the
// march's blocks take equal shares of the strips' rows (with what a strip's start costs, k_hydro_march.cu), at
// 0.38 us a row, 0.42 counted as odd widths take longer.  Whole steps, us, the model's choice marked:
//                    256^2  384^2  512^2  600^2  724^2  1001x613  900x800  1024^2  1200x1000  12 worlds  40 worlds
//   1 (52x9)         129*   233    298    409    536     660       710     945      1098       625        1194
//   2 (52x12)        143    178    225    290    379     447       479     640       721       451         780
//   3 (52x24)        162    168*   237    251*   346*    428       484     572       648       428         754
//   4 (52x28)        173    178    251    269    368     392*      453     545       621       396*        682*
//   5 (52x20)        157    208    222*   307    379     457       461     593       656       454         766
//   9 (march)        253           283    323    390     433       443*    533*      581*      474         750
// (12 worlds 200 to 300 wide, 0.55 M cells; 40 of 128 to 256, 1.08 M.)  60 such worlds (1.6 M) take 986 with the march, which
// it chooses, against 957; 100 (2.5 M) 1461 against 1471; 20 of 240x400 882 against 1039.
static int default_hydro_variant(const Batch &b, bool split)
{
    // 50 dt >= 1.5: the march's transport reaches two cells; no two at once.  20 sub-iterations with 1 / 2 / 3 / 4, us:
    // 256^2 138 / 142 / 176 / 221, 512^2 215 / 198 / 217 / 272, 701x503 276 / 254 / 267 / 288, 1024^2 643 / 546 / 504 /
    // 538, 2048^2 2711 / 2067 / 1806 / 1840, 4096^2 10489 / 7869 / 6706 / 6671.
    if (split)
        return b.total <= (size_t)1 << 17 ? 1 : b.total <= (size_t)1 << 20 ? 3 : 4;
    constexpr double kSms = 152.0;
    struct Shape {
        int ty, held;
        double us[3];  // a wave of 1, 2, 3 tiles an SM
    };
    static const Shape shapes[5] = {
        {9, 1, {5.6}}, {12, 3, {8.3, 11.5, 15.0}}, {24, 2, {10.2, 16.2}}, {28, 2, {11.3, 17.6}}, {20, 2, {9.7, 14.7}}};
    int best = 1;
    double best_us = INFINITY;
    for (int v = 0; v < 5; ++v) {
        double tiles = 0.0;
        for (const tecto_world *w : b.members)
            tiles += (double)((w->W + 51) / 52) * (double)((w->H + shapes[v].ty - 1) / shapes[v].ty);
        const double wave = kSms * shapes[v].held, full = floor(tiles / wave), rest = ceil((tiles - full * wave) / kSms);
        const double us = full * shapes[v].us[shapes[v].held - 1] + (rest > 0.0 ? shapes[v].us[(int)rest - 1] : 0.0);
        if (us < best_us) {
            best_us = us;
            best = v + 1;
        }
    }
    // strip-rows of two at once and of one, with the rows that starting a strip costs
    double rows2 = 0.0, start2 = 0.0, rows1 = 0.0, start1 = 0.0;
    for (const tecto_world *w : b.members) {
        const double n2 = (w->W + kMarchTwoInner - 1) / kMarchTwoInner, n1 = (w->W + kMarchInner - 1) / kMarchInner;
        rows2 += n2 * w->H;
        start2 += n2 * 36.0;
        rows1 += n1 * w->H;
        start1 += n1 * 24.0;
    }
    const double march = 5.0 * rows2 <= 6.0 * rows1 ? 0.42 * ((rows2 + start2) / kSms + 36.0)
                                                    : 2.0 * 0.46 * ((rows1 + start1) / (2.0 * kSms) + 24.0);
    return march < best_us ? kHydroMarchVariant : best;
}

static void choose_tuning(Batch &b, int *variant, int *rb, int *tvariant)
{
    *tvariant = thermal_variant_for(b.settings);
    if (*tvariant == 0) *tvariant = b.tuned_thermal;
    if (*tvariant == 0) {
        const size_t march = thermal_packed(b.settings.kernel) ? kThermalMarchMinCells : kThermalScalarMarchMinCells;
        *tvariant = b.total >= march                ? kThermalMarchVariant
                    : b.total <= kThermalSmallCells ? kThermalSmallVariant
                                                    : kDefaultThermalVariant;
    }
    *variant = hydro_variant_for(b.settings);
    if (*variant == 0) *variant = b.tuned_hydro;
    // Variants 1 and 7, tiles of 8 and 4 rows, are shapes for batches that leave SMs idle; larger ones take 4.  20
    // sub-iterations with 1 / 7 / 4, us: 256^2 62 / 123 / 104, 512^2 216 / 304 / 168, 1024^2 785 / 1004 / 389, 4096^2
    // 12833 / 16821 / 5839; the split path 138 / 143 / 221, 215 / 277 / 272, 643 / 909 / 538, 10489 / 16037 / 6671, and
    // 701x503 274 / 341 / 286.
    const bool split = !hydro_fused(b, b.settings.step.hydraulicDt);
    if ((*variant == 1 || *variant == 7) && b.total > (split ? kShortTileSplitCells : kShortTileCells)) *variant = 4;
    if (*variant == 0) {
        if (b.dirty) b.hydro_default[0] = b.hydro_default[1] = 0;  // of other members
        int &d = b.hydro_default[split];
        if (d == 0) d = default_hydro_variant(b, split);
        *variant = d;
    }
    *rb = b.settings.step.sortRadixBits;
    if (!valid_radix_bits(*rb)) *rb = valid_radix_bits(b.tuned_rb) ? b.tuned_rb : default_radix_bits(b.total);
}

int batch_prepare(Batch &b, cudaStream_t st)
{
    if (b.dirty && !b.members.empty()) {  // membership changed: cached autotuner choice, if any
        size_t cells = 0;
        b.long_side = 0;
        for (const tecto_world *w : b.members) {
            cells += w->N;
            b.long_side = std::max(b.long_side, std::max(w->W, w->H));
        }
        b.total = cells;
        // A choice of another size says less than the defaults' model: taken from an octave away at most in all.
        // (2048^2 with the tiles that 1024^2 was tuned to 1980 us a step, with the default 1490.)
        constexpr int kTunedSteps = 2;
        int th = 0, tr = 0, tt = 0, steps = 0;
        if (tune_lookup(b.device, cells, b.members.size(), &th, &tr, &tt, &steps)) {
            const bool near = steps <= kTunedSteps;
            b.tuned_hydro = near ? th : 0;
            b.tuned_rb = near ? tr : 0;
            b.tuned_thermal = near ? tt : 0;
        }
    }
    int variant = 0, rb = 0, tvariant = 0;
    choose_tuning(b, &variant, &rb, &tvariant);
    if (!b.dirty && variant == b.hydro_variant && rb == b.sort.radix_bits && tvariant == b.thermal_variant)
        return TECTO_OK;
    if (b.members.empty()) {
        set_error("batch has no worlds");
        return TECTO_ERR_INVALID;
    }
    int rc = ensure_kernel_attributes();
    if (rc != TECTO_OK) return rc;
    if ((rc = sort_kernel_attributes()) != TECTO_OK) return rc;
    drop_graphs(b);
    b.hydro_variant = variant;
    b.thermal_variant = tvariant;
    const size_t n = b.members.size();
    std::vector<uint32_t> vbase(n + 1);
    size_t total = 0;
    for (size_t i = 0; i < n; ++i) {
        vbase[i] = (uint32_t)total;
        total += b.members[i]->N;
    }
    if (total > (size_t)kValueMask) {
        set_error("batch holds more than 2^30 cells");
        return TECTO_ERR_INVALID;
    }
    vbase[n] = (uint32_t)total;
    b.total = total;
    std::vector<WorldDev> table(n);
    for (size_t i = 0; i < n; ++i) {
        b.members[i]->dev.vbase = vbase[i];
        table[i] = b.members[i]->dev;
    }
    std::vector<uint2> tiles[TK_COUNT];
    size_t need = a256(n * sizeof(WorldDev)) + a256((n + 1) * 4);
    for (int k = 0; k < TK_COUNT; ++k) {
        build_tiles(b, k, tiles[k]);
        b.ntiles[k] = (int)tiles[k].size();
        need += a256(tiles[k].size() * sizeof(uint2));
    }
    std::vector<uint4> strips[ST_COUNT];
    for (int k = 0; k < ST_COUNT; ++k) {
        const int inner = k == ST_THERMAL ? kThermalInner : k == ST_HYDRO_TWO ? kMarchTwoInner : kMarchInner;
        strips[k] = build_strips(b, inner, &b.strips[k].rows);
        b.strips[k].n = (int)strips[k].size();
        need += a256(strips[k].size() * sizeof(uint4));
    }
    if (need > b.table_bytes) {
        if (b.table_arena) cudaFree(b.table_arena);
        b.table_arena = nullptr;
        b.table_bytes = 0;
        TECTO_CUDA(cudaMalloc(&b.table_arena, need));
        b.table_bytes = need;
    }
    // the tables as one image and one copy: a first pass 210 -> 181 us against a copy a table
    std::vector<char> image(need);
    size_t at = 0;
    const auto put = [&](const void *data, size_t bytes) {
        memcpy(image.data() + at, data, bytes);
        char *p = (char *)b.table_arena + at;
        at += a256(bytes);
        return (void *)p;
    };
    b.d_worlds = (WorldDev *)put(table.data(), n * sizeof(WorldDev));
    b.d_vbase = (uint32_t *)put(vbase.data(), (n + 1) * 4);
    for (int k = 0; k < TK_COUNT; ++k) b.d_tiles[k] = (uint2 *)put(tiles[k].data(), tiles[k].size() * sizeof(uint2));
    for (int k = 0; k < ST_COUNT; ++k) b.strips[k].d = (uint4 *)put(strips[k].data(), strips[k].size() * sizeof(uint4));
    TECTO_CUDA(cudaMemcpyAsync(b.table_arena, image.data(), need, cudaMemcpyHostToDevice, st));
    // batch-level buffers: key/value ping-pong for `capacity` cells, the control block, then the
    // sort scratch of the current size and digit width
    const int kb = key_bits_for(total);
    {
        const size_t cap = std::max(b.capacity, total);
        const size_t need = 4 * a256(cap * 4) + a256(sizeof(BatchCtl)) + a256(sort_scratch_bytes(total, kb, rb));
        if (need > b.arena_bytes) {
            if (b.arena) cudaFree(b.arena);
            b.arena = nullptr;
            b.capacity = 0;
            b.arena_bytes = 0;
            TECTO_CUDA(cudaMalloc(&b.arena, need));
            TECTO_CUDA(cudaMemsetAsync(b.arena, 0, need, st));
            const size_t arr = a256(cap * 4);
            char *q = (char *)b.arena;
            b.keys[0] = (uint32_t *)q;
            b.keys[1] = (uint32_t *)(q + arr);
            b.vals[0] = (uint32_t *)(q + 2 * arr);
            b.vals[1] = (uint32_t *)(q + 3 * arr);
            b.bctl = (BatchCtl *)(q + 4 * arr);
            b.capacity = cap;
            b.arena_bytes = need;
        }
    }
    {
        char *q = (char *)b.arena + 4 * a256(b.capacity * 4) + a256(sizeof(BatchCtl));
        sort_scratch_carve(q, total, kb, rb, &b.sort);
    }
    if ((rc = uplift_ref_prepare(b, st)) != TECTO_OK) return rc;
    // the error word may now sit where a larger batch kept look-back status words
    TECTO_CUDA(cudaMemsetAsync(b.sort.error, 0, 4, st));
    TECTO_CUDA(cudaStreamSynchronize(st));
    b.dirty = false;
    return TECTO_OK;
}

// ccl: 0 none, 1 every member (the caller checked it is due), 2 members whose counter is due
int batch_enqueue_step(Batch &b, cudaStream_t st, int ccl)
{
    int rc;
    const tecto_settings &s = b.settings;
    if ((rc = launch_plates(b, st)) != TECTO_OK) return rc;
    if ((rc = launch_sort_keys(b, st)) != TECTO_OK) return rc;
    if ((rc = launch_words(b, st)) != TECTO_OK) return rc;
    if ((rc = launch_type_matrix(b, st)) != TECTO_OK) return rc;
    if ((rc = launch_resolve(b, false, st)) != TECTO_OK) return rc;
    if (s.step.upliftMode == TECTO_UPLIFT_REFERENCE && (rc = launch_uplift_ref(b, st)) != TECTO_OK) return rc;
    if ((rc = launch_thermal(b, s.step.thermalIterations, st)) != TECTO_OK) return rc;
    if ((rc = launch_hydraulic(b, s.step.hydraulicIterations, s.step.hydraulicDt, st)) != TECTO_OK) return rc;
    // the labelling and the policy read the iteration counter: with either it advances after them
    const bool bump = !ccl && !s.step.platePolicy;
    if ((rc = launch_finish(b, true, bump, st)) != TECTO_OK) return rc;
    if (ccl && (rc = launch_ccl(b, s.step.cclConnectivity, ccl == 2, st)) != TECTO_OK) return rc;
    if (s.step.platePolicy && (rc = launch_plate_policy(b, ccl, st)) != TECTO_OK) return rc;
    return bump ? TECTO_OK : launch_bump_iteration(b, st);
}

static void sync_members(Batch &b)
{
    for (tecto_world *w : b.members) {
        w->cur_h = b.cur_h;
        w->cur_wsf = b.cur_wsf;
        w->cur_id = b.cur_id;
    }
}

int batch_step(Batch &b, int nsteps, cudaStream_t st) { return batch_step_graph(b, nsteps, st, true); }

// use_graph false: plain launches (worth it right after a membership change, when a captured
// graph would be used once)
int batch_step_graph(Batch &b, int nsteps, cudaStream_t st, bool use_graph)
{
    int rc = batch_prepare(b, st);
    if (rc != TECTO_OK) return rc;
    const int period = b.settings.sim.iterationsForCCL > 0 ? b.settings.sim.iterationsForCCL : 1;
    for (int s = 0; s < nsteps; ++s) {
        int ccl;
        if (b.members.size() == 1) ccl = (b.members[0]->iteration % (uint32_t)period == 0) ? 1 : 0;
        else ccl = 2;
        const uint64_t before = b.launches;
        if (st == nullptr || !use_graph) {  // the legacy stream cannot be captured
            if ((rc = batch_enqueue_step(b, st, ccl)) != TECTO_OK) return rc;
        } else {
            const int key = b.cur_h | (b.cur_wsf << 1) | (b.cur_id << 2) | ((ccl == 1 ? 1 : 0) << 3);
            if (!b.graph_valid[key]) {
                cudaGraph_t g = nullptr;
                TECTO_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
                rc = batch_enqueue_step(b, st, ccl);
                const cudaError_t ce = cudaStreamEndCapture(st, &g);
                if (rc != TECTO_OK) {
                    if (g) cudaGraphDestroy(g);
                    return rc;
                }
                if (ce != cudaSuccess) return cuda_fail(ce, "cudaStreamEndCapture");
                cudaGraphExec_t ex = nullptr;
                const cudaError_t ie = cudaGraphInstantiate(&ex, g, 0);
                cudaGraphDestroy(g);
                if (ie != cudaSuccess) return cuda_fail(ie, "cudaGraphInstantiate");
                b.graphs[key] = ex;
                b.graph_valid[key] = true;
                b.graph_end[key][0] = b.cur_h;
                b.graph_end[key][1] = b.cur_wsf;
                b.graph_end[key][2] = b.cur_id;
                b.graph_end[key][3] = b.sort_final;
                b.graph_launches[key] = b.launches - before;
                TECTO_CUDA(cudaGraphLaunch(ex, st));
            } else {
                TECTO_CUDA(cudaGraphLaunch(b.graphs[key], st));
                b.cur_h = b.graph_end[key][0];
                b.cur_wsf = b.graph_end[key][1];
                b.cur_id = b.graph_end[key][2];
                b.sort_final = b.graph_end[key][3];
                b.launches += b.graph_launches[key];
            }
        }
        const uint64_t step_launches = b.launches - before;
        for (tecto_world *w : b.members) {
            w->iteration += 1;
            w->launches += step_launches;
        }
        sync_members(b);
    }
    return TECTO_OK;
}

}  // namespace tecto

using namespace tecto;

extern "C" {

int tecto_selftest_tiles(int width, int height, int world, int tile_x, int tile_y, unsigned long long *bad)
{
    if (width < 1 || height < 1 || (long long)width * height > 1ll << 30 || world < 0 || world >= kMaxBatchWorlds ||
        tile_x < 1 || tile_y < 1 || tile_x > 1 << 16 || tile_y > 1 << 16 || !bad)
        return TECTO_ERR_INVALID;
    const size_t nx = ((size_t)width + tile_x - 1) / tile_x, ny = ((size_t)height + tile_y - 1) / tile_y;
    if (nx > 1u << 26 || ny > 1u << 28 || nx * ny > 1u << 27) return TECTO_ERR_INVALID;  // no phase has that many
    std::vector<uint2> tiles;
    add_tiles(world, width, height, tile_x, tile_y, tiles);
    *bad = tiles.size() > nx * ny ? tiles.size() - nx * ny : nx * ny - tiles.size();
    for (size_t i = 0; i < tiles.size(); ++i) {
        int w, x, y;
        tile_of(tiles[i], &w, &x, &y);
        if (w != world || (size_t)x != i % nx || (size_t)y != i / nx) *bad += 1;
    }
    return TECTO_OK;
}

int tecto_batch_create(tecto_batch **out)
{
    if (!out) return TECTO_ERR_INVALID;
    *out = new (std::nothrow) tecto_batch();
    return *out ? TECTO_OK : TECTO_ERR_OOM;
}

int tecto_batch_destroy(tecto_batch *batch)
{
    if (!batch) return TECTO_OK;
    for (tecto_world *w : batch->b.members) w->in_batch = nullptr;
    batch_release(batch->b);
    delete batch;
    return TECTO_OK;
}

int tecto_batch_add(tecto_batch *batch, tecto_world *world, tecto_stream_t stream)
{
    if (!batch || !world) return TECTO_ERR_INVALID;
    if (world->in_batch && world->in_batch != world->own) {
        set_error("world already belongs to a batch");
        return TECTO_ERR_INVALID;
    }
    const int rc = batch_join(batch->b, world, (cudaStream_t)stream);
    if (rc == TECTO_OK) world->in_batch = &batch->b;
    return rc;
}

int tecto_batch_remove(tecto_batch *batch, tecto_world *world)
{
    if (!batch || !world) return TECTO_ERR_INVALID;
    const int rc = batch_leave(batch->b, world);
    if (rc == TECTO_OK) world->in_batch = nullptr;
    return rc;
}

int tecto_batch_step(tecto_batch *batch, int nSteps, tecto_stream_t stream)
{
    if (!batch || nSteps < 0) return TECTO_ERR_INVALID;
    if (batch->b.members.empty()) return TECTO_OK;
    return batch_step(batch->b, nSteps, (cudaStream_t)stream);
}

int tecto_batch_phase_hydraulic(tecto_batch *batch, int iterations, float dt, tecto_stream_t stream)
{
    if (!batch || iterations < 0 || !std::isfinite(dt)) return TECTO_ERR_INVALID;
    Batch &b = batch->b;
    if (b.members.empty()) return TECTO_OK;
    const cudaStream_t st = (cudaStream_t)stream;
    int rc = batch_prepare(b, st);
    if (rc != TECTO_OK) return rc;
    const uint64_t before = b.launches;
    rc = launch_hydraulic(b, iterations, dt, st);
    for (tecto_world *w : b.members) w->launches += b.launches - before;
    sync_members(b);
    return rc;
}

int tecto_batch_phase_thermal(tecto_batch *batch, int iterations, tecto_stream_t stream)
{
    if (!batch || iterations < 0) return TECTO_ERR_INVALID;
    Batch &b = batch->b;
    if (b.members.empty()) return TECTO_OK;
    const cudaStream_t st = (cudaStream_t)stream;
    int rc = batch_prepare(b, st);
    if (rc != TECTO_OK) return rc;
    const uint64_t before = b.launches;
    rc = launch_thermal(b, iterations, st);
    for (tecto_world *w : b.members) w->launches += b.launches - before;
    sync_members(b);
    return rc;
}

int tecto_batch_size(const tecto_batch *batch, int *worlds, size_t *cells)
{
    if (!batch) return TECTO_ERR_INVALID;
    size_t c = 0;
    for (const tecto_world *w : batch->b.members) c += w->N;
    if (worlds) *worlds = (int)batch->b.members.size();
    if (cells) *cells = c;
    return TECTO_OK;
}

int tecto_batch_launch_count(const tecto_batch *batch, uint64_t *count)
{
    if (!batch || !count) return TECTO_ERR_INVALID;
    *count = batch->b.launches;
    return TECTO_OK;
}

int tecto_batch_check(tecto_batch *batch, tecto_stream_t stream)
{
    if (!batch) return TECTO_ERR_INVALID;
    for (tecto_world *w : batch->b.members) {
        const int rc = tecto_world_check(w, stream);
        if (rc != TECTO_OK) return rc;
    }
    if (batch->b.sort.error) {
        uint32_t e = 0;
        TECTO_CUDA(cudaMemcpy(&e, batch->b.sort.error, 4, cudaMemcpyDeviceToHost));
        if (e) {
            cudaMemset(batch->b.sort.error, 0, 4);
            set_error("a bounded device-side wait gave up");
            return TECTO_ERR_DEVICE_TIMEOUT;
        }
    }
    return TECTO_OK;
}

}  // extern "C"
