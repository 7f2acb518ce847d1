// C ABI of the library (include/stencil_b200.h): argument checks, kernel choice,
// tensor-map setup and error reporting around the sm_100a kernels.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <cmath>
#include <cstdio>
#include <map>
#include <mutex>
#include <string>
#include <tuple>

#include "dispatch.h"
#include "kernels.h"
#include "stencil_b200.h"

// Library-wide device error word (one per device context); kernels receive its
// address and record bounded-wait failures in it.
__device__ int g_sb200_device_error = 0;

namespace sb200 {

namespace {

thread_local std::string t_last_error;

int fail(int code, const std::string& msg) {
    t_last_error = msg;
    return code;
}

int cuda_fail(cudaError_t e, const char* where) {
    return fail(SB200_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
}

std::mutex g_dev_mu;
int* g_err_ptr[64] = {};

int* device_error_ptr() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lock(g_dev_mu);
    if (!g_err_ptr[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_sb200_device_error) != cudaSuccess) return nullptr;
        g_err_ptr[dev] = static_cast<int*>(p);
    }
    return g_err_ptr[dev];
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int to_desc(const sb200_grid* g, GridDesc* d) {
    if (!g) return fail(SB200_ERR_INVALID, "grid descriptor is NULL");
    if (g->nx < 0 || g->ny < 0 || g->nz < 0)
        return fail(SB200_ERR_INVALID, "negative grid extent");
    if (g->nx > (1 << 30) || g->ny > (1 << 30) || g->nz > (1 << 30))
        return fail(SB200_ERR_INVALID, "grid extent above 2^30");
    if (!(g->dx > 0.f) || !(g->dy > 0.f) || !(g->dz > 0.f) || !std::isfinite(g->dx) ||
        !std::isfinite(g->dy) || !std::isfinite(g->dz))
        return fail(SB200_ERR_INVALID, "grid spacing must be positive and finite");
    if (!std::isfinite(g->dt)) return fail(SB200_ERR_INVALID, "dt must be finite");
    d->nx = g->nx;
    d->ny = g->ny;
    d->nz = g->nz;
    d->dx = g->dx;
    d->dy = g->dy;
    d->dz = g->dz;
    d->dt = g->dt;
    return SB200_OK;
}

// ── pencil configuration: override or heuristic ──────────────────────────────

struct Override {
    int variant = -1;
    int zchunks = 1;
};
std::mutex g_cfg_mu;
Override g_override[4];

bool valid_kind(int kind) {
    return kind == SB200_KIND_WAVE_F32 || kind == SB200_KIND_HEAT_F32 ||
           kind == SB200_KIND_WAVE_F16 || kind == SB200_KIND_WAVE2_F32;
}

int variant_count(int kind) {
    if (kind == SB200_KIND_WAVE2_F32) return leap2_variant_count();
    return kind == SB200_KIND_WAVE_F16 ? pencil_f16_variant_count()
                                       : pencil_f32_variant_count(kind == SB200_KIND_HEAT_F32);
}

const char* variant_name(int kind, int v) {
    if (kind == SB200_KIND_WAVE2_F32) return leap2_variant_name(v);
    if (kind == SB200_KIND_WAVE_F16) return pencil_f16_variant_name(v);
    return pencil_f32_variant_name(kind == SB200_KIND_HEAT_F32, v);
}

int sm_count() {
    int dev = 0, n = 148;
    if (cudaGetDevice(&dev) == cudaSuccess)
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n;
}

// ── untuned choice: a cost model over tiles and z splits ──────────────────────

// Cost of sweeping an interior of inz planes in chunks of zlen with `tiles` columns, on
// SMs that hold `resident` CTAs each, in planes of a fully occupied SM: whole waves of
// zlen + start planes (start: what filling a CTA's rings costs), and a last wave in which
// the busiest SM holds k CTAs: they take (k / resident)^0.62 of a full wave's time (fewer
// CTAs hide less latency).
double split_cost(int64_t tiles, int inz, int zlen, int resident, int sms, double start) {
    const int64_t ctas = tiles * ((inz + zlen - 1) / zlen);
    const int64_t slots = int64_t(sms) * resident;
    const int64_t rest = ctas % slots;
    double waves = double(ctas / slots);
    if (rest) waves += std::pow(double((rest + sms - 1) / sms) / resident, 0.62);
    return waves * (zlen + start);
}

// What a step costs beside other runs (Sharing, dispatch.h): its part of the sweeping, at
// least its latency over the steps that overlap it, and a tenth of its latency on top.
constexpr double kOverlap[] = {1.0, 1.25, 3.0};

// (cost, z chunks) of every distinct chunk length, cheapest first.
std::vector<std::pair<double, int>> rank_splits(int64_t tiles, int inz, int resident, double start,
                                                int sharing) {
    const int sms = std::max(1, sm_count());
    resident = std::max(1, resident);
    std::vector<std::pair<double, int>> out;
    int last = 0;
    for (int n = 1; n <= std::min(inz, 512); ++n) {
        const int zlen = (inz + n - 1) / n;
        if (zlen == last) continue;
        last = zlen;
        const int zc = (inz + zlen - 1) / zlen;
        const double alone = split_cost(tiles, inz, zlen, resident, sms, start);
        const double work = double(tiles) * zc / (double(sms) * resident) * (zlen + start);
        out.emplace_back(sharing ? std::max(work, alone / kOverlap[sharing]) + 0.1 * alone : alone, zc);
    }
    std::stable_sort(out.begin(), out.end());
    if (out.empty()) out.emplace_back(1.0, 1);
    return out;
}

// Tiles an untuned launch chooses from, with the cost of a point relative to the table's
// other tiles where the step's fields fit L2 (126 MB) and where they do not (0: not
// taken).  Model and weights were fitted to 22 grids from 64^3 to 1024^3 (cubes, thin and
// flat boxes; graph replays), every tile at 11 to 23 splits: the picks are on average 1.0
// % (FP32), 2.3 % (heat) and 1.1 % (FP16) from the best of them, at worst 6 to 8 %.
// What the tables say:
//   * acoustic, beyond L2: 16 warps per SM and wide rows.  One 64 x 32 CTA of 8 warps per
//     SM was the default; it follows the SM clock, and full-range data holds that at 1.55
//     GHz under the 1000 W cap.  1024^3, sustained: 2930 us (t64x32_r2_s8_a3), 2830
//     (t64x32_r2_s6_a2, two CTAs), 2790 (t128x16_r2_s6_a2), 2670 (t128x32_r2_s7_a2, 1.33
//     staged words a point instead of 1.41);
//   * small grids: as many short CTAs as there are slots (acoustic 64^3 4.9 -> 3.2 us,
//     320^3 96 -> 84 us; heat 160^3 10.5 -> 8.1 us; FP16 96^3 6.0 -> 5.2 us).
//   * reference order: 59 separately rounded operations a point, bound by issue and power;
//     the one-row tile covers odd extents best, two-row tiles spend fewer instructions a
//     point (acoustic 384^3 178 us with t32x16_r1_s8_a4, 174 / 174 / 170 with the other
//     three in the table's order; 512^3 438 against 410 / 408 / 415; 160 x 150 x 170 14.1
//     against 17.7 / 19.1 / 21.2; heat 512^3 301 against 288, 160 x 150 x 170 12.1 against
//     13.7).
//   * runs at once, each on its stream, all take one tile: CTAs of unlike kernels do not
//     share the SMs well, and short chunks that fill an idle device only add planes on a full
//     one.  48 runs of 96 to 192 cells, us per step of all: each its own choice 652, the
//     same splits on t64x32_r2_s6_a2 418, with 8 chunks 386 (t128x16_r2_s6_a2 420,
//     t32x32_r2_s8_a4 421); FP16 339, h64x16_s8_a4 265 (h64x32_s8_a2 278); heat 298,
//     t64x16_r2_s8 274; reference order 499, t32x16_r1_s8_a4 403-416 (t64x32_r2_s6_a2 439).
struct Candidate {
    const char* name;
    double in_l2, beyond;
};
struct Family {
    double start;
    int step_bytes;  // per cell: the fields a step keeps in use
    Candidate tiles[4];
    const char* shared;       // the tile of runs that share the device
    const char* many_beyond;  // and that of many, beyond L2
};
// Kinds of choice beyond the public ones: the reference order on the pencil tiles, the
// composition pre-pass, and the ragged kernels.
enum Internal : int { kExactWave = 4, kExactHeat, kPrepass, kRaggedWave, kRaggedHeat };
bool reference_order(int kind) { return kind == kExactWave || kind == kExactHeat; }
// The public kind whose override holds for a kind (of the ragged kernels, its z split).
int public_kind(int kind) {
    return kind == kExactHeat || kind == kRaggedHeat ? SB200_KIND_HEAT_F32
           : kind >= kExactWave                      ? SB200_KIND_WAVE_F32
                                                     : kind;
}

const Family kFamilies[] = {
    // SB200_KIND_WAVE_F32
    {2.1, 12,
     {{"t32x32_r2_s8_a4", 1.38, 0}, {"t64x32_r2_s6_a2", 1.04, 1.074}, {"t128x16_r2_s6_a2", 1.0, 0},
      {"t128x32_r2_s7_a2", 0, 1.0}},
     "t64x32_r2_s6_a2", "t64x32_r2_s6_a2"},
    // SB200_KIND_HEAT_F32
    {6.7, 8, {{"t32x32_r2_s8", 1.05, 0}, {"t64x16_r2_s8", 1.0, 1.114}, {"t128x16_r2_s8", 0, 1.0}},
     "t64x16_r2_s8", "t128x16_r2_s8"},
    // SB200_KIND_WAVE_F16
    {4.3, 6, {{"h64x16_s8_a4", 0, 1.02}, {"h64x32_s8_a2", 1.1, 0}, {"h128x16_s8_a2", 1.0, 1.0}},
     "h64x16_s8_a4", "h64x16_s8_a4"},
    {},  // SB200_KIND_WAVE2_F32: one tile
    // kExactWave
    {2.1, 12,
     {{"t32x16_r1_s8_a4", 1.0, 1.0}, {"t64x32_r2_s6_a2", 0.95, 0.95},
      {"t128x16_r2_s6_a2", 0.94, 0.94}, {"t128x32_r2_s7_a2", 0.92, 0.92}},
     "t32x16_r1_s8_a4", "t32x16_r1_s8_a4"},
    // kExactHeat
    {2.1, 8, {{"t32x16_r1_s8", 1.0, 1.0}, {"t64x16_r2_s8", 0.96, 0.96}}, "t32x16_r1_s8",
     "t32x16_r1_s8"},
    // kPrepass beyond L2, 32 interior planes and more (else as the acoustic step: 2048 x 1025
    // x 17 74 us, with this choice 81).  It writes two fields and pays more for a chunk's
    // start; the acoustic step's choice took 10 to 14 % longer than the one 64 x 32 CTA per SM
    // before it on some grids (192 x 1024 x 1024 805 and 715 us, 440^3 310 and 283).  Over 22
    // grids now at most 4 % longer than the better of the two, 715 and 281.
    {10, 12, {{"t64x32_r2_s8_a3", 0, 1.02}, {"t128x32_r2_s7_a2", 0, 0.96}}, "", ""},
};
constexpr double kL2Bytes = 126e6;
constexpr int64_t kSharedCells = 48000000;

int variant_by_name(int kind, const char* name) {
    for (int v = 0; v < variant_count(kind); ++v)
        if (std::strcmp(variant_name(kind, v), name) == 0) return v;
    return -1;
}

int64_t column_tiles(int kind, int v, const GridDesc& g) {
    return kind == SB200_KIND_WAVE2_F32  ? leap2_ctas(v, g, 1)
           : kind == SB200_KIND_WAVE_F16 ? pencil_f16_ctas(v, g, 1)
                                         : pencil_f32_ctas(kind == SB200_KIND_HEAT_F32, v, g, 1);
}

int resident_ctas(int kind, int v) {
    return kind == SB200_KIND_WAVE2_F32  ? leap2_resident(v)
           : kind == SB200_KIND_WAVE_F16 ? pencil_f16_resident(v)
                                         : pencil_f32_resident(kind == SB200_KIND_HEAT_F32, v);
}

// The cheapest tile and split of a family (a public kind's or a reference-order one).
PencilConfig cheapest(int family, const GridDesc& g, int sharing) {
    const bool beyond = double(g.size()) * kFamilies[family].step_bytes > kL2Bytes;
    if (family == kPrepass && (!beyond || g.nz < 40)) family = SB200_KIND_WAVE_F32;
    const Family& f = kFamilies[family];
    const bool exact = reference_order(family);
    const int kind = public_kind(family);
    PencilConfig best;
    double cost = 0;
    for (const Candidate& c : f.tiles) {
        double weight = beyond ? c.beyond : c.in_l2;
        if (sharing && c.name)
            weight = std::strcmp(c.name, sharing == kMany && beyond ? f.many_beyond : f.shared) == 0;
        const int v = c.name && weight > 0 ? variant_by_name(kind, c.name) : -1;
        if (v < 0) continue;
        const PencilBoxes b = kind == SB200_KIND_WAVE_F16
                                  ? pencil_f16_boxes(v)
                                  : pencil_f32_boxes(kind == SB200_KIND_HEAT_F32, v);
        const int resident = exact ? pencil_f32_resident(kind == SB200_KIND_HEAT_F32, v, true)
                                   : resident_ctas(kind, v);
        const auto s =
            rank_splits(column_tiles(kind, v, g), static_cast<int>(g.nz - 8), resident, f.start, sharing)
                .front();
        const double t = s.first * weight * b.points * resident;
        if (cost == 0 || t < cost) {
            cost = t;
            best.variant = v;
            best.zchunks = s.second;
        }
    }
    return best;
}

// For steps whose caller says nothing of others: the other streams (up to 4) that steps on
// the device went to since the last one on `stream`, if that is among the last 32 (the
// first step on a stream, a capture's for instance, is taken to be alone).  Steps of unlike
// grids on several streams meet on the SMs as runs do (four of 96 to 192 cells 55.8 us a
// round with each its own choice, 40.5 before the cost model, 33.3 now).
constexpr int kFromStreams = -1;
int streams_beside(void* stream) {
    constexpr unsigned kLast = 32;
    struct Ring {
        std::atomic<uintptr_t> stream[kLast] = {};  // + 1; 0: none yet
        std::atomic<unsigned> at{0};
    };
    static Ring rings[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    Ring& r = rings[dev & 63];
    const uintptr_t mine = reinterpret_cast<uintptr_t>(stream) + 1;
    const unsigned at = r.at.fetch_add(1, std::memory_order_relaxed);
    uintptr_t seen[4];
    int n = 0;
    bool again = false;
    for (unsigned k = 1; k < kLast && !again; ++k) {
        const uintptr_t v = r.stream[(at - k) % kLast].load(std::memory_order_relaxed);
        again = v == mine;
        if (!again && v && n < 4 && std::find(seen, seen + n, v) == seen + n) seen[n++] = v;
    }
    r.stream[at % kLast].store(mine, std::memory_order_relaxed);
    return again ? n : 0;
}

PencilConfig choose(int kind, const GridDesc& g, int sharing = kAlone) {
    {
        std::lock_guard<std::mutex> lock(g_cfg_mu);
        // (the reference order keeps its own tile where it has no form of the given one)
        const Override o = g_override[public_kind(kind)];
        if (o.variant >= 0) {
            PencilConfig c;
            c.variant = !reference_order(kind) || pencil_f32_has_exact(kind == kExactHeat, o.variant)
                            ? o.variant
                            : cheapest(kind, g, sharing).variant;
            c.zchunks = std::max(1, o.zchunks);
            return c;
        }
    }
    // steps that fill the device many times over gain nothing by agreeing on a tile (four of
    // 384 to 640 cells, each its own and shared: acoustic 1225 and 1289 us, heat 767 and 852,
    // reference order 1459 and 1588; of 200 to 320 cells 148.8 and 148.6, eight 383 and 353)
    if (g.size() > kSharedCells) sharing = kAlone;
    PencilConfig c;
    if ((kind < 4 || kind == kPrepass) && tuned_choice(public_kind(kind), g, &c)) return c;
    // Heuristic pick, memoised per (kind, extents, device, sharing): launches stay cheap
    // on the host.
    static std::mutex memo_mu;
    static std::map<std::tuple<int, int64_t, int64_t, int64_t, int, int>, PencilConfig> memo;
    int dev = 0;
    cudaGetDevice(&dev);
    const auto key = std::make_tuple(kind, g.nx, g.ny, g.nz, dev, sharing);
    std::lock_guard<std::mutex> lock(memo_mu);
    auto it = memo.find(key);
    if (it != memo.end()) return it->second;
    const int inz = static_cast<int>(g.nz - 8);
    const double start = kFamilies[SB200_KIND_WAVE_F32].start;
    if (kind >= kRaggedWave) {
        c.zchunks = rank_splits(ragged_ctas(g, 1), inz, ragged_resident(kind == kRaggedHeat, g), start,
                                sharing)
                        .front()
                        .second;
    } else if (kind == SB200_KIND_WAVE2_F32) {
        c.variant = std::max(0, variant_by_name(kind, "l32x32_r1_s8"));
        c.zchunks = zchunk_ranking(kind, c.variant, g, 1).front();
    } else {
        c = cheapest(kind, g, sharing);
    }
    memo[key] = c;
    return c;
}

// Interior points from which reference-order steps run on staged planes; below, the
// one-thread-per-point kernel, which fills no rings first.  Acoustic step in a graph, one
// thread per point against staged, us: aligned 64^3 3.1 and 3.8, 72^3 3.5 and 4.0, 80^3 5.5
// and 4.7, 88^3 6.3 and 4.8; ragged 72^3 4.6 and 4.5, 80^3 5.4 and 5.8, 88^3 6.3 and 5.8
// (heat crosses at the same sizes).
constexpr int64_t kPencilPoints = int64_t(5) << 16, kRaggedPoints = int64_t(7) << 16;

// Whether reference-order steps of a grid are worth staging: enough points, and not too few
// rows for the tiles.  The staged kernels compute whole tiles of at least 16 rows, the
// one-thread-per-point kernel rows of 32 columns; a point of the latter costs about 3
// (ragged rows; from 3.0 on) or 3.5 of the former.  Acoustic step, one thread per point
// against staged, us: 264 columns of 3000 - 8 planes with 4 rows (4 tile points to one) 26.7
// and 35.2, 5 rows (3.2) 36.9 and 35.3, 6 rows 42.4 and 35.4; 265 columns (ragged; 3.6 and
// 3.0 to one) with 5 rows 41.0 and 45.8, with 6 47.1 and 45.9.  A single row took up to 4.6
// times as long staged (73 x 9 x 20000: 24.7 and 114).  Grids too tall for a launch of the
// one-thread-per-point kernel are staged all the same.
bool staged_pays(const GridDesc& g, bool ragged) {
    if (g.interior() < (ragged ? kRaggedPoints : kPencilPoints)) return false;
    if (!naive_fits(g)) return true;
    const int64_t lanes = (g.nx - 8 + 31) / 32 * 32, rows = g.ny - 8;
    return ragged ? ragged_covered(g) <= 3 * lanes * rows
                  : 2 * ((rows + 15) / 16 * 16) <= 7 * rows;
}

bool pencil_ok(const GridDesc& g, std::initializer_list<const void*> ptrs) {
    if (g.nx % 4 != 0) return false;
    for (const void* p : ptrs)
        if (p && !aligned16(p)) return false;
    return true;
}

int finish_launch(cudaError_t e, const char* where) {
    if (e != cudaSuccess) return cuda_fail(e, where);
    return SB200_OK;
}

// Encodes the tensor maps a pencil variant reads: the haloed box over the
// stencil field and, where the variant stages them by TMA, the tile box over
// p_prev and vel2.
int pencil_maps(bool heat, int v, const GridDesc& g, const void* field, const void* prev,
                const void* vel2, PencilMaps* m, const char* where) {
    const PencilBoxes b = pencil_f32_boxes(heat, v);
    int rc = tensor_map_3d(&m->p, field, g.nx, g.ny, g.nz, 4, b.halo_x, b.halo_y);
    m->prev = m->p;
    m->vel2 = m->p;
    if (!rc && b.aux_tma) {
        rc = tensor_map_3d(&m->prev, prev, g.nx, g.ny, g.nz, 4, b.tile_x, b.tile_y);
        if (!rc) rc = tensor_map_3d(&m->vel2, vel2, g.nx, g.ny, g.nz, 4, b.tile_x, b.tile_y);
    }
    if (rc)
        return fail(SB200_ERR_CUDA, std::string(where) + ": tensor map encode failed (" +
                                        std::to_string(rc) + ")");
    return SB200_OK;
}

int ragged_maps(bool heat, const GridDesc& g, const void* field, const void* prev, const void* vel2,
                PencilMaps* m, const char* where) {
    const PencilBoxes b = ragged_boxes(heat, g);
    const int64_t rows = g.ny * g.nz;
    int rc = tensor_map_rows4(&m->p, field, g.nx, rows, b.halo_x, b.halo_y);
    m->prev = m->p;
    m->vel2 = m->p;
    if (!rc && b.aux_tma) {
        rc = tensor_map_rows4(&m->prev, prev, g.nx, rows, b.tile_x, b.tile_y);
        if (!rc) rc = tensor_map_rows4(&m->vel2, vel2, g.nx, rows, b.tile_x, b.tile_y);
    }
    if (rc)
        return fail(SB200_ERR_CUDA, std::string(where) + ": tensor map encode failed (" +
                                        std::to_string(rc) + ")");
    return SB200_OK;
}

int wave_step(const float* p, const float* p_prev, const float* vel2, float* p_next,
              const sb200_grid* grid, const SourceDesc& src, void* stream, bool exact,
              const char* where, int sharing = kFromStreams) {
    const int64_t src_index = src.idx;
    GridDesc g;
    if (int rc = to_desc(grid, &g)) return rc;
    if (!p || !p_prev || !vel2 || !p_next)
        return fail(SB200_ERR_INVALID, std::string(where) + ": NULL field pointer");
    if (p_next == p)
        return fail(SB200_ERR_INVALID, std::string(where) + ": p_next must not alias p_cur");
    if (src_index >= g.size())
        return fail(SB200_ERR_INVALID, std::string(where) + ": source index outside the grid");
    if (!g.has_interior()) return SB200_OK;  // no interior point: nothing to update
    if (sharing == kFromStreams) sharing = sharing_of(streams_beside(stream));
    auto st = static_cast<cudaStream_t>(stream);
    if ((!exact || staged_pays(g, false)) && pencil_ok(g, {p, p_prev, vel2, p_next})) {
        const PencilConfig cfg = choose(exact ? int(kExactWave) : int(SB200_KIND_WAVE_F32), g, sharing);
        PencilMaps maps;
        if (int rc = pencil_maps(false, cfg.variant, g, p, p_prev, vel2, &maps, where)) return rc;
        return finish_launch(launch_wave_pencil_f32(maps, p_prev, vel2, p_next, g, src, cfg,
                                                    device_error_ptr(), st, exact),
                             where);
    }
    if (staged_pays(g, true) && ragged_ok(g) && aligned16(p) && aligned16(p_prev) && aligned16(vel2)) {
        PencilMaps maps;
        if (int rc = ragged_maps(false, g, p, p_prev, vel2, &maps, where)) return rc;
        return finish_launch(launch_wave_ragged_f32(maps, p_next, g, src,
                                                    choose(kRaggedWave, g, sharing).zchunks,
                                                    device_error_ptr(), st),
                             where);
    }
    return finish_launch(launch_wave_naive(p, p_prev, vel2, p_next, g, src, st), where);
}

int heat_step(const float* u, float* u_next, const sb200_grid* grid, float alpha, void* stream,
              bool exact, const char* where, int sharing = kFromStreams) {
    GridDesc g;
    if (int rc = to_desc(grid, &g)) return rc;
    if (!u || !u_next) return fail(SB200_ERR_INVALID, std::string(where) + ": NULL field pointer");
    if (u == u_next)
        return fail(SB200_ERR_INVALID, std::string(where) + ": u_next must not alias u");
    if (!std::isfinite(alpha))
        return fail(SB200_ERR_INVALID, std::string(where) + ": alpha must be finite");
    if (!g.has_interior()) return SB200_OK;
    if (sharing == kFromStreams) sharing = sharing_of(streams_beside(stream));
    const float alpha_dt = alpha * g.dt;
    auto st = static_cast<cudaStream_t>(stream);
    PencilMaps maps;
    if ((!exact || staged_pays(g, false)) && pencil_ok(g, {u, u_next})) {
        const PencilConfig cfg = choose(exact ? int(kExactHeat) : int(SB200_KIND_HEAT_F32), g, sharing);
        if (int rc = pencil_maps(true, cfg.variant, g, u, nullptr, nullptr, &maps, where)) return rc;
        return finish_launch(launch_heat_pencil_f32(maps, u_next, g, alpha_dt, cfg,
                                                    device_error_ptr(), st, exact),
                             where);
    }
    if (staged_pays(g, true) && ragged_ok(g) && aligned16(u)) {
        if (int rc = ragged_maps(true, g, u, nullptr, nullptr, &maps, where)) return rc;
        return finish_launch(launch_heat_ragged_f32(maps, u_next, g, alpha_dt,
                                                    choose(kRaggedHeat, g, sharing).zchunks,
                                                    device_error_ptr(), st),
                             where);
    }
    return finish_launch(launch_heat_naive(u, u_next, g, alpha_dt, st), where);
}

// Two acoustic steps in one sweep (leap2_f32.cu).  outputs_may_alias lets the
// tuner time it with one scratch buffer for both outputs (their values unused).
int wave_step2(const float* p, const float* p_prev, const float* vel2, float* out1, float* out2,
               const sb200_grid* grid, const SourceDesc& src, float w1, void* stream,
               bool outputs_may_alias, const char* where) {
    GridDesc g;
    if (int rc = to_desc(grid, &g)) return rc;
    if (!p || !p_prev || !vel2 || !out1 || !out2)
        return fail(SB200_ERR_INVALID, std::string(where) + ": NULL field pointer");
    if (p == p_prev || (out1 == out2 && !outputs_may_alias))
        return fail(SB200_ERR_INVALID, std::string(where) + ": the five fields must be distinct");
    for (const float* o : {static_cast<const float*>(out1), static_cast<const float*>(out2)})
        if (o == p || o == p_prev || o == vel2)
            return fail(SB200_ERR_INVALID,
                        std::string(where) + ": an output aliases an input (five distinct fields)");
    if (src.idx >= g.size())
        return fail(SB200_ERR_INVALID, std::string(where) + ": source index outside the grid");
    if (!g.has_interior()) return SB200_OK;
    if (!pencil_ok(g, {p, p_prev, vel2, out1, out2}))
        return fail(SB200_ERR_UNSUPPORTED,
                    std::string(where) + ": needs nx % 4 == 0 and 16-byte aligned fields");
    const PencilConfig cfg = choose(SB200_KIND_WAVE2_F32, g);
    const PencilBoxes b = leap2_boxes(cfg.variant);
    PencilMaps maps;
    int rc = tensor_map_3d(&maps.p, p, g.nx, g.ny, g.nz, 4, b.halo_x, b.halo_y);
    if (!rc) rc = tensor_map_3d(&maps.prev, p_prev, g.nx, g.ny, g.nz, 4, b.tile_x, b.tile_y);
    if (!rc) rc = tensor_map_3d(&maps.vel2, vel2, g.nx, g.ny, g.nz, 4, b.tile_x, b.tile_y);
    if (rc)
        return fail(SB200_ERR_CUDA, std::string(where) + ": tensor map encode failed (" +
                                        std::to_string(rc) + ")");
    return finish_launch(launch_leap2_f32(maps, out1, out2, g, src, w1, cfg, device_error_ptr(),
                                          static_cast<cudaStream_t>(stream)),
                         where);
}

SourceDesc host_source(int64_t idx, float amp) {
    SourceDesc s;
    s.idx = idx;
    s.w = amp;
    return s;
}

int wave_step_f16(const uint16_t* p, uint16_t* p_prev_next, const uint16_t* k,
                  const sb200_grid* grid, const SourceDesc& src, const sb200_f16_scale* scale,
                  int phase, void* stream, int sharing = kFromStreams) {
    const char* where = "sb200_wave_step_f16";
    GridDesc g;
    if (int rc = to_desc(grid, &g)) return rc;
    if (!p || !p_prev_next || !k || !scale)
        return fail(SB200_ERR_INVALID, std::string(where) + ": NULL pointer");
    if (p == p_prev_next)
        return fail(SB200_ERR_INVALID, std::string(where) + ": p_next must not alias p");
    if (phase < 0 || phase > 2) return fail(SB200_ERR_INVALID, std::string(where) + ": bad phase");
    if (src.idx >= g.size())
        return fail(SB200_ERR_INVALID, std::string(where) + ": source index outside the grid");
    if (src.idx >= 0 && src.wavelet && !src.step)
        return fail(SB200_ERR_INVALID, std::string(where) + ": wavelet without step pointer");
    if (!g.has_interior()) return SB200_OK;
    if (g.nx % 8 != 0 || !aligned16(p) || !aligned16(p_prev_next) || !aligned16(k))
        return fail(SB200_ERR_UNSUPPORTED,
                    std::string(where) + ": needs nx % 8 == 0 and 16-byte aligned fields");
    if (sharing == kFromStreams) sharing = sharing_of(streams_beside(stream));
    const PencilConfig cfg = choose(SB200_KIND_WAVE_F16, g, sharing);
    const PencilBoxes b = pencil_f16_boxes(cfg.variant);
    PencilMaps maps;
    int rc = tensor_map_3d(&maps.p, p, g.nx, g.ny, g.nz, 2, b.halo_x, b.halo_y);
    if (!rc) rc = tensor_map_3d(&maps.prev, p_prev_next, g.nx, g.ny, g.nz, 2, b.tile_x, b.tile_y);
    if (!rc) rc = tensor_map_3d(&maps.vel2, k, g.nx, g.ny, g.nz, 2, b.tile_x, b.tile_y);
    if (rc)
        return fail(SB200_ERR_CUDA, std::string(where) + ": tensor map encode failed (" +
                                        std::to_string(rc) + ")");
    return finish_launch(
        launch_wave_pencil_f16(maps, p_prev_next, g, src, reinterpret_cast<const F16Scale*>(scale),
                               phase, cfg, device_error_ptr(), static_cast<cudaStream_t>(stream)),
        where);
}

}  // namespace

// Step dispatch with a full source descriptor (trace included), for the run
// engine; the public entry points wrap these.
int dispatch_wave_f32(const float* p, const float* p_prev, const float* vel2, float* p_next,
                      const sb200_grid* grid, const SourceDesc& src, void* stream, bool exact,
                      int sharing) {
    return wave_step(p, p_prev, vel2, p_next, grid, src, stream, exact,
                     exact ? "sb200_wave_step_exact_f32" : "sb200_wave_step_f32", sharing);
}

int dispatch_heat_f32(const float* u, float* u_next, const sb200_grid* grid, float alpha,
                      void* stream, bool exact, int sharing) {
    return heat_step(u, u_next, grid, alpha, stream, exact,
                     exact ? "sb200_heat_step_exact_f32" : "sb200_heat_step_f32", sharing);
}

int prepare_step(const sb200_grid* grid, bool heat, bool half, bool exact, int sharing) {
    GridDesc g;
    if (int rc = to_desc(grid, &g)) return rc;
    if (!g.has_interior()) return SB200_OK;
    device_error_ptr();
    if (half) {
        pencil_f16_resident(choose(SB200_KIND_WAVE_F16, g, sharing).variant);
    } else if (g.nx % 4 == 0 && (!exact || staged_pays(g, false))) {
        const int kind = heat ? (exact ? int(kExactHeat) : int(SB200_KIND_HEAT_F32))
                              : (exact ? int(kExactWave) : int(SB200_KIND_WAVE_F32));
        pencil_f32_resident(heat, choose(kind, g, sharing).variant, exact);
    } else if (staged_pays(g, true) && ragged_ok(g)) {
        choose(heat ? kRaggedHeat : kRaggedWave, g, sharing);
        ragged_resident(heat, g);
    }
    return SB200_OK;
}

int dispatch_wave2_f32(const float* p, const float* p_prev, const float* vel2, float* out1,
                       float* out2, const sb200_grid* grid, const SourceDesc& src, float w1,
                       void* stream, bool outputs_may_alias) {
    return wave_step2(p, p_prev, vel2, out1, out2, grid, src, w1, stream, outputs_may_alias,
                      "sb200_wave_step2_f32");
}

int dispatch_wave_f16(const uint16_t* p, uint16_t* p_prev_next, const uint16_t* k,
                      const sb200_grid* grid, const SourceDesc& src, const sb200_f16_scale* scale,
                      int phase, void* stream, int sharing) {
    return wave_step_f16(p, p_prev_next, k, grid, src, scale, phase, stream, sharing);
}

int set_error(int code, const std::string& msg) { return fail(code, msg); }

int* device_error_word() { return device_error_ptr(); }

std::vector<int> zchunk_ranking(int kind, int v, const GridDesc& g, int max_n) {
    // (two steps per sweep: a chunk reads 16 halo planes)
    const auto ranked =
        rank_splits(column_tiles(kind, v, g), static_cast<int>(g.nz - 8), resident_ctas(kind, v),
                    kind == SB200_KIND_WAVE2_F32 ? 6.0 : kFamilies[kind].start, kAlone);
    std::vector<int> out;
    for (const auto& s : ranked)
        if (static_cast<int>(out.size()) < max_n) out.push_back(s.second);
    return out;
}

}  // namespace sb200

using namespace sb200;

extern "C" {

int sb200_version(void) { return 100; }

const char* sb200_last_error(void) { return t_last_error.c_str(); }

int sb200_device_error(int clear) {
    int* p = device_error_ptr();
    if (!p) return fail(SB200_ERR_CUDA, "sb200_device_error: no usable CUDA device");
    int v = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_sb200_device_error, sizeof(int));
    if (e != cudaSuccess) return cuda_fail(e, "sb200_device_error");
    if (clear && v) {
        const int zero = 0;
        e = cudaMemcpyToSymbol(g_sb200_device_error, &zero, sizeof(int));
        if (e != cudaSuccess) return cuda_fail(e, "sb200_device_error");
    }
    return v;
}

int sb200_upload_fd_coefficients(void) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaSetDevice(dev);  // initialises the primary context
    if (e != cudaSuccess) return cuda_fail(e, "sb200_upload_fd_coefficients");
    return SB200_OK;
}

int sb200_launch_naive(const float* p_cur, const float* p_prev, const float* vel2,
                       float* p_next, const sb200_grid* grid, void* stream) {
    return wave_step(p_cur, p_prev, vel2, p_next, grid, host_source(-1, 0.f), stream, true,
                     "sb200_launch_naive");
}

int sb200_launch_tiled(const float* p_cur, const float* p_prev, const float* vel2,
                       float* p_next, const sb200_grid* grid, void* stream) {
    return wave_step(p_cur, p_prev, vel2, p_next, grid, host_source(-1, 0.f), stream, false,
                     "sb200_launch_tiled");
}

int sb200_launch_slab(const float* p_cur, const float* p_prev, const float* vel2,
                      float* p_next, const sb200_grid* grid, void* stream) {
    return wave_step(p_cur, p_prev, vel2, p_next, grid, host_source(-1, 0.f), stream, false,
                     "sb200_launch_slab");
}

int sb200_wave_step_f32(const float* p, const float* p_prev, const float* vel2, float* p_next,
                        const sb200_grid* grid, int64_t src_index, float src_amp,
                        void* stream) {
    return wave_step(p, p_prev, vel2, p_next, grid, host_source(src_index, src_amp), stream,
                     false, "sb200_wave_step_f32");
}

int sb200_wave_step2_f32(const float* p, const float* p_prev, const float* vel2, float* p_next,
                         float* p_next2, const sb200_grid* grid, int64_t src_index,
                         float src_amp0, float src_amp1, void* stream) {
    return wave_step2(p, p_prev, vel2, p_next, p_next2, grid, host_source(src_index, src_amp0),
                      src_amp1, stream, false, "sb200_wave_step2_f32");
}

int sb200_wave_step2_dev_f32(const float* p, const float* p_prev, const float* vel2,
                             float* p_next, float* p_next2, const sb200_grid* grid,
                             int64_t src_index, const float* wavelet, const int* step,
                             int step_offset, float* trace, void* stream) {
    if (src_index >= 0 && (!wavelet || !step))
        return fail(SB200_ERR_INVALID, "sb200_wave_step2_dev_f32: NULL wavelet / step pointer");
    SourceDesc s;
    s.idx = src_index;
    s.wavelet = wavelet;
    s.step = step;
    s.step_offset = step_offset;
    s.trace = trace;
    return wave_step2(p, p_prev, vel2, p_next, p_next2, grid, s, 0.f, stream, false,
                      "sb200_wave_step2_dev_f32");
}

int sb200_wave_step_exact_f32(const float* p, const float* p_prev, const float* vel2,
                              float* p_next, const sb200_grid* grid, int64_t src_index,
                              float src_amp, void* stream) {
    return wave_step(p, p_prev, vel2, p_next, grid, host_source(src_index, src_amp), stream,
                     true, "sb200_wave_step_exact_f32");
}

int sb200_wave_step_dev_f32(const float* p, const float* p_prev, const float* vel2,
                            float* p_next, const sb200_grid* grid, int64_t src_index,
                            const float* wavelet, const int* step, int step_offset, int exact,
                            void* stream) {
    if (src_index >= 0 && (!wavelet || !step))
        return fail(SB200_ERR_INVALID, "sb200_wave_step_dev_f32: NULL wavelet / step pointer");
    SourceDesc s;
    s.idx = src_index;
    s.wavelet = wavelet;
    s.step = step;
    s.step_offset = step_offset;
    return wave_step(p, p_prev, vel2, p_next, grid, s, stream, exact != 0,
                     "sb200_wave_step_dev_f32");
}

int sb200_set_device_int(int* dst, int value, void* stream) {
    if (!dst) return fail(SB200_ERR_INVALID, "sb200_set_device_int: NULL pointer");
    return finish_launch(launch_set_int(dst, value, static_cast<cudaStream_t>(stream)),
                         "sb200_set_device_int");
}

int sb200_heat_step_exact_f32(const float* u, float* u_next, const sb200_grid* grid,
                              float alpha, void* stream) {
    return heat_step(u, u_next, grid, alpha, stream, true, "sb200_heat_step_exact_f32");
}

int sb200_heat_step_f32(const float* u, float* u_next, const sb200_grid* grid, float alpha,
                        void* stream) {
    return heat_step(u, u_next, grid, alpha, stream, false, "sb200_heat_step_f32");
}

int sb200_wave_prepass_f32(const float* p, float* p_prev, const float* vel2, float* r,
                           const sb200_grid* grid, float beta, void* stream) {
    const char* where = "sb200_wave_prepass_f32";
    GridDesc g;
    if (int rc = to_desc(grid, &g)) return rc;
    if (!p || !p_prev || !vel2 || !r)
        return fail(SB200_ERR_INVALID, std::string(where) + ": NULL field pointer");
    if (r == p || r == p_prev || p == p_prev)
        return fail(SB200_ERR_INVALID, std::string(where) + ": r, p and p_prev must be distinct");
    if (!std::isfinite(beta))
        return fail(SB200_ERR_INVALID, std::string(where) + ": beta must be finite");
    if (!g.has_interior()) return SB200_OK;
    if (!pencil_ok(g, {p, p_prev, vel2, r}))
        return fail(SB200_ERR_UNSUPPORTED,
                    std::string(where) + ": needs nx % 4 == 0 and 16-byte aligned fields");
    const PencilConfig cfg = choose(kPrepass, g);
    PencilMaps maps;
    if (int rc = pencil_maps(false, cfg.variant, g, p, p_prev, vel2, &maps, where)) return rc;
    return finish_launch(launch_prepass_pencil_f32(maps, p_prev, vel2, r, g, beta, cfg,
                                                   device_error_ptr(),
                                                   static_cast<cudaStream_t>(stream)),
                         where);
}

int sb200_f16_pack(const float* src, uint16_t* dst, int64_t n, float scale, void* stream) {
    if (!src || !dst || n < 0) return fail(SB200_ERR_INVALID, "sb200_f16_pack: bad arguments");
    if (!(scale > 0.f) || !std::isfinite(scale))
        return fail(SB200_ERR_INVALID, "sb200_f16_pack: scale must be positive");
    if (n == 0) return SB200_OK;
    return finish_launch(launch_f16_pack(src, dst, n, scale, static_cast<cudaStream_t>(stream)),
                         "sb200_f16_pack");
}

int sb200_f16_unpack(const uint16_t* src, float* dst, int64_t n, float scale, void* stream) {
    if (!src || !dst || n < 0)
        return fail(SB200_ERR_INVALID, "sb200_f16_unpack: bad arguments");
    if (!(scale > 0.f) || !std::isfinite(scale))
        return fail(SB200_ERR_INVALID, "sb200_f16_unpack: scale must be positive");
    if (n == 0) return SB200_OK;
    return finish_launch(launch_f16_unpack(src, dst, n, scale, static_cast<cudaStream_t>(stream)),
                         "sb200_f16_unpack");
}

int sb200_k_field_bf16(const float* vel2, uint16_t* k, const sb200_grid* grid, void* stream) {
    GridDesc g;
    if (int rc = to_desc(grid, &g)) return rc;
    if (!vel2 || !k) return fail(SB200_ERR_INVALID, "sb200_k_field_bf16: NULL pointer");
    if (!(g.dt > 0.f)) return fail(SB200_ERR_INVALID, "sb200_k_field_bf16: dt must be positive");
    if (g.size() == 0) return SB200_OK;
    const float f = static_cast<float>(double(g.dt) * g.dt / (double(g.dx) * g.dx));
    return finish_launch(launch_k_bf16(vel2, k, g.size(), f, static_cast<cudaStream_t>(stream)),
                         "sb200_k_field_bf16");
}

int sb200_wave_step_f16(const uint16_t* p, uint16_t* p_prev_next, const uint16_t* k,
                        const sb200_grid* grid, int64_t src_index, float src_amp,
                        const float* wavelet, const int* step, int step_offset,
                        const sb200_f16_scale* scale, int phase, void* stream) {
    SourceDesc src;
    src.idx = src_index;
    src.w = src_amp;
    src.wavelet = wavelet;
    src.step = step;
    src.step_offset = step_offset;
    return wave_step_f16(p, p_prev_next, k, grid, src, scale, phase, stream);
}

int sb200_f16_renorm(const double* stats3, sb200_f16_scale* scale, const float* bound,
                     const int* step, float bound_host, float target, void* stream) {
    if (!stats3 || !scale || (bound && !step))
        return fail(SB200_ERR_INVALID, "sb200_f16_renorm: NULL pointer");
    if (!(target > 0.f) || !(bound_host >= 0.f))
        return fail(SB200_ERR_INVALID, "sb200_f16_renorm: bad target / bound");
    return finish_launch(launch_f16_renorm(stats3, reinterpret_cast<F16Scale*>(scale), bound,
                                           step, bound_host, target,
                                           static_cast<cudaStream_t>(stream)),
                         "sb200_f16_renorm");
}

int64_t sb200_field_stats_scratch_len(const sb200_grid* grid) {
    GridDesc g;
    if (int rc = to_desc(grid, &g)) return rc;
    if (!g.has_interior()) return fail(SB200_ERR_INVALID, "grid has no interior");
    return 3 * static_cast<int64_t>(stats_blocks(g));
}

namespace {
int field_stats(const void* field, bool half, const sb200_grid* grid, float scale, double* out3,
                double* scratch, int64_t scratch_len, void* stream, const char* where) {
    GridDesc g;
    if (int rc = to_desc(grid, &g)) return rc;
    if (!field || !out3 || !scratch)
        return fail(SB200_ERR_INVALID, std::string(where) + ": NULL pointer");
    if (!g.has_interior()) return fail(SB200_ERR_INVALID, std::string(where) + ": no interior");
    if (!(scale > 0.f) || !std::isfinite(scale))
        return fail(SB200_ERR_INVALID, std::string(where) + ": scale must be positive");
    if (scratch_len < 3 * static_cast<int64_t>(stats_blocks(g)))
        return fail(SB200_ERR_INVALID, std::string(where) + ": scratch too small (need " +
                                           std::to_string(3 * stats_blocks(g)) + " doubles)");
    return finish_launch(launch_field_stats(field, half, g, scale, out3, scratch,
                                            static_cast<cudaStream_t>(stream)),
                         where);
}
}  // namespace

int sb200_field_stats_f32(const float* field, const sb200_grid* grid, double* out3,
                          double* scratch, int64_t scratch_len, void* stream) {
    return field_stats(field, false, grid, 1.0f, out3, scratch, scratch_len, stream,
                       "sb200_field_stats_f32");
}

int sb200_field_stats_f16(const uint16_t* field, const sb200_grid* grid, float scale,
                          double* out3, double* scratch, int64_t scratch_len, void* stream) {
    return field_stats(field, true, grid, scale, out3, scratch, scratch_len, stream,
                       "sb200_field_stats_f16");
}

int sb200_pencil_variant_count(int kind) {
    if (!valid_kind(kind)) return fail(SB200_ERR_INVALID, "unknown kernel kind");
    return variant_count(kind);
}

const char* sb200_pencil_variant_name(int kind, int variant) {
    if (!valid_kind(kind)) return nullptr;
    return variant_name(kind, variant);
}

int sb200_set_pencil_override(int kind, int variant, int zchunks) {
    if (!valid_kind(kind)) return fail(SB200_ERR_INVALID, "unknown kernel kind");
    if (variant >= variant_count(kind))
        return fail(SB200_ERR_INVALID, "variant out of range");
    if (zchunks < 1) return fail(SB200_ERR_INVALID, "zchunks must be >= 1");
    std::lock_guard<std::mutex> lock(g_cfg_mu);
    g_override[kind].variant = variant;
    g_override[kind].zchunks = zchunks;
    return SB200_OK;
}

int sb200_pencil_choice(int kind, const sb200_grid* grid, int* variant, int* zchunks) {
    if (!valid_kind(kind)) return fail(SB200_ERR_INVALID, "unknown kernel kind");
    GridDesc g;
    if (int rc = to_desc(grid, &g)) return rc;
    if (!variant || !zchunks) return fail(SB200_ERR_INVALID, "NULL output pointer");
    if (!g.has_interior()) return fail(SB200_ERR_INVALID, "grid has no interior");
    const PencilConfig c = choose(kind, g);
    *variant = c.variant;
    *zchunks = c.zchunks;
    return SB200_OK;
}

}  // extern "C"
