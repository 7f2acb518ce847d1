// Acoustic and heat steps of grids whose rows are no multiple of 16 bytes
// (nx % 4 != 0), in the reference's operation order.
//
// The bits are launch_naive's (src/kernels/stencil_naive.cu:49-89, in the order of its
// CPU branch, 151-169): every product and sum is rounded by itself.
//
// A tiled TMA copy needs strides and a start that are multiples of 16 bytes.  Four
// rows together always are: seen as a matrix of 4 nx words by (ny nz) / 4, row r of
// the field is the piece at x = (r % 4) nx of line r / 4, and every fourth row of a
// tile is one line below the other.  So an x-y plane of a tile comes by four copies,
// one per row residue, each started at the 16-byte boundary at or below its first
// word; a row then sits (r nx) % 4 words into its staged line.  Words a copy brings
// beyond a row's end belong to the next row, and rows beyond the last whole group of
// four are halo of the last plane: no stored point reads either.
//
// Work unit: a CTA owns a 64 x 16 tile of interior columns and marches z over one
// chunk.  A lane is a column in x and holds 4 rows (two packed f32x2 pairs), so shared
// and global accesses are 32 consecutive words at any alignment, a lane's row residues
// are compile-time, and the 4 rows above and below serve 4 points.  Planes of p fill an
// 8-stage ring, p_prev and vel2 tiles a 4-stage ring; plane z + 4 and the tiles of z are
// one group on one mbarrier, 4 groups in flight, warp k issuing residue k.  The z
// neighbours live in an 8-deep register queue (the pair z - 4, z + 4 is added as plane
// z + 4 takes plane z - 4's slot; plane loop unrolled by 8, so every stage and phase is
// compile-time); one CTA barrier per plane.
//
// Why lanes are columns: a float4 of x per thread, as in the pencil kernel, would need
// 16-byte aligned rows in shared memory; rows copied by 4-byte cp.async instead cost 97
// instructions per point, half of them copies and addresses (245 us at 401 x 357 x 301).
// Here 73 instructions and 14 words of shared memory per point (79 with a 9-deep queue
// and stages computed from the plane's number).  Acoustic step measured, against the
// one-thread-per-point kernel that ran before: 401 x 357 x 301 152 (9-deep queue: 161)
// against 328 us (its bytes at the copy rate: 98 us).  Bound by issue and power.
#include <algorithm>

#include "kernels.h"
#include "sb200_common.cuh"

namespace sb200 {

namespace {

constexpr int RPT = 4;         // rows per lane
constexpr int RS = 8, RG = 4;  // staged planes of p; groups in flight
static_assert(RS == 2 * R && RG == R, "a group's stage is the one its plane z - 4 leaves");

template <int TX, int TY>
struct RaggedShape {
    static constexpr int NT = TX * TY / RPT;
    static constexpr int PW = TX + 2 * R + 4;    // words per staged row of p (3 of alignment)
    static constexpr int PH = (TY + 2 * R) / 4;  // staged rows per residue
    static constexpr int AW = TX + 4, AH = TY / 4;  // p_prev / vel2: no halo
    static constexpr int PBLOCK = (PW * PH * 4 + 127) / 128 * 32;  // words per residue
    static constexpr int ABLOCK = (AW * AH * 4 + 127) / 128 * 32;  // (128-byte steps)
    static constexpr int PPLANE = 4 * PBLOCK, ATILE = 4 * ABLOCK;
    static constexpr size_t smem(bool heat) {
        return size_t(RS * PPLANE + (heat ? 0 : RG * 2 * ATILE)) * 4 + 128;
    }
    static_assert(TX % 32 == 0 && TY % 4 == 0, "a warp is 32 columns of one row group");
    static_assert(NT >= 128, "warp k issues row residue k");
};

struct RaggedArgs {
    float* next;
    int nx, ny, nz;
    int64_t sy, sz;
    int tiles_x, tiles_y, zlen;
    float inv_dx2, inv_dy2, inv_dz2;
    float k;        // wave: dt^2; heat: alpha*dt
    float one;      // 1: a product meets its sum as fma(product, one, sum), which rounds
                    // as an add and cannot be contracted (the compiler contracts
                    // mul.rn.f32x2 + add.rn.f32x2)
    int src_x, src_y, src_z;  // -1 when there is no source
    float src_w;
    const float* wavelet;
    const int* step;
    int step_off;
    float* trace;
    int* err;
};

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x,
                                            int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}

// Word at byte offset `off` of shared memory.
__device__ __forceinline__ float lds_at(const char* p, int off) {
    return *reinterpret_cast<const float*>(p + off);
}

__device__ __forceinline__ void stg_if(float* p, float v, bool pred) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.global.f32 [%0], %1;\n\t}" ::"l"(p),
                 "f"(v), "r"(static_cast<uint32_t>(pred))
                 : "memory");
}

template <int TX, int TY, bool HEAT>
__global__ void __launch_bounds__(RaggedShape<TX, TY>::NT, 512 / RaggedShape<TX, TY>::NT)
    ragged_f32_kernel(const __grid_constant__ CUtensorMap pmap,
                      const __grid_constant__ CUtensorMap qmap,
                      const __grid_constant__ CUtensorMap vmap, const RaggedArgs a) {
    using P = RaggedShape<TX, TY>;
    constexpr int PW = P::PW, PH = P::PH, AW = P::AW, AH = P::AH;
    constexpr int PBLOCK = P::PBLOCK, ABLOCK = P::ABLOCK, PPLANE = P::PPLANE, ATILE = P::ATILE;
    extern __shared__ unsigned char dsmem[];
    __shared__ __align__(8) uint64_t start, full[RG];
    float* sm = reinterpret_cast<float*>(smem_align<128>(dsmem));
    float* aux = sm + RS * PPLANE;  // RG stages of [p_prev tile | vel2 tile]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        prefetch_tmap(&pmap);
        if (!HEAT) {
            prefetch_tmap(&qmap);
            prefetch_tmap(&vmap);
        }
        mbar_init(&start, 4);
#pragma unroll
        for (int s = 0; s < RG; ++s) mbar_init(&full[s], 4);
        fence_barrier_init();
    }
    launch_order();
    __syncthreads();

    int b = blockIdx.x;
    const int tx = b % a.tiles_x;
    b /= a.tiles_x;
    const int ty = b % a.tiles_y;
    const int zc = b / a.tiles_y;
    const int x0 = R + tx * TX, y0 = R + ty * TY;  // both multiples of 4
    const int zb = R + zc * a.zlen;
    const int nint = min(a.zlen, a.nz - R - zb);

    // Lane 0 of warp k < 4 issues row residue k: plane j of the chunk (z = zb - 4 + j) into
    // stage j % 8, and group g = plane g + 8 and p_prev / vel2 of iteration g.
    const bool issuer = lane == 0 && warp < 4;
    auto issue_plane = [&](int j, uint64_t* bar) {
        const int row = (zb - R + j) * a.ny + y0 - R + warp;
        tma_load_2d(sm + (j % RS) * PPLANE + warp * PBLOCK, &pmap, bar,
                    ((row & 3) * a.nx + x0 - R) & ~3, row >> 2);
    };
    int groups = 0;  // groups issued so far
    auto issue_group = [&](int g) {
        uint64_t* bar = &full[g % RG];
        mbar_arrive_expect_tx(bar, PW * PH * 4u + (HEAT ? 0u : 2 * AW * AH * 4u));
        issue_plane(g + 2 * R, bar);
        if (!HEAT) {
            const int row = (zb + g) * a.ny + y0 + warp;
            const int x = ((row & 3) * a.nx + x0) & ~3;
            float* st = aux + (g % RG) * 2 * ATILE + warp * ABLOCK;
            tma_load_2d(st, &qmap, bar, x, row >> 2);
            tma_load_2d(st + ATILE, &vmap, bar, x, row >> 2);
        }
        groups = g + 1;
    };
    if (issuer) {
        mbar_arrive_expect_tx(&start, 2 * R * PW * PH * 4u);
        for (int j = 0; j < 2 * R; ++j) issue_plane(j, &start);
    }

    const int lx = tid % TX, ly = RPT * (tid / TX);
    const int gx = x0 + lx, gy = y0 + ly;
    const bool xin = gx < a.nx - R;
    bool rin[RPT];
#pragma unroll
    for (int j = 0; j < RPT; ++j) rin[j] = xin && gy + j < a.ny - R;
    // The source's iteration and row if this lane owns it.
    const int src_j = a.src_y - gy;
    const int src_i =
        !HEAT && gx == a.src_x && xin && src_j >= 0 && src_j < RPT && a.src_y < a.ny - R
            ? a.src_z - zb
            : -1;
    // Byte offsets of this lane's column, own row group: staged plane, p_prev / vel2 tile.
    const int poff = 4 * ((ly / 4 + 1) * PW + lx + R);
    const int aoff = 4 * (ly / 4 * AW + lx);
    // Row residue k of plane z starts 4 (((z ny + k) nx) % 4) bytes into its line (x0 and
    // y0 are multiples of 4).  One byte of `sh` per residue, advanced from plane to plane;
    // plane z + 4 has plane z's.
    auto shifts = [&](int z) {
        uint32_t w = 0;
        for (int k = 0; k < 4; ++k)
            w |= uint32_t(((((z & 3) * (a.ny & 3) + k) * (a.nx & 3)) & 3) * 4) << (8 * k);
        return w;
    };
    const uint32_t sh_step = uint32_t((((a.ny & 3) * (a.nx & 3)) & 3) * 4) * 0x01010101u;

    float2 q[8][RPT / 2];  // plane j of the chunk in slot j % 8
    bool bad = !mbar_wait(&start, 0);
    uint32_t sh = shifts(zb - R);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const char* pl = reinterpret_cast<const char*>(sm + j * PPLANE) + poff;
#pragma unroll
        for (int h = 0; h < RPT / 2; ++h)
            q[j][h] = make_float2(lds_at(pl + ((sh >> (16 * h)) & 0xff), 4 * (2 * h) * PBLOCK),
                                  lds_at(pl + ((sh >> (16 * h + 8)) & 0xff), 4 * (2 * h + 1) * PBLOCK));
        sh = (sh + sh_step) & 0x0c0c0c0cu;
    }
    sh = shifts(zb);
    bool abort_run = __syncthreads_or(bad) != 0;
    // Planes 0..3 are only queue feed: their stages are free again.
    if (!abort_run && issuer)
        for (int g = 0; g < RG && g < nint; ++g) issue_group(g);

    const float2 c2[R + 1] = {dup2(C0), dup2(C1), dup2(C2), dup2(C3), dup2(C4)};
    const float2 ix2 = dup2(a.inv_dx2), iy2 = dup2(a.inv_dy2), iz2 = dup2(a.inv_dz2);
    const float2 k2 = dup2(a.k), one = dup2(a.one), neg1 = dup2(-1.f);
    float* dst = a.next + int64_t(zb) * a.sz + int64_t(gy) * a.sy + gx;
    const char* const pbase = reinterpret_cast<const char*>(sm) + poff;
    const char* const abase = reinterpret_cast<const char*>(aux) + aoff;
    for (int i0 = 0; i0 < nint && !abort_run; i0 += 8) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = i0 + u;
            if (i < nint && !abort_run) {
                // This lane's column by residue.  The stages of the centre plane i + 4, of the
                // fed plane i + 8 and of the aux tiles are compile-time offsets.
                constexpr int kBytes = 4 * PPLANE;
                const int cen = (u + 4) % RS * kBytes, fed = u * kBytes;
                uint32_t s[4];
                const char* pc[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    s[k] = __byte_perm(sh, 0, 0x4440 + k);
                    pc[k] = pbase + s[k];
                }
                sh = (sh + sh_step) & 0x0c0c0c0cu;
                if (!mbar_wait(&full[u % RG], u / RG)) bad = true;
                // Plane z + 4 meets plane z - 4 and takes its slot.
                float2 z4[RPT / 2];
#pragma unroll
                for (int h = 0; h < RPT / 2; ++h) {
                    const float2 f =
                        make_float2(lds_at(pc[2 * h], fed + 4 * (2 * h) * PBLOCK),
                                    lds_at(pc[2 * h + 1], fed + 4 * (2 * h + 1) * PBLOCK));
                    z4[h] = add2(f, q[u][h]);
                    q[u][h] = f;
                }
                // Row pairs (-4, -3) .. (6, 7): the own ones are the queue's centre.
                float2 row[6];
#pragma unroll
                for (int m = 0; m < 6; ++m)
                    row[m] = m == 2 || m == 3
                                 ? q[(u + 4) % 8][m - 2]
                                 : make_float2(lds_at(pc[2 * (m & 1)],
                                                      cen + 4 * (2 * (m & 1) * PBLOCK + (m / 2 - 1) * PW)),
                                               lds_at(pc[2 * (m & 1) + 1],
                                                      cen + 4 * ((2 * (m & 1) + 1) * PBLOCK +
                                                                 (m / 2 - 1) * PW)));
                auto row_at = [&](int e) { return e & 1 ? row[e / 2].y : row[e / 2].x; };
                float2 o[RPT / 2], kv[RPT / 2];
#pragma unroll
                for (int h = 0; h < RPT / 2; ++h) {
                    const float2 c = q[(u + 4) % 8][h];
                    const int e = R + 2 * h;  // the pair's first row in row_at
                    const int o0 = cen + 4 * 2 * h * PBLOCK, o1 = cen + 4 * (2 * h + 1) * PBLOCK;
                    auto x_at = [&](int d) {
                        return make_float2(lds_at(pc[2 * h], o0 + 4 * d),
                                           lds_at(pc[2 * h + 1], o1 + 4 * d));
                    };
                    const float2 t = mul2(c2[0], c);
                    float2 l_x = mul2(t, ix2), l_y = mul2(t, iy2), l_z = mul2(t, iz2);
#pragma unroll
                    for (int r = 1; r <= R; ++r) {
                        l_x = fma2(mul2(mul2(c2[r], add2(x_at(r), x_at(-r))), ix2), one, l_x);
                        const float2 sy = r & 1 ? make_float2(row_at(e + r) + row_at(e - r),
                                                              row_at(e + 1 + r) + row_at(e + 1 - r))
                                                : add2(row[(e + r) / 2], row[(e - r) / 2]);
                        l_y = fma2(mul2(mul2(c2[r], sy), iy2), one, l_y);
                        const float2 sz =
                            r == R ? z4[h] : add2(q[(u + 4 + r) % 8][h], q[(u + 4 - r) % 8][h]);
                        l_z = fma2(mul2(mul2(c2[r], sz), iz2), one, l_z);
                    }
                    const float2 lap = add2(add2(l_x, l_y), l_z);
                    if (HEAT) {
                        // 2u - u is exact: the reference's heat arithmetic is u + k*lap
                        o[h] = fma2(mul2(k2, lap), one, c);
                    } else {
                        const char* a0 = abase + s[2 * h];
                        const char* a1 = abase + s[2 * h + 1];
                        const int st = u % RG * 2 * ATILE * 4;
                        const int b0 = st + 4 * 2 * h * ABLOCK, b1 = st + 4 * (2 * h + 1) * ABLOCK;
                        kv[h] = mul2(k2, make_float2(lds_at(a0, b0 + 4 * ATILE),
                                                     lds_at(a1, b1 + 4 * ATILE)));
                        // 2c - p_prev in one rounding (2c is exact)
                        const float2 d =
                            fma2(neg1, make_float2(lds_at(a0, b0), lds_at(a1, b1)), add2(c, c));
                        o[h] = fma2(mul2(kv[h], lap), one, d);
                    }
                }
                if (!HEAT && i == src_i) {
                    const float w = a.wavelet ? a.wavelet[*a.step + a.step_off] : a.src_w;
#pragma unroll
                    for (int j = 0; j < RPT; ++j)
                        if (j == src_j) {
                            float& v = j & 1 ? o[j / 2].y : o[j / 2].x;
                            v = __fadd_rn(v, __fmul_rn(j & 1 ? kv[j / 2].y : kv[j / 2].x, w));
                            if (a.trace) a.trace[(a.step ? *a.step : 0) + a.step_off] = v;
                        }
                }
                float* dj = dst;
#pragma unroll
                for (int j = 0; j < RPT; ++j) {
                    stg_if(dj, j & 1 ? o[j / 2].y : o[j / 2].x, rin[j]);
                    dj += a.sy;
                }
                dst += a.sz;
                abort_run = __syncthreads_or(bad) != 0;
                if (!abort_run && issuer && i + RG < nint) issue_group(i + RG);
            }
        }
    }
    if (abort_run && tid == 0) {
        record_error(a.err, kDevWaitTimeout);
        // Let every copy still in flight land before the shared memory is released (the
        // warps issue alike; each barrier has at most one phase outstanding).
        (void)mbar_wait(&start, 0);
        for (int g = max(0, groups - RG); g < groups; ++g)
            (void)mbar_wait(&full[g % RG], (g / RG) & 1);
    }
}

using LaunchFn = cudaError_t (*)(const PencilMaps&, const RaggedArgs&, unsigned, cudaStream_t);

// CTAs per SM; the first call per device sets the shared-memory attribute.
template <int TX, int TY, bool HEAT>
int resident() {
    using P = RaggedShape<TX, TY>;
    static int cached[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (cached[dev & 63] > 0) return cached[dev & 63];
    auto kern = ragged_f32_kernel<TX, TY, HEAT>;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(P::smem(HEAT))) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, P::NT, P::smem(HEAT)) ==
            cudaSuccess &&
        n > 0) {
        cached[dev & 63] = n;
        return n;
    }
    cudaGetLastError();
    return 512 / P::NT;
}

template <int TX, int TY, bool HEAT>
cudaError_t launch(const PencilMaps& m, const RaggedArgs& a, unsigned ctas, cudaStream_t stream) {
    using P = RaggedShape<TX, TY>;
    resident<TX, TY, HEAT>();
    return launch_after(ragged_f32_kernel<TX, TY, HEAT>, ctas, P::NT, P::smem(HEAT), stream, m.p,
                        m.prev, m.vel2, a);
}

struct Shape {
    int tx, ty, pw, ph, aw, ah;
    LaunchFn launch[2];  // [heat]
    int (*resident[2])();
};

template <int TX, int TY>
constexpr Shape shape_of() {
    using P = RaggedShape<TX, TY>;
    return {TX, TY, P::PW, P::PH, P::AW, P::AH,
            {&launch<TX, TY, false>, &launch<TX, TY, true>},
            {&resident<TX, TY, false>, &resident<TX, TY, true>}};
}

const Shape kShapes[] = {shape_of<64, 16>(), shape_of<32, 32>()};

// Points of a plane that a shape's tiles cover.
int64_t covered(const Shape& s, const GridDesc& g) {
    const int64_t x = (g.nx - 2 * R + s.tx - 1) / s.tx, y = (g.ny - 2 * R + s.ty - 1) / s.ty;
    return x * s.tx * y * s.ty;
}

// The shape whose tiles cover fewer points outside the interior; where they cover the
// same, the wider one (acoustic: 401 x 357 x 301 covers 448 or 416 columns and runs 156
// or 150 us; 383^3 covers the same points and runs 195 or 198 us).
const Shape& shape_for(const GridDesc& g) {
    return covered(kShapes[1], g) < covered(kShapes[0], g) ? kShapes[1] : kShapes[0];
}

RaggedArgs make_args(float* next, const GridDesc& g, float k, int zchunks, int* err) {
    const Shape& s = shape_for(g);
    RaggedArgs a{};
    a.next = next;
    a.nx = static_cast<int>(g.nx);
    a.ny = static_cast<int>(g.ny);
    a.nz = static_cast<int>(g.nz);
    a.sy = g.nx;
    a.sz = g.nx * g.ny;
    a.tiles_x = static_cast<int>((g.nx - 2 * R + s.tx - 1) / s.tx);
    a.tiles_y = static_cast<int>((g.ny - 2 * R + s.ty - 1) / s.ty);
    const int inz = static_cast<int>(g.nz - 2 * R);
    const int zc = std::max(1, std::min(zchunks, inz));
    a.zlen = (inz + zc - 1) / zc;
    // Host-side reciprocals in float, as the reference launcher computes them
    // (stencil_naive.cu:96-99).
    a.inv_dx2 = 1.0f / (g.dx * g.dx);
    a.inv_dy2 = 1.0f / (g.dy * g.dy);
    a.inv_dz2 = 1.0f / (g.dz * g.dz);
    a.k = k;
    a.one = 1.0f;
    a.src_x = a.src_y = a.src_z = -1;
    a.err = err;
    return a;
}

unsigned ctas_of(const RaggedArgs& a, const GridDesc& g) {
    const int inz = static_cast<int>(g.nz - 2 * R);
    return static_cast<unsigned>(int64_t(a.tiles_x) * a.tiles_y * ((inz + a.zlen - 1) / a.zlen));
}

}  // namespace

// Rows of the field must be countable in 32 bits, and four of them addressable as one
// TMA line.
bool ragged_ok(const GridDesc& g) {
    return g.nx < (int64_t(1) << 28) && g.ny * g.nz < (int64_t(1) << 30) && g.ny * g.nz >= 4;
}

int64_t ragged_covered(const GridDesc& g) { return covered(shape_for(g), g); }

PencilBoxes ragged_boxes(bool heat, const GridDesc& g) {
    const Shape& s = shape_for(g);
    PencilBoxes b;
    b.halo_x = s.pw;
    b.halo_y = s.ph;
    b.tile_x = s.aw;
    b.tile_y = s.ah;
    b.aux_tma = !heat;
    return b;
}

int ragged_resident(bool heat, const GridDesc& g) {
    return shape_for(g).resident[heat]();
}

int64_t ragged_ctas(const GridDesc& g, int zchunks) {
    return ctas_of(make_args(nullptr, g, 0.f, zchunks, nullptr), g);
}

cudaError_t launch_wave_ragged_f32(const PencilMaps& maps, float* next, const GridDesc& g,
                                   const SourceDesc& src, int zchunks, int* err,
                                   cudaStream_t stream) {
    RaggedArgs a = make_args(next, g, g.dt * g.dt, zchunks, err);
    if (src.idx >= 0) {
        a.src_x = static_cast<int>(src.idx % g.nx);
        a.src_y = static_cast<int>((src.idx / g.nx) % g.ny);
        a.src_z = static_cast<int>(src.idx / (g.nx * g.ny));
        a.src_w = src.w;
        a.wavelet = src.wavelet;
        a.step = src.step;
        a.step_off = src.step_offset;
        a.trace = src.trace;
    }
    return shape_for(g).launch[false](maps, a, ctas_of(a, g), stream);
}

cudaError_t launch_heat_ragged_f32(const PencilMaps& maps, float* u_next, const GridDesc& g,
                                   float alpha_dt, int zchunks, int* err,
                                   cudaStream_t stream) {
    const RaggedArgs a = make_args(u_next, g, alpha_dt, zchunks, err);
    return shape_for(g).launch[true](maps, a, ctas_of(a, g), stream);
}

}  // namespace sb200
