// Cell-aggregated scatter of one unit (4 x 4 x 8 cells) by a sweep along x,
// shared by P2G (pm_p2g.cu) and the adjoint of G2P (pm_adjoint.cu).
//
// A CTA of 8 warps takes one non-empty unit.  Lane l of every warp stands for
// the cell (y, z) = (l / 8, l % 8) of an x-layer; warp w for one set of node
// planes: warps 0..2 the quadratic planes X = w mod 3, warps 3..7 the cubic
// planes X = w - 3 mod 5.  At layer x each warp therefore has exactly one
// plane to add to (a cell's quadratic stencil covers planes x .. x+2, its
// cubic stencils x-1 .. x+3), whatever the layer.  A lane sums its cell's
// particles in float registers, 9 or 25 nodes per component; after the layer the
// lanes' sums meet in a plane of exact 64-bit fixed point in shared memory that
// only this warp uses (plain loads and stores: the two 32-bit shared atomics per
// sum that several warps on one tile need were half of the former kernel), and
// when no later layer reaches the plane it goes to the global grid with one
// 64-bit atomic per nonzero node component.
//
// Within a unit the warps run without barriers: row k of a layer is the k-th
// particle of each of its 32 cells, one per lane, and every lane copies its own
// particle's payload (asynchronously, a few rows ahead) into its own slot of
// the warp's ring in shared memory and reads only that.  (Staging rows once for
// all warps, with their weights, takes fewer instructions, but a barrier every
// 4 rows, at which the adding-up and the staging of single warps stop all.)
//
// Float sums: a cell's particles in id order, the sum restarted (what there is
// added to the plane) at every 256th particle of the cell's 4^3-cell sub-block in
// Morton order of its cells.  The sums of a substep are thus fixed by the
// particles alone, not by the order of arrival, the launch or the batch.
//
// Bound by instruction issue (68%) and the FMA pipe.  1M displaced particles, 6 to
// 11 per cell: 114 us, the former tile kernel 129; on a regular lattice of 8 per
// cell 102 and 99.5, and below 2 per cell it is the slower one too (a layer's sums
// go to the planes for all 32 cells: 885k at 1 per cell 332 us and 280).  It gains
// where cells hold more or units are few: with the counted binning 8.8M particles at
// 27 per cell go from 6,400 to 5,090 us per two substeps, 138k from 1,205 to 598
// us per six.
#pragma once

#include "pm_common.cuh"

namespace pm {

constexpr int kSweepThreads = 256;
constexpr int kSweepQ = 3, kSweepC = 5;       // warps on quadratic / cubic planes
constexpr int kUnitX = 4, kUnitY = 4, kUnitZ = 8;
constexpr int kQRows = kUnitY + 2, kQCols = kUnitZ + 2;   // nodes of a quadratic plane
constexpr int kCRows = kUnitY + 4, kCCols = kUnitZ + 4;   // nodes of a cubic plane
constexpr int kPlaneCols = 16;                // words of a plane row (see plane_word)
constexpr int kFewCells = 2, kCloud = 24;     // below kCloud particles to a unit: layers of so few cells one by one
constexpr int kRing = 4;                      // rows of a warp's ring, kRing - 1 on their way

// Word of node (row, col) of a plane.  Odd rows are rotated by half: the 16
// lanes of a 64-bit access cover 8 columns of two neighbouring rows, which
// then lie in different halves of the banks.
__device__ __forceinline__ int plane_word(int row, int col) {
    return row * kPlaneCols + ((col + 8 * (row & 1)) & (kPlaneCols - 1));
}

// Asynchronous copies to shared memory; the words past `bytes` (0: all) are filled with zeros.
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
                 "l"(gmem), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
                 "l"(gmem), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {   // until at most N of this thread's groups are under way
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Payload of a particle, 4 parts of 16 bytes and one of 4:
//   {fx, d} {v, m} {a00, a10, a01, a11} {a02, a12, a20, a21} {a22}
// node o of its quadratic stencil receives w (v + a (o - fx) dx) and w m, a node
// of its cubic stencil w d and w (the adjoint: d times the Laplacian's weights).
// In global memory in blocks of 32 places (one row of a layer in the row layout):
// part 0 of all, parts 1 and 2 of each side by side, part 3, part 4.  A particle
// whose neighbours in the state lie elsewhere thus writes four sectors: 1M
// particles in no order 509 us per substep with part after part (five sectors),
// 489 so; the regular slab's sweep, which reads whole rows either way, is the
// same to 0.4%.  (Parts 0 and 1, 2 and 3 side by side, three sectors: 476, but
// the cubic planes' warps, which read part 0 alone, make the slab 1.1% slower.)
constexpr int kPayBlock = kPayBytes * 32;
__device__ __forceinline__ int pay_part(int k, int i) {   // byte of part k of the block's place i
    return k == 0 ? 16 * i : (k == 3 ? 1536 + 16 * i : (k == 4 ? 2048 + 4 * i : 496 + 16 * k + 32 * i));
}
__device__ __forceinline__ char *pay_block(const void *payload, long long place) {
    return (char *)payload + (place >> 5) * kPayBlock;
}
__device__ __forceinline__ void pay_store(void *payload, long long place, const float4 (&p)[4], float a22) {
    char *b = pay_block(payload, place);
    const int i = (int)(place & 31);
#pragma unroll
    for (int k = 0; k < 4; ++k) *(float4 *)(b + pay_part(k, i)) = p[k];
    *(float *)(b + pay_part(4, i)) = a22;
}
// Place of the k-th particle of a cell from its first place.
__device__ __forceinline__ long long place_of(int first, int k) {
    return first < 0 ? (first & ~kCellRows) + 32LL * k : (long long)first + k;
}

struct QuadSlot {                             // a row in a ring: the payload block
    float4 p[4][32];
    float az2[32];
};
struct CubicSlot {                            // part 0 only
    float4 p0[32];
};

struct SweepShared {
    QuadSlot qring[kSweepQ][kRing];
    CubicSlot cring[kSweepC][kRing];
    long long qpl[kSweepQ][4][kQRows * kPlaneCols];   // zero between flushes
    long long cpl[kSweepC][2][kCRows * kPlaneCols];
    float2 spill[8][26];                      // a lane's sums on their way to its warp's plane
    unsigned char split[kUnitCells];          // particles of the sub-block before the cell, mod 256
    int2 cell[kUnitCells];                    // {first place (kCellRows), particles}; regular cells only (0 otherwise)
    int2 raw[kUnitCells];                     // the next unit's cells
    int layer_rows[kUnitX];                   // rows of a layer; negative: at most kFewCells cells (see sweep_layer)
    float dx;
    float scale[4];                           // fixed-point scales of {momentum, mass, w d, w}
    long long *g_quad, *g_cubic;              // global sums of the first node of the unit's plane 0
    long long ng;
    long long *g0_quad, *g0_cubic, gblock;    // scatter_clamped's: global sums of node 0, the scene's first grid block
    float inv_dx;
    unsigned clamped_layers;                  // layers of the units that scatter_clamped takes
    int2 next;                                // the next item (see sweep_item)
    unsigned char mark[36];                   // grid blocks s-1 .. s+1, s-1 .. s+1, s-1 .. s+2 of the unit
};

// Items of the work: the units of the list, but the last one per CTA of the
// launch (all, if there are fewer) layer by layer, so that the CTAs end together
// and a short list spreads over the SMs: 1M particles, 1,377 units on 444 CTAs,
// 340 us per substep without the single layers, 333 with them.  (A layer by itself
// adds its 3 and 5 planes to the grid, a whole unit its 6 and 8.)
struct SweepItems {
    unsigned whole, all;                      // whole units first, then single layers
};
__device__ __forceinline__ SweepItems sweep_items(unsigned n_units) {
    const unsigned single = min(n_units, gridDim.x);
    return {n_units - single, n_units - single + single * kUnitX};
}
// Item i: {place in the list, first layer and, times 256, the one after the last}, {-1, 0} past the end.
__device__ __forceinline__ int2 sweep_item(unsigned i, SweepItems n) {
    if (i >= n.all) return make_int2(-1, 0);
    if (i < n.whole) return make_int2((int)i, kUnitX << 8);
    const unsigned j = i - n.whole;
    return make_int2((int)(n.whole + j / kUnitX), (int)(j % kUnitX) * 257 + 256);
}
__device__ __forceinline__ int2 sweep_unit(unsigned i, SweepItems n, const int *__restrict__ work) {   // {unit, layers}
    const int2 item = sweep_item(i, n);
    return make_int2(item.x >= 0 ? work[item.x] : -1, item.y);
}

// SweepShared::layer_rows of a layer, cnt: this lane's cell.
__device__ __forceinline__ int layer_code(int cnt, bool cloud) {
    const int rows = __reduce_max_sync(0xffffffffu, cnt), cells = __popc(__ballot_sync(0xffffffffu, cnt > 0));
    return cloud && cells <= kFewCells ? -rows : rows;
}

// Starts the copy of the payload of a block's place i into this lane's words of a
// ring slot; lanes without a particle get zeros.
__device__ __forceinline__ void row_copy(QuadSlot &s, const char *block, int i, bool on, int lane) {
    const int bytes = on ? 16 : 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) cp_async16(&s.p[k][lane], block + pay_part(k, i), bytes);
    cp_async4(&s.az2[lane], block + pay_part(4, i), bytes >> 2);
}
__device__ __forceinline__ void row_copy(CubicSlot &s, const char *block, int i, bool on, int lane) {
    cp_async16(&s.p0[lane], block + pay_part(0, i), on ? 16 : 0);
}

// Adds NC sums to a node's word (byte address `at`) in NC planes `stride` bytes apart.
template <int NC>
__device__ __forceinline__ void plane_words_add(char *at, int stride, const long long (&q)[NC]) {
    long long o[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) o[k] = *(long long *)(at + k * stride);
#pragma unroll
    for (int k = 0; k < NC; ++k) *(long long *)(at + k * stride) = fix_add(o[k], q[k]);
    __syncwarp();
}
constexpr int kOddRow = 64, kRowBytes = 8 * kPlaneCols;   // rows an odd number apart: xor kOddRow (see plane_word)

__device__ __forceinline__ void red_add(long long *g, long long q) {   // g: global memory
    asm volatile("red.global.add.u64 [%0], %1;" ::"l"(__cvta_generic_to_global(g)), "l"(q) : "memory");
}
// Sends a plane's nonzero words to the global sums (node (r, c) at
// gp + gs (r ng + c)) and clears them.  A float sum that is not a number or
// infinite was converted to +-2^63 or 2^63 - 1 and has wrapped the word's top
// bit: without that bit (a unit's finite sums stay below 2^62, see
// kDenseSubblock) it counts for nothing, so that a particle gone astray does not
// throw its neighbours about.
template <int NC, int ROWS, int COLS, int NP>
__device__ __forceinline__ void plane_out(long long (&pl)[NP][ROWS * kPlaneCols], long long *gp, int gs, long long ng,
                                          int lane) {
    for (int t = lane; t < ROWS * COLS; t += 32) {
        const int r = t / COLS, c = t - r * COLS, i = plane_word(r, c);
        long long *g = gp + gs * (r * ng + c);
#pragma unroll
        for (int k = 0; k < NC; ++k) {
            const long long v = pl[k][i];
            if (v != 0) {
                pl[k][i] = 0;
                const long long q = (long long)((unsigned long long)v << 1) >> 1;
                if (q != 0) red_add(g + k, q);
            }
        }
    }
    __syncwarp();
}

// A warp's sums of one quadratic plane: [oy][oz], components (0, 1) and (2, mass).
// ADJ: without mass, and the global sums are 4 words per node {3 components, lap}.
template <bool ADJ>
struct QuadSums {
    using Slot = QuadSlot;
    static constexpr int NC = ADJ ? 3 : 4, kStride = 8 * kQRows * kPlaneCols;
    float2 a[3][3][2];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) a[i][j][0] = a[i][j][1] = make_float2(0.0f, 0.0f);
    }
    // A particle's contribution to the 9 nodes of plane ox of its cell.
    __device__ __forceinline__ void row(const QuadSlot &s, int lane, int ox, float dx) {
        const float4 p0 = s.p[0][lane], p1 = s.p[1][lane], p2 = s.p[2][lane], p3 = s.p[3][lane];
        const float az2 = s.az2[lane];
        float wy[3], wz[3];
        qw(p0.y, wy);
        qw(p0.z, wz);
        // qw's weight of node ox alone
        const float t = ox == 0 ? 1.5f - p0.x : (ox == 1 ? p0.x - 1.0f : p0.x - 0.5f);
        const float wx = ox == 1 ? fmaf(-t, t, 0.75f) : 0.5f * (t * t);
        const float dxo = ((float)ox - p0.x) * dx;
        const float2 ay01 = make_float2(p2.z, p2.w), az01 = make_float2(p3.x, p3.y);
        const float2 base01 = fma2(make_float2(p2.x, p2.y), bc2(dxo), make_float2(p1.x, p1.y));
        const float base2 = fmaf(p3.z, dxo, p1.z);
        float2 b01[3], b2m[3], wz2[3];
#pragma unroll
        for (int oz = 0; oz < 3; ++oz) {
            const float dz = ((float)oz - p0.z) * dx;
            wz2[oz] = bc2(wz[oz]);
            b01[oz] = mul2(wz2[oz], fma2(az01, bc2(dz), base01));
            b2m[oz] = make_float2(wz[oz] * fmaf(az2, dz, base2), ADJ ? 0.0f : wz[oz] * p1.w);
        }
#pragma unroll
        for (int oy = 0; oy < 3; ++oy) {
            const float wxy = wx * wy[oy];
            const float wdy = wxy * (((float)oy - p0.y) * dx);
            const float2 w2 = bc2(wxy), s01 = mul2(bc2(wdy), ay01);
            const float s2 = wdy * p3.w;
#pragma unroll
            for (int oz = 0; oz < 3; ++oz) {
                a[oy][oz][0] = fma2(s01, wz2[oz], fma2(w2, b01[oz], a[oy][oz][0]));
                if (ADJ)
                    a[oy][oz][1].x = fmaf(wxy, b2m[oz].x, a[oy][oz][1].x);
                else
                    a[oy][oz][1] = fma2(w2, b2m[oz], a[oy][oz][1]);
                a[oy][oz][1].x = fmaf(s2, wz[oz], a[oy][oz][1].x);
            }
        }
    }
    static __device__ __forceinline__ void to_q(const SweepShared &sh, float2 u, float2 v, long long (&q)[NC]) {
        const float sm = sh.scale[0];
        q[0] = to_fix(u.x, sm);
        q[1] = to_fix(u.y, sm);
        q[2] = to_fix(v.x, sm);
        if (!ADJ) q[NC - 1] = to_fix(v.y, sh.scale[1]);
    }
    // All lanes' sums into the warp's plane.
    __device__ __forceinline__ void add(SweepShared &sh, int wid, int lane) {
        const int y = lane >> 3, z = lane & 7;
        char *pl = (char *)sh.qpl[wid];
#pragma unroll
        for (int oz = 0; oz < 3; ++oz) {
            const int i = 8 * plane_word(y, z + oz);
#pragma unroll
            for (int oy = 0; oy < 3; ++oy) {
                long long q[NC];
                to_q(sh, a[oy][oz][0], a[oy][oz][1], q);
                plane_words_add<NC>(pl + ((oy & 1) ? i ^ kOddRow : i) + oy * kRowBytes, kStride, q);
            }
        }
        clear();
    }
    // The sums of lane l alone: one node per lane.
    __device__ __forceinline__ void add_lane(SweepShared &sh, int wid, int lane, int l) {
        float2 *sp = sh.spill[wid];
        if (lane == l) {
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                sp[2 * i] = a[i / 3][i % 3][0];
                sp[2 * i + 1] = a[i / 3][i % 3][1];
            }
            clear();
        }
        __syncwarp();
        if (lane < 9) {
            long long q[NC];
            to_q(sh, sp[2 * lane], sp[2 * lane + 1], q);
            const int i = plane_word((l >> 3) + lane / 3, (l & 7) + lane % 3);
#pragma unroll
            for (int k = 0; k < NC; ++k) sh.qpl[wid][k][i] = fix_add(sh.qpl[wid][k][i], q[k]);
        }
        __syncwarp();
    }
    __device__ __forceinline__ void out(SweepShared &sh, int wid, int lane, int X) {
        plane_out<NC, kQRows, kQCols>(sh.qpl[wid], sh.g_quad + 4 * X * sh.ng * sh.ng, 4, sh.ng, lane);
    }
};

// A warp's sums of one cubic plane: [ny][nz], pairs (sum w d, sum w).
struct CubicSums {
    using Slot = CubicSlot;
    static constexpr int kStride = 8 * kCRows * kPlaneCols;
    float2 a[5][5];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < 5; ++i)
#pragma unroll
            for (int j = 0; j < 5; ++j) a[i][j] = make_float2(0.0f, 0.0f);
    }
    __device__ __forceinline__ void row(const CubicSlot &s, int lane, int ox, float) {
        const float4 p0 = s.p0[lane];
        float ey[5], ez[5];
        cw5(p0.y, ey);
        cw5(p0.z, ez);
        // a lane without a particle has fx = 0 (fx >= 0.5 otherwise)
        const float wx = p0.x != 0.0f ? cw5_node(ox, p0.x) : 0.0f;
        float2 ez2[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) ez2[k] = make_float2(p0.w * ez[k], ez[k]);
#pragma unroll
        for (int ny = 0; ny < 5; ++ny) {
            const float2 w2 = bc2(wx * ey[ny]);
#pragma unroll
            for (int nz = 0; nz < 5; ++nz) a[ny][nz] = fma2(w2, ez2[nz], a[ny][nz]);
        }
    }
    __device__ __forceinline__ void add(SweepShared &sh, int wid, int lane) {
        const int y = lane >> 3, z = lane & 7;
        char *pl = (char *)sh.cpl[wid - kSweepQ];
        const float sd = sh.scale[2], sw = sh.scale[3];
#pragma unroll
        for (int nz = 0; nz < 5; ++nz) {
            const int i = 8 * plane_word(y, z + nz);
#pragma unroll
            for (int ny = 0; ny < 5; ++ny) {
                const long long q[2] = {to_fix(a[ny][nz].x, sd), to_fix(a[ny][nz].y, sw)};
                plane_words_add<2>(pl + ((ny & 1) ? i ^ kOddRow : i) + ny * kRowBytes, kStride, q);
            }
        }
        clear();
    }
    __device__ __forceinline__ void add_lane(SweepShared &sh, int wid, int lane, int l) {
        float2 *sp = sh.spill[wid];
        if (lane == l) {
#pragma unroll
            for (int i = 0; i < 25; ++i) sp[i] = a[i / 5][i % 5];
            clear();
        }
        __syncwarp();
        if (lane < 25) {
            const float2 v = sp[lane];
            const int i = plane_word((l >> 3) + lane / 5, (l & 7) + lane % 5);
            long long(&pl)[2][kCRows * kPlaneCols] = sh.cpl[wid - kSweepQ];
            pl[0][i] = fix_add(pl[0][i], to_fix(v.x, sh.scale[2]));
            pl[1][i] = fix_add(pl[1][i], to_fix(v.y, sh.scale[3]));
        }
        __syncwarp();
    }
    __device__ __forceinline__ void out(SweepShared &sh, int wid, int lane, int X) {
        plane_out<2, kCRows, kCCols>(sh.cpl[wid - kSweepQ], sh.g_cubic + 2 * X * sh.ng * sh.ng, 2, sh.ng, lane);
    }
};

// The adjoint's cubic plane: sum d (w''x wy wz + wx w''y wz + wx wy w''z), [ny],
// paired over z: nodes 0, 1 and 2, 3; node 4 alone.
struct CubicLapSums {
    using Slot = CubicSlot;
    float2 a01[5], a23[5];
    float a4[5];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            a01[k] = a23[k] = make_float2(0.0f, 0.0f);
            a4[k] = 0.0f;
        }
    }
    __device__ __forceinline__ void row(const CubicSlot &s, int lane, int ox, float) {
        const float4 p0 = s.p0[lane];                // a lane without a particle has d = 0
        float ey[5], ez[5], fy[5], fz[5];
        cw5(p0.y, ey);
        cw5(p0.z, ez);
        cw5_2(p0.y, fy);
        cw5_2(p0.z, fz);
        const float ax = p0.w * cw5_2_node(ox, p0.x), bx2 = p0.w * cw5_node(ox, p0.x);   // d w''x, d wx
        const float2 ez01 = make_float2(ez[0], ez[1]), ez23 = make_float2(ez[2], ez[3]);
        const float2 fz01 = make_float2(fz[0], fz[1]), fz23 = make_float2(fz[2], fz[3]);
#pragma unroll
        for (int ny = 0; ny < 5; ++ny) {
            const float wy = ey[ny], w2y = fy[ny];
            const float t1 = ax * wy + bx2 * w2y;   // (w''x wy + wx w''y) d
            const float t2 = bx2 * wy;              // wx wy d
            const float2 t12 = bc2(t1), t22 = bc2(t2);
            a01[ny] = fma2(t22, fz01, fma2(t12, ez01, a01[ny]));
            a23[ny] = fma2(t22, fz23, fma2(t12, ez23, a23[ny]));
            a4[ny] = fmaf(t2, fz[4], fmaf(t1, ez[4], a4[ny]));
        }
    }
    __device__ __forceinline__ void add(SweepShared &sh, int wid, int lane) {
        const int y = lane >> 3, z = lane & 7;
        char *pl = (char *)sh.cpl[wid - kSweepQ];
        const float sd = sh.scale[2];
#pragma unroll
        for (int nz = 0; nz < 5; ++nz) {
            const int i = 8 * plane_word(y, z + nz);
#pragma unroll
            for (int ny = 0; ny < 5; ++ny) {
                const float v = nz == 0 ? a01[ny].x : nz == 1 ? a01[ny].y : nz == 2 ? a23[ny].x : nz == 3 ? a23[ny].y : a4[ny];
                const long long q[1] = {to_fix(v, sd)};
                plane_words_add<1>(pl + ((ny & 1) ? i ^ kOddRow : i) + ny * kRowBytes, 0, q);
            }
        }
        clear();
    }
    __device__ __forceinline__ void add_lane(SweepShared &sh, int wid, int lane, int l) {
        float *sp = (float *)sh.spill[wid];
        if (lane == l) {
#pragma unroll
            for (int ny = 0; ny < 5; ++ny) {
                sp[5 * ny] = a01[ny].x;
                sp[5 * ny + 1] = a01[ny].y;
                sp[5 * ny + 2] = a23[ny].x;
                sp[5 * ny + 3] = a23[ny].y;
                sp[5 * ny + 4] = a4[ny];
            }
            clear();
        }
        __syncwarp();
        if (lane < 25) {
            long long &at = sh.cpl[wid - kSweepQ][0][plane_word((l >> 3) + lane / 5, (l & 7) + lane % 5)];
            at = fix_add(at, to_fix(sp[lane], sh.scale[2]));
        }
        __syncwarp();
    }
    __device__ __forceinline__ void out(SweepShared &sh, int wid, int lane, int X) {
        plane_out<1, kCRows, kCCols>(sh.cpl[wid - kSweepQ], sh.g_cubic + 4 * X * sh.ng * sh.ng, 4, sh.ng, lane);
    }
};

// Adds the rows of one layer (this lane's cell: `cell`, and `split`, see
// SweepShared) to a warp's sums.  IN_ROWS: the layer's layout, known for the
// whole layer.  few: the layer's sums go to the plane here, cell by cell with the
// nodes over the lanes, not with the cells over the lanes node by node (add): a
// cloud of 100k particles, 7 to a unit, 566 us per substep and 484.  (Only in
// clouds: for the thin layers of bodies' surfaces it is the longer chain, 12 small
// scenes 340 and 344 us.)
template <bool IN_ROWS, class SUMS>
__device__ __forceinline__ void sweep_layer(SweepShared &sh, SUMS &sums, typename SUMS::Slot *ring, const char *payload,
                                            int2 cell, int split, int rows, bool few, int ox, int wid, int lane) {
    const int first = cell.x & ~kCellRows;
    const float dx = sh.dx;
    const char *src = pay_block(payload, first);   // in rows: place k of the cell is the lane's of the k-th block on
    auto copy = [&](int k) {
        const bool on = k < cell.y;
        if (IN_ROWS) {
            row_copy(ring[k & (kRing - 1)], src, lane, on, lane);
            src += kPayBlock;
        } else {
            const int s = on ? first + k : 0;
            row_copy(ring[k & (kRing - 1)], pay_block(payload, s), s & 31, on, lane);
        }
    };
#pragma unroll
    for (int k = 0; k < kRing - 1; ++k) {
        if (k < rows) copy(k);
        cp_async_commit();
    }
    int restart = 256 - split;              // this lane's next particle that starts a new sum
    int k = 0;
    for (;;) {
        const int until = __reduce_min_sync(0xffffffffu, restart < cell.y ? restart : rows);
#pragma unroll 1
        for (; k < until; ++k) {
            cp_async_wait<kRing - 2>();
            sums.row(ring[k & (kRing - 1)], lane, ox, dx);
            if (k + kRing - 1 < rows) copy(k + kRing - 1);   // into the slot of the row before this one
            cp_async_commit();
        }
        const bool end = k >= rows;
        if (end && (IN_ROWS || !few)) break;     // (a layer in rows has at least 16 cells)
        const bool mine = end ? cell.y > 0 : restart == k;
        for (unsigned m = __ballot_sync(0xffffffffu, mine); m; m &= m - 1) sums.add_lane(sh, wid, lane, __ffs(m) - 1);
        if (end) break;
        if (mine) restart += 256;
    }
}

// The sweep of one warp (wid: its number in the CTA, set: among the N interleaved
// sets of planes) over layers x0 .. x1 - 1.  FEW: whether layer_code marks thin
// layers of clouds (the adjoint, mostly of bodies, saves the test: 0.4% of the slab's
// gradients).  (The reductions of values that all lanes share tell the compiler
// that they do.)
template <class SUMS, int N, bool FEW>
__device__ __forceinline__ void sweep_warp(SweepShared &sh, typename SUMS::Slot *ring, const char *payload, int wid,
                                           int set, int lane, int x0, int x1) {
    SUMS sums;
    sums.clear();
    bool dirty = false;
    int ox = (set + 4 * N - x0) % N;                       // this warp's plane: X = x + ox
#pragma unroll 1
    for (int x = x0; x < x1; ++x) {
        const int code = __reduce_max_sync(0xffffffffu, sh.layer_rows[x]);
        if (code != 0) {
            const bool few = FEW && code < 0;
            const int rows = FEW ? abs(code) : code;
            const int2 cell = sh.cell[32 * x + lane];
            const int split = sh.split[32 * x + lane];
            if (__any_sync(0xffffffffu, cell.x < 0))
                sweep_layer<true>(sh, sums, ring, payload, cell, split, rows, few, ox, wid, lane);
            else
                sweep_layer<false>(sh, sums, ring, payload, cell, split, rows, few, ox, wid, lane);
            if (!few) sums.add(sh, wid, lane);
            dirty = true;
        }
        if (dirty && (ox == 0 || x == x1 - 1)) {           // no later layer reaches this plane
            sums.out(sh, wid, lane, x + ox);
            dirty = false;
        }
        ox = ox == 0 ? N - 1 : ox - 1;
    }
}

// ------------------------------------------------------------ clamped nodes
// Cells whose stencils need the reference's clamped nodes (anisompm.py:716-724,
// 771-776; base cell outside [1, n_grid - 4], payload part 0 {x, d}) are left out
// of the sweep and scattered by the same CTAs when they have run out of items, a
// layer of a unit (its cells in sh.cell) at a time.  One warp takes up to kClampRun
// particles of a cell, one after another, and every lane keeps the exact sums of
// its nodes: lane l quadratic node l of 27, cubic nodes l, l + 32, .. of the 125
// that the cell's particles can reach, which go to the grid when the run ends or
// the particles' base cell changes (outside the domain cells share their place in
// the table).  MARK::node is called for every node that the sums go to.  ADJ: see
// QuadSums; the cubic sums are CubicLapSums'.
//
// A thread per particle with its 236 atomics, a cell of the layer after another,
// made a substep of a body resting on the upper end of the domain (131k particles,
// 8 per cell) 595 us, this 82; with four layers pressed into the last one (164k)
// 1,090 us and 130.  (Called from within the sweep's loop it costs the sweep of bodies
// that touch no edge 5 to 15%, in registers.)
__device__ __forceinline__ bool clamped_cell(const int c[3], int ng) {
    bool reg = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) reg = reg && c[a] >= 1 && c[a] <= ng - 4;
    return !reg;
}
// Whether a unit with first cell org has such cells.
__device__ __forceinline__ bool clamped_unit(const int org[3], int ng) {
    return org[0] == 0 || org[1] == 0 || org[2] == 0 || org[0] + kUnitX > ng - 3 || org[1] + kUnitY > ng - 3 ||
           org[2] + kUnitZ > ng - 3;
}
// First cell of unit u; blk: its sort block within the scene, nb sort blocks per axis.
__device__ __forceinline__ void unit_origin(int u, unsigned blk, int nb, int org[3]) {
    org[0] = (int)(blk / ((unsigned)nb * nb)) * kSortBlock + ((u >> 1) & 1) * kUnitX;
    org[1] = (int)(blk / nb % nb) * kSortBlock + (u & 1) * kUnitY;
    org[2] = (int)(blk % nb) * kSortBlock;
}
constexpr int kClampRun = 32;
template <bool ADJ, class MARK>
__device__ __noinline__ void scatter_clamped(SweepShared &sh, const WS *w, const char *payload) {
    constexpr int NQ = ADJ ? 3 : 4, NC = ADJ ? 1 : 2, GC = ADJ ? 4 : 2, CN = 4;   // CN: cubic nodes of a lane
    constexpr unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, o[3] = {lane / 9, lane / 3 % 3, lane % 3};
    const int ng = (int)sh.ng;
    const float inv_dx = sh.inv_dx, dx = sh.dx;
    QuadSlot &slot = (&sh.qring[0][0])[wid];       // the rings are idle
    const int2 mine = sh.cell[lane];
    int run = 0;
    for (unsigned todo = __ballot_sync(all, mine.y > 0); todo; todo &= todo - 1) {
        const int l = __ffs(todo) - 1;
        const int first = __shfl_sync(all, mine.x, l), cnt = __shfl_sync(all, mine.y, l);
        for (int k0 = 0; k0 < cnt; k0 += kClampRun, ++run) {
            if ((run & 7) != wid) continue;
            // lane k: the run's k-th particle, to shared memory; its base cell and place between the nodes
            const int n = min(cnt - k0, kClampRun);
            float f[3] = {0.0f, 0.0f, 0.0f};
            int b[3] = {0, 0, 0};
            __syncwarp();                          // the run before is done with
            if (lane < n) {
                const long long s = place_of(first, k0 + lane);
                const char *block = pay_block(payload, s);
                const int i = (int)(s & 31);
                const float4 p0 = *(const float4 *)(block + pay_part(0, i));
                slot.p[0][lane] = p0;
#pragma unroll
                for (int k = 1; k < 4; ++k) slot.p[k][lane] = *(const float4 *)(block + pay_part(k, i));
                slot.az2[lane] = *(const float *)(block + pay_part(4, i));
                const float xp[3] = {p0.x, p0.y, p0.z};
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const float X = __fmul_rn(xp[a], inv_dx), fb = floorf(__fsub_rn(X, 0.5f));
                    b[a] = sat_base(fb, ng);
                    f[a] = __fsub_rn(X, fb);
                }
            }
            __syncwarp();
            bool other = false;                    // another base cell than the particle before
#pragma unroll
            for (int a = 0; a < 3; ++a) other |= __shfl_up_sync(all, b[a], 1) != b[a];
            const unsigned ends = __ballot_sync(all, lane == 0 || lane >= n || other) >> 1;   // bit k: k is the last of its base
            long long q[NQ], c[CN][NC];
#pragma unroll
            for (int i = 0; i < NQ; ++i) q[i] = 0;
#pragma unroll
            for (int j = 0; j < CN; ++j)
#pragma unroll
                for (int i = 0; i < NC; ++i) c[j][i] = 0;
            for (int k = 0; k < n; ++k) {
                const float4 p1 = slot.p[1][k], p2 = slot.p[2][k], p3 = slot.p[3][k];
                const float a22 = slot.az2[k], d = slot.p[0][k].w;
                const float fk[3] = {__shfl_sync(all, f[0], k), __shfl_sync(all, f[1], k), __shfl_sync(all, f[2], k)};
                // lane 5 a + i: the cubic weight of axis a, node i
                const float fl = lane < 5 ? fk[0] : (lane < 10 ? fk[1] : fk[2]);
                const int il = lane < 5 ? lane : (lane < 10 ? lane - 5 : lane - 10);
                const float wl = cw5_node(il, fl), wl2 = ADJ ? cw5_2_node(il, fl) : 0.0f;
                {   // quadratic: this lane's node (lanes 27 and up: not used)
                    float wq[3], D[3];
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        const float t = o[a] == 0 ? 1.5f - fk[a] : (o[a] == 1 ? fk[a] - 1.0f : fk[a] - 0.5f);
                        wq[a] = o[a] == 1 ? 0.75f - t * t : 0.5f * (t * t);
                        D[a] = ((float)o[a] - fk[a]) * dx;
                    }
                    const float wk = wq[0] * wq[1] * wq[2], sm = sh.scale[0];
                    const float a0 = p2.x * D[0] + p2.z * D[1] + p3.x * D[2];
                    const float a1 = p2.y * D[0] + p2.w * D[1] + p3.y * D[2];
                    const float a2 = p3.z * D[0] + p3.w * D[1] + a22 * D[2];
                    q[0] = fix_add(q[0], to_fix(wk * (p1.x + a0), sm));
                    q[1] = fix_add(q[1], to_fix(wk * (p1.y + a1), sm));
                    q[2] = fix_add(q[2], to_fix(wk * (p1.z + a2), sm));
                    if (!ADJ) q[NQ - 1] = fix_add(q[NQ - 1], to_fix(wk * p1.w, sh.scale[1]));
                }
#pragma unroll
                for (int j = 0; j < CN; ++j) {     // (lanes past the 125th node: any weight, not used)
                    const int m = min(lane + 32 * j, 124), nx = m / 25, ny = 5 + m / 5 % 5, nz = 10 + m % 5;
                    const float wx = __shfl_sync(all, wl, nx), wy = __shfl_sync(all, wl, ny), wz = __shfl_sync(all, wl, nz);
                    if (ADJ) {
                        const float vx = __shfl_sync(all, wl2, nx), vy = __shfl_sync(all, wl2, ny),
                                    vz = __shfl_sync(all, wl2, nz);
                        const float ab = d * (vx * wy + wx * vy), e = d * (wx * wy);
                        c[j][0] = fix_add(c[j][0], to_fix(ab * wz + e * vz, sh.scale[2]));
                    } else {
                        const float wk = wx * wy * wz;
                        c[j][0] = fix_add(c[j][0], to_fix(wk * d, sh.scale[2]));
                        c[j][NC - 1] = fix_add(c[j][NC - 1], to_fix(wk, sh.scale[3]));
                    }
                }
                if (k < n - 1 && !(ends >> k & 1)) continue;
                const int bk[3] = {__shfl_sync(all, b[0], k), __shfl_sync(all, b[1], k), __shfl_sync(all, b[2], k)};
                if (lane < 27) {
                    const int x = clampi(bk[0] + o[0], 0, ng - 1), y = clampi(bk[1] + o[1], 0, ng - 1),
                              z = clampi(bk[2] + o[2], 0, ng - 1);
                    long long *g = sh.g0_quad + 4 * (((long long)x * ng + y) * ng + z);
#pragma unroll
                    for (int i = 0; i < NQ; ++i) {
                        if (q[i] != 0) red_add(g + i, q[i]);
                        q[i] = 0;
                    }
                    MARK::node(sh, w, x, y, z);
                }
#pragma unroll
                for (int j = 0; j < CN; ++j) {
                    const int m = lane + 32 * j;
                    if (m < 125) {
                        const int x = clampi(bk[0] - 1 + m / 25, 0, ng - 1), y = clampi(bk[1] - 1 + m / 5 % 5, 0, ng - 1),
                                  z = clampi(bk[2] - 1 + m % 5, 0, ng - 1);
                        long long *g = sh.g0_cubic + GC * (((long long)x * ng + y) * ng + z);
#pragma unroll
                        for (int i = 0; i < NC; ++i) {
                            if (c[j][i] != 0) red_add(g + i, c[j][i]);
                            c[j][i] = 0;
                        }
                        MARK::node(sh, w, x, y, z);
                    }
                }
                __syncwarp();
            }
        }
    }
}

}  // namespace pm
