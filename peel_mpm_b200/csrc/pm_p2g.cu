// Binning, constitutive update and P2G.
//
// Binning is by counting, in a table over the substep's cells: k_count gives
// every particle its arrival number in its cell and lists the non-empty units
// (4 x 4 x 8 cells), k_offsets gives every unit's cells their payload places,
// k_place and k_rank turn arrival numbers into places in id order, so that what
// follows does not depend on the order of arrival.  (A stable radix sort of cell
// keys took 9 or 10 latency-bound launches, 90 us of the 1M-particle substep,
// against 50 here.)
//
// k_stress, one thread per particle in particle order (coalesced state
// reads): particle BC, polar decomposition (Jacobi eigensolve of F^T F),
// fixed-corotated Kirchhoff stress, anisotropic phase-field damage (the
// Cauchy stress's eigensystem taken from the polar decomposition, a Jacobi
// solve only for nearly singular F), degradation and the APIC affine term;
// the P2G payload goes to the particle's place, and the substep's bounds on one
// node contribution (momentum, mass, damage) are raised in the control block.
//
// k_p2g_sweep, persistent CTAs taking units from the list: every cell's
// contributions to its 27 quadratic ({mv, m}) and 125 cubic ({sum w d, sum w})
// nodes are summed in float registers by a sweep along x and added as exact fixed
// point (pm_sweep.cuh); integer addition is associative, so the grid sums, and
// with them the whole substep, are the same bits whatever order the atomics run
// in.  The 4^3 grid blocks touched are marked and listed.  Cells whose stencils
// need the reference's edge clamping (base cell outside [1, n_grid-4]) go straight
// to the global grid instead (scatter_clamped).
//
// Reference: anisompm.py:601-724 (constitutive, damage, P2G) and 768-776
// (cubic damage scatter).
#include "pm_kernels.cuh"
#include "pm_sweep.cuh"

namespace pm {

__device__ __forceinline__ float clamp_min(float v, float lo) { return v < lo ? lo : v; }   // torch.clamp(min=)
__device__ __forceinline__ float relu(float v) { return v > 0.0f ? v : (v != v ? v : 0.0f); }
// torch.maximum: NaN if either operand is NaN
__device__ __forceinline__ float tmax(float a, float b) { return (a != a || b != b) ? a + b : (a > b ? a : b); }

// Constitutive update of particle p (anisompm.py:614-706).  Writes tau and
// updates F (f_clamp), d, D_hist and the diagnostics in place.
// When `rec` is set (recording a substep for the adjoint) the polar
// decomposition (R, V, S) and, on damage steps, phi are written to its planes:
// rec[k * rs + p] for R (k 0..8), V (9..17), S (18..20), phi (21).
// Per-particle inputs of the constitutive update, all loaded before any
// store (the state planes share one buffer, so a store would otherwise keep
// later loads from being issued early).  The inputs of the affine term and
// the payload (C, v, x, vol0, mass, grip) are loaded after it: they are not
// needed earlier, and holding them across the eigensolve costs registers.
struct StressIn {
    float F[9], A0[9];
    float d, lap, Dh, mu, lam, sc, eta, zeta, l0, res;
    bool allow;
};

__device__ __forceinline__ void constitutive(const pm_params &prm, const Parts &P, long long p, bool do_damage,
                                             const StressIn &in, float tau[9], float &d_out, float *rec = nullptr,
                                             long long rs = 0) {
    const long long ps = P.ps;
    float F[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) F[k] = in.F[k];
    float Cg[9];   // C = F^T F (615)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) Cg[3 * i + j] = F[i] * F[j] + F[3 + i] * F[3 + j] + F[6 + i] * F[6 + j];
    float lamC[3], V[9];
    sym_eig3<5>(Cg, lamC, V);                                        // (616)
    float S[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) S[i] = sqrtf(clamp_min(lamC[i], 1e-12f));   // (617)
    float W[9], R[9];
    bool u_ok;
    mm3(F, V, W);                                                    // (619)
    {
        float wn[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            wn[j] = sqrtf(W[j] * W[j] + W[3 + j] * W[3 + j] + W[6 + j] * W[6 + j]);
            const float rn = 1.0f / (wn[j] + 1e-12f);                 // one division per column
#pragma unroll
            for (int i = 0; i < 3; ++i) W[3 * i + j] *= rn;          // (620)
        }
        u_ok = polar_u_ok(wn);
    }
    mmt3(W, V, R);                                                   // R = What V^T (621)
    if (rec) {
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            rec[k * rs + p] = R[k];
            rec[(9 + k) * rs + p] = V[k];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) rec[(18 + k) * rs + p] = S[k];
    }
    if (prm.use_f_clamp) {                                           // (622-636)
        f_clamp_F(F, V, S, (float)prm.f_clamp_lo, (float)prm.f_clamp_hi, F);
#pragma unroll
        for (int k = 0; k < 9; ++k) P.Fo[k * ps + p] = F[k];
    }
    const float J = clamp_min(S[0] * S[1] * S[2], 1e-6f);            // (637)
    const float mu = in.mu, lam = in.lam;
    float tdev[9];
    {
        float FmR[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) FmR[k] = (2.0f * mu) * (F[k] - R[k]);
        mmt3(FmR, F, tdev);                                          // 2mu (F-R) F^T (643)
    }
    const float tv = lam * (J - 1.0f) * J;                           // (644)

    if (do_damage) {                                                 // (647-685)
        float sg[9];
        const float rJ = 1.0f / J;
#pragma unroll
        for (int k = 0; k < 9; ++k) sg[k] = (tdev[k] + ((k % 4 == 0) ? tv : 0.0f)) * rJ;
        float sgs[9];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) sgs[3 * i + j] = 0.5f * (sg[3 * i + j] + sg[3 * j + i]);
        float ev[3], EV[9];
        if (u_ok)   // (652: sym_eig of sig)
            stress_eig_polar(W, sgs, ev, EV);
        else
            sym_eig3<5>(sgs, ev, EV);
        float sp[9];
        {
            float ED[9];
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const float e = ev[j] < 0.0f ? 0.0f : ev[j];
#pragma unroll
                for (int i = 0; i < 3; ++i) ED[3 * i + j] = EV[3 * i + j] * e;
            }
            mmt3(ED, EV, sp);                                        // sigma+ (654-655)
        }
        float A[9];
        {
            float A0[9], RA[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) A0[k] = in.A0[k];
            mm3(R, A0, RA);
            mmt3(RA, R, A);                                          // A = R A0 R^T (661)
        }
        float M[9];
        mm3(A, sp, M);
        const float trMM = (M[0] * M[0] + M[1] * M[3] + M[2] * M[6]) + (M[3] * M[1] + M[4] * M[4] + M[5] * M[7]) +
                           (M[6] * M[2] + M[7] * M[5] + M[8] * M[8]);
        const float sc = in.sc;
        const float phi = trMM / (sc * sc);                          // (663-664)
        if (rec) rec[21 * rs + p] = phi;
        if (P.phi) P.phi[p] = phi;
        if (P.phi_shear) {                                           // (670-673)
            float phs = 0.0f;
            if (P.n_interface) {
                const float n0 = P.n_interface[p], n1 = P.n_interface[ps + p], n2 = P.n_interface[2 * ps + p];
                const float s0 = sp[0] * n0 + sp[1] * n1 + sp[2] * n2;
                const float s1 = sp[3] * n0 + sp[4] * n1 + sp[5] * n2;
                const float s2 = sp[6] * n0 + sp[7] * n1 + sp[8] * n2;
                const float tn = s0 * n0 + s1 * n1 + s2 * n2;
                const float t0 = s0 - tn * n0, t1 = s1 - tn * n1, t2 = s2 - tn * n2;
                const float q = sqrtf(t0 * t0 + t1 * t1 + t2 * t2) / sc;
                phs = q * q;
            }
            P.phi_shear[p] = phs;
        }
        const float drive = in.zeta * relu(phi - 1.0f);
        const float dh0 = in.Dh;
        const float Dh = tmax(dh0, drive);
        P.Dho[p] = Dh;                                               // history max (679)
        const float d = in.d;
        const float l0 = in.l0;
        const float resist = d - (l0 * l0) * in.lap;
        const float ddot = relu((1.0f - d) * Dh - resist);           // (681-682)
        const float dt_dmg = (float)(prm.dt * (double)prm.damage_every);
        float dn = d + (dt_dmg / in.eta) * ddot;
        dn = dn < 0.0f ? 0.0f : dn;
        dn = dn > 1.0f ? 1.0f : dn;                                  // (683-684)
        if (in.allow) {                                              // monotone, where allowed (685)
            d_out = tmax(dn, d);
            P.d_o[p] = d_out;
        }
    }
    const float d = d_out;
    const float res = in.res;
    const float omd = 1.0f - d;
    const float g = (omd * omd) * (1.0f - res) + res;                // (688)
    const float vdeg = (J >= 1.0f) ? g : 1.0f;                       // (690)
#pragma unroll
    for (int k = 0; k < 9; ++k) tau[k] = g * tdev[k] + ((k % 4 == 0) ? vdeg * tv : 0.0f);
    if (P.interface_mask && P.interface_mask[p]) {
        // directional_kirchhoff(tau_dev + tau_vol, F, d, n, g, g, tension_gate=True)
        // (anisompm.py:190-227 via 697-703)
        float tc[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) tc[k] = tdev[k] + ((k % 4 == 0) ? tv : 0.0f);
        const float n0 = P.n_interface[p], n1 = P.n_interface[ps + p], n2 = P.n_interface[2 * ps + p];
        float m[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) m[i] = F[3 * i] * n0 + F[3 * i + 1] * n1 + F[3 * i + 2] * n2;
        const float mn = sqrtf(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]) + 1e-9f;
#pragma unroll
        for (int i = 0; i < 3; ++i) m[i] = m[i] / mn;
        float Pm[9], Qm[9];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                Pm[3 * i + j] = m[i] * m[j];
                Qm[3 * i + j] = ((i == j) ? 1.0f : 0.0f) - Pm[3 * i + j];
            }
        float T1[9], perp[9], sh1[9], sh2[9], par[9];
        mm3(Pm, tc, T1);
        mm3(T1, Pm, perp);
        mm3(T1, Qm, sh1);
        mm3(Qm, tc, T1);
        mm3(T1, Pm, sh2);
        mm3(T1, Qm, par);
        float tm0 = m[0] * tc[0] + m[1] * tc[3] + m[2] * tc[6];
        float tm1 = m[0] * tc[1] + m[1] * tc[4] + m[2] * tc[7];
        float tm2 = m[0] * tc[2] + m[1] * tc[5] + m[2] * tc[8];
        const float snn = tm0 * m[0] + tm1 * m[1] + tm2 * m[2];
        const float gI = (snn > 0.0f) ? g : 1.0f;
#pragma unroll
        for (int k = 0; k < 9; ++k) tau[k] = par[k] + gI * perp[k] + g * (sh1[k] + sh2[k]);
    }
    if (prm.record_stress) {
        if (P.tau_last) {
#pragma unroll
            for (int k = 0; k < 9; ++k) P.tau_last[k * ps + p] = tau[k];
        }
        if (P.J_last) P.J_last[p] = J;
    }
}

// ------------------------------------------------------------------ binning
// Key of particle p's cell in the substep's cell table.
template <class SC>
__device__ __forceinline__ unsigned cell_of(const SC &sc, int sid, const float xp[3], int ng, float inv_dx) {
    int qb[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) qb[a] = sat_base(floorf(__fsub_rn(__fmul_rn(xp[a], inv_dx), 0.5f)), ng);
    return (sc.sblock_base(sid) << kSortBlockBits) + unit_key(qb, ng);
}

// Particles per cell, in the substep's own cell table: every particle takes
// its arrival number in its cell (one atomic per warp and cell), the first
// particle of a unit puts the unit on the work list, and allow.any() is
// raised.  CTAs are aligned to scenes: 256 particles each, four per thread so
// that the chains of load, atomic and list entry of four particles overlap.
constexpr int kCountThreads = 64, kCountItems = 256 / kCountThreads;
template <class SC>
__global__ void __launch_bounds__(kCountThreads) k_count(const SC sc, const float *__restrict__ x, long long n,
                                                         long long ps, const unsigned char *__restrict__ allow,
                                                         const WS w) {
    const int sid = sc.of_cta(blockIdx.x), lane = threadIdx.x & 31;
    const pm_params &prm = sc.params(sid);
    const long long p0 = sc.p_begin(sid) + ((long long)blockIdx.x - sc.cta_base(sid)) * 256 + threadIdx.x;
    const long long end = sc.p_end(sid, n);
    const int ng = prm.n_grid;
    const float inv_dx = (float)prm.inv_dx;
    unsigned key[kCountItems], peers[kCountItems];
    int base[kCountItems];
    bool any = false;
#pragma unroll
    for (int g = 0; g < kCountItems; ++g) {
        const long long p = p0 + g * kCountThreads;
        key[g] = 0xffffffffu;
        if (p < end) {
            const float xp[3] = {x[p], x[ps + p], x[2 * ps + p]};
            any |= allow[p] != 0;
            key[g] = cell_of(sc, sid, xp, ng, inv_dx);
        }
    }
#pragma unroll
    for (int g = 0; g < kCountItems; ++g) {
        peers[g] = __match_any_sync(0xffffffffu, key[g]);
        base[g] = 0;
        if (p0 + g * kCountThreads < end && lane == __ffs(peers[g]) - 1)
            base[g] = atomicAdd(&w.cells[key[g]].y, __popc(peers[g]));
    }
#pragma unroll
    for (int g = 0; g < kCountItems; ++g) {
        const long long p = p0 + g * kCountThreads;
        const int leader = __ffs(peers[g]) - 1;
        if (p < end && lane == leader && base[g] == 0 && atomicAdd(&w.utot[key[g] / kUnitCells], 1) == 0) {
            const unsigned i = atomicAdd(&w.ctrl->n_work, 1u);
            if (i < (unsigned long long)n) w.work[i] = (int)(key[g] / kUnitCells);   // bounded even without a clock reset
        }
        const int b = __shfl_sync(0xffffffffu, base[g], leader);
        if (p < end) w.slot[p] = b + __popc(peers[g] & lanemask_lt());
    }
    // one store per scene in the main: a store per warp queues on the one word
    if (__syncthreads_or(any) && threadIdx.x == 0 && *(volatile int *)&w.ctrl[sid].any_allow == 0)
        w.ctrl[sid].any_allow = 1;
}

// Gives every listed unit's layers (32 cells) a run of payload places and the
// cells their first place; runs lie in any order (the grid sums are exact).  A
// layer goes in rows, from the front of the payload, if those take at most
// kPayPlaces places per particle, else cell after cell, from the back, so that
// the two never meet.  Also counts the 4^3-cell sub-blocks beyond the fixed-point
// headroom and lists the units with cells that need clamped nodes.  One warp per
// unit, one lane per cell of a layer.
template <class SC>
__global__ void __launch_bounds__(256) k_offsets(const SC sc, const WS w, long long n) {
    __shared__ __align__(16) int s_morton[8][kUnitCells];   // read as int4 too
    const unsigned n_work = min(w.ctrl->n_work, (unsigned)min(n, (long long)0x7fffffff));
    const int lane = threadIdx.x & 31;
    int *morton = s_morton[threadIdx.x >> 5];
    const int y = lane >> 3, z = lane & 7;
    const int mz = (z >> 2) * 64 + (y >> 1) * 16 + ((z >> 1) & 1) * 8 + (y & 1) * 2 + (z & 1);   // x bits: 32 and 4
    for (unsigned i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n_work; i += (gridDim.x * blockDim.x) >> 5) {
        const int u = w.work[i];
        int2 *cells = w.cells + (long long)u * kUnitCells + lane;
        int c[kUnitX], first[kUnitX], rows_size = 0, flat_size = 0;
#pragma unroll
        for (int x = 0; x < kUnitX; ++x) c[x] = cells[32 * x].y;
#pragma unroll
        for (int x = 0; x < kUnitX; ++x) {
            int incl = c[x];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const int total = __shfl_sync(0xffffffffu, incl, 31), rows = __reduce_max_sync(0xffffffffu, c[x]);
            const bool in_rows = rows <= total * kPayPlaces / 32;
            first[x] = in_rows ? (rows_size + lane) | kCellRows : flat_size + incl - c[x];
            rows_size += in_rows ? rows * 32 : 0;
            flat_size += in_rows ? 0 : total;
        }
        int base = 0, end = 0;
        if (lane == 0) {
            if (rows_size > 0) base = (int)atomicAdd(&w.ctrl->run_next, (unsigned)rows_size);
            if (flat_size > 0) end = (int)(w.pay_places - atomicAdd(&w.ctrl->run_end, (unsigned)flat_size)) - flat_size;
        }
        base = __shfl_sync(0xffffffffu, base, 0);
        end = __shfl_sync(0xffffffffu, end, 0);
#pragma unroll
        for (int x = 0; x < kUnitX; ++x) {
            const int f = first[x] + (first[x] < 0 ? base : end);
            cells[32 * x].x = f;
            if (w.rec_cells) w.rec_cells[(long long)i * kUnitCells + 32 * x + lane] = make_int2(f, c[x]);
        }
        {   // particles before each cell in Morton order of its sub-block (16 lanes, 4 cells each, to a sub-block)
            __syncwarp();
#pragma unroll
            for (int x = 0; x < kUnitX; ++x) morton[mz + (x >> 1) * 32 + (x & 1) * 4] = c[x];
            __syncwarp();
            int4 m = ((int4 *)morton)[lane];
            const int sum = m.x + m.y + m.z + m.w;
            int incl = sum;
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o, 16);
                if ((lane & 15) >= o) incl += v;
            }
            const int before = incl - sum;
            __syncwarp();
            ((int4 *)morton)[lane] = make_int4(before, before + m.x, before + m.x + m.y, before + m.x + m.y + m.z);
            __syncwarp();
#pragma unroll
            for (int x = 0; x < kUnitX; ++x) {
                const unsigned char b = (unsigned char)(morton[mz + (x >> 1) * 32 + (x & 1) * 4] & 255);
                w.split[(long long)u * kUnitCells + 32 * x + lane] = b;
                if (w.rec_split) w.rec_split[(long long)i * kUnitCells + 32 * x + lane] = b;
            }
        }
        const int sid = sc.of_sblock((unsigned)u / kBlockUnits);
        const int ng = sc.params(sid).n_grid;
        int org[3];
        unit_origin(u, (unsigned)u / kBlockUnits - sc.sblock_base(sid), sort_blocks_per_axis(ng), org);
        if (clamped_unit(org, ng)) {
            bool any = false;
#pragma unroll
            for (int x = 0; x < kUnitX; ++x) {
                const int g[3] = {org[0] + x, org[1] + y, org[2] + z};
                any |= c[x] > 0 && clamped_cell(g, ng);
            }
            if (__any_sync(0xffffffffu, any) && lane == 0) {
                const unsigned at = atomicAdd(&w.ctrl->n_clamped, 1u);
                if (at < n_work) w.clamped[at] = (int)i;   // bounded even without a clock reset
            }
        }
        const int mine = c[0] + c[1] + c[2] + c[3];
        const int low = __reduce_add_sync(0xffffffffu, (lane & 7) < 4 ? mine : 0);
        const int high = __reduce_add_sync(0xffffffffu, (lane & 7) < 4 ? 0 : mine);
        if (lane == 0 && max(low, high) > kDenseSubblock)
            atomicAdd(&w.ctrl[sid].dense_subblocks,
                      (low > kDenseSubblock ? 1u : 0u) + (high > kDenseSubblock ? 1u : 0u));
    }
}

// Particle ids by place, in order of arrival.  Particles of cells of more than
// kRankRows particles are marked in w.slot (see k_rank).
constexpr int kRankRows = 64, kRankWarps = 4, kRankRun = kRankRows * 32 / kRankWarps;
template <class SC>
__global__ void __launch_bounds__(256) k_place(const SC sc, const float *__restrict__ x, long long n, long long ps,
                                               const WS w) {
    const int sid = sc.of_cta(blockIdx.x);
    const pm_params &prm = sc.params(sid);
    const long long p = sc.p_begin(sid) + ((long long)blockIdx.x - sc.cta_base(sid)) * 256 + threadIdx.x;
    if (p >= sc.p_end(sid, n)) return;
    const float xp[3] = {x[p], x[ps + p], x[2 * ps + p]};
    const int slot = w.slot[p];
    const int2 cell = w.cells[cell_of(sc, sid, xp, prm.n_grid, (float)prm.inv_dx)];
    const long long at = place_of(cell.x, slot);
    w.ids[at] = (int)p;
    if (cell.y > kRankRows) w.slot[p] = -1;
}

// Sorts the ids of a layer's cells `more` (cell: this lane's), each in runs of
// kRankRun, a warp to a run (buf: this warp's).
__device__ __noinline__ void sort_runs(int *ids, int2 cell, unsigned more, int *buf) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int run = 0; more; more &= more - 1) {
        const int l = __ffs(more) - 1;
        const int first = __shfl_sync(0xffffffffu, cell.x, l), total = __shfl_sync(0xffffffffu, cell.y, l);
        const int base = first & ~kCellRows, step = first < 0 ? 32 : 1;
        for (int k0 = 0; k0 < total; k0 += kRankRun, ++run) {
            if (run % kRankWarps != wid) continue;
            const int n = min(kRankRun, total - k0);
            for (int k = lane; k < kRankRun; k += 32) buf[k] = k < n ? ids[base + (k0 + k) * step] : 0x7fffffff;
            __syncwarp();
            for (int k = 2; k <= kRankRun; k *= 2)           // bitonic
                for (int j = k / 2; j > 0; j /= 2) {
                    for (int q = lane; q < kRankRun / 2; q += 32) {
                        const int a = 2 * q - (q & (j - 1)), va = buf[a], vb = buf[a + j];
                        if ((va > vb) == ((a & k) == 0)) {
                            buf[a] = vb;
                            buf[a + j] = va;
                        }
                    }
                    __syncwarp();
                }
            for (int k = lane; k < n; k += 32) ids[base + (k0 + k) * step] = buf[k];
            __syncwarp();
        }
    }
}

// Gives every particle its payload place (w.slot): in its cell's run by rank of
// its id, so that a cell's float sums run over its particles in id order
// whatever the order of arrival.  One CTA per layer, one lane per cell, the ids in
// shared memory, a column per cell; every warp ranks every kRankWarps-th
// particle of the cells.  (With one warp to a layer the chain of a cell's
// particles squared was the time where units are few: 34 us for 138k particles
// at 27 per cell, 11 here; sorting the columns by insertion, or skipping
// columns that arrived in order, was slower: longer chains.)  Cells of more than
// kRankRows particles are left to k_stress, where every particle counts for
// itself, reading the ids from global memory (for every cell: 956 us there against
// 715 and 85 here, 8.8M particles at 27 per cell); of more than kRankRun in runs that
// are sorted here, so that it counts by halving: 2,000 particles without a position,
// in one cell, 190 us there and 33 now, and no cell need be left in order of
// arrival.  (Runs from kRankRows on: 512k particles at 125 per cell 255 us per
// substep against 224, 885k at 216 per cell 359 against 380.)
__global__ void __launch_bounds__(32 * kRankWarps) k_rank(const WS w, long long n) {
    __shared__ int ids[kRankRows][32];
    const unsigned n_layers = min(w.ctrl->n_work, (unsigned)min(n, (long long)0x1fffffff)) * kUnitX;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    bool crowded = false;
    for (unsigned i = blockIdx.x; i < n_layers; i += gridDim.x) {
        const int2 cell = w.cells[(long long)w.work[i / kUnitX] * kUnitCells + 32 * (i % kUnitX) + lane];
        const int cnt = cell.y <= kRankRows ? cell.y : 0;
        const int *src = w.ids + (cell.x & ~kCellRows);
        const int step = cell.x < 0 ? 32 : 1;
        __syncthreads();                     // the layer before is ranked
#pragma unroll 4
        for (int k = wid; k < cnt; k += kRankWarps) ids[k][lane] = src[k * step];
        __syncthreads();
        for (int k0 = wid; k0 < cnt; k0 += 4 * kRankWarps) {   // four at a time: one read for four comparisons
            int id[4], rank[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int k = k0 + q * kRankWarps;
                id[q] = k < cnt ? ids[k][lane] : -1;
                rank[q] = 0;
            }
#pragma unroll 4
            for (int j = 0; j < cnt; ++j) {
                const int other = ids[j][lane];
#pragma unroll
                for (int q = 0; q < 4; ++q) rank[q] += other < id[q];
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (id[q] >= 0) w.slot[id[q]] = (cell.x & ~kCellRows) + rank[q] * step;
        }
        crowded |= cell.y > kRankRun;
    }
    if (!__syncthreads_or(crowded)) return;  // the columns are ranked
    for (unsigned i = blockIdx.x; i < n_layers; i += gridDim.x) {
        const int2 cell = w.cells[(long long)w.work[i / kUnitX] * kUnitCells + 32 * (i % kUnitX) + lane];
        const unsigned more = __ballot_sync(0xffffffffu, cell.y > kRankRun);   // the same in every warp
        if (more) sort_runs(w.ids, cell, more, &ids[0][0] + wid * kRankRun);
    }
}

// One thread per particle in particle order: particle BC, constitutive update,
// damage update, degradation and the APIC affine term (anisompm.py:601-713);
// the P2G payload goes to the particle's place in its cell, in id order (its
// rank among the cell's ids: the float sums of a cell then do not depend on the
// order of arrival in k_count), 4 parts of 16 bytes and one of 4:
//   {fx | x, d} {m v, m} {a00, a10, a01, a11} {a02, a12, a20, a21} {a22}, a = affine,
// with fx = X - floor(X - 0.5) per axis for particles whose stencil needs no
// clamping (base cell in [1, n_grid-4]) and the position x otherwise.
// MINB: resident CTAs per SM the registers are budgeted for (3: 80 registers;
// 4: 64 registers with a few spills), a tunable.
template <class SC, int MINB>
__global__ void __launch_bounds__(256, MINB) k_stress(const SC sc, const Parts P, const WS w) {
    // particle order: the state reads and writes are coalesced; CTAs are aligned to scenes
    const int sid = sc.of_cta(blockIdx.x);
    const long long p = sc.p_begin(sid) + ((long long)blockIdx.x - sc.cta_base(sid)) * 256 + threadIdx.x;
    if (p >= sc.p_end(sid, P.n)) return;
    const pm_params &prm = sc.params(sid);
    const long long ps = P.ps;
    const int ng = prm.n_grid;
    const float inv_dx = (float)prm.inv_dx;
    const Ctrl *ctrl = w.ctrl + sid;
    const bool do_damage = ctrl->any_allow != 0 && (ctrl->step % (long long)prm.damage_every) == 0;
    StressIn in;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        in.F[k] = P.F[k * ps + p];
        in.A0[k] = do_damage ? P.A0[k * ps + p] : 0.0f;
    }
    in.d = P.d[p];
    in.lap = P.lap[p];
    in.Dh = P.D_hist[p];
    in.mu = P.mu[p];
    in.lam = P.lam[p];
    in.sc = P.sigma_c[p];
    in.eta = P.eta[p];
    in.zeta = P.zeta[p];
    in.l0 = P.l0[p];
    in.res = P.residual[p];
    in.allow = P.allow[p] != 0;
    float tau[9];
    float d_new = in.d;
    constitutive(prm, P, p, do_damage, in, tau, d_new, w.tape_pol, w.tape_aff_stride);
    if (P.d_o != P.d) {   // out of place: every particle's d and D_hist go to the output state
        P.d_o[p] = d_new;
        if (!do_damage) P.Dho[p] = in.Dh;
    }
    float Cp[9], v[3], xp[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) xp[k] = P.x[k * ps + p];
#pragma unroll
    for (int k = 0; k < 9; ++k) Cp[k] = P.C[k * ps + p];
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = P.v[k * ps + p];
    const float vol0 = P.vol0[p], m = P.mass[p];
    float fx[3];
    bool reg = true;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const float X = __fmul_rn(xp[ax], inv_dx);
        const float fb = floorf(__fsub_rn(X, 0.5f));
        reg = reg && (fb >= 1.0f) && (fb <= (float)(ng - 4));
        fx[ax] = __fsub_rn(X, fb);                                   // in [0.5, 1.5)
    }
    long long s = w.slot[p];
    if (s < 0) {                                                     // a cell of more than kRankRows particles
        const int2 cell = w.cells[cell_of(sc, sid, xp, ng, inv_dx)];
        const int *ids = w.ids + (cell.x & ~kCellRows);
        const long long step = cell.x < 0 ? 32 : 1;
        int rank = 0;
        if (cell.y <= kRankRun) {
            for (int k = 0; k < cell.y; ++k) rank += ids[k * step] < (int)p;
        } else {                                                     // sorted runs: how many ids of each are smaller
            for (int k0 = 0; k0 < cell.y; k0 += kRankRun) {
                int lo = k0, hi = min(k0 + kRankRun, cell.y);
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (ids[mid * step] < (int)p) lo = mid + 1; else hi = mid;
                }
                rank += lo - k0;
            }
        }
        s = place_of(cell.x, rank);
        w.slot[p] = (int)s;                                          // (a recorded substep keeps it)
    }
    {                                                                // particle BCs (601-602)
        const int g = P.grip_tag ? P.grip_tag[p] : -1;
        if (g >= 0 && g < prm.n_grips) {
            const double f = prm.grips[g].ramp > 0.0 ? fmin(ctrl->time / prm.grips[g].ramp, 1.0) : 1.0;
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) v[ax] = (float)(prm.grips[g].vel[ax] * f);
        }
    }
    // stress_coeff = -dt*vol0*4*inv_dx*inv_dx; affine = coeff*tau + m*C (711-713)
    const float coeff =
        __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn((float)(-prm.dt), vol0), 4.0f), inv_dx), inv_dx);
    float aff[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) aff[k] = coeff * tau[k] + m * Cp[k];
    {
        const float4 part[4] = {reg ? make_float4(fx[0], fx[1], fx[2], d_new) : make_float4(xp[0], xp[1], xp[2], d_new),
                                make_float4(m * v[0], m * v[1], m * v[2], m), make_float4(aff[0], aff[3], aff[1], aff[4]),
                                make_float4(aff[2], aff[5], aff[6], aff[7])};
        pay_store(w.payload, s, part, aff[8]);
    }
    {   // bounds of one node contribution: |w (m v + aff dpos)| with w <= 1 and |dpos| <= 1.5 dx per axis
        const float hx = 1.5f * (float)prm.dx;
        float bm = 0.0f;
#pragma unroll
        for (int c = 0; c < 3; ++c)
            bm = fmaxf(bm, fabsf(m * v[c]) + hx * (fabsf(aff[3 * c]) + fabsf(aff[3 * c + 1]) + fabsf(aff[3 * c + 2])));
        unsigned bmom = bound_bits(bm), bmass = bound_bits(m), bdmg = bound_bits(d_new);
        Ctrl *cw = w.ctrl + sid;
        // any partition of the warp is correct here: each group raises the
        // bounds to its own maximum, in the slot of its warp
        const unsigned am = __activemask();
        const int bslot = (int)(((blockIdx.x << 3) + (threadIdx.x >> 5)) & (kBoundSlots - 1));
        bmom = __reduce_max_sync(am, bmom);
        bmass = __reduce_max_sync(am, bmass);
        bdmg = __reduce_max_sync(am, bdmg);
        if ((threadIdx.x & 31) == (unsigned)(__ffs(am) - 1)) {
            atomicMax(&cw->bound_slots[0][bslot], bmom);
            atomicMax(&cw->bound_slots[1][bslot], bmass);
            atomicMax(&cw->bound_slots[2][bslot], bdmg);
        }
    }
    if (w.tape_aff) {
#pragma unroll
        for (int k = 0; k < 9; ++k) w.tape_aff[k * w.tape_aff_stride + p] = aff[k];
    }
}

// ------------------------------------------------------------------ scatter
// Marks grid block gb (numbered over all scenes); 0 if it was unmarked.
__device__ __forceinline__ unsigned mark_block(unsigned char *mask, long long gb) {
    const unsigned bit = 1u << (8 * (int)(gb & 3));
    return atomicOr((unsigned *)(mask + (gb & ~3LL)), bit) & bit;
}
__device__ __forceinline__ void list_block(const WS &w, long long gb, unsigned slot) {
    if (slot < (unsigned long long)w.n_blocks) w.block_list[slot] = (int)gb;   // bounded even without a clock reset
}
__device__ __forceinline__ void mark_node_block(const WS &w, long long gb0, int nbs, int x, int y, int z) {
    const long long gb = gb0 + ((long long)(x >> 2) * nbs + (y >> 2)) * nbs + (z >> 2);
    if (*(volatile unsigned char *)(w.block_mask + gb) == 0 && mark_block(w.block_mask, gb) == 0)
        list_block(w, gb, atomicAdd(&w.ctrl->n_active, 1u));
}

struct NodeMark {   // of scatter_clamped
    static __device__ __forceinline__ void node(const SweepShared &sh, const WS *w, int x, int y, int z) {
        mark_node_block(*w, sh.gblock, ((int)sh.ng + kBlockEdge - 1) / kBlockEdge, x, y, z);
    }
};

// Folds a scene's bound slots of quantity v (kept for the grid update too).
__device__ __forceinline__ void fold_bounds(SweepShared &sh, const WS &w, int sid, int v, int lane) {
    unsigned m = 0;
#pragma unroll
    for (int k = 0; k < kBoundSlots / 32; ++k) m = max(m, w.ctrl[sid].bound_slots[v][k * 32 + lane]);
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) {
        sh.scale[v] = fix_scale(m).scale;
        (v == 0 ? w.ctrl[sid].mom_bound : v == 1 ? w.ctrl[sid].mass_bound : w.ctrl[sid].dmg_bound) = m;
    }
}

template <class SC>
__global__ void __launch_bounds__(kSweepThreads, 3) k_p2g_sweep(const __grid_constant__ SC sc,
                                                                const __grid_constant__ WS w, long long n) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    SweepShared &sh = *(SweepShared *)s_raw;
    int tid;   // read once: the compiler would read the special register again in every row
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
    const int lane = tid & 31, wid = __reduce_max_sync(0xffffffffu, tid >> 5);
    Ctrl *ctrl0 = w.ctrl;
    const unsigned n_units = min(ctrl0->n_work, (unsigned)min(n, (long long)0x1fffffff));
    const SweepItems items = sweep_items(n_units);
    const bool cloud = n < (long long)kCloud * n_units;
    for (int i = tid; i < kSweepQ * 4 * kQRows * kPlaneCols; i += kSweepThreads) sh.qpl[0][0][i] = 0;
    for (int i = tid; i < kSweepC * 2 * kCRows * kPlaneCols; i += kSweepThreads) sh.cpl[0][0][i] = 0;
    if (tid < 36) sh.mark[tid] = 0;
    if (tid == 0) {
        sh.scale[3] = fix_scale(__float_as_uint(1.0f)).scale;
        sh.clamped_layers = min(ctrl0->n_clamped, n_units) * kUnitX;
        sh.next = sweep_unit(gridDim.x + atomicAdd(&ctrl0->work_next, 1u), items, w.work);
    }
    int2 now = sweep_unit(blockIdx.x, items, w.work);    // the first item is the CTA's own
    int scene = -1;
    if (now.x >= 0 && wid >= (now.y & 255) && wid < now.y >> 8)
        cp_async8(&sh.raw[tid], w.cells + (long long)now.x * kUnitCells + tid);
    cp_async_commit();
    __syncthreads();
    while (now.x >= 0) {
        const int u = now.x, x0 = now.y & 255, x1 = now.y >> 8;
        const unsigned gblk = (unsigned)u / kBlockUnits;
        const int sid = sc.of_sblock(gblk);                  // sort blocks never span scenes
        const pm_params &prm = sc.params(sid);
        const int ng = prm.n_grid, nb = sort_blocks_per_axis(ng), nbs = (ng + kBlockEdge - 1) / kBlockEdge;
        const unsigned blk = gblk - sc.sblock_base(sid);
        int org[3];
        unit_origin(u, blk, nb, org);
        if (sid != scene && wid >= 4 && wid < 7) fold_bounds(sh, w, sid, wid - 4, lane);
        scene = sid;
        long long *g_mom = w.g_mom + 4 * sc.node_base(sid);
        long long *g_dmg = w.g_dmg + 2 * sc.node_base(sid);
        if (tid == kSweepThreads - 1) {
            sh.ng = ng;
            sh.dx = (float)prm.dx;
            sh.g_quad = g_mom + 4 * (((long long)org[0] * ng + org[1]) * ng + org[2]);
            sh.g_cubic = g_dmg + 2 * (((long long)(org[0] - 1) * ng + org[1] - 1) * ng + org[2] - 1);
        }
        // the unit's cells; the table goes back to zero for the next substep
        const int2 next = sh.next;
        if (wid >= x0 && wid < x1) {
            cp_async_wait<0>();
            const int2 cell = sh.raw[tid];
            const int c[3] = {tid >> 5, (tid >> 3) & 3, tid & 7}, g[3] = {org[0] + c[0], org[1] + c[1], org[2] + c[2]};
            const bool reg = !clamped_cell(g, ng);
            if (reg) w.cells[(long long)u * kUnitCells + tid] = make_int2(0, 0);   // (the others: below)
            const int cnt = reg ? cell.y : 0;
            sh.cell[tid] = make_int2(cell.x, cnt);
            sh.split[tid] = w.split[(long long)u * kUnitCells + tid];
            const int code = layer_code(cnt, cloud);
            if (lane == 0) sh.layer_rows[wid] = code;
            if (cnt > 0) {
                // the cell's stencils (quadratic nodes c..c+2, cubic c-1..c+3 per
                // axis) span grid blocks (c-1)/4 .. (c+3)/4: marked whatever the
                // sums, so that the grid update writes every node a gather reads (a
                // node whose contributions all round to zero still gets its zero
                // velocity and damage)
                const int b0 = c[0] > 0, b1 = c[1] > 0, b2 = (c[2] + 3) >> 2;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    sh.mark[((b0 + (k >> 2)) * 3 + b1 + ((k >> 1) & 1)) * 4 + b2 + (k & 1)] = 1;
            }
        } else if (tid == kUnitCells && x0 == 0) {
            w.utot[u] = 0;
        }
        __syncthreads();
        const long long gb0 = sc.gblock_base(sid);
        // the item after the next is taken, the next one's cells are on their way and the blocks are marked, while
        // this one is swept
        unsigned take = 0, was = ~0u;
        if (tid == kSweepThreads - 1) take = gridDim.x + atomicAdd(&ctrl0->work_next, 1u);
        int gb = 0;
        if (tid < 36 && sh.mark[tid]) {
            sh.mark[tid] = 0;
            const int bx = (org[0] >> 2) - 1 + tid / 12, by = (org[1] >> 2) - 1 + (tid >> 2) % 3,
                      bz = (org[2] >> 2) - 1 + (tid & 3);
            if (bx >= 0 && by >= 0 && bz >= 0 && bx < nbs && by < nbs && bz < nbs) {
                gb = (int)(gb0 + ((long long)bx * nbs + by) * nbs + bz);
                was = mark_block(w.block_mask, gb);
            }
        }
        if (next.x >= 0 && wid >= (next.y & 255) && wid < next.y >> 8)
            cp_async8(&sh.raw[tid], w.cells + (long long)next.x * kUnitCells + tid);
        cp_async_commit();
        if (wid < kSweepQ)
            sweep_warp<QuadSums<false>, kSweepQ, true>(sh, sh.qring[wid], (const char *)w.payload, wid, wid, lane, x0, x1);
        else
            sweep_warp<CubicSums, kSweepC, true>(sh, sh.cring[wid - kSweepQ], (const char *)w.payload, wid, wid - kSweepQ,
                                             lane, x0, x1);
        if (tid < 64) {                   // the blocks this item is the first to touch join the list
            const bool fresh = was == 0;
            const unsigned fb = __ballot_sync(0xffffffffu, fresh);
            unsigned at = 0;
            if (lane == 0 && fb) at = atomicAdd(&ctrl0->n_active, (unsigned)__popc(fb));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (fresh) list_block(w, gb, at + __popc(fb & lanemask_lt()));
        } else if (tid == kSweepThreads - 1) {
            sh.next = sweep_unit(take, items, w.work);
        }
        __syncthreads();                  // the item's shared state is done with
        now = next;
    }
    for (unsigned i = blockIdx.x; i < sh.clamped_layers; i += gridDim.x) {
        const int u = w.work[w.clamped[i / kUnitX]], layer = (int)(i % kUnitX);
        const unsigned gblk = (unsigned)u / kBlockUnits;
        const int sid = sc.of_sblock(gblk);
        const pm_params &prm = sc.params(sid);
        const int ng = prm.n_grid;
        int org[3];
        unit_origin(u, gblk - sc.sblock_base(sid), sort_blocks_per_axis(ng), org);
        if (sid != scene && wid >= 4 && wid < 7) fold_bounds(sh, w, sid, wid - 4, lane);
        scene = sid;
        bool any = false;
        if (tid < 32) {
            int2 *at = w.cells + (long long)u * kUnitCells + 32 * layer + tid;
            const int g[3] = {org[0] + layer, org[1] + (tid >> 3), org[2] + (tid & 7)};
            int2 cell = make_int2(0, 0);
            if (clamped_cell(g, ng)) {
                cell = *at;
                *at = make_int2(0, 0);
            }
            any = cell.y > 0;
            sh.cell[tid] = cell;
        } else if (tid == 32) {
            sh.ng = ng;
            sh.dx = (float)prm.dx;
            sh.inv_dx = (float)prm.inv_dx;
            sh.g0_quad = w.g_mom + 4 * sc.node_base(sid);
            sh.g0_cubic = w.g_dmg + 2 * sc.node_base(sid);
            sh.gblock = sc.gblock_base(sid);
        }
        if (__syncthreads_or(any)) scatter_clamped<false, NodeMark>(sh, &w, (const char *)w.payload);
        __syncthreads();
    }
}

int resident_slots(const void *kernel, int threads, size_t smem) {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem);
    return std::max(1, sms * std::max(per, 1));
}

// One-time kernel attribute set-up for the current device (not a stream
// operation, so it must not first happen inside a stream capture).
void prepare_p2g() {
    static int done[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(k_p2g_sweep<PlainScenes>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(SweepShared));
        cudaFuncSetAttribute(k_p2g_sweep<BatchScenes>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(SweepShared));
        done[dev] = 1;
    }
}

// n_ctas: 256-particle CTAs over all scenes (each scene's particles start a new
// CTA); the plain form derives it from P.n.  Persistent P2G CTAs: every
// resident slot of the device (units are taken from the list dynamically), or
// `ctas_per_sm` (1..3) per SM.
template <class SC>
void launch_p2g(const SC &sc, const Parts &P, const WS &w, cudaStream_t s, long long n_ctas, int ctas_per_sm,
                int stress_ctas) {
    if (P.n <= 0) return;
    prepare_p2g();
    const unsigned ctas = (unsigned)(n_ctas >= 0 ? n_ctas : (P.n + 255) / 256);
    k_count<SC><<<ctas, kCountThreads, 0, s>>>(sc, P.x, P.n, P.ps, P.allow, w);
    k_offsets<SC><<<(unsigned)std::min<long long>((P.n + 255) / 256, 148LL * 4), 256, 0, s>>>(sc, w, P.n);
    k_place<SC><<<ctas, 256, 0, s>>>(sc, P.x, P.n, P.ps, w);
    k_rank<<<(unsigned)std::min<long long>(P.n, 148LL * (2048 / (32 * kRankWarps))), 32 * kRankWarps, 0, s>>>(w, P.n);
    if (stress_ctas == 4)
        k_stress<SC, 4><<<ctas, 256, 0, s>>>(sc, P, w);
    else
        k_stress<SC, 3><<<ctas, 256, 0, s>>>(sc, P, w);
    static int slots_dev[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    int slots = (dev >= 0 && dev < 64) ? slots_dev[dev] : 0;
    if (slots <= 0) {
        slots = resident_slots((const void *)k_p2g_sweep<SC>, kSweepThreads, sizeof(SweepShared));
        if (dev >= 0 && dev < 64) slots_dev[dev] = slots;
    }
    if (ctas_per_sm > 0) {   // the cap
        int sms = 148;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        slots = std::min(slots, sms * ctas_per_sm);
    }
    const unsigned blocks = (unsigned)std::max<long long>(1, std::min<long long>(slots, P.n));
    k_p2g_sweep<SC><<<blocks, kSweepThreads, sizeof(SweepShared), s>>>(sc, w, P.n);
}
template void launch_p2g<PlainScenes>(const PlainScenes &, const Parts &, const WS &, cudaStream_t, long long, int, int);
template void launch_p2g<BatchScenes>(const BatchScenes &, const Parts &, const WS &, cudaStream_t, long long, int, int);

}  // namespace pm
