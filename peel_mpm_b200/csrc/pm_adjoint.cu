// Reverse-mode adjoint of one plain substep (anisompm.py:593-803) for the
// differentiable form: given the adjoints of the state after substep t
// (x', v', F', C', d', lap', D_hist'), produce the adjoints of the state
// before it and accumulate the gradients of the per-particle parameters mu,
// lam, sigma_c and A0.
//
// The forward substep t is first recorded (pm_substep_record) into a tape
// slot: grid velocity and mass {v, m}, the normalised damage field gd, the
// cubic weight sums, the active 4^3 block list and the step's clock.  The
// adjoint then runs four kernels:
//   k_adj_pre       per particle (particle order): the G2P tail adjoint and
//                   the G2P adjoint's scatter payload, written to the
//                   particle's recorded place of the forward substep,
//                   and the bounds that fix the fixed-point units;
//   k_adj_sweep     G2P adjoint as a scatter over the recorded unit list (the
//                   forward P2G's sweep): the adjoint of the grid velocity and
//                   damage field in int64 fixed point, so the sums do not
//                   depend on the atomics' order and a backward pass is
//                   reproducible bit for bit;
//   k_adj_grid      grid-update adjoint over the recorded active blocks
//                   (normalisation by mass and by the cubic weight sum);
//   k_adj_particle  P2G adjoint as a gather plus the constitutive adjoint
//                   (particle order): recomputes the particle's constitutive
//                   update, gathers the grid adjoints, and runs the polar,
//                   stress, damage and eigen-split adjoints.
// Non-smooth operations take the branch the forward took (relu, max and clamp
// pass the adjoint where the forward passed the value; base cells are
// piecewise constant).  The strain limit (f_clamp) is differentiated as a
// function of the singular values (f_clamp_adj), grid colliders from the
// recorded pre-collider grid velocity (resolve_adj), and the directional
// stress at interface particles by dir_adjoint.
#include "pm_kernels.cuh"
#include "pm_sweep.cuh"

namespace pm {

namespace {

__device__ __forceinline__ float relu_f(float v) { return v > 0.0f ? v : 0.0f; }

// Tape header of one slot.
struct TapeHead {
    unsigned n_active;
    int any_allow;
    long long step;
    double time;
    unsigned n_work;    // non-empty units of the substep
    unsigned n_clamped; // of these, the ones with cells that need clamped nodes
    float col_origin[PM_MAX_COLLIDERS][3];   // the substep's collider origins and velocities
    float col_vel[PM_MAX_COLLIDERS][3];
};

// Control block of one adjoint substep: the bounds of the scatter's
// contributions (float bits) and the dynamic work cursor.
struct AdjCtrl {
    unsigned mom_bound, lap_bound, work_next, pad;
    unsigned slots[2][kBoundSlots];   // per-warp-slot bounds, folded by k_adj_sweep
};

// Quadratic weights with their derivatives wrt the local coordinate fx.
struct QuadD {
    int b[3];
    float fx[3];
    float w[3][3], dw[3][3];
};
__device__ __forceinline__ void quad_weights_d(const float x[3], float inv_dx, int ng, QuadD &q) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float X = __fmul_rn(x[a], inv_dx);
        const float fb = floorf(__fsub_rn(X, 0.5f));
        q.b[a] = sat_base(fb, ng);
        const float f = __fsub_rn(X, fb);
        q.fx[a] = f;
        const float t0 = 1.5f - f, t1 = f - 1.0f, t2 = f - 0.5f;
        q.w[0][a] = 0.5f * (t0 * t0);
        q.w[1][a] = 0.75f - t1 * t1;
        q.w[2][a] = 0.5f * (t2 * t2);
        q.dw[0][a] = -t0;
        q.dw[1][a] = -2.0f * t1;
        q.dw[2][a] = t2;
    }
}

// Cubic weights, second derivatives and the derivatives of both wrt f.
struct CubicD {
    int b[3];
    float w[4][3], w2[4][3], dw[4][3], dw2[4][3];
};
__device__ __forceinline__ void cubic_weights_d(const float x[3], float inv_dx, int ng, CubicD &c) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float X = __fmul_rn(x[a], inv_dx);
        const float fb = floorf(X);
        c.b[a] = sat_base(fb, ng) - 1;
        const float f = __fsub_rn(X, fb);
        const float one = 1.0f - f;
        c.w[0][a] = (1.0f / 6.0f) * (one * one * one);
        c.w[1][a] = (2.0f / 3.0f - f * f) + 0.5f * (f * f * f);
        c.w[2][a] = (2.0f / 3.0f - one * one) + 0.5f * (one * one * one);
        c.w[3][a] = (1.0f / 6.0f) * (f * f * f);
        c.w2[0][a] = one;
        c.w2[1][a] = 3.0f * f - 2.0f;
        c.w2[2][a] = 1.0f - 3.0f * f;
        c.w2[3][a] = f;
        c.dw[0][a] = -0.5f * one * one;
        c.dw[1][a] = -2.0f * f + 1.5f * f * f;
        c.dw[2][a] = 2.0f * one - 1.5f * one * one;
        c.dw[3][a] = 0.5f * f * f;
        c.dw2[0][a] = -1.0f;
        c.dw2[1][a] = 3.0f;
        c.dw2[2][a] = -3.0f;
        c.dw2[3][a] = 1.0f;
    }
}

__device__ __forceinline__ int node_of(int x, int y, int z, int ng) {
    return (clampi(x, 0, ng - 1) * ng + clampi(y, 0, ng - 1)) * ng + clampi(z, 0, ng - 1);
}

struct AdjIn {
    float xb[3], vb[3], Cb[9], Fb[9], db, lapb, Dhb;
};
__device__ __forceinline__ void load_adj(const pm_state_adj &A, long long p, AdjIn &a) {
    const long long s = A.plane_stride;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        a.xb[k] = A.x[k * s + p];
        a.vb[k] = A.v[k * s + p];
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        a.Cb[k] = A.C[k * s + p];
        a.Fb[k] = A.F[k * s + p];
    }
    a.db = A.d[p];
    a.lapb = A.lap[p];
    a.Dhb = A.D_hist[p];
}

// Adjoint of the end of G2P: x' = clamp(x + dt v'), F' = (I + dt C') F.
// Returns the total adjoints of v' and C' and the pass-through mask of x.
__device__ __forceinline__ void g2p_tail_adj(const pm_params &prm, const float xp[3], const float vpost[3],
                                             const float Fpre[9], const AdjIn &a, float vt[3], float Ct[9],
                                             bool inside[3]) {
    const float dt = (float)prm.dt;
    const float pad = (float)(2.0 * prm.dx), hi = (float)(prm.grid_lim - 2.0 * prm.dx);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float t = xp[k] + dt * vpost[k];
        inside[k] = (t >= pad) && (t <= hi);
        vt[k] = a.vb[k] + (inside[k] ? dt * a.xb[k] : 0.0f);
    }
    // C' enters F' = (I + dt C') F: Cbar += dt Fbar' F^T
    float FbFt[9];
    mmt3(a.Fb, Fpre, FbFt);
#pragma unroll
    for (int k = 0; k < 9; ++k) Ct[k] = a.Cb[k] + dt * FbFt[k];
}

// The F that G2P updated: with the strain limit, the limited F rebuilt from
// the taped V and S as the forward built it.
__device__ __forceinline__ void g2p_input_F(const pm_params &prm, const float *__restrict__ tpol, long long rs,
                                            long long p, float F[9]) {
    if (!prm.use_f_clamp) return;
    float V[9], S[3];
#pragma unroll
    for (int k = 0; k < 9; ++k) V[k] = tpol[(9 + k) * rs + p];
#pragma unroll
    for (int k = 0; k < 3; ++k) S[k] = tpol[(18 + k) * rs + p];
    f_clamp_F(F, V, S, (float)prm.f_clamp_lo, (float)prm.f_clamp_hi, F);
}

// ---------------------------------------------------------------- k_adj_pre
// Adjoint of v' = sum w v_i, C' = K sum w v_i dpos^T and lap' = sum L gd_i has
// the form of a P2G scatter: node i receives w (vt + K Ct dpos) and
// lb (w''x wy wz + wx w''y wz + wx wy w''z) with lb = L lapbar.  This kernel
// forms each particle's payload {fx | x, lb}, {vt, 0}, K Ct at its recorded place.
__global__ void __launch_bounds__(256) k_adj_pre(const pm_params prm, const Parts pre, const Parts post,
                                                 const pm_state_adj ain, const int *__restrict__ iperm,
                                                 void *__restrict__ pay, AdjCtrl *actl,
                                                 const float *__restrict__ tpol, long long rs) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= pre.n) return;
    const long long ps = pre.ps;
    const int ng = prm.n_grid;
    const float inv_dx = (float)prm.inv_dx, dx = (float)prm.dx;
    const float K = (float)(4.0 * prm.inv_dx * prm.inv_dx);
    const float L2 = (float)(prm.inv_dx * prm.inv_dx);
    float xp[3], vpost[3], F[9];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        xp[k] = pre.x[k * ps + p];
        vpost[k] = post.v[k * ps + p];
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) F[k] = pre.F[k * ps + p];
    g2p_input_F(prm, tpol, rs, p, F);
    AdjIn a;
    load_adj(ain, p, a);
    float vt[3], Ct[9];
    bool inside[3];
    g2p_tail_adj(prm, xp, vpost, F, a, vt, Ct, inside);
    float kc[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) kc[k] = K * Ct[k];
    const float lb = a.lapb * L2;
    float fx[3];
    bool reg = true;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const float X = __fmul_rn(xp[ax], inv_dx);
        const float fb = floorf(__fsub_rn(X, 0.5f));
        reg = reg && (fb >= 1.0f) && (fb <= (float)(ng - 4));
        fx[ax] = __fsub_rn(X, fb);
    }
    {
        const float4 part[4] = {reg ? make_float4(fx[0], fx[1], fx[2], lb) : make_float4(xp[0], xp[1], xp[2], lb),
                                make_float4(vt[0], vt[1], vt[2], 0.0f), make_float4(kc[0], kc[3], kc[1], kc[4]),
                                make_float4(kc[2], kc[5], kc[6], kc[7])};
        pay_store(pay, iperm[p], part, kc[8]);
    }
    // bounds of one node contribution: |w (vt + K Ct dpos)| with w <= 1,
    // |dpos| <= 1.5 dx per axis (the cubic stencil's quadratic part), and
    // |lb W''| with |w''x wy wz + wx w''y wz + wx wy w''z| <= 3 (|w''| <= 2, w <= 2/3)
    const float hx = 1.5f * dx;
    float bm = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c)
        bm = fmaxf(bm, fabsf(vt[c]) + hx * (fabsf(kc[3 * c]) + fabsf(kc[3 * c + 1]) + fabsf(kc[3 * c + 2])));
    unsigned bmom = bound_bits(bm), blap = bound_bits(3.0f * lb);
    const unsigned am = __activemask();
    bmom = __reduce_max_sync(am, bmom);
    blap = __reduce_max_sync(am, blap);
    if ((threadIdx.x & 31) == (unsigned)(__ffs(am) - 1)) {
        const int slot = (int)(((blockIdx.x << 3) + (threadIdx.x >> 5)) & (kBoundSlots - 1));
        atomicMax(&actl->slots[0][slot], bmom);
        atomicMax(&actl->slots[1][slot], blap);
    }
}

// ---------------------------------------------------------------- k_adj_sweep
struct NoMark {
    static __device__ __forceinline__ void node(const SweepShared &, const WS *, int, int, int) {}
};
// The G2P adjoint scatter over the forward substep's non-empty units, with the
// forward P2G's sweep (pm_sweep.cuh): quadratic planes sum w (vt + K Ct dpos)
// into the momentum adjoint, cubic planes lb W'' into the damage adjoint, int64
// fixed point.  The adjoint touches exactly the nodes the forward P2G touched,
// so no block marks are needed.
__global__ void __launch_bounds__(kSweepThreads, 3) k_adj_sweep(const __grid_constant__ pm_params prm,
                                                                const int *__restrict__ work,
                                                                const int *__restrict__ clamped,
                                                                const int2 *__restrict__ cells,
                                                                const unsigned char *__restrict__ split,
                                                                const TapeHead *head,
                                                                void *pay, AdjCtrl *actl, long long *__restrict__ acc,
                                                                long long n) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    SweepShared &sh = *(SweepShared *)s_raw;
    int tid;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
    const int lane = tid & 31, wid = __reduce_max_sync(0xffffffffu, tid >> 5);
    const unsigned n_units = min(head->n_work, (unsigned)min(n, (long long)0x1fffffff));
    const SweepItems items = sweep_items(n_units);
    const int ng = prm.n_grid, nb = sort_blocks_per_axis(ng);
    for (int i = tid; i < kSweepQ * 4 * kQRows * kPlaneCols; i += kSweepThreads) sh.qpl[0][0][i] = 0;
    for (int i = tid; i < kSweepC * 2 * kCRows * kPlaneCols; i += kSweepThreads) sh.cpl[0][0][i] = 0;
    if (tid == 0) sh.clamped_layers = min(head->n_clamped, n_units) * kUnitX;
    if (wid >= 4 && wid < 6) {            // fold the bound slots (kept for the grid adjoint too)
        unsigned m = 0;
#pragma unroll
        for (int k = 0; k < kBoundSlots / 32; ++k) m = max(m, actl->slots[wid - 4][k * 32 + lane]);
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) {
            sh.scale[2 * (wid - 4)] = fix_scale(m).scale;
            if (wid == 4) actl->mom_bound = m;
            else actl->lap_bound = m;
        }
    }
    __syncthreads();
    int2 now = sweep_item(blockIdx.x, items);   // the first item is the CTA's own
    while (now.x >= 0) {
        const int i = now.x, u = work[i], x0 = now.y & 255, x1 = now.y >> 8;
        const unsigned blk = (unsigned)u / kBlockUnits;
        int org[3];
        unit_origin(u, blk, nb, org);
        if (wid >= x0 && wid < x1) {
            const int2 cell = cells[(long long)i * kUnitCells + tid];
            const int g[3] = {org[0] + (tid >> 5), org[1] + ((tid >> 3) & 3), org[2] + (tid & 7)};
            const int cnt = clamped_cell(g, ng) ? 0 : cell.y;
            sh.cell[tid] = make_int2(cell.x, cnt);
            sh.split[tid] = split[(long long)i * kUnitCells + tid];
            const int code = layer_code(cnt, false);
            if (lane == 0) sh.layer_rows[wid] = code;
        }
        if (tid == kSweepThreads - 1) {
            sh.ng = ng;
            sh.dx = (float)prm.dx;
            sh.g_quad = acc + 4 * (((long long)org[0] * ng + org[1]) * ng + org[2]);
            sh.g_cubic = acc + 4 * (((long long)(org[0] - 1) * ng + org[1] - 1) * ng + org[2] - 1) + 3;
        }
        __syncthreads();
        unsigned take = 0;                // the next item is taken while this one is swept
        if (tid == kSweepThreads - 1) take = gridDim.x + atomicAdd(&actl->work_next, 1u);
        if (wid < kSweepQ)
            sweep_warp<QuadSums<true>, kSweepQ, false>(sh, sh.qring[wid], (const char *)pay, wid, wid, lane, x0, x1);
        else
            sweep_warp<CubicLapSums, kSweepC, false>(sh, sh.cring[wid - kSweepQ], (const char *)pay, wid, wid - kSweepQ, lane, x0,
                                             x1);
        if (tid == kSweepThreads - 1) sh.next = sweep_item(take, items);
        __syncthreads();
        now = sh.next;
    }
    for (unsigned j = blockIdx.x; j < sh.clamped_layers; j += gridDim.x) {
        const int i = clamped[j / kUnitX], u = work[i], layer = (int)(j % kUnitX);
        int org[3];
        unit_origin(u, (unsigned)u / kBlockUnits, nb, org);
        bool any = false;
        if (tid < 32) {
            const int g[3] = {org[0] + layer, org[1] + (tid >> 3), org[2] + (tid & 7)};
            int2 cell = make_int2(0, 0);
            if (clamped_cell(g, ng)) cell = cells[(long long)i * kUnitCells + 32 * layer + tid];
            any = cell.y > 0;
            sh.cell[tid] = cell;
        } else if (tid == 32) {
            sh.ng = ng;
            sh.dx = (float)prm.dx;
            sh.inv_dx = (float)prm.inv_dx;
            sh.g0_quad = acc;
            sh.g0_cubic = acc + 3;
        }
        if (__syncthreads_or(any)) scatter_clamped<true, NoMark>(sh, nullptr, (const char *)pay);
        __syncthreads();
    }
}

// Adjoint of resolve() (the reference's _resolve, anisompm.py:811-825) at
// input velocity v: vb holds the adjoint of the output on entry and of the
// input on return.  Sticky: the output is the collider velocity, a constant.
// Slip: torch's subgradient conventions, clamp passing where its input lies
// inside the bounds inclusive (vn <= 0 for the inward part, scale >= 0 for
// the friction factor) and the norm passing nothing at zero.
__device__ __forceinline__ void resolve_adj(const float v[3], const float vc[3], const float nn[3], bool sticky,
                                            float fr, float vb[3]) {
    if (sticky) {
        vb[0] = vb[1] = vb[2] = 0.0f;
        return;
    }
    const float r[3] = {v[0] - vc[0], v[1] - vc[1], v[2] - vc[2]};
    const float vn = r[0] * nn[0] + r[1] * nn[1] + r[2] * nn[2];
    const float inward = vn < 0.0f ? vn : 0.0f;
    const float t[3] = {r[0] - vn * nn[0], r[1] - vn * nn[1], r[2] - vn * nn[2]};
    const float keepb = vb[0] * nn[0] + vb[1] * nn[1] + vb[2] * nn[2];
    float tb[3] = {vb[0], vb[1], vb[2]};
    float inwardb = -keepb;
    if (fr > 0.0f) {
        const float vtm = sqrtf(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]);
        const float den = vtm + 1e-9f;
        const float sraw = 1.0f + fr * inward / den;
        const float sc = sraw < 0.0f ? 0.0f : sraw;
        const float scb = tb[0] * t[0] + tb[1] * t[1] + tb[2] * t[2];
#pragma unroll
        for (int a = 0; a < 3; ++a) tb[a] *= sc;
        if (sraw >= 0.0f) {
            inwardb += scb * fr / den;
            const float vtmb = -scb * fr * inward / (den * den);
            if (vtm > 0.0f) {
#pragma unroll
                for (int a = 0; a < 3; ++a) tb[a] += vtmb * t[a] / vtm;
            }
        }
    }
    float vnb = keepb - (tb[0] * nn[0] + tb[1] * nn[1] + tb[2] * nn[2]);
    if (vn <= 0.0f) vnb += inwardb;
#pragma unroll
    for (int a = 0; a < 3; ++a) vb[a] = tb[a] + vnb * nn[a];
}

// ---------------------------------------------------------------- k_adj_grid
// Grid-update adjoint over the recorded active blocks.  Forward (active node,
// m > 1e-12): v = (mv / m + dt g) * damp; gd = sum wd / sum w when sum w >
// 1e-12.  Writes A = {mvbar, mbar}, B = {sumwd bar, sumw bar, gd, 0} and
// clears acc.
__global__ void __launch_bounds__(256) k_adj_grid(const pm_params prm, const int *__restrict__ blocks,
                                                  const TapeHead *head, const float4 *__restrict__ gvel,
                                                  const float4 *__restrict__ vpre,
                                                  const float *__restrict__ ggd, const float *__restrict__ gsw,
                                                  long long *__restrict__ acc, const AdjCtrl *actl,
                                                  float4 *__restrict__ A, float4 *__restrict__ B,
                                                  long long n_blocks) {
    const float umom = fix_scale(actl->mom_bound).unit, ulap = fix_scale(actl->lap_bound).unit;
    const long long nact = min((long long)head->n_active, n_blocks);
    const long long items = nact * 64;
    const int ng = prm.n_grid, nbs = (ng + kBlockEdge - 1) / kBlockEdge;
    const float dt = (float)prm.dt, damp = (float)prm.grid_damp, dx = (float)prm.dx;
    const float dg[3] = {damp * dt * (float)prm.gravity[0], damp * dt * (float)prm.gravity[1],
                         damp * dt * (float)prm.gravity[2]};
    for (long long it = (long long)blockIdx.x * blockDim.x + threadIdx.x; it < items;
         it += (long long)gridDim.x * blockDim.x) {
        const int b = blocks[it >> 6];
        const int l = (int)(it & 63);
        const int bx = b / (nbs * nbs), by = (b / nbs) % nbs, bz = b % nbs;
        const int ix = bx * kBlockEdge + (l >> 4), iy = by * kBlockEdge + ((l >> 2) & 3), iz = bz * kBlockEdge + (l & 3);
        if (ix >= ng || iy >= ng || iz >= ng) continue;
        const long long node = ((long long)ix * ng + iy) * ng + iz;
        longlong2 *an = (longlong2 *)(acc + 4 * node);
        const longlong2 a01 = an[0], a23 = an[1];
        an[0] = make_longlong2(0, 0);
        an[1] = make_longlong2(0, 0);
        const float4 ab = make_float4(from_fix(a01.x, umom), from_fix(a01.y, umom), from_fix(a23.x, umom),
                                      from_fix(a23.y, ulap));
        float4 gv = gvel[node];
        float4 ao = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (gv.w > 1e-12f) {
            float vb[3] = {ab.x, ab.y, ab.z};
            if (vpre && prm.n_colliders > 0) {
                // colliders (anisompm.py:737-746): rerun them from the recorded
                // pre-collider velocity, keeping each one's input, then walk
                // them back
                const float4 vp = vpre[node];
                const float pos[3] = {(float)ix * dx, (float)iy * dx, (float)iz * dx};
                float vs[PM_MAX_COLLIDERS][3], nrm[PM_MAX_COLLIDERS][3];
                unsigned hit = 0u;
                float v[3] = {vp.x, vp.y, vp.z};
                for (int c = 0; c < prm.n_colliders; ++c) {
                    vs[c][0] = v[0]; vs[c][1] = v[1]; vs[c][2] = v[2];
                    if (collider_hit(prm.colliders[c], head->col_origin[c], pos, nrm[c])) {
                        hit |= 1u << c;
                        resolve(v, head->col_vel[c], nrm[c], prm.colliders[c].mode == 1,
                                (float)prm.colliders[c].friction);
                    }
                }
                for (int c = prm.n_colliders - 1; c >= 0; --c)
                    if (hit & (1u << c))
                        resolve_adj(vs[c], head->col_vel[c], nrm[c], prm.colliders[c].mode == 1,
                                    (float)prm.colliders[c].friction, vb);
                gv.x = vp.x; gv.y = vp.y; gv.z = vp.z;   // the velocity the mass and momentum made
            }
            const float im = 1.0f / gv.w;
            const float u0 = damp * vb[0], u1 = damp * vb[1], u2 = damp * vb[2];
            ao.x = u0 * im; ao.y = u1 * im; ao.z = u2 * im;
            // mv / m = v / damp - dt g:  mbar = -damp vbar . (mv/m) / m
            ao.w = -(vb[0] * (gv.x - dg[0]) + vb[1] * (gv.y - dg[1]) + vb[2] * (gv.z - dg[2])) * im;
        }
        A[node] = ao;
        const float sw = gsw[node], gd = ggd[node];
        float4 bo = make_float4(0.0f, 0.0f, gd, 0.0f);
        if (sw > 1e-12f) {
            bo.x = ab.w / sw;
            bo.y = -ab.w * gd / sw;
        }
        B[node] = bo;
    }
}

// ---------------------------------------------------------------- constitutive
// What the adjoint keeps of the forward constitutive update.  The damage
// driving geometry (Cauchy stress eigensystem, sigma+, A, M) is not kept: it
// is needed only where the history drive is active, and is recomputed there.
struct Cons {
    float F[9], V[9], S[3], Sc[3], R[9], lamC[3];   // F: after the strain limit; S before it, Sc after
    bool fclamp, iface;
    float n0[3];   // interface normal (iface)
    float J, Jraw, tdev[9], tv;
    bool dmg;
    float phi, drive, Dh0, Dh1, d0, lap, arg, cc, u, dn, d1, g, vdeg, res, sc, zeta, l0;
    bool allow;
};

// Damage driving geometry (anisompm.py:650-664): sig = sym(tdev + tv I) / J,
// its eigensystem, sigma+ = Q relu(e) Q^T, A = R A0 R^T, M = A sigma+ and
// phi = tr(M M) / sigma_c^2.
struct DamageGeom {
    float sig[9], ev[3], Q[9], sp[9], A[9], M[9], A0[9];
    float phi;
};
__device__ __forceinline__ void damage_geom(const float R[9], const float V[9], const float S[3], const float tdev[9],
                                            float tv, float J, float sc, const Parts &P, long long p,
                                            DamageGeom &g) {
    const long long ps = P.ps;
    float sg[9];
    const float rJ = 1.0f / J;   // as the forward computes it
#pragma unroll
    for (int k = 0; k < 9; ++k) sg[k] = (tdev[k] + ((k % 4 == 0) ? tv : 0.0f)) * rJ;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) g.sig[3 * i + j] = 0.5f * (sg[3 * i + j] + sg[3 * j + i]);
    {   // eigensystem as the forward took it: U = R V from the taped polar decomposition
        float U[9];
        mm3(R, V, U);
        if (polar_u_ok(S))
            stress_eig_polar(U, g.sig, g.ev, g.Q);
        else
            sym_eig3<5>(g.sig, g.ev, g.Q);
    }
    {
        float ED[9];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const float e = g.ev[j] < 0.0f ? 0.0f : g.ev[j];
#pragma unroll
            for (int i = 0; i < 3; ++i) ED[3 * i + j] = g.Q[3 * i + j] * e;
        }
        mmt3(ED, g.Q, g.sp);
    }
    {
        float RA[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) g.A0[k] = P.A0[k * ps + p];
        mm3(R, g.A0, RA);
        mmt3(RA, R, g.A);
    }
    mm3(g.A, g.sp, g.M);
    const float trMM = (g.M[0] * g.M[0] + g.M[1] * g.M[3] + g.M[2] * g.M[6]) +
                       (g.M[3] * g.M[1] + g.M[4] * g.M[4] + g.M[5] * g.M[7]) +
                       (g.M[6] * g.M[2] + g.M[7] * g.M[5] + g.M[8] * g.M[8]);
    g.phi = trMM / (sc * sc);
}


// Forward constitutive update without interface particles, as the forward
// kernel computes it (the strain limit included), keeping the intermediates.  The polar
// decomposition (R, V, S) and, on damage steps, phi come from the tape that
// the recorded forward wrote (pol[k * rs + p]: R 0..8, V 9..17, S 18..20,
// phi 21), so neither eigensolve is repeated here.
// EXT: the strain limit and interface particles are compiled in (a kernel
// without them keeps fewer registers live).
template <bool EXT>
__device__ __forceinline__ void cons_forward(const pm_params &prm, const Parts &P, long long p, bool do_damage,
                                             Cons &c, float tau[9], const float *__restrict__ pol, long long rs) {
    const long long ps = P.ps;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        c.F[k] = P.F[k * ps + p];
        c.R[k] = pol[k * rs + p];
        c.V[k] = pol[(9 + k) * rs + p];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        c.S[i] = pol[(18 + i) * rs + p];
        c.lamC[i] = c.S[i] > sqrtf(1e-12f) ? 1.0f : 0.0f;   // 0 where S = sqrt(max(lamC, 1e-12)) clamped
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) c.Sc[i] = c.S[i];
    c.fclamp = EXT && prm.use_f_clamp != 0;
    if (c.fclamp) f_clamp_F(c.F, c.V, c.Sc, (float)prm.f_clamp_lo, (float)prm.f_clamp_hi, c.F);
    c.Jraw = c.Sc[0] * c.Sc[1] * c.Sc[2];
    c.J = c.Jraw < 1e-6f ? 1e-6f : c.Jraw;
    const float mu = P.mu[p], lam = P.lam[p];
    {
        float FmR[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) FmR[k] = (2.0f * mu) * (c.F[k] - c.R[k]);
        mmt3(FmR, c.F, c.tdev);
    }
    c.tv = lam * (c.J - 1.0f) * c.J;
    c.dmg = do_damage;
    c.d0 = P.d[p];
    c.Dh0 = P.D_hist[p];
    c.d1 = c.d0;
    c.Dh1 = c.Dh0;
    c.allow = P.allow[p] != 0;
    if (do_damage) {
        c.sc = P.sigma_c[p];
        c.phi = pol[21 * rs + p];
        c.zeta = P.zeta[p];
        c.drive = c.zeta * relu_f(c.phi - 1.0f);
        c.Dh1 = c.drive > c.Dh0 ? c.drive : c.Dh0;
        c.l0 = P.l0[p];
        c.lap = P.lap[p];
        const float resist = c.d0 - (c.l0 * c.l0) * c.lap;
        c.arg = (1.0f - c.d0) * c.Dh1 - resist;
        const float ddot = relu_f(c.arg);
        const float dt_dmg = (float)(prm.dt * (double)prm.damage_every);
        c.cc = dt_dmg / P.eta[p];
        c.u = c.d0 + c.cc * ddot;
        c.dn = c.u < 0.0f ? 0.0f : (c.u > 1.0f ? 1.0f : c.u);
        if (c.allow) c.d1 = c.dn > c.d0 ? c.dn : c.d0;
    }
    c.res = P.residual[p];
    const float omd = 1.0f - c.d1;
    c.g = (omd * omd) * (1.0f - c.res) + c.res;
    c.vdeg = (c.J >= 1.0f) ? c.g : 1.0f;
#pragma unroll
    for (int k = 0; k < 9; ++k) tau[k] = c.g * c.tdev[k] + ((k % 4 == 0) ? c.vdeg * c.tv : 0.0f);
    c.iface = EXT && P.interface_mask && P.interface_mask[p];
    if (c.iface) {
        c.n0[0] = P.n_interface[p];
        c.n0[1] = P.n_interface[ps + p];
        c.n0[2] = P.n_interface[2 * ps + p];
    }
}

// Adjoint of the directional (delamination) stress at an interface particle
// (directional_kirchhoff, anisompm.py:190-227 via 697-703): tau = Q tc Q +
// gI P tc P + g (P tc Q + Q tc P) with tc = tdev + tv I, P = m m^T, Q = I - P,
// m = F n0 / (|F n0| + 1e-9) and gI = g where m^T tc m > 0, else 1.  Given
// taub: the adjoints of g (gb), tdev, tv and the direct part of F (Fb, added).
__device__ __forceinline__ void dir_adjoint(const Cons &c, const float taub[9], float &gb, float tdevb[9],
                                            float &tvb, float Fb[9]) {
    float tc[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) tc[k] = c.tdev[k] + ((k % 4 == 0) ? c.tv : 0.0f);
    float u[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) u[i] = c.F[3 * i] * c.n0[0] + c.F[3 * i + 1] * c.n0[1] + c.F[3 * i + 2] * c.n0[2];
    const float un = sqrtf(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
    const float mn = un + 1e-9f;
    const float m[3] = {u[0] / mn, u[1] / mn, u[2] / mn};
    float Pm[9], Qm[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            Pm[3 * i + j] = m[i] * m[j];
            Qm[3 * i + j] = ((i == j) ? 1.0f : 0.0f) - Pm[3 * i + j];
        }
    float snn = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) snn += m[i] * tc[3 * i + j] * m[j];
    const bool tens = snn > 0.0f;
    const float gI = tens ? c.g : 1.0f;
    // pieces of the forward, for the adjoint of g
    float T1[9], perp[9], shs[9], X[9];
    mm3(Pm, tc, T1);                        // P tc
    mm3(T1, Pm, perp);                      // P tc P
    mm3(T1, Qm, shs);                       // P tc Q
    mm3(Qm, tc, T1);                        // Q tc
    mm3(T1, Pm, X);                         // Q tc P
    gb = 0.0f;
#pragma unroll
    for (int k = 0; k < 9; ++k) gb += taub[k] * (shs[k] + X[k] + (tens ? perp[k] : 0.0f));
    // tcb = Q taub Q + gI P taub P + g (P taub Q + Q taub P)
    float PT[9], QT[9], A1[9], A2[9], A3[9], A4[9];
    mm3(Pm, taub, PT);
    mm3(Qm, taub, QT);
    mm3(QT, Qm, A1);
    mm3(PT, Pm, A2);
    mm3(PT, Qm, A3);
    mm3(QT, Pm, A4);
    float trc = 0.0f;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const float tcb = A1[k] + gI * A2[k] + c.g * (A3[k] + A4[k]);
        tdevb[k] = tcb;
        if (k % 4 == 0) trc += tcb;
    }
    tvb = trc;
    // Pbar, Qbar from the four products (P, Q symmetric; Xbar of each piece:
    // par taub, perp gI taub, both shears g taub)
    float Pb[9], Qb[9];
    {
        float tcP[9], tcQ[9], tcT[9];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) tcT[3 * i + j] = tc[3 * j + i];
        mm3(tcT, Pm, tcP);                  // tc^T P
        mm3(tcT, Qm, tcQ);                  // tc^T Q
        float PtcT[9], QtcT[9];
        mm3(Pm, tcT, PtcT);                 // P tc^T
        mm3(Qm, tcT, QtcT);                 // Q tc^T
        float B1[9], B2[9], B3[9], B4[9], B5[9], B6[9], B7[9], B8[9];
        mm3(taub, PtcT, B1);                // perp: Xb P tc^T
        mm3(tcP, taub, B2);                 //       tc^T P Xb
        mm3(taub, QtcT, B3);                // sh1 = P tc Q: Pb += Xb Q tc^T
        mm3(tcP, taub, B4);                 //               Qb += tc^T P Xb
        mm3(taub, PtcT, B5);                // sh2 = Q tc P: Qb += Xb P tc^T
        mm3(tcQ, taub, B6);                 //               Pb += tc^T Q Xb
        mm3(taub, QtcT, B7);                // par = Q tc Q: Qb += Xb Q tc^T
        mm3(tcQ, taub, B8);                 //               Qb += tc^T Q Xb
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            Pb[k] = gI * (B1[k] + B2[k]) + c.g * (B3[k] + B6[k]);
            Qb[k] = c.g * (B4[k] + B5[k]) + B7[k] + B8[k];
        }
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) Pb[k] -= Qb[k];   // Q = I - P
    float mb[3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
        mb[i] = (Pb[3 * i] + Pb[i]) * m[0] + (Pb[3 * i + 1] + Pb[3 + i]) * m[1] + (Pb[3 * i + 2] + Pb[6 + i]) * m[2];
    const float mbu = mb[0] * u[0] + mb[1] * u[1] + mb[2] * u[2];
    const float cu = un > 0.0f ? mbu / (un * mn * mn) : 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float ub = mb[i] / mn - cu * u[i];
#pragma unroll
        for (int j = 0; j < 3; ++j) Fb[3 * i + j] += ub * c.n0[j];
    }
}

// Adjoint of the eigen split sp = Q diag(relu(e)) Q^T of the symmetric sig:
// sigbar = Q (Gam o (Q^T sym(spbar) Q)) Q^T with Gam_ii = [e_i > 0] and
// Gam_ij = (relu(e_i) - relu(e_j)) / (e_i - e_j), guarded for near-equal
// eigenvalues by the mean of the diagonal terms (Daleckii-Krein formula for
// the isotropic matrix function relu).
__device__ __forceinline__ void eigsplit_adj(const float ev[3], const float Q[9], const float spb[9], float sgb[9]) {
    float Sy[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) Sy[3 * i + j] = 0.5f * (spb[3 * i + j] + spb[3 * j + i]);
    float T[9], Bq[9];
    mm3(Sy, Q, T);                       // Sy Q
    // Bq = Q^T (Sy Q)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) Bq[3 * i + j] = Q[i] * T[j] + Q[3 + i] * T[3 + j] + Q[6 + i] * T[6 + j];
    float gd[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) gd[i] = ev[i] >= 0.0f ? 1.0f : 0.0f;   // clamp(min=0) passes at 0
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            float gm;
            if (i == j) {
                gm = gd[i];
            } else {
                const float de = ev[i] - ev[j];
                const float scale = fabsf(ev[i]) + fabsf(ev[j]);
                if (fabsf(de) > 1e-6f * scale && fabsf(de) > 1e-30f)
                    gm = (relu_f(ev[i]) - relu_f(ev[j])) / de;
                else
                    gm = 0.5f * (gd[i] + gd[j]);
            }
            Bq[3 * i + j] *= gm;
        }
    // sgb = Q Bq Q^T
    mm3(Q, Bq, T);
    mmt3(T, Q, sgb);
}

// Fb: the adjoint of the pre-substep F; with the strain limit, the adjoint
// of the limited F (direct terms only) and, apart, the polar rotation's
// contribution to the pre-substep F (Fp) and the adjoint of the limited
// singular values (Scb), which f_clamp_adj combines.
struct ConsAdj {
    float Fb[9], Fp[9], Scb[3], mub, lamb, scb, A0b[9], d0b, lapb, Dh0b;
};

// Reverse of cons_forward given taubar, the adjoint of the updated damage d1
// and of the updated history D_hist1.
__device__ __forceinline__ void cons_adjoint(const Cons &c, const float mu, const float lam, const float taub[9],
                                             float d1b, float Dh1b, const Parts &P, long long p, ConsAdj &o) {
    float gb = 0.0f, tdevb[9], tvb, Fbd[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) Fbd[k] = 0.0f;
    if (c.iface) {
        dir_adjoint(c, taub, gb, tdevb, tvb, Fbd);
    } else {   // tau = g tdev + vdeg tv I
        const float trt = taub[0] + taub[4] + taub[8];
#pragma unroll
        for (int k = 0; k < 9; ++k) gb += taub[k] * c.tdev[k];
        if (c.J >= 1.0f) gb += c.tv * trt;
#pragma unroll
        for (int k = 0; k < 9; ++k) tdevb[k] = c.g * taub[k];
        tvb = c.vdeg * trt;
    }
    d1b += gb * (-2.0f * (1.0f - c.d1) * (1.0f - c.res));
    float Jb = 0.0f, Rb[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        Rb[k] = 0.0f;
        o.A0b[k] = 0.0f;
    }
    o.d0b = 0.0f;
    o.lapb = 0.0f;
    o.Dh0b = 0.0f;
    o.scb = 0.0f;
    if (c.dmg) {
        // torch.maximum sends half of the adjoint to each operand on a tie;
        // clamp passes it on [lo, hi] inclusive; relu only where the input > 0
        float dnb = 0.0f;
        if (!c.allow || c.dn < c.d0) {
            o.d0b += d1b;
        } else if (c.dn > c.d0) {
            dnb = d1b;
        } else {
            dnb = 0.5f * d1b;
            o.d0b += 0.5f * d1b;
        }
        float ddotb = 0.0f;
        if (c.u >= 0.0f && c.u <= 1.0f) {
            o.d0b += dnb;
            ddotb = c.cc * dnb;
        }
        float Dh1t = Dh1b;
        if (c.arg > 0.0f) {
            Dh1t += (1.0f - c.d0) * ddotb;
            o.d0b += -(c.Dh1 + 1.0f) * ddotb;
            o.lapb += (c.l0 * c.l0) * ddotb;
        }
        float driveb = 0.0f;
        if (c.drive > c.Dh0) {
            driveb = Dh1t;
        } else if (c.drive < c.Dh0) {
            o.Dh0b += Dh1t;
        } else {
            driveb = 0.5f * Dh1t;
            o.Dh0b += 0.5f * Dh1t;
        }
        const float phib = (c.phi > 1.0f) ? c.zeta * driveb : 0.0f;
        if (phib != 0.0f) {
            DamageGeom dg;
            damage_geom(c.R, c.V, c.S, c.tdev, c.tv, c.J, c.sc, P, p, dg);
            const float isc2 = 1.0f / (c.sc * c.sc);
            o.scb += -2.0f * c.phi / c.sc * phib;
            float Mb[9];
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) Mb[3 * i + j] = 2.0f * phib * isc2 * dg.M[3 * j + i];
            float Ab[9], spb[9];
            mmt3(Mb, dg.sp, Ab);                    // Mb sp^T
            // spb = A^T Mb
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    spb[3 * i + j] = dg.A[i] * Mb[j] + dg.A[3 + i] * Mb[3 + j] + dg.A[6 + i] * Mb[6 + j];
            // A = R A0 R^T:  Rb += Ab R A0^T + Ab^T R A0;  A0b += R^T Ab R
            {
                float T1[9], T2[9], RA0t[9], RA0[9];
                mmt3(c.R, dg.A0, RA0t);             // R A0^T
                mm3(c.R, dg.A0, RA0);               // R A0
                mm3(Ab, RA0t, T1);
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j)
                        T2[3 * i + j] = Ab[i] * RA0[j] + Ab[3 + i] * RA0[3 + j] + Ab[6 + i] * RA0[6 + j];   // Ab^T RA0
#pragma unroll
                for (int k = 0; k < 9; ++k) Rb[k] += T1[k] + T2[k];
                float AbR[9];
                mm3(Ab, c.R, AbR);
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j)
                        o.A0b[3 * i + j] = c.R[i] * AbR[j] + c.R[3 + i] * AbR[3 + j] + c.R[6 + i] * AbR[6 + j];
            }
            float sgb[9];
            eigsplit_adj(dg.ev, dg.Q, spb, sgb);
            // sig = sym(tdev + tv I) / J
            const float iJ = 1.0f / c.J;
            float dots = 0.0f;
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                tdevb[k] += sgb[k] * iJ;
                dots += sgb[k] * dg.sig[k];
            }
            tvb += (sgb[0] + sgb[4] + sgb[8]) * iJ;
            Jb += -dots * iJ;
        }
    } else {
        o.d0b += d1b;
        o.Dh0b += Dh1b;
    }
    // tv = lam (J - 1) J
    o.lamb = tvb * (c.J - 1.0f) * c.J;
    Jb += tvb * lam * (2.0f * c.J - 1.0f);
    // tdev = 2 mu (F - R) F^T
    float FmR[9], FmRFt[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) FmR[k] = c.F[k] - c.R[k];
    mmt3(FmR, c.F, FmRFt);
    float mub = 0.0f;
#pragma unroll
    for (int k = 0; k < 9; ++k) mub += tdevb[k] * FmRFt[k];
    o.mub = 2.0f * mub;
    float TF[9], TtFmR[9];
    mm3(tdevb, c.F, TF);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            TtFmR[3 * i + j] = tdevb[i] * FmR[j] + tdevb[3 + i] * FmR[3 + j] + tdevb[6 + i] * FmR[6 + j];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        o.Fb[k] = (2.0f * mu) * (TF[k] + TtFmR[k]) + Fbd[k];
        Rb[k] += -(2.0f * mu) * TF[k];
    }
    // J = max(S0 S1 S2, 1e-6); S = sqrt(max(lamC, 1e-12))
    float Sb[3] = {0.0f, 0.0f, 0.0f};
    if (c.Jraw > 1e-6f) {
        Sb[0] = Jb * c.Sc[1] * c.Sc[2];
        Sb[1] = Jb * c.Sc[0] * c.Sc[2];
        Sb[2] = Jb * c.Sc[0] * c.Sc[1];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        if (c.lamC[i] == 0.0f) Sb[i] = 0.0f;
        o.Scb[i] = Sb[i];
        if (c.fclamp) Sb[i] = 0.0f;   // through the limited values: f_clamp_adj
    }
    // polar F = R U: Fbar += R V (G + diag(Sbar)) V^T with
    // G_ij = (B_ij - B_ji) / (S_i + S_j), B = V^T R^T Rbar V
    float RtRb[9], T[9], Bm[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            RtRb[3 * i + j] = c.R[i] * Rb[j] + c.R[3 + i] * Rb[3 + j] + c.R[6 + i] * Rb[6 + j];
    mm3(RtRb, c.V, T);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) Bm[3 * i + j] = c.V[i] * T[j] + c.V[3 + i] * T[3 + j] + c.V[6 + i] * T[6 + j];
    float G[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            if (i == j) {
                G[3 * i + j] = Sb[i];
            } else {
                float den = c.S[i] + c.S[j];
                den = den < 1e-6f ? 1e-6f : den;
                G[3 * i + j] = (Bm[3 * i + j] - Bm[3 * j + i]) / den;
            }
        }
    float RV[9], RVG[9], Fp[9];
    mm3(c.R, c.V, RV);
    mm3(RV, G, RVG);
    mmt3(RVG, c.V, Fp);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        o.Fp[k] = Fp[k];
        if (!c.fclamp) o.Fb[k] += Fp[k];
    }
}

// Adjoint of the strain limit F -> Fc = U g(S) V^T (anisompm.py:622-636 with
// U = R V, S the singular values before the limit, g = clamp(., lo, hi)),
// given Fcb (the adjoint of Fc) and Scb (of g(S)): returns U G V^T with
// X = U^T Fcb V, G_ii = g'(S_i) (X_ii + Scb_i) and, off the diagonal, the
// divided differences of a singular-value function:
// G_ij = a (X_ij + X_ji)/2 + b (X_ij - X_ji)/2, a = (g_i - g_j)/(S_i - S_j)
// (the mean of g' at equal values), b = (g_i + g_j)/(S_i + S_j).  g' passes
// on [lo, hi] inclusive, as torch's clamp does.
__device__ __forceinline__ void f_clamp_adj(const Cons &c, float lo, float hi, const float Fcb[9],
                                            const float Scb[3], float out[9]) {
    float U[9], T[9], X[9], G[9], g[3], gp[3];
    mm3(c.R, c.V, U);
    mm3(Fcb, c.V, T);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) X[3 * i + j] = U[i] * T[j] + U[3 + i] * T[3 + j] + U[6 + i] * T[6 + j];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        g[i] = c.Sc[i];
        gp[i] = (c.S[i] >= lo && c.S[i] <= hi) ? 1.0f : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            if (i == j) {
                G[3 * i + i] = c.lamC[i] != 0.0f ? gp[i] * (X[3 * i + i] + Scb[i]) : 0.0f;
            } else {
                const float ds = c.S[i] - c.S[j];
                const float a = fabsf(ds) > 1e-6f * fmaxf(c.S[i], c.S[j]) ? (g[i] - g[j]) / ds : 0.5f * (gp[i] + gp[j]);
                const float den = fmaxf(c.S[i] + c.S[j], 1e-6f);
                const float b = (g[i] + g[j]) / den;
                const float xs = 0.5f * (X[3 * i + j] + X[3 * j + i]), xa = 0.5f * (X[3 * i + j] - X[3 * j + i]);
                G[3 * i + j] = a * xs + b * xa;
            }
        }
    float UG[9];
    mm3(U, G, UG);
    mmt3(UG, c.V, out);
}

constexpr int kAQ = 512;    // staged quadratic nodes per CTA ({v, m} and {mvbar, mbar}: 32 B each)
constexpr int kAC = 1024;   // staged cubic nodes per CTA (16 B each)

// Gathers of k_adj_particle for one particle, from the CTA's shared-memory
// tile (TILE) or from global memory with the reference's clamped indices.
// Both are folded over z, then y, then x, sums that share a weight or a value in
// packed pairs (b.w holds b.z again in the tile): 1M particles 316 us with the
// x and y weights multiplied out per row, 299 now.  The kernel is bound by latency
// at 16 warps per SM (45% of issue slots): with 3 CTAs per SM, without spills, the
// backward of 8 substeps took 370 us longer, with 5 as long.
template <bool TILE>
__device__ __forceinline__ void adj_gather(const float xp[3], float inv_dx, float dx, float K, int ng,
                                           const float vt[3], const float Ct[9], const float mv[3], float m,
                                           const float aff[9], float d1, float lb, const float4 *sv,
                                           const float4 *sa, const float4 *sb, const int lo[3], const int qd[3],
                                           const int cd[3], const float4 *__restrict__ gvel,
                                           const float4 *__restrict__ A, const float4 *__restrict__ B,
                                           float xb[3], float vsum[3], float mvb[3], float affb[9], float &d1b) {
    {
        // Per node o: wbar = g . u + an . c + an.w m with u = vt + K Ct dpos and
        // c = mv + aff dpos; the sums over the 27 nodes are contracted over z
        // first (Z0 = sum_z wz wbar, Z1 = sum_z w'z wbar, Gz = sum_z wz g,
        // Az = sum_z wz an, Azd = sum_z wz dpos_z an), then folded with the x
        // and y weights per (x, y) row.
        QuadD q;
        quad_weights_d(xp, inv_dx, ng, q);
        float DX[3], DY[3], DZ[3];
#pragma unroll
        for (int o = 0; o < 3; ++o) {
            DX[o] = ((float)o - q.fx[0]) * dx;
            DY[o] = ((float)o - q.fx[1]) * dx;
            DZ[o] = ((float)o - q.fx[2]) * dx;
        }
        const float2 zero = make_float2(0.0f, 0.0f);
        // components x and y in packed pairs, z with its dpos_z moment
        const float2 C0 = make_float2(K * Ct[0], K * Ct[3]), C1 = make_float2(K * Ct[1], K * Ct[4]),
                     C2 = make_float2(K * Ct[2], K * Ct[5]);
        const float2 a0 = make_float2(aff[0], aff[3]), a1 = make_float2(aff[1], aff[4]), a2 = make_float2(aff[2], aff[5]);
        const float C20 = K * Ct[6], C21 = K * Ct[7], C22 = K * Ct[8];
        float2 vs01 = zero, mv01 = zero, ax01 = zero, ay01 = zero, az01 = zero, mvaz2 = zero;
        float vs2 = 0.0f, ax2 = 0.0f, ay2 = 0.0f;
        float z0[2] = {0.0f, 0.0f}, z1 = 0.0f;   // per axis of xbar
#pragma unroll
        for (int ox = 0; ox < 3; ++ox) {
            const float2 ux01 = fma2(C0, bc2(DX[ox]), make_float2(vt[0], vt[1]));
            const float2 cx01 = fma2(a0, bc2(DX[ox]), make_float2(mv[0], mv[1]));
            const float ux2 = vt[2] + C20 * DX[ox], cx2 = mv[2] + aff[6] * DX[ox];
#pragma unroll
            for (int oy = 0; oy < 3; ++oy) {
                const float2 uxy01 = fma2(C1, bc2(DY[oy]), ux01), cxy01 = fma2(a1, bc2(DY[oy]), cx01);
                const float uxy2 = ux2 + C21 * DY[oy], cxy2 = cx2 + aff[7] * DY[oy];
                float2 Z = zero, G01 = zero, A01 = zero, Ad01 = zero, AAd2 = zero;   // Z: (Z0, Z1); AAd2: (Az, Azd).z
                float G2 = 0.0f;
                const int row = TILE ? ((q.b[0] + ox - lo[0]) * qd[1] + (q.b[1] + oy - lo[1])) * qd[2] + q.b[2] - lo[2] : 0;
#pragma unroll
                for (int oz = 0; oz < 3; ++oz) {
                    float4 g, an;
                    if (TILE) {
                        g = sv[row + oz];
                        an = sa[row + oz];
                    } else {
                        const int node = node_of(q.b[0] + ox, q.b[1] + oy, q.b[2] + oz, ng);
                        g = __ldg(&gvel[node]);
                        an = __ldg(&A[node]);
                    }
                    const float2 g01 = make_float2(g.x, g.y), an01 = make_float2(an.x, an.y);
                    const float2 u01 = fma2(C2, bc2(DZ[oz]), uxy01), c01 = fma2(a2, bc2(DZ[oz]), cxy01);
                    const float u2 = uxy2 + C22 * DZ[oz], c2 = cxy2 + aff[8] * DZ[oz];
                    const float2 t = fma2(an01, c01, mul2(g01, u01));
                    const float wbar = (t.x + t.y) + (g.z * u2 + (an.z * c2 + an.w * m));
                    const float wz = q.w[oz][2], wzd = wz * DZ[oz];
                    Z = fma2(make_float2(wz, q.dw[oz][2]), bc2(wbar), Z);
                    G01 = fma2(bc2(wz), g01, G01);
                    G2 += wz * g.z;
                    A01 = fma2(bc2(wz), an01, A01);
                    Ad01 = fma2(bc2(wzd), an01, Ad01);
                    AAd2 = fma2(make_float2(wz, wzd), bc2(an.z), AAd2);
                }
                const float wx = q.w[ox][0], wy = q.w[oy][1], wxy = wx * wy;
                z0[0] += q.dw[ox][0] * wy * Z.x;
                z0[1] += wx * q.dw[oy][1] * Z.x;
                z1 += wxy * Z.y;
                const float wxyx = wxy * DX[ox], wxyy = wxy * DY[oy];
                const float2 w2 = bc2(wxy);
                vs01 = fma2(w2, G01, vs01);
                vs2 += wxy * G2;
                mv01 = fma2(w2, A01, mv01);
                ax01 = fma2(bc2(wxyx), A01, ax01);
                ay01 = fma2(bc2(wxyy), A01, ay01);
                az01 = fma2(w2, Ad01, az01);
                mvaz2 = fma2(w2, AAd2, mvaz2);
                ax2 += wxyx * AAd2.x;
                ay2 += wxyy * AAd2.x;
            }
        }
        vsum[0] = vs01.x; vsum[1] = vs01.y; vsum[2] = vs2;
        mvb[0] = mv01.x;  mvb[1] = mv01.y;  mvb[2] = mvaz2.x;
        affb[0] = ax01.x; affb[1] = ay01.x; affb[2] = az01.x;
        affb[3] = ax01.y; affb[4] = ay01.y; affb[5] = az01.y;
        affb[6] = ax2;    affb[7] = ay2;    affb[8] = mvaz2.y;
        xb[0] += inv_dx * z0[0];
        xb[1] += inv_dx * z0[1];
        xb[2] += inv_dx * z1;
    }
    {
        CubicD cw;
        cubic_weights_d(xp, inv_dx, ng, cw);
        // Per node: wbar = b.x d1 + b.y, and b.z for the Laplacian's position part.
        // Folded over z, then y, then x, in packed pairs where two sums share a
        // weight or a value.
        float dsum = 0.0f;
        float x0 = 0.0f, x1 = 0.0f, x2 = 0.0f;
        const float2 zero = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int ox = 0; ox < 4; ++ox) {
            // sums over y: wy (swd, swb); wy (g0, g2); w2y (g0, g2) + wy (g1, g3); dwy swb; wy sdwb; dwy g0; dw2y g0 + dwy g1
            float2 W = zero, G = zero, GS = zero;
            float dW = 0.0f, wD = 0.0f, dG = 0.0f, tG = 0.0f;
#pragma unroll
            for (int oy = 0; oy < 4; ++oy) {
                const int row = TILE ? ((cw.b[0] + ox - lo[0] + 1) * cd[1] + (cw.b[1] + oy - lo[1] + 1)) * cd[2] +
                                           cw.b[2] - lo[2] + 1
                                     : (clampi(cw.b[0] + ox, 0, ng - 1) * ng + clampi(cw.b[1] + oy, 0, ng - 1)) * ng;
                float2 sw = zero, g02 = zero, g13 = zero;   // sums over z: w (b.x, wbar); (w, dw) b.z; (w2, dw2) b.z
                float sdwb = 0.0f;
#pragma unroll
                for (int oz = 0; oz < 4; ++oz) {
                    const float4 bn = TILE ? sb[row + oz] : __ldg(&B[row + clampi(cw.b[2] + oz, 0, ng - 1)]);
                    const float wbar = bn.x * d1 + bn.y;
                    const float2 zz = make_float2(bn.z, TILE ? bn.w : bn.z);
                    sw = fma2(bc2(cw.w[oz][2]), make_float2(bn.x, wbar), sw);
                    sdwb += cw.dw[oz][2] * wbar;
                    g02 = fma2(make_float2(cw.w[oz][2], cw.dw[oz][2]), zz, g02);
                    g13 = fma2(make_float2(cw.w2[oz][2], cw.dw2[oz][2]), zz, g13);
                }
                const float wy = cw.w[oy][1], dwy = cw.dw[oy][1];
                W = fma2(bc2(wy), sw, W);
                G = fma2(bc2(wy), g02, G);
                GS = fma2(bc2(cw.w2[oy][1]), g02, fma2(bc2(wy), g13, GS));
                dW += dwy * sw.y;
                wD += wy * sdwb;
                dG += dwy * g02.x;
                tG += cw.dw2[oy][1] * g02.x + dwy * g13.x;
            }
            const float wx = cw.w[ox][0], dwx = cw.dw[ox][0], sx = cw.w2[ox][0], tx = cw.dw2[ox][0];
            dsum += wx * W.x;
            x0 += inv_dx * dwx * W.y + lb * (tx * G.x + dwx * GS.x);
            x1 += inv_dx * wx * dW + lb * (sx * dG + wx * tG);
            x2 += inv_dx * wx * wD + lb * (sx * G.y + wx * GS.y);
        }
        xb[0] += x0;
        xb[1] += x1;
        xb[2] += x2;
        d1b += dsum;
    }
}

// ---------------------------------------------------------------- k_adj_particle
// The gathers come first, with the forward's APIC affine term read from the
// tape, so the constitutive recompute and its adjoint run last with none of
// the gather state live.  The output adjoint of F is written in two parts:
// (I + dt C')^T Fbar' before the gathers, the constitutive part added at the
// end (same thread, same address).
template <bool EXT>
__global__ void __launch_bounds__(128, 4) k_adj_particle(const pm_params prm, const Parts pre, const Parts post,
                                                         const pm_state_adj ain, const pm_state_adj aout,
                                                         const pm_param_adj grads, const TapeHead *head,
                                                         const float4 *__restrict__ gvel,
                                                         const float4 *__restrict__ A, const float4 *__restrict__ B,
                                                         const float *__restrict__ taff, const float *__restrict__ tpol,
                                                         long long taff_stride) {
    __shared__ float4 sv[kAQ], sa[kAQ], sb[kAC];
    __shared__ int s_box[6];
    const int tid = threadIdx.x;
    const long long p = (long long)blockIdx.x * blockDim.x + tid;
    const bool valid = p < pre.n;
    const long long ps = pre.ps, as = ain.plane_stride, os = aout.plane_stride;
    const int ng = prm.n_grid;
    const float inv_dx = (float)prm.inv_dx, dx = (float)prm.dx, dt = (float)prm.dt;
    const float K = (float)(4.0 * prm.inv_dx * prm.inv_dx);
    const float L2 = (float)(prm.inv_dx * prm.inv_dx);
    float xp[3] = {0.0f, 0.0f, 0.0f};
    // ---- stage the CTA's grid footprint (as k_g2p does): {v, m} and the
    // momentum adjoints of the quadratic nodes of the regular particles' base
    // cells' bounding box, the damage adjoints of its cubic nodes
    bool reg = valid;
    int qb[3] = {0, 0, 0};
    if (valid) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            xp[k] = pre.x[k * ps + p];
            const float fb = floorf(__fsub_rn(__fmul_rn(xp[k], inv_dx), 0.5f));
            reg = reg && (fb >= 1.0f) && (fb <= (float)(ng - 4));
            qb[k] = reg ? (int)fb : 0;
        }
    }
    if (tid < 6) s_box[tid] = tid < 3 ? 0x7fffffff : -0x7fffffff;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int mn = __reduce_min_sync(0xffffffffu, reg ? qb[k] : 0x7fffffff);
        const int mx = __reduce_max_sync(0xffffffffu, reg ? qb[k] : -0x7fffffff);
        if ((tid & 31) == 0) {
            atomicMin(&s_box[k], mn);
            atomicMax(&s_box[3 + k], mx);
        }
    }
    __syncthreads();
    const int lo[3] = {s_box[0], s_box[1], s_box[2]};
    const bool any = s_box[3] >= lo[0];
    const int qd[3] = {s_box[3] - lo[0] + 3, s_box[4] - lo[1] + 3, s_box[5] - lo[2] + 3};
    const int cd[3] = {qd[0] + 2, qd[1] + 2, qd[2] + 2};
    const int qn = any ? qd[0] * qd[1] * qd[2] : 0, cn = any ? cd[0] * cd[1] * cd[2] : 0;
    const bool tile = any && qn <= kAQ && cn <= kAC;
    if (tile) {   // regular nodes lie inside the grid
        const FastDiv qyz = make_fastdiv(qd[1] * qd[2]), qz = make_fastdiv(qd[2]);
        for (int i = tid; i < qn; i += blockDim.x) {
            const int ix = fdiv(i, qyz), r = i - ix * qyz.d, iy = fdiv(r, qz);
            const int gx = lo[0] + ix, gy = lo[1] + iy, gz = lo[2] + r - iy * qz.d;
            const long long node = ((long long)gx * ng + gy) * ng + gz;
            sv[i] = gvel[node];
            sa[i] = A[node];
        }
        const FastDiv cyz = make_fastdiv(cd[1] * cd[2]), cz = make_fastdiv(cd[2]);
        for (int i = tid; i < cn; i += blockDim.x) {
            const int ix = fdiv(i, cyz), r = i - ix * cyz.d, iy = fdiv(r, cz);
            const int gx = lo[0] - 1 + ix, gy = lo[1] - 1 + iy, gz = lo[2] - 1 + r - iy * cz.d;
            float4 b = B[((long long)gx * ng + gy) * ng + gz];
            b.w = b.z;                       // a packed operand
            sb[i] = b;
        }
    }
    __syncthreads();
    if (!valid) return;
    const TapeHead h = *head;
    float xb[3] = {0.0f, 0.0f, 0.0f};
    float vt[3], Ct[9];
    {
        float vpost[3], F[9];
#pragma unroll
        for (int k = 0; k < 3; ++k) vpost[k] = post.v[k * ps + p];
#pragma unroll
        for (int k = 0; k < 9; ++k) F[k] = pre.F[k * ps + p];
        if (EXT) g2p_input_F(prm, tpol, taff_stride, p, F);
        AdjIn a;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            a.xb[k] = ain.x[k * as + p];
            a.vb[k] = ain.v[k * as + p];
        }
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            a.Cb[k] = ain.C[k * as + p];
            a.Fb[k] = ain.F[k * as + p];
        }
        bool inside[3];
        g2p_tail_adj(prm, xp, vpost, F, a, vt, Ct, inside);
#pragma unroll
        for (int k = 0; k < 3; ++k) xb[k] = inside[k] ? a.xb[k] : 0.0f;   // x' = clamp(x + dt v')
        // F' = (I + dt C') F:  Fbar = (I + dt C')^T Fbar' (+ the constitutive part below)
        float Cp[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) Cp[k] = post.C[k * ps + p];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j)
                aout.F[(3 * i + j) * os + p] =
                    a.Fb[3 * i + j] + dt * (Cp[i] * a.Fb[j] + Cp[3 + i] * a.Fb[3 + j] + Cp[6 + i] * a.Fb[6 + j]);
    }
    // ---- P2G inputs of the forward: velocity after the grips, mass, affine term
    float v[3] = {pre.v[p], pre.v[ps + p], pre.v[2 * ps + p]};
    bool gripped = false;
    if (pre.grip_tag) {
        const int gi = pre.grip_tag[p];
        if (gi >= 0 && gi < prm.n_grips) {
            gripped = true;
            const double f = prm.grips[gi].ramp > 0.0 ? fmin(h.time / prm.grips[gi].ramp, 1.0) : 1.0;
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) v[ax] = (float)(prm.grips[gi].vel[ax] * f);
        }
    }
    const float m = pre.mass[p];
    const float mv[3] = {m * v[0], m * v[1], m * v[2]};
    float aff[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) aff[k] = taff[k * taff_stride + p];
    // ---- gathers (quadratic: G2P adjoint position part and P2G adjoint;
    // cubic: damage scatter adjoint and the Laplacian's position part)
    float vsum[3], mvb[3], affb[9];
    float d1b = ain.d[p];
    {
        const float d1 = post.d[p];
        const float lb = ain.lap[p] * L2 * inv_dx;
        if (reg && tile)
            adj_gather<true>(xp, inv_dx, dx, K, ng, vt, Ct, mv, m, aff, d1, lb, sv, sa, sb, lo, qd, cd, gvel, A, B,
                             xb, vsum, mvb, affb, d1b);
        else
            adj_gather<false>(xp, inv_dx, dx, K, ng, vt, Ct, mv, m, aff, d1, lb, sv, sa, sb, lo, qd, cd, gvel, A, B,
                              xb, vsum, mvb, affb, d1b);
    }
    // dpos = node - x:  xbar -= K Cbar^T sum(w v_i) + aff^T sum(w mvbar_i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
        xb[j] -= K * (Ct[j] * vsum[0] + Ct[3 + j] * vsum[1] + Ct[6 + j] * vsum[2]) +
                 (aff[j] * mvb[0] + aff[3 + j] * mvb[1] + aff[6 + j] * mvb[2]);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        aout.x[k * os + p] = xb[k];
        aout.v[k * os + p] = gripped ? 0.0f : m * mvb[k];
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) aout.C[k * os + p] = m * affb[k];
    // ---- constitutive recompute and adjoint
    const bool do_damage = h.any_allow != 0 && (h.step % (long long)prm.damage_every) == 0;
    const float coeff =
        __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn((float)(-prm.dt), pre.vol0[p]), 4.0f), inv_dx), inv_dx);
    float taub[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) taub[k] = coeff * affb[k];
    Cons c;
    float tau[9];
    cons_forward<EXT>(prm, pre, p, do_damage, c, tau, tpol, taff_stride);
    ConsAdj o;
    cons_adjoint(c, pre.mu[p], pre.lam[p], taub, d1b, ain.D_hist[p], pre, p, o);
    if (c.fclamp) {
        // the G2P part above and the stress's direct part are adjoints of the
        // limited F: through the limit to the pre-substep F, plus the polar
        // rotation's part
        float Fcb[9], F0b[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) Fcb[k] = aout.F[k * os + p] + o.Fb[k];
        f_clamp_adj(c, (float)prm.f_clamp_lo, (float)prm.f_clamp_hi, Fcb, o.Scb, F0b);
#pragma unroll
        for (int k = 0; k < 9; ++k) aout.F[k * os + p] = F0b[k] + o.Fp[k];
    } else {
#pragma unroll
        for (int k = 0; k < 9; ++k) aout.F[k * os + p] += o.Fb[k];
    }
    aout.d[p] = o.d0b;
    aout.lap[p] = o.lapb;
    aout.D_hist[p] = o.Dh0b;
    const long long gs = grads.plane_stride;
    if (grads.mu) grads.mu[p] += o.mub;
    if (grads.lam) grads.lam[p] += o.lamb;
    // sigma_c and A0 enter only through an active damage drive: most
    // particles add zero, so skip their read-modify-write
    if (grads.sigma_c && o.scb != 0.0f) grads.sigma_c[p] += o.scb;
    if (grads.A0) {
        bool nz = false;
#pragma unroll
        for (int k = 0; k < 9; ++k) nz = nz || o.A0b[k] != 0.0f;
        if (nz) {
#pragma unroll
            for (int k = 0; k < 9; ++k) grads.A0[k * gs + p] += o.A0b[k];
        }
    }
}

__global__ void k_tape_head(const Ctrl *ctrl, TapeHead *head, long long n) {
    if (threadIdx.x == 0) {
        head->n_active = ctrl->n_active;
        head->any_allow = ctrl->any_allow;
        head->step = ctrl->step;
        head->time = ctrl->time;
        head->n_work = (unsigned)min((long long)ctrl->n_work, n);
        head->n_clamped = (unsigned)min((long long)ctrl->n_clamped, n);
    }
    if (threadIdx.x < PM_MAX_COLLIDERS) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            head->col_origin[threadIdx.x][a] = ctrl->col_origin[threadIdx.x][a];
            head->col_vel[threadIdx.x][a] = ctrl->col_vel[threadIdx.x][a];
        }
    }
}

}  // namespace

// One-time kernel attribute set-up for the current device (not a stream
// operation; pm_prepare runs it before any capture).
void prepare_adjoint() {
    static int done[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(k_adj_sweep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SweepShared));
        done[dev] = 1;
    }
}

// ------------------------------------------------------------------ tape layout
TapeLayout make_tape_layout(long long n, int ng, int slots, int flags) {
    TapeLayout T;
    const size_t A = 256;
    const long long G = (long long)ng * ng * ng;
    const int nbs = (ng + kBlockEdge - 1) / kBlockEdge;
    const long long nb = (long long)nbs * nbs * nbs;
    const long long nb8 = sort_blocks_per_axis(ng);
    const long long units = listed_units(n, nb8 * nb8 * nb8);
    const long long np = (n + 63) / 64 * 64 > 0 ? (n + 63) / 64 * 64 : 64;
    size_t o = 0;
    T.head = o;    o = align_up(o + sizeof(TapeHead) * (size_t)(slots > 0 ? slots : 1), A);
    T.actl = o;    o = align_up(o + sizeof(AdjCtrl), A);
    T.acc = o;     o = align_up(o + 32 * (size_t)G, A);     // 4 x int64 per node
    T.adj_q = o;   o = align_up(o + 16 * (size_t)G, A);
    T.adj_c = o;   o = align_up(o + 16 * (size_t)G, A);
    T.apay = o;    o = align_up(o + kPayBytes * (size_t)(kPayPlaces * np), A);   // (np is a multiple of 32)
    T.slot0 = o;
    size_t s = 0;
    T.vel = s;     s = align_up(s + 16 * (size_t)G, A);
    T.gd = s;      s = align_up(s + 4 * (size_t)G, A);
    T.sw = s;      s = align_up(s + 4 * (size_t)G, A);
    T.vpre = s;    s = align_up(s + ((flags & PM_TAPE_COLLIDERS) ? 16 * (size_t)G : 0), A);   // pre-collider v
    T.blocks = s;  s = align_up(s + 4 * (size_t)nb, A);
    T.iperm = s;   s = align_up(s + 4 * (size_t)np, A);
    T.work = s;    s = align_up(s + 4 * (size_t)np, A);
    T.clamped = s; s = align_up(s + 4 * (size_t)units, A);
    T.split = s;   s = align_up(s + (size_t)kUnitCells * (size_t)units, A);
    T.cells = s;   s = align_up(s + 8 * (size_t)kUnitCells * (size_t)units, A);
    T.aff = s;     s = align_up(s + 36 * (size_t)np, A);
    T.pol = s;     s = align_up(s + 88 * (size_t)np, A);
    T.aff_stride = np;
    T.slot_bytes = s;
    T.total = o + s * (size_t)(slots > 0 ? slots : 1);
    T.n_blocks = nb;
    T.slots = slots;
    T.flags = flags;
    return T;
}

void record_redirect(const TapeLayout &T, void *tape, int slot, WS &w) {
    char *b = (char *)tape + T.slot0 + T.slot_bytes * (size_t)slot;
    w.g_vel = (float4 *)(b + T.vel);
    w.g_gd = (float *)(b + T.gd);
    w.g_sw = (float *)(b + T.sw);
    w.g_vpre = (T.flags & PM_TAPE_COLLIDERS) ? (float4 *)(b + T.vpre) : nullptr;
    w.block_list = (int *)(b + T.blocks);
    w.slot = (int *)(b + T.iperm);       // the particles' places, the unit list and its cells stay on the tape
    w.work = (int *)(b + T.work);
    w.clamped = (int *)(b + T.clamped);
    w.rec_cells = (int2 *)(b + T.cells);
    w.rec_split = (unsigned char *)(b + T.split);
    w.tape_aff = (float *)(b + T.aff);
    w.tape_pol = (float *)(b + T.pol);
    w.tape_aff_stride = T.aff_stride;
}

void launch_tape_head(const TapeLayout &T, void *tape, int slot, const WS &w, long long n, cudaStream_t s) {
    k_tape_head<<<1, 32, 0, s>>>(w.ctrl, (TapeHead *)((char *)tape + T.head) + slot, n);
}

void launch_adjoint(const pm_params &prm, const Parts &pre, const Parts &post, const pm_state_adj &ain,
                    const pm_state_adj &aout, const pm_param_adj &grads, const TapeLayout &T, void *tape, int slot,
                    cudaStream_t s) {
    char *base = (char *)tape;
    char *b = base + T.slot0 + T.slot_bytes * (size_t)slot;
    const TapeHead *h = (const TapeHead *)(base + T.head) + slot;
    AdjCtrl *actl = (AdjCtrl *)(base + T.actl);
    long long *acc = (long long *)(base + T.acc);
    void *apay = base + T.apay;
    float4 *Aq = (float4 *)(base + T.adj_q);
    float4 *Bc = (float4 *)(base + T.adj_c);
    const float4 *gvel = (const float4 *)(b + T.vel);
    const float *ggd = (const float *)(b + T.gd);
    const float *gsw = (const float *)(b + T.sw);
    const int *blocks = (const int *)(b + T.blocks);
    const long long n = pre.n;
    if (n <= 0) return;
    prepare_adjoint();
    cudaMemsetAsync(actl, 0, sizeof(AdjCtrl), s);
    k_adj_pre<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(prm, pre, post, ain, (const int *)(b + T.iperm), apay, actl,
                                                          (const float *)(b + T.pol), T.aff_stride);
    {
        static int slots_dev[64] = {0};
        int dev = 0;
        cudaGetDevice(&dev);
        int slots = (dev >= 0 && dev < 64) ? slots_dev[dev] : 0;
        if (slots <= 0) {
            slots = resident_slots((const void *)k_adj_sweep, kSweepThreads, sizeof(SweepShared));
            if (dev >= 0 && dev < 64) slots_dev[dev] = slots;
        }
        k_adj_sweep<<<(unsigned)std::min<long long>(slots, n), kSweepThreads, sizeof(SweepShared), s>>>(
            prm, (const int *)(b + T.work), (const int *)(b + T.clamped), (const int2 *)(b + T.cells),
            (const unsigned char *)(b + T.split), h, apay, actl, acc, n);
    }
    const long long max_items = T.n_blocks * 64;
    const int gb = (int)std::max<long long>(1, std::min<long long>((max_items + 255) / 256, 148LL * 8));
    const float4 *vpre = (T.flags & PM_TAPE_COLLIDERS) ? (const float4 *)(b + T.vpre) : nullptr;
    k_adj_grid<<<gb, 256, 0, s>>>(prm, blocks, h, gvel, vpre, ggd, gsw, acc, actl, Aq, Bc, T.n_blocks);
    const float *taff = (const float *)(b + T.aff);
    const float *tpol = (const float *)(b + T.pol);
    const unsigned pb = (unsigned)((n + 127) / 128);
    if (prm.use_f_clamp || pre.interface_mask)
        k_adj_particle<true><<<pb, 128, 0, s>>>(prm, pre, post, ain, aout, grads, h, gvel, Aq, Bc, taff, tpol,
                                                T.aff_stride);
    else
        k_adj_particle<false><<<pb, 128, 0, s>>>(prm, pre, post, ain, aout, grads, h, gvel, Aq, Bc, taff, tpol,
                                                 T.aff_stride);
}

}  // namespace pm
