// Gaussian-splat renderer (render.py:71-162 of the reference): EWA projection
// of 3D gaussians to screen-space gaussians, then the reference's two-pass
// soft z-buffer -- per pixel the nearest splat depth, then a blend of all
// splats weighted by exp(-(z - z_min) / tau) -- and coverage compositing over
// a background.  The image is a headless device buffer (H, W, 3).
//
// Screen tiles of 16x16 pixels.  k_splat_project (one thread per gaussian:
// camera transform, Jacobian, 2D covariance + 0.3 dilation, conic, radius,
// culling) packs each drawn splat into 48 bytes and counts it into every tile
// its (2r+1)^2 footprint square touches; k_tile_alloc and k_splat_emit build
// per-tile splat lists; k_splat_tiles runs one warp per
// 8x8 part of a tile, two pixels per lane: the soft z-buffer walks the tile's
// list once, the splats that reach the part through shared memory, with the
// pixels' state in registers, and each pixel is composed at the end -- no per-pixel atomics, no clear of pixel buffers.
// tau from the median depth selects it digit by digit from the depth keys.
#include "pm_kernels.cuh"

namespace pm {
namespace {

constexpr int kTile = 16;                 // screen tile edge, pixels
constexpr int kSubTile = 8;               // edge of the part of a tile that a warp draws

struct RenderWS {
    float4 *sp;        // [3n] per splat: {u, v, c00, c01}, {c11, z, u0, v0 (int bits)}, {r, g, b, rad (int bits)}
    unsigned *count;   // [0] drawn splats, [1] list overflow (never set when the capacity bound holds), [2] list length
    float *tau;        // [0] tau, [1] 1 / max(tau, 1e-6)
    unsigned *keys;    // [n] depth keys (z bits; all ones: not drawn)
    unsigned *hist;    // [kMedianPasses][kMedianBins] keys by digit, then {prefix, rank, CTAs done per pass}
    unsigned *tcnt;    // [ntiles] splats per tile
    unsigned *tfill;   // [ntiles] emit cursors, absolute
    unsigned *tstart;  // [ntiles] first list entry of the tile
    int *tlist;        // [cap] splat ids grouped by tile
    long long cap;
    int ntx, nty;
};

// The median's digits: 11, 11 and 10 bits from the top.
constexpr int kMedianPasses = 3, kMedianBins = 2048, kMedianWords = kMedianPasses * kMedianBins + 2 + kMedianPasses;

__device__ __forceinline__ void splat_tiles(int u0, int v0, int rad, int W, int H, int &tx0, int &ty0, int &nx,
                                            int &ny) {
    const int x0 = max(u0 - rad, 0), x1 = min(u0 + rad, W - 1);
    const int y0 = max(v0 - rad, 0), y1 = min(v0 + rad, H - 1);
    tx0 = x0 / kTile;
    ty0 = y0 / kTile;
    nx = x1 / kTile - tx0 + 1;
    ny = y1 / kTile - ty0 + 1;
}

// Clears the counters; tau is the given one, or 1 until a median replaces it.
__global__ void __launch_bounds__(256) k_splat_clear(RenderWS r, int ntiles, float tau_given) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 4) r.count[i] = 0;
    if (i < kMedianWords) r.hist[i] = 0;
    if (i < ntiles) r.tcnt[i] = 0;
    if (i == 0) {
        const float tau = tau_given > 0.0f ? tau_given : 1.0f;
        r.tau[0] = tau;
        r.tau[1] = 1.0f / (tau > 1e-6f ? tau : 1e-6f);
    }
}

// Each lane walks the tiles of its own splat; lanes of a warp that hit the
// same tile in the same step (neighbouring gaussians) add to it with one atomic.
struct TileWalk {
    int tx0, ty0, nx, ny, ntx;
    __device__ __forceinline__ int tile(int k, bool on) const {
        const int ky = on ? k / nx : 0;
        return on ? (ty0 + ky) * ntx + tx0 + (k - ky * nx) : -1;
    }
};

__global__ void __launch_bounds__(256) k_splat_project(const pm_camera cam, const pm_render_params rp,
                                                       const float *__restrict__ xyz, const float *__restrict__ cov,
                                                       const float *__restrict__ color, long long n, RenderWS r) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float X[3] = {xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]};
    float Xc[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) Xc[j] = (X[0] * cam.R[j] + X[1] * cam.R[3 + j] + X[2] * cam.R[6 + j]) + cam.T[j];
    const float z = Xc[2];
    bool ok = z > rp.near;
    float u = 0.0f, v = 0.0f, c00 = 0.0f, c01 = 0.0f, c11 = 0.0f;
    int u0 = 0, v0 = 0, rad = 0;
    if (ok) {
        const float cx = 0.5f * (float)cam.width, cy = 0.5f * (float)cam.height;
        u = cam.fx * Xc[0] / z + cx;
        v = cam.fy * Xc[1] / z + cy;
        const float invz = 1.0f / z;
        // J (2x3): [fx/z, 0, -fx x / z^2; 0, fy/z, -fy y / z^2]
        const float J00 = cam.fx * invz, J02 = -cam.fx * Xc[0] * invz * invz;
        const float J11 = cam.fy * invz, J12 = -cam.fy * Xc[1] * invz * invz;
        // cov_cam = R^T cov R * s^2 (Rt = R^T)
        float Sg[9], T1[9], Cc[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) Sg[k] = cov[9 * i + k];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b)   // T1 = Rt Sg, Rt[a][k] = R[k][a]
                T1[3 * a + b] = cam.R[a] * Sg[b] + cam.R[3 + a] * Sg[3 + b] + cam.R[6 + a] * Sg[6 + b];
        const float s2 = rp.scale_modifier * rp.scale_modifier;
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b)   // Cc = T1 Rt^T = T1 R, Rt^T[k][b] = R[k][b]
                Cc[3 * a + b] = (T1[3 * a] * cam.R[b] + T1[3 * a + 1] * cam.R[3 + b] + T1[3 * a + 2] * cam.R[6 + b]) * s2;
        // cov2d = J Cc J^T
        const float M00 = J00 * Cc[0] + J02 * Cc[6], M01 = J00 * Cc[1] + J02 * Cc[7], M02 = J00 * Cc[2] + J02 * Cc[8];
        const float M11 = J11 * Cc[4] + J12 * Cc[7], M12 = J11 * Cc[5] + J12 * Cc[8], M10 = J11 * Cc[3] + J12 * Cc[6];
        const float a = (M00 * J00 + M02 * J02) + 0.3f;
        const float b = M01 * J11 + M02 * J12;
        const float d = (M11 * J11 + M12 * J12) + 0.3f;
        (void)M10;
        const float det = a * d - b * b;
        const float mid = 0.5f * (a + d);
        const float disc = mid * mid - det;
        const float lam = mid + sqrtf(disc > 0.0f ? disc : 0.0f);
        const float raw = 3.0f * sqrtf(lam > 1e-6f ? lam : 1e-6f);
        u0 = (int)floorf(u);
        v0 = (int)floorf(v);
        rad = (int)ceilf(raw);
        rad = rad < 1 ? 1 : (rad > rp.r_max ? rp.r_max : rad);
        ok = det > 1e-9f && raw < rp.max_raw_radius && u0 + rad >= 0 && u0 - rad < cam.width && v0 + rad >= 0 &&
             v0 - rad < cam.height;
        if (ok) {
            const float inv_det = 1.0f / det;
            c00 = d * inv_det;
            c01 = -b * inv_det;
            c11 = a * inv_det;
        }
    }
    const int rd = ok ? rad : 0;
    r.sp[3 * i] = make_float4(u, v, c00, c01);
    r.sp[3 * i + 1] = make_float4(c11, z, __int_as_float(u0), __int_as_float(v0));
    if (ok)
        r.sp[3 * i + 2] = make_float4(color[3 * i], color[3 * i + 1], color[3 * i + 2], __int_as_float(rd));
    else
        r.sp[3 * i + 2] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(0));
    // depth key for the median of the drawn splats (z > near > 0: the float bits order like the values)
    r.keys[i] = ok ? __float_as_uint(z) : 0xffffffffu;
    const unsigned act = __activemask(), drawn = __ballot_sync(act, ok);
    if ((threadIdx.x & 31) == (unsigned)(__ffs(act) - 1) && drawn) atomicAdd(r.count, (unsigned)__popc(drawn));
    // tile counts of the footprint square
    TileWalk t{0, 0, 0, 0, r.ntx};
    if (ok) splat_tiles(u0, v0, rd, cam.width, cam.height, t.tx0, t.ty0, t.nx, t.ny);
    const int nt = t.nx * t.ny;
    const int steps = __reduce_max_sync(act, nt);
    const int lane = threadIdx.x & 31;
    for (int k = 0; k < steps; ++k) {
        const int tile = t.tile(k, k < nt);
        const unsigned peers = __match_any_sync(act, tile);
        if (tile >= 0 && lane == __ffs(peers) - 1) atomicAdd(&r.tcnt[tile], (unsigned)__popc(peers));
    }
}

// tau = 0.02 * median depth of the drawn splats (torch.median: the lower middle
// element), by selection: one pass over the keys per digit counts those that
// share the digits found so far, and the last CTA to finish finds the digit that
// holds the wanted rank.  (A whole radix sort of the keys for this one value took
// 89 of the 500 us of 262k gaussians; the three passes take 25.)
constexpr int kMedianThreads = 1024;
template <int PASS>
__global__ void __launch_bounds__(kMedianThreads) k_median(RenderWS r, long long n) {
    constexpr int kShift = PASS == 0 ? 21 : (PASS == 1 ? 10 : 0), kBits = PASS == 2 ? 10 : 11;
    __shared__ unsigned cnt[kMedianBins], wsum[kMedianThreads / 32];
    __shared__ bool last;
    const int tid = threadIdx.x, lane = tid & 31;
    unsigned *hist = r.hist + PASS * kMedianBins, *sel = r.hist + kMedianPasses * kMedianBins;
    const unsigned prefix = PASS == 0 ? 0u : sel[0];
    for (int i = tid; i < kMedianBins; i += kMedianThreads) cnt[i] = 0;
    __syncthreads();
    const long long stride = (long long)gridDim.x * kMedianThreads;
#pragma unroll 4
    for (long long base = (long long)blockIdx.x * kMedianThreads; base < n; base += stride) {
        const unsigned key = base + tid < n ? r.keys[base + tid] : 0u;
        bool on = base + tid < n;
        if (PASS > 0) on = on && (key >> (PASS == 1 ? 21 : 10)) == prefix;
        const int bin = on ? (int)((key >> kShift) & ((1u << kBits) - 1u)) : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, bin);   // depths share their leading digits
        if (on && lane == __ffs(peers) - 1) atomicAdd(&cnt[bin], (unsigned)__popc(peers));
    }
    __syncthreads();
    for (int i = tid; i < kMedianBins; i += kMedianThreads)
        if (cnt[i]) atomicAdd(&hist[i], cnt[i]);
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(&sel[2 + PASS], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    const unsigned drawn = *(volatile unsigned *)r.count;
    if (drawn == 0) return;                                // tau stays 1
    const unsigned rank = PASS == 0 ? (drawn - 1) / 2 : *(volatile unsigned *)(sel + 1);
    constexpr int kOwn = kMedianBins / kMedianThreads;
    unsigned c[kOwn], sum = 0;
#pragma unroll
    for (int k = 0; k < kOwn; ++k) {
        c[k] = __ldcg(&hist[kOwn * tid + k]);
        sum += c[k];
    }
    unsigned incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[tid >> 5] = incl;
    __syncthreads();
    unsigned before = incl - sum;
    for (int k = 0; k < tid >> 5; ++k) before += wsum[k];
#pragma unroll
    for (int k = 0; k < kOwn; ++k) {
        if (rank >= before && rank - before < c[k]) {      // one thread, one bin
            const unsigned found = (prefix << kBits) | (unsigned)(kOwn * tid + k);
            sel[0] = found;
            sel[1] = rank - before;
            if (PASS == kMedianPasses - 1) {
                const float tau = 0.02f * __uint_as_float(found);
                r.tau[0] = tau;
                r.tau[1] = 1.0f / (tau > 1e-6f ? tau : 1e-6f);
            }
        }
        before += c[k];
    }
}

// Gives every tile its part of the list: a scan within a CTA's tiles, one atomic
// per CTA for where they begin (the parts lie in any order).  (One CTA scanning
// all 14,400 tiles took 16 us, this 3.)
__global__ void __launch_bounds__(256) k_tile_alloc(RenderWS r, int ntiles) {
    __shared__ unsigned wsum[8], first;
    const int tid = threadIdx.x, lane = tid & 31, i = blockIdx.x * 256 + tid;
    const unsigned v = i < ntiles ? r.tcnt[i] : 0u;
    unsigned incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[tid >> 5] = incl;
    __syncthreads();
    unsigned before = 0, all = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        before += k < (tid >> 5) ? wsum[k] : 0u;
        all += wsum[k];
    }
    if (tid == 0) first = atomicAdd(r.count + 2, all);
    __syncthreads();
    if (i < ntiles) r.tstart[i] = r.tfill[i] = first + before + incl - v;
}

// Per-tile lists: every drawn splat id into each tile of its footprint square,
// four tiles at a time, their reservations under way together.  Lanes of a warp
// that hit the same tile in the same step (neighbouring gaussians) reserve
// with one atomic.
__global__ void __launch_bounds__(256) k_splat_emit(const pm_camera cam, long long n, RenderWS r) {
    constexpr int G = 4;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p1 = r.sp[3 * i + 1], p2 = r.sp[3 * i + 2];
    const int rd = __float_as_int(p2.w);
    TileWalk t{0, 0, 0, 0, r.ntx};
    if (rd > 0)
        splat_tiles(__float_as_int(p1.z), __float_as_int(p1.w), rd, cam.width, cam.height, t.tx0, t.ty0, t.nx, t.ny);
    const int nt = t.nx * t.ny;
    const unsigned act = __activemask();
    const int steps = __reduce_max_sync(act, nt), lane = threadIdx.x & 31;
    for (int k0 = 0; k0 < steps; k0 += G) {
        int tile[G];
        unsigned peers[G], base[G];
#pragma unroll
        for (int q = 0; q < G; ++q) {
            tile[q] = t.tile(k0 + q, k0 + q < nt);
            peers[q] = __match_any_sync(act, tile[q]);
            base[q] = 0;
            if (tile[q] >= 0 && lane == __ffs(peers[q]) - 1)
                base[q] = atomicAdd(&r.tfill[tile[q]], (unsigned)__popc(peers[q]));
        }
#pragma unroll
        for (int q = 0; q < G; ++q) {
            const long long at =
                (long long)__shfl_sync(act, base[q], __ffs(peers[q]) - 1) + __popc(peers[q] & lanemask_lt());
            if (tile[q] >= 0) {
                if (at < r.cap)
                    r.tlist[at] = (int)i;
                else
                    r.count[1] = 1;
            }
        }
    }
}

// One warp per 8x8 part of a tile (4 parts and warps per CTA), two pixels per lane
// (rows y and y + 4).  A splat counts at a pixel when the pixel lies in its
// footprint square and alpha = exp(min(power, 0)) exceeds 1/255.  The
// reference's two passes -- nearest depth z_min, then sums of c w and w with w =
// alpha exp(-(z - z_min) / tau) -- are done in one, the sums relative to a
// nearest depth so far and rescaled when a nearer splat arrives, which is the
// same sum up to rounding.  The coverage 1 - exp(sum log(max(1 - alpha, 1e-6)))
// is taken as 1 - prod max(1 - alpha, 1e-6): the same quantity, and a product
// that underflows gives coverage 1.0f exactly as the sum of logs does.  The
// exponentials use ex2.approx (a few ulp; the image tolerance is 1e-4 absolute).
//
// draw_part takes the list 32 splats at a time: every lane tests one splat against
// the whole part (footprint square, and the largest power in it) and computes
// what all pixels share, above all the depth weight, relative to the nearest
// depth of the part instead of the pixel: one exponential per splat in place of
// one per pixel.  What remains is drawn by all lanes without branches, the two
// pixels in packed pairs.  The weights then span the part's depth range; where
// that exceeds kMaxRange tau (float32 would lose the nearest splats of the
// farther pixels), or a colour is not finite (a zero weight would spread it),
// draw_part_general does the part again with a nearest depth per pixel.
//
// Bound by instruction issue.  262k splats of 7 pixels radius on 1280x720: 346 us
// with 8x8 lists, every splat of the list tested per pixel and two exponentials
// per pixel (80 instructions per splat and part), 150 us now; beyond kMaxRange, whole
// renders of as many splats take 425 us against 490.  Lists of 16x16
// pixels halve the list work (emit 30 -> 15, project 27 -> 16 us); the parts then
// test more splats, but a warp tests 32 at a time.
constexpr int kTileWarps = 4;

struct PixAcc {
    float zmin, c0, c1, c2, w, rev;   // rev: prod max(1 - alpha, 1e-6)
};

__device__ __forceinline__ void pix_add(PixAcc &p, const float4 &A, const float4 &B, const float4 &Cc, int px, int py,
                                        float inv_tau) {
    const int rd = __float_as_int(Cc.w);
    if (abs(px - __float_as_int(B.z)) > rd || abs(py - __float_as_int(B.w)) > rd) return;
    const float dx = ((float)px + 0.5f) - A.x, dy = ((float)py + 0.5f) - A.y;
    const float power = fmaf(-0.5f, fmaf(A.z * dx, dx, __fmul_rn(B.x * dy, dy)), -__fmul_rn(A.w * dx, dy));
    if (power < -6.0f) return;
    const float ga = __expf(power < 0.0f ? power : 0.0f);
    if (!(ga > (1.0f / 255.0f))) return;
    float w;
    if (B.y < p.zmin) {
        const float sc = p.w > 0.0f ? __expf(-(p.zmin - B.y) * inv_tau) : 0.0f;
        p.c0 *= sc; p.c1 *= sc; p.c2 *= sc; p.w *= sc;
        p.zmin = B.y;
        w = ga;   // exp(0)
    } else {
        w = ga * __expf(-(B.y - p.zmin) * inv_tau);
    }
    p.c0 += Cc.x * w;
    p.c1 += Cc.y * w;
    p.c2 += Cc.z * w;
    p.w += w;
    const float om = 1.0f - ga;
    p.rev *= om > 1e-6f ? om : 1e-6f;
}

// has: the weight above which a pixel counts as drawn on.
__device__ __forceinline__ void pix_store(const PixAcc &p, float has, const pm_camera &cam, const pm_render_params &rp,
                                          int px, int py, float *img) {
    if (px >= cam.width || py >= cam.height) return;
    const float cover = 1.0f - p.rev;
    const float csum[3] = {p.c0, p.c1, p.c2};
    float *o = img + 3 * ((long long)py * cam.width + px);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float rgb = p.w > has ? csum[c] / p.w : rp.bg[c];
        const float v = rgb * cover + rp.bg[c] * (1.0f - cover);
        o[c] = v < 0.0f ? 0.0f : (v > 1.0f ? 1.0f : v);
    }
}

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
constexpr float kLog2e = 1.4426950408889634f, kMaxRange = 60.0f;

struct PartShared {                       // one warp's splats
    float4 a[32];                         // {u, v, c00, c01}
    float4 b[32];                         // {u0 + 0.5, v0 + 0.5, rad, blue}
    float4 c[32];                         // {c11, c11, depth weight, depth weight}
    float4 d[32];                         // {red, red, green, green}
};

// Whether a splat can count at a pixel of the part with first pixel (x0, y0): the
// footprint square, and the largest power over the part's rectangle of pixel
// centres, 0 with the splat's centre inside, else on the sides that face it; below
// -6 (alpha 0.0025, under 1/255), rounding aside, it cannot.
__device__ __forceinline__ bool reaches(const float4 &P0, const float4 &P1, const float4 &P2, int x0, int y0) {
    const int u0 = __float_as_int(P1.z), v0 = __float_as_int(P1.w), rd = __float_as_int(P2.w);
    const float X0 = ((float)x0 + 0.5f) - P0.x, X1 = X0 + (float)(kSubTile - 1);
    const float Y0 = ((float)y0 + 0.5f) - P0.y, Y1 = Y0 + (float)(kSubTile - 1);
    const float ex = fminf(fmaxf(0.0f, X0), X1), ey = fminf(fmaxf(0.0f, Y0), Y1);
    const float a = P0.z, b = P0.w, c = P1.x, inf = __int_as_float(0x7f800000);
    const float sy = fminf(fmaxf(__fdividef(-b * ex, c), Y0), Y1);
    const float sx = fminf(fmaxf(__fdividef(-b * ey, a), X0), X1);
    const float fx = -0.5f * (a * ex * ex + c * sy * sy) - b * ex * sy;
    const float fy = -0.5f * (a * sx * sx + c * ey * ey) - b * sx * ey;
    float most = ex != 0.0f ? fx : -inf;
    if (ey != 0.0f) most = fmaxf(most, fy);
    if (ex == 0.0f && ey == 0.0f) most = 0.0f;
    const float size = a * fmaxf(ex * ex, sx * sx) + c * fmaxf(ey * ey, sy * sy);
    const bool sane = a > 1e-20f && c > 1e-20f && size < 1e20f;
    return u0 + rd >= x0 && u0 - rd <= x0 + kSubTile - 1 && v0 + rd >= y0 && v0 - rd <= y0 + kSubTile - 1 &&
           !(sane && most < -6.0f - 1e-5f * size);
}

__device__ __noinline__ void draw_part_general(const pm_camera &cam, const pm_render_params &rp, const RenderWS &r,
                                               PartShared &sh, unsigned beg, unsigned end, float inv_tau, int x0,
                                               int y0, int px, int py0, float *img) {
    const int lane = threadIdx.x & 31, py1 = py0 + 4;
    const float inf = __int_as_float(0x7f800000);
    PixAcc a = {inf, 0.0f, 0.0f, 0.0f, 0.0f, 1.0f}, b = a;
    for (unsigned base = beg; base < end; base += 32) {
        bool keep = base + lane < end;
        float4 P0, P1, P2;
        if (keep) {
            const long long g = r.tlist[base + lane];
            P0 = r.sp[3 * g];
            P1 = r.sp[3 * g + 1];
            P2 = r.sp[3 * g + 2];
            keep = reaches(P0, P1, P2, x0, y0);
        }
        const unsigned kept = __ballot_sync(0xffffffffu, keep);
        const int cnt = __popc(kept);
        __syncwarp();
        if (keep) {
            const int at = __popc(kept & lanemask_lt());
            sh.a[at] = P0;
            sh.b[at] = P1;
            sh.c[at] = P2;
        }
        __syncwarp();
        for (int j = 0; j < cnt; ++j) {
            const float4 A = sh.a[j], B = sh.b[j], Cc = sh.c[j];
            pix_add(a, A, B, Cc, px, py0, inv_tau);
            pix_add(b, A, B, Cc, px, py1, inv_tau);
        }
    }
    pix_store(a, 1e-8f, cam, rp, px, py0, img);
    pix_store(b, 1e-8f, cam, rp, px, py1, img);
}

// The part with first pixel (x0, y0); false: left to draw_part_general.
__device__ __forceinline__ bool draw_part(const pm_camera &cam, const pm_render_params &rp, const RenderWS &r,
                                          PartShared &sh, unsigned beg, unsigned end, float inv_tau, int x0, int y0,
                                          int px, int py0, float *img) {
    const int lane = threadIdx.x & 31;
    const unsigned all = 0xffffffffu;
    const float inf = __int_as_float(0x7f800000);
    const float pxc = (float)px + 0.5f, pyc0 = (float)py0 + 0.5f, pyc1 = (float)(py0 + 4) + 0.5f;
    const float tau2 = inv_tau * kLog2e;
    float2 c0 = make_float2(0.0f, 0.0f), c1 = c0, c2 = c0, w = c0, rev = make_float2(1.0f, 1.0f);
    float zref = inf, zfar = 0.0f;
    // the splats of the next batch, and the ids of the one after, are on their way while one is drawn
    float4 P0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), P1 = P0, P2 = P0;
    auto fetch = [&](int g) {
        P0 = r.sp[3 * (long long)g];
        P1 = r.sp[3 * (long long)g + 1];
        P2 = r.sp[3 * (long long)g + 2];
    };
    if (beg + lane < end) fetch(r.tlist[beg + lane]);
    int g = beg + 32 + lane < end ? r.tlist[beg + 32 + lane] : 0;
    for (unsigned base = beg; base < end; base += 32) {
        bool keep = base + lane < end;
        const float z = P1.y;
        keep = keep && reaches(P0, P1, P2, x0, y0);
        const bool odd = keep && !(fabsf(P2.x) + fabsf(P2.y) + fabsf(P2.z) < inf && z > 0.0f);
        if (__any_sync(all, odd)) return false;
        const unsigned kept = __ballot_sync(all, keep);
        const int cnt = __popc(kept);
        if (cnt > 0) {
            const float zn = fminf(zref, __uint_as_float(__reduce_min_sync(all, keep ? __float_as_uint(z) : 0x7f800000u)));
            zfar = fmaxf(zfar, __uint_as_float(__reduce_max_sync(all, keep ? __float_as_uint(z) : 0u)));
            if (!((zfar - zn) * inv_tau <= kMaxRange)) return false;
            if (zn < zref) {
                // nothing to rescale the first time (and infinity times 1 / tau = 0, tau infinite, is not a number)
                const float sc = zref < inf ? ex2(-(zref - zn) * tau2) : 0.0f;
                const float2 sc2 = bc2(sc);
                c0 = mul2(c0, sc2);
                c1 = mul2(c1, sc2);
                c2 = mul2(c2, sc2);
                w = mul2(w, sc2);
                zref = zn;
            }
            __syncwarp();                                    // the batch before is drawn
            if (keep) {
                const int at = __popc(kept & lanemask_lt());
                // 2^t from its whole and its broken part: t itself is off by as many ulps as it is large
                const float dz = zref - z, t = dz * tau2, whole = rintf(t), part = fmaf(dz, tau2, -whole);
                const float e = ex2(part) * __int_as_float(((int)whole + 127) << 23);
                sh.a[at] = P0;
                sh.b[at] = make_float4((float)__float_as_int(P1.z) + 0.5f, (float)__float_as_int(P1.w) + 0.5f,
                                       (float)__float_as_int(P2.w), P2.z);
                sh.c[at] = make_float4(P1.x, P1.x, e, e);
                sh.d[at] = make_float4(P2.x, P2.x, P2.y, P2.y);
            }
            __syncwarp();
        }
        if (base + 32 + lane < end) fetch(g);
        g = base + 64 + lane < end ? r.tlist[base + 64 + lane] : 0;
#pragma unroll 2
        for (int j = 0; j < cnt; ++j) {
            const float4 A = sh.a[j], B = sh.b[j], C = sh.c[j], D = sh.d[j];
            const float dx = pxc - A.x;
            const float2 dy = make_float2(pyc0 - A.y, pyc1 - A.y);
            // power with pix_add's roundings, operation by operation: the same pixels pass 1/255
            const float2 q = fma2(bc2(A.z * dx), bc2(dx), mul2(mul2(make_float2(C.x, C.y), dy), dy));
            const float2 power = fma2(bc2(-0.5f), q, mul2(bc2(-(A.w * dx)), dy));
            const float2 p2 = mul2(make_float2(fminf(power.x, 0.0f), fminf(power.y, 0.0f)), bc2(kLog2e));
            float2 ga = make_float2(ex2(p2.x), ex2(p2.y));
            const bool in = fabsf(pxc - B.x) <= B.z;
            const bool on0 = in && fabsf(pyc0 - B.y) <= B.z && ga.x > (1.0f / 255.0f);
            const bool on1 = in && fabsf(pyc1 - B.y) <= B.z && ga.y > (1.0f / 255.0f);
            ga = make_float2(on0 ? ga.x : 0.0f, on1 ? ga.y : 0.0f);
            const float2 wt = mul2(ga, make_float2(C.z, C.w));
            c0 = fma2(make_float2(D.x, D.y), wt, c0);
            c1 = fma2(make_float2(D.z, D.w), wt, c1);
            c2 = make_float2(fmaf(B.w, wt.x, c2.x), fmaf(B.w, wt.y, c2.y));
            w = add2(w, wt);
            const float2 om = add2(bc2(1.0f), make_float2(-ga.x, -ga.y));
            rev = mul2(rev, make_float2(fmaxf(om.x, 1e-6f), fmaxf(om.y, 1e-6f)));
        }
    }
    pix_store(PixAcc{zref, c0.x, c1.x, c2.x, w.x, rev.x}, 0.0f, cam, rp, px, py0, img);
    pix_store(PixAcc{zref, c0.y, c1.y, c2.y, w.y, rev.y}, 0.0f, cam, rp, px, py0 + 4, img);
    return true;
}

__global__ void __launch_bounds__(32 * kTileWarps) k_splat_tiles(const pm_camera cam, const pm_render_params rp,
                                                                 const RenderWS r, float *__restrict__ img) {
    __shared__ PartShared sh[kTileWarps];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, tile = blockIdx.x;
    const int x0 = (tile % r.ntx) * kTile + (wid & 1) * kSubTile, y0 = (tile / r.ntx) * kTile + (wid >> 1) * kSubTile;
    if (x0 >= cam.width || y0 >= cam.height) return;   // whole warps only; no block-wide barrier below
    const int px = x0 + (lane & (kSubTile - 1)), py0 = y0 + (lane >> 3);
    const unsigned beg = r.tstart[tile], end = beg + r.tcnt[tile];
    const float inv_tau = r.tau[1];
    if (!draw_part(cam, rp, r, sh[wid], beg, end, inv_tau, x0, y0, px, py0, img))
        draw_part_general(cam, rp, r, sh[wid], beg, end, inv_tau, x0, y0, px, py0, img);
}

struct RenderLayout {
    size_t sp, count, tau, keys, hist, tcnt, tfill, tstart, tlist, total;
    long long cap;
    int ntx, nty;
};

// Tiles a footprint square of side 2 r_max + 1 can touch, per axis:
// floor(2 r_max / kTile) + 2, and never more than the screen has.
RenderLayout make_render_layout(long long n, int width, int height, int r_max) {
    RenderLayout R;
    R.ntx = (width + kTile - 1) / kTile;
    R.nty = (height + kTile - 1) / kTile;
    const long long ntiles = (long long)R.ntx * R.nty;
    const long long per_axis = 2LL * (r_max > 1 ? r_max : 1) / kTile + 2;
    const long long per = std::min(per_axis, (long long)R.ntx) * std::min(per_axis, (long long)R.nty);
    R.cap = std::max<long long>(1, n * per);
    const size_t A = 256, nn = (size_t)(n > 0 ? n : 1), nt = (size_t)ntiles;
    size_t o = 0;
    R.sp = o;     o = align_up(o + 48 * nn, A);
    R.count = o;  o = align_up(o + 16, A);
    R.tau = o;    o = align_up(o + 16, A);
    R.keys = o;   o = align_up(o + 4 * nn, A);
    R.hist = o;   o = align_up(o + 4 * kMedianWords, A);
    R.tcnt = o;   o = align_up(o + 4 * nt, A);
    R.tfill = o;  o = align_up(o + 4 * nt, A);
    R.tstart = o; o = align_up(o + 4 * nt, A);
    R.tlist = o;  o = align_up(o + 4 * (size_t)R.cap, A);
    R.total = o;
    return R;
}


// Gaussian carrying (run_orange.py:116-133): gaussian i bound to particle
// b = bind[i] moves with the particle's affine motion: position
// A (x_b) + t + F_b off0_i, covariance F_b cov0_i F_b^T, colour darkened by
// damage, color0_i (1 - tint d_b).
__global__ void __launch_bounds__(256) k_carry(const Parts P, const int *__restrict__ bind, const float *__restrict__ off0,
                                               const float *__restrict__ cov0, const float *__restrict__ color0,
                                               long long g_n, const float *__restrict__ affine, float tint,
                                               float *__restrict__ pos, float *__restrict__ cov,
                                               float *__restrict__ color) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g_n) return;
    const long long b = bind[i];
    if (b < 0 || b >= P.n) {   // an unbound gaussian: NaN outputs (the host wrapper rejects such bindings)
        const float q = __int_as_float(0x7fc00000);
#pragma unroll
        for (int k = 0; k < 3; ++k) pos[3 * i + k] = color[3 * i + k] = q;
#pragma unroll
        for (int k = 0; k < 9; ++k) cov[9 * i + k] = q;
        return;
    }
    const long long ps = P.ps;
    float F[9], xp[3];
#pragma unroll
    for (int k = 0; k < 9; ++k) F[k] = P.F[k * ps + b];
#pragma unroll
    for (int a = 0; a < 3; ++a) xp[a] = P.x[a * ps + b];
    const float o[3] = {off0[3 * i], off0[3 * i + 1], off0[3 * i + 2]};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float w = (affine[4 * a] * xp[0] + affine[4 * a + 1] * xp[1] + affine[4 * a + 2] * xp[2]) + affine[4 * a + 3];
        pos[3 * i + a] = w + (F[3 * a] * o[0] + F[3 * a + 1] * o[1] + F[3 * a + 2] * o[2]);
    }
    float S[9], T1[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) S[k] = cov0[9 * i + k];
    mm3(F, S, T1);
    mmt3(T1, F, S);
#pragma unroll
    for (int k = 0; k < 9; ++k) cov[9 * i + k] = S[k];
    const float shade = tint > 0.0f ? 1.0f - tint * P.d[b] : 1.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c) color[3 * i + c] = color0[3 * i + c] * shade;
}

}  // namespace

void launch_carry(const Parts &P, const int *bind, const float *off0, const float *cov0, const float *color0,
                  long long g_n, const float *affine, float tint, float *pos, float *cov, float *color,
                  cudaStream_t s) {
    if (g_n <= 0) return;
    k_carry<<<(unsigned)((g_n + 255) / 256), 256, 0, s>>>(P, bind, off0, cov0, color0, g_n, affine, tint, pos, cov,
                                                          color);
}

size_t render_workspace_bytes(long long n, int width, int height, int r_max) {
    return make_render_layout(n, width, height, r_max).total;
}

void launch_render(const pm_camera &cam, const pm_render_params &rp, const float *xyz, const float *cov,
                   const float *color, long long n, float *img, void *ws, cudaStream_t s) {
    const RenderLayout L = make_render_layout(n, cam.width, cam.height, rp.r_max);
    char *b = (char *)ws;
    RenderWS r;
    r.sp = (float4 *)(b + L.sp);
    r.count = (unsigned *)(b + L.count);
    r.tau = (float *)(b + L.tau);
    r.keys = (unsigned *)(b + L.keys);
    r.hist = (unsigned *)(b + L.hist);
    r.tcnt = (unsigned *)(b + L.tcnt);
    r.tfill = (unsigned *)(b + L.tfill);
    r.tstart = (unsigned *)(b + L.tstart);
    r.tlist = (int *)(b + L.tlist);
    r.cap = L.cap;
    r.ntx = L.ntx;
    r.nty = L.nty;
    const int ntiles = L.ntx * L.nty;
    k_splat_clear<<<(unsigned)((std::max(ntiles, kMedianWords) + 255) / 256), 256, 0, s>>>(r, ntiles, rp.tau);
    if (n > 0) k_splat_project<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(cam, rp, xyz, cov, color, n, r);
    if (!(rp.tau > 0.0f) && n > 0) {
        const unsigned ctas = (unsigned)std::min<long long>((n + 4 * kMedianThreads - 1) / (4 * kMedianThreads), 148LL);
        k_median<0><<<ctas, kMedianThreads, 0, s>>>(r, n);
        k_median<1><<<ctas, kMedianThreads, 0, s>>>(r, n);
        k_median<2><<<ctas, kMedianThreads, 0, s>>>(r, n);
    }
    k_tile_alloc<<<(unsigned)((ntiles + 255) / 256), 256, 0, s>>>(r, ntiles);
    if (n > 0) k_splat_emit<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(cam, n, r);
    k_splat_tiles<<<(unsigned)ntiles, 32 * kTileWarps, 0, s>>>(cam, rp, r, img);
}

}  // namespace pm
