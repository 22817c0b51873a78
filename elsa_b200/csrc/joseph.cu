// Joseph's method (driving-direction ray stepping with bilinear interpolation) for sm_100a.
//
// Reference semantics: projectors/JosephsMethod.cpp:37-198 and
// projectors/DrivingDirectionTraversal.cpp:6-106 (elsa's CPU path, the parity target). Per ray r
// with n samples and step length L:
//   forward  y[r] = L * sum_j bilinear(x, plane k0 + j*dir, (pa_j, pb_j))
//   adjoint  x[v] = sum_r sum_j y[r] * L * w_v(r, j)
// Taps outside the volume contribute zero (the reference masks them, :60-97).
//
// Sample positions. The reference advances pos += step in float after every sample
// (DrivingDirectionTraversal.cpp:265). With a constant step every addition rounds the same way
// inside a binade, so the accumulated position drifts linearly from pos0 + j*step (about 1e-3
// voxel after 256 steps at 256^3) -- far more than the 1e-5 parity budget allows. Both kernels
// therefore reproduce the accumulation bit for bit: the forward accumulates along each ray, and
// the adjoint starts every ray segment from a checkpoint (the exact accumulated position at the
// ray's first sample in each slab of kCheckpointDepth planes, computed once per geometry) and
// accumulates from there.
//
// Forward: joseph_tma.cu in 3D; in 2D a warp takes 32 neighbouring rays through a checkpoint slab,
// reading zero-padded copies of the image's rows and columns (the image itself for small problems).
//
// Adjoint (default): atomic-free and deterministic. Each warp owns one brick (2D: tile) of the
// volume in shared memory for a chunk of the views. For every view it visits the rays of the
// brick's detector window so that lanes never meet: rays whose pixel indices are congruent modulo
// m stay more than two voxels apart on every plane (m is validated per geometry at construction),
// so their bilinear taps never overlap and shared memory is updated without atomics. In 3D the
// lanes take one such class at a time; in 2D 32 neighbouring rays, those of different classes on
// different planes. Every voxel receives its contributions in a fixed order, with the positions
// and weights of the forward kernel.
// The launch knob kKnobAdjointScatter = 1 selects a thread-per-ray scatter instead (the forward's
// sample loop with atomic adds to the four taps), slower in 2D (512^2 / 720 views: 1.74 ms against
// 0.54) and 3D, where four global atomics per sample exceed what the L2 sustains. A shared-memory
// variant (several warps per brick adding with shared atomics, no ray classes) measured 65.5 ms
// against 54.8 ms at 256^3 / 360 views and was dropped.
#include "joseph_tma.cuh"
#include "projector.hpp"
#include "raysetup.cuh"
#include "solvers.hpp"

#include <algorithm>
#include <atomic>
#include <mutex>
#include <cmath>
#include <cstring>

#ifndef ELSA_ADJ_MIN_BLOCKS
#define ELSA_ADJ_MIN_BLOCKS 1 // resident one-warp blocks per SM asked of the register allocator
#endif
#ifndef ELSA_ADJ_BATCH
#define ELSA_ADJ_BATCH 3 // class rays per lane fetched together by the adjoints (3D axis bricks at 256^3 / 360 views: 1: 37.5 ms, 2: 33.5, 3: 33.0)
#endif
#ifndef ELSA_AXIS_TD
#define ELSA_AXIS_TD 16 // depth along the driving axis of the 3D adjoint's axis bricks
#endif
#ifndef ELSA_AXIS_TW
#define ELSA_AXIS_TW 32 // edge along the non-driving axis over which a detector row's rays spread
#endif
#ifndef ELSA_AXIS_TV
#define ELSA_AXIS_TV 8 // edge along the other non-driving axis
#endif
#ifndef ELSA_SPLAT_UNROLL
#define ELSA_SPLAT_UNROLL 2 // unroll factor of the adjoint's per-sample loop (1: 72.8 ms, 2: 63.4 ms, 4: 68.9 ms at 256^3)
#endif

namespace elsa_b200
{
    namespace
    {
        constexpr int kForwardThreads = 256;    // default rays per block of the gather forward
        constexpr int kMaxForwardThreads = 512; // largest block the autotuner may choose
        constexpr int kSplatUnroll = ELSA_SPLAT_UNROLL;
        constexpr int kMinClass = 2;
        constexpr int kMaxClass = 8;
        // Joseph brick windows: the brick grown by half a voxel (the reach of a bilinear tap)
        // plus slack for the accumulated-position drift (at most n steps of half an ulp of a
        // coordinate below n: n^2 2^-24 voxel, 0.004 at n = 256), doubled, and 0.05 voxel for the
        // rounding of the float rays; 0.05 pixel of margin for the projection of the corners.
        inline float windowGrow(const VolumeShape& vol)
        {
            const float n = static_cast<float>(std::max(vol.n[0], std::max(vol.n[1], vol.n[2])));
            return 0.55f + 2.0f * n * n * 5.9604645e-8f;
        }
        constexpr float kWindowPixelMargin = 0.05f;

        struct Weights {
            int ia, ib;
            float wa, cwa, wb, cwb;
        };

        // Bilinear weights at non-driving position (pa, pb), as JosephsMethod.cpp:37-52:
        // floor of pos - 0.5, complement weight (pos - floor) - 0.5, weight 1 - complement.
        __device__ __forceinline__ void tapWeights(float pa, float pb, Weights& w)
        {
            const float fa = floorf(__fsub_rn(pa, 0.5f));
            const float fb = floorf(__fsub_rn(pb, 0.5f));
            w.cwa = __fsub_rn(__fsub_rn(pa, fa), 0.5f);
            w.cwb = __fsub_rn(__fsub_rn(pb, fb), 0.5f);
            w.wa = __fsub_rn(1.0f, w.cwa);
            w.wb = __fsub_rn(1.0f, w.cwb);
            w.ia = static_cast<int>(fa);
            w.ib = static_cast<int>(fb);
        }

        __device__ __forceinline__ int floorDiv(int a, int b)
        {
            return a >= 0 ? a / b : -((-a + b - 1) / b);
        }

        // Adjoint by atomic scatter: the forward's sample loop, one thread per ray, adding
        // y[r] * len * (tap weight) to the in-volume taps of every sample (x zeroed beforehand);
        // the tap values are those of the brick-owner adjoint, the order of the additions varies.
        template <int DIM>
        __global__ void __launch_bounds__(kMaxForwardThreads)
            josephScatterKernel(const JosephRay* __restrict__ rays, int64_t nrays,
                                const float* __restrict__ y, VolumeShape vol,
                                float* __restrict__ x)
        {
            const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (r >= nrays)
                return;
            const JosephRay R = rays[r];
            if (R.n == 0)
                return;
            const float yl = __ldg(y + r) * R.len;
            if (yl == 0.0f)
                return;
            const int g = R.meta & 3;
            const int dir = (R.meta & 4) ? -1 : 1;
            int a, b;
            nonDrivingAxes(g, a, b);
            const int64_t plane = static_cast<int64_t>(vol.n[0]) * vol.n[1];
            const int64_t sg = g == 0 ? 1 : (g == 1 ? vol.n[0] : plane);
            const int64_t sa = a == 0 ? 1 : (a == 1 ? vol.n[0] : plane);
            const int ng = g == 0 ? vol.n[0] : (g == 1 ? vol.n[1] : vol.n[2]);
            const int na = a == 0 ? vol.n[0] : (a == 1 ? vol.n[1] : vol.n[2]);
            const int64_t sb = DIM == 3 ? (b == 1 ? vol.n[0] : plane) : 0;
            const int nb = DIM == 3 ? (b == 1 ? vol.n[1] : vol.n[2]) : 1;
            float pa = R.pa, pb = R.pb;
            int k = R.k0;
            for (int j = 0; j < R.n; ++j, k += dir, pa = __fadd_rn(pa, R.sa),
                     pb = __fadd_rn(pb, R.sb)) {
                if (static_cast<unsigned>(k) >= static_cast<unsigned>(ng))
                    continue;
                Weights w;
                tapWeights(pa, pb, w);
                float* base = x + k * sg;
                const bool a0 = static_cast<unsigned>(w.ia) < static_cast<unsigned>(na);
                const bool a1 = static_cast<unsigned>(w.ia + 1) < static_cast<unsigned>(na);
                if (DIM == 2) {
                    if (a0)
                        atomicAdd(base + w.ia * sa, yl * w.wa);
                    if (a1)
                        atomicAdd(base + (w.ia + 1) * sa, yl * w.cwa);
                } else {
                    const bool b0 = static_cast<unsigned>(w.ib) < static_cast<unsigned>(nb);
                    const bool b1 = static_cast<unsigned>(w.ib + 1) < static_cast<unsigned>(nb);
                    float* p0 = base + w.ia * sa + w.ib * sb;
                    if (a0 && b0)
                        atomicAdd(p0, yl * (w.wa * w.wb));
                    if (a1 && b0)
                        atomicAdd(p0 + sa, yl * (w.cwa * w.wb));
                    if (a0 && b1)
                        atomicAdd(p0 + sb, yl * (w.wa * w.cwb));
                    if (a1 && b1)
                        atomicAdd(p0 + sa + sb, yl * (w.cwa * w.cwb));
                }
            }
        }

        // elsa's default CUDA adjoint (JosephsMethodCUDA with fast = true,
        // TraverseJosephsCUDA.cu:218-287): a voxel-driven backprojection, not the transpose of the
        // forward. For voxel centre c and view p: pixel = B_p (c - o_p) with B_p the leading
        // DIM x DIM block of the projection matrix and o_p = -Binv_p p4_p, divided by its last
        // coordinate; the sinogram is read through a layered texture (linear filtering, border
        // addressing) and the views are summed in order. The float operations are the reference
        // kernel's: its x coordinates come from 32 lanes per (y, z) row, lane t taking voxels
        // t + 32 s and advancing the first difference by adding 32 once per step s (voxels past
        // the last multiple of 32 computed directly), and its matrix-vector product
        // ((b0 r0 + b1 r1) + b2 r2, Matrix.cuh:12-32) is contracted as fma(b2, r2, fma(b0, r0,
        // b1 r1)). The layout is the reference's too, a row per 32 lanes, but with kRows rows per
        // block and the sums of kChunk steps in registers instead of shared memory.
        template <int DIM>
        __device__ __forceinline__ float fastSample(cudaTextureObject_t sino, const float* T,
                                                    float r0, float r1, float r2, int p)
        {
            if (DIM == 3) {
                const float q0 = __fmaf_rn(T[6], r2, __fmaf_rn(T[0], r0, __fmul_rn(T[3], r1)));
                const float q1 = __fmaf_rn(T[7], r2, __fmaf_rn(T[1], r0, __fmul_rn(T[4], r1)));
                const float q2 = __fmaf_rn(T[8], r2, __fmaf_rn(T[2], r0, __fmul_rn(T[5], r1)));
                return tex2DLayered<float>(sino, __fdiv_rn(q0, q2), __fdiv_rn(q1, q2), p);
            }
            const float q0 = __fmaf_rn(T[0], r0, __fmul_rn(T[2], r1));
            const float q1 = __fmaf_rn(T[1], r0, __fmul_rn(T[3], r1));
            return tex1DLayered<float>(sino, __fdiv_rn(q0, q1), p);
        }

        constexpr int kFastRows = 4;   // (y, z) rows per block of the fast adjoint
        constexpr int kFastChunk = 8;  // steps per lane summed in registers at once

        template <int DIM>
        __global__ void __launch_bounds__(32 * kFastRows)
            josephFastAdjointKernel(cudaTextureObject_t sino, const float* __restrict__ table,
                                    int np, VolumeShape vol, float* __restrict__ x)
        {
            constexpr int kT = DIM == 3 ? 12 : 6; // block (column-major) + origin
            extern __shared__ float tab[];        // kT floats per view
            for (int i = threadIdx.y * 32 + threadIdx.x; i < kT * np; i += 32 * kFastRows)
                tab[i] = table[i];
            __syncthreads();
            const int lane = threadIdx.x;
            const int row = blockIdx.x * kFastRows + threadIdx.y;
            const int nrows = vol.n[1] * (DIM == 3 ? vol.n[2] : 1);
            if (row >= nrows)
                return;
            // rows z fastest, as the reference's grid: neighbouring blocks then read neighbouring
            // detector rows of a view through the texture cache
            const int nz = DIM == 3 ? vol.n[2] : 1;
            const int zi = row % nz, yi = row / nz;
            const int nsteps = vol.n[0] / 32, rem = vol.n[0] - nsteps * 32;
            const float c1 = static_cast<float>(yi) + 0.5f;
            const float c2 = static_cast<float>(zi) + 0.5f;
            float* out = x + static_cast<int64_t>(vol.n[0]) * (yi + static_cast<int64_t>(vol.n[1]) * zi);
            const float c0 = static_cast<float>(lane) + 0.5f;
            for (int s0 = 0; s0 < nsteps; s0 += kFastChunk) {
                const int cnt = min(kFastChunk, nsteps - s0);
                float acc[kFastChunk];
#pragma unroll
                for (int k = 0; k < kFastChunk; ++k)
                    acc[k] = 0.0f;
                for (int p = 0; p < np; ++p) {
                    const float* T = tab + kT * p;
                    float r0 = __fsub_rn(c0, T[DIM * DIM]);
                    for (int s = 0; s < s0; ++s)
                        r0 = __fadd_rn(r0, 32.0f);
                    const float r1 = __fsub_rn(c1, T[DIM * DIM + 1]);
                    const float r2 = DIM == 3 ? __fsub_rn(c2, T[11]) : 0.0f;
#pragma unroll
                    for (int k = 0; k < kFastChunk; ++k) {
                        if (k < cnt)
                            acc[k] = __fadd_rn(acc[k], fastSample<DIM>(sino, T, r0, r1, r2, p));
                        r0 = __fadd_rn(r0, 32.0f);
                    }
                }
#pragma unroll
                for (int k = 0; k < kFastChunk; ++k)
                    if (k < cnt)
                        out[lane + 32 * (s0 + k)] = acc[k];
            }
            if (lane < rem) {
                const int xi = nsteps * 32 + lane;
                const float cr = static_cast<float>(xi) + 0.5f;
                float acc = 0.0f;
                for (int p = 0; p < np; ++p) {
                    const float* T = tab + kT * p;
                    const float r0 = __fsub_rn(cr, T[DIM * DIM]);
                    const float r1 = __fsub_rn(c1, T[DIM * DIM + 1]);
                    const float r2 = DIM == 3 ? __fsub_rn(c2, T[11]) : 0.0f;
                    acc = __fadd_rn(acc, fastSample<DIM>(sino, T, r0, r1, r2, p));
                }
                out[xi] = acc;
            }
        }

        // Detector window of every (brick, view): projection of the brick grown by one voxel,
        // plus one pixel of margin. Falls back to the whole detector when a corner lies behind
        // the source.
        // Number of entries of the ascending table t[0..n) that are < x (le: <= x).
        __device__ __forceinline__ int countBelow(const float* __restrict__ t, int n, float x,
                                                  bool le)
        {
            int lo = 0, hi = n;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (le ? (t[mid] <= x) : (t[mid] < x))
                    lo = mid + 1;
                else
                    hi = mid;
            }
            return lo;
        }

        // grow > 0 (tight mode, flat detectors): the window holds exactly the pixels whose
        // centres lie in the projection of the brick grown by `grow` voxels on every side, plus
        // `pixMargin` pixels (the float rays deviate from the exact pixel-centre rays by far less
        // than both). A Joseph sample on driving plane k touches the brick only if its position
        // lies within half a voxel of the brick in both non-driving axes (taps floor(p - 0.5)
        // and floor(p - 0.5) + 1), so grow = 0.5 plus the accumulated-position slack suffices.
        // grow = 0: the conservative window (brick grown by one voxel, one pixel of margin).
        __global__ void josephWindowKernel(const float* __restrict__ poses, VolumeShape vol,
                                           DetectorShape det, int3 brick, int3 nBricks,
                                           CurvedMap cm, float grow, float pixMargin,
                                           RayWindow* __restrict__ out)
        {
            const int nb = nBricks.x * nBricks.y * nBricks.z;
            const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (t >= static_cast<int64_t>(nb) * det.np)
                return;
            const int bi = static_cast<int>(t % nb);
            const int p = static_cast<int>(t / nb);
            const float* P = poses + static_cast<int64_t>(p) * 40;
            const int bxi = bi % nBricks.x, byi = (bi / nBricks.x) % nBricks.y,
                      bzi = bi / (nBricks.x * nBricks.y);
            const bool tight = grow > 0.0f && !cm.planarU;
            const float g = tight ? grow : 1.0f;
            const float lo0 = static_cast<float>(bxi * brick.x) - g;
            const float lo1 = static_cast<float>(byi * brick.y) - g;
            const float lo2 = static_cast<float>(bzi * brick.z) - g;
            const float hi0 = static_cast<float>(bxi * brick.x + brick.x) + g;
            const float hi1 = static_cast<float>(byi * brick.y + brick.y) + g;
            const float hi2 = static_cast<float>(bzi * brick.z + brick.z) + g;
            float umin = 1e30f, umax = -1e30f, vmin = 1e30f, vmax = -1e30f;
            bool behind = false;
            const int corners = vol.dim == 3 ? 8 : 4;
            for (int c = 0; c < corners; ++c) {
                const float X = (c & 1) ? hi0 : lo0;
                const float Y = (c & 2) ? hi1 : lo1;
                if (vol.dim == 3) {
                    const float Z = (c & 4) ? hi2 : lo2;
                    const float h0 = P[0] * X + P[1] * Y + P[2] * Z + P[3];
                    const float h1 = P[4] * X + P[5] * Y + P[6] * Z + P[7];
                    const float h2 = P[8] * X + P[9] * Y + P[10] * Z + P[11];
                    if (!(h2 > 1e-6f)) {
                        behind = true;
                        break;
                    }
                    const float u = h0 / h2, v = h1 / h2;
                    umin = fminf(umin, u), umax = fmaxf(umax, u);
                    vmin = fminf(vmin, v), vmax = fmaxf(vmax, v);
                } else {
                    const float h0 = P[0] * X + P[1] * Y + P[2];
                    const float h1 = P[3] * X + P[4] * Y + P[5];
                    if (!(h1 > 1e-6f)) {
                        behind = true;
                        break;
                    }
                    const float u = h0 / h1;
                    umin = fminf(umin, u), umax = fmaxf(umax, u);
                    vmin = 0.0f, vmax = 0.0f;
                }
            }
            RayWindow w;
            if (behind) {
                w.u0 = 0, w.u1 = det.nu - 1, w.v0 = 0, w.v1 = det.nv - 1;
            } else if (cm.planarU) {
                // curved detector: the rays of pixel column u pass planar coordinate
                // planarU[u] (ascending), and rows are stretched by a factor in [fmin, fmax]
                // about the detector's centre row
                const int below = countBelow(cm.planarU, det.nu, umin, true);
                const int before = countBelow(cm.planarU, det.nu, umax, false);
                w.u0 = max(0, below - 2);
                w.u1 = min(det.nu - 1, before + 1);
                if (vol.dim == 3) {
                    const float cy = 0.5f * static_cast<float>(det.nv);
                    const float lo = cy + fminf((vmin - cy) / cm.fmin, (vmin - cy) / cm.fmax);
                    const float hi = cy + fmaxf((vmax - cy) / cm.fmin, (vmax - cy) / cm.fmax);
                    const float vLo = fmaxf(floorf(lo - 0.5f) - 1.0f, -1.0f);
                    const float vHi = fminf(ceilf(hi - 0.5f) + 1.0f, static_cast<float>(det.nv));
                    w.v0 = max(0, static_cast<int>(vLo));
                    w.v1 = min(det.nv - 1, static_cast<int>(vHi));
                } else {
                    w.v0 = 0, w.v1 = 0;
                }
            } else if (tight) {
                // pixels whose centres i + 0.5 lie in [umin - margin, umax + margin]
                const float uLo = fmaxf(ceilf(umin - 0.5f - pixMargin), -1.0f);
                const float uHi = fminf(floorf(umax - 0.5f + pixMargin), static_cast<float>(det.nu));
                w.u0 = max(0, static_cast<int>(uLo));
                w.u1 = min(det.nu - 1, static_cast<int>(uHi));
                if (vol.dim == 3) {
                    const float vLo = fmaxf(ceilf(vmin - 0.5f - pixMargin), -1.0f);
                    const float vHi =
                        fminf(floorf(vmax - 0.5f + pixMargin), static_cast<float>(det.nv));
                    w.v0 = max(0, static_cast<int>(vLo));
                    w.v1 = min(det.nv - 1, static_cast<int>(vHi));
                } else {
                    w.v0 = 0, w.v1 = 0;
                }
            } else {
                // pixel i has its centre at i + 0.5
                const float uLo = fmaxf(floorf(umin - 0.5f) - 1.0f, -1.0f);
                const float uHi = fminf(ceilf(umax - 0.5f) + 1.0f, static_cast<float>(det.nu));
                w.u0 = max(0, static_cast<int>(uLo));
                w.u1 = min(det.nu - 1, static_cast<int>(uHi));
                if (vol.dim == 3) {
                    const float vLo = fmaxf(floorf(vmin - 0.5f) - 1.0f, -1.0f);
                    const float vHi =
                        fminf(ceilf(vmax - 0.5f) + 1.0f, static_cast<float>(det.nv));
                    w.v0 = max(0, static_cast<int>(vLo));
                    w.v1 = min(det.nv - 1, static_cast<int>(vHi));
                } else {
                    w.v0 = 0, w.v1 = 0;
                }
            }
            out[t] = w;
        }

        // Check of the brick windows (test support, elsa_projector_info key 8): every tap of
        // every sample must lie in a brick whose window for the ray's view contains the ray.
        // Counts the taps that violate this.
        __global__ void josephWindowCheckKernel(const JosephRay* __restrict__ rays,
                                                const RayWindow* __restrict__ windows,
                                                VolumeShape vol, DetectorShape det, int3 brick,
                                                int3 nBricks, int onlyAxis,
                                                unsigned long long* __restrict__ misses)
        {
            const int64_t nrays = static_cast<int64_t>(det.nu) * det.nv * det.np;
            const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (r >= nrays)
                return;
            const JosephRay R = rays[r];
            if (R.n == 0 || (onlyAxis >= 0 && (R.meta & 3) != onlyAxis))
                return;
            const int u = static_cast<int>(r % det.nu);
            const int v = static_cast<int>((r / det.nu) % det.nv);
            const int p = static_cast<int>(r / (static_cast<int64_t>(det.nu) * det.nv));
            const int nb = nBricks.x * nBricks.y * nBricks.z;
            const int g = R.meta & 3;
            const int dir = (R.meta & 4) ? -1 : 1;
            int a, b;
            nonDrivingAxes(g, a, b);
            const int bext[3] = {brick.x, brick.y, brick.z};
            float pa = R.pa, pb = R.pb;
            int k = R.k0;
            unsigned long long bad = 0;
            int lastBrick = -1;
            for (int j = 0; j < R.n; ++j, k += dir, pa = __fadd_rn(pa, R.sa),
                     pb = __fadd_rn(pb, R.sb)) {
                const int ia = static_cast<int>(floorf(__fsub_rn(pa, 0.5f)));
                const int ib = static_cast<int>(floorf(__fsub_rn(pb, 0.5f)));
                for (int t = 0; t < (vol.dim == 3 ? 4 : 2); ++t) {
                    int c[3];
                    c[g] = k;
                    c[a] = ia + (t & 1);
                    if (vol.dim == 3)
                        c[b] = ib + (t >> 1);
                    else
                        c[2] = 0;
                    bool in = true;
                    for (int i = 0; i < vol.dim; ++i)
                        in = in && c[i] >= 0 && c[i] < vol.n[i];
                    if (!in)
                        continue;
                    const int bi = c[0] / bext[0] + nBricks.x *
                                   (c[1] / bext[1] + nBricks.y * (vol.dim == 3 ? c[2] / bext[2] : 0));
                    if (bi == lastBrick)
                        continue;
                    const RayWindow w = windows[static_cast<int64_t>(p) * nb + bi];
                    if (u < w.u0 || u > w.u1 || v < w.v0 || v > w.v1)
                        ++bad;
                    else
                        lastBrick = bi;
                }
            }
            if (bad)
                atomicAdd(misses, bad);
        }

        // Approximate non-driving position of ray R on driving plane k (pos0 + j*step). It
        // differs from the accumulated position by at most n/2 ulp, which the separation margin
        // below absorbs.
        __device__ __forceinline__ float planePos(const JosephRay& R, int k, bool second)
        {
            const int dir = (R.meta & 4) ? -1 : 1;
            const float fj = static_cast<float>((k - R.k0) * dir);
            return second ? fmaf(fj, R.sb, R.pb) : fmaf(fj, R.sa, R.pa);
        }

        // True when rays R and S (same driving axis) stay more than two voxels apart in one
        // non-driving coordinate over their common planes, so their bilinear taps are disjoint.
        __device__ bool separated(const JosephRay& R, const JosephRay& S, int dim)
        {
            const int dr = (R.meta & 4) ? -1 : 1, ds = (S.meta & 4) ? -1 : 1;
            const int r0 = R.k0, r1 = R.k0 + (R.n - 1) * dr;
            const int s0 = S.k0, s1 = S.k0 + (S.n - 1) * ds;
            const int lo = max(min(r0, r1), min(s0, s1));
            const int hi = min(max(r0, r1), max(s0, s1));
            if (lo > hi)
                return true;
            const float margin = 2.05f;
            const float da0 = planePos(R, lo, false) - planePos(S, lo, false);
            const float da1 = planePos(R, hi, false) - planePos(S, hi, false);
            if ((da0 > margin && da1 > margin) || (da0 < -margin && da1 < -margin))
                return true;
            if (dim == 3) {
                const float db0 = planePos(R, lo, true) - planePos(S, lo, true);
                const float db1 = planePos(R, hi, true) - planePos(S, hi, true);
                if ((db0 > margin && db1 > margin) || (db0 < -margin && db1 < -margin))
                    return true;
            }
            return false;
        }

        // Records the driving axes present per view and, per candidate class spacing m, whether
        // two same-class neighbours could share a bilinear tap.
        __global__ void josephClassCheckKernel(const JosephRay* __restrict__ rays,
                                               DetectorShape det, int dim,
                                               unsigned* __restrict__ viewAxes,
                                               unsigned* __restrict__ badSpacing,
                                               unsigned long long* __restrict__ samples)
        {
            const int64_t nrays = static_cast<int64_t>(det.nu) * det.nv * det.np;
            const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (r >= nrays)
                return;
            const JosephRay R = rays[r];
            if (R.n == 0)
                return;
            const int u = static_cast<int>(r % det.nu);
            const int v = static_cast<int>((r / det.nu) % det.nv);
            const int p = static_cast<int>(r / (static_cast<int64_t>(det.nu) * det.nv));
            atomicOr(viewAxes + p, 1u << (R.meta & 3));
            atomicAdd(samples, static_cast<unsigned long long>(R.n));
            unsigned bad = 0;
            for (int m = kMinClass; m <= kMaxClass; ++m) {
                // pairs that the adjoint may process concurrently: same row m apart, and rows m
                // apart with any offset inside a 32-ray segment (plus one)
                const int noffs = dim == 3 ? 2 + 65 : 1;
                for (int o = 0; o < noffs; ++o) {
                    const int du = o == 0 ? m : (o == 1 ? 33 : o - 2 - 32);
                    const int dv = o < 2 ? 0 : m;
                    const int u2 = u + du, v2 = v + dv;
                    if (u2 < 0 || u2 >= det.nu || v2 < 0 || v2 >= det.nv)
                        continue;
                    const JosephRay S = rays[u2 + static_cast<int64_t>(det.nu) *
                                                       (v2 + static_cast<int64_t>(det.nv) * p)];
                    if (S.n == 0 || (S.meta & 3) != (R.meta & 3))
                        continue;
                    if (!separated(R, S, dim))
                        bad |= 1u << m;
                }
            }
            if (bad)
                atomicOr(badSpacing, bad);
        }

        // Exact accumulated position of every ray at its first sample in each driving-axis slab
        // of `depth` planes. Slab-major layout: row floor(k/depth) + 1, column = ray index, so a
        // warp of neighbouring rays reads one contiguous run.
        __global__ void josephCheckpointKernel(const JosephRay* __restrict__ rays, int64_t nrays,
                                               int depth, int slabRows,
                                               float2* __restrict__ checkpoints)
        {
            const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (r >= nrays)
                return;
            const JosephRay R = rays[r];
            if (R.n == 0)
                return;
            const int dir = (R.meta & 4) ? -1 : 1;
            float pa = R.pa, pb = R.pb;
            int k = R.k0, slab = floorDiv(R.k0, depth) - dir;
            for (int j = 0; j < R.n; ++j, k += dir) {
                const int s = floorDiv(k, depth);
                if (s != slab) {
                    slab = s;
                    // rows 0 .. slabRows-1 cover k in [-depth, (slabRows-1)*depth); the host
                    // sizes slabRows for every sample of an N-plane volume
                    if (s + 1 >= 0 && s + 1 < slabRows)
                        checkpoints[(s + 1) * nrays + r] = make_float2(pa, pb);
                }
                pa = __fadd_rn(pa, R.sa);
                pb = __fadd_rn(pb, R.sb);
            }
        }

        // Sample range [jLo, jHi] of ray R inside driving planes [kLo, kHi]; false if empty.
        __device__ __forceinline__ bool sampleRange(const JosephRay& R, int kLo, int kHi, int& jLo,
                                                    int& jHi)
        {
            const int dir = (R.meta & 4) ? -1 : 1;
            if (dir > 0) {
                jLo = max(0, kLo - R.k0);
                jHi = min(R.n - 1, kHi - R.k0);
            } else {
                jLo = max(0, R.k0 - kHi);
                jHi = min(R.n - 1, R.k0 - kLo);
            }
            return jLo <= jHi;
        }

        // ---- 2D on padded copies and square tiles ------------------------------------------------
        // Forward. A sample of a ray along axis G reads two neighbouring pixels of image line k
        // (a row for G = y, a column for G = x). The image is copied twice per call, as rows and
        // as columns, each line between kLinePad zeros, so that the 32 neighbouring rays of a
        // warp read consecutive words whatever their axis and taps outside the image need no
        // test. A warp takes 32 rays through one checkpoint slab of planes, starting from the
        // exact accumulated positions of the checkpoints; the slabs' sums are added in slab
        // order. Bound by issue and L2 latency: one thread per ray reading the image itself took
        // 0.87 ms at 512^2 / 720 views / 730 pixels (half of the views read one word per sector),
        // this takes 0.24 ms.
        constexpr int kLinePad = 8;
        __host__ __device__ inline int linePitch(int n) { return (n + 2 * kLinePad + 3) / 4 * 4; }

        // rows: ny lines of linePitch(nx); columns: nx lines of linePitch(ny). 32 x 8 threads per
        // 32 x 32 block of the image.
        __global__ void padLinesKernel(const float* __restrict__ x, int nx, int ny,
                                       float* __restrict__ rows, float* __restrict__ columns)
        {
            __shared__ float t[32][33];
            const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
            const int pitchX = linePitch(nx), pitchY = linePitch(ny);
            for (int j = threadIdx.y; j < 32; j += 8) {
                const int ix = x0 + threadIdx.x, iy = y0 + j;
                const float v =
                    ix < nx && iy < ny ? x[ix + static_cast<int64_t>(nx) * iy] : 0.0f;
                t[j][threadIdx.x] = v;
                if (ix < nx && iy < ny)
                    rows[static_cast<int64_t>(iy) * pitchX + kLinePad + ix] = v;
            }
            __syncthreads();
            for (int j = threadIdx.y; j < 32; j += 8) {
                const int ix = x0 + j, iy = y0 + threadIdx.x;
                if (ix < nx && iy < ny)
                    columns[static_cast<int64_t>(ix) * pitchY + kLinePad + iy] = t[threadIdx.x][j];
            }
        }

        // `count` samples from position p on, line `q` (its pixel 0) advancing by `lineStep`.
        template <bool Clamp>
        __device__ __forceinline__ float lineSamples(const float* q, int64_t lineStep, float p,
                                                     float s, int count, int n)
        {
            float acc = 0.0f;
#pragma unroll 8
            for (int j = 0; j < count; ++j) {
                int i;
                const float h = __fsub_rn(p, 0.5f);
                const float cw = __fsub_rn(h, floorSmall(h, i));
                if (Clamp)
                    i = min(max(i, -2), n);
                acc = __fmaf_rn(__fsub_rn(1.0f, cw), __ldg(q + i), acc);
                acc = __fmaf_rn(cw, __ldg(q + i + 1), acc);
                p = __fadd_rn(p, s);
                q += lineStep;
            }
            return acc;
        }

        // The same samples from the image itself: line k's pixel i at q + i * tapStep.
        __device__ __forceinline__ float imageSamples(const float* q, int lineStep, int tapStep,
                                                      float p, float s, int count, int n)
        {
            float acc = 0.0f;
            for (int j = 0; j < count; ++j) {
                int i;
                const float h = __fsub_rn(p, 0.5f);
                const float cw = __fsub_rn(h, floorSmall(h, i));
                const bool in0 = static_cast<unsigned>(i) < static_cast<unsigned>(n);
                const bool in1 = static_cast<unsigned>(i + 1) < static_cast<unsigned>(n);
                const float v0 = in0 ? __ldg(q + i * tapStep) : 0.0f;
                const float v1 = in1 ? __ldg(q + (i + 1) * tapStep) : 0.0f;
                acc = __fmaf_rn(__fsub_rn(1.0f, cw), v0, acc);
                acc = __fmaf_rn(cw, v1, acc);
                p = __fadd_rn(p, s);
                q += lineStep;
            }
            return acc;
        }

        // blockDim.x = 32 lanes (neighbouring rays of one view), blockDim.y = warps: `groups` groups
        // of warps, one view each, the warps of a group dividing its slabs. A block's views follow
        // one another, so its groups read nearly the same lines from L1. Padded: from rows and
        // columns; otherwise from the image (rows), for images so small that the launch that pads them
        // is not repaid.
        template <bool Padded>
        __global__ void __launch_bounds__(kMaxForwardThreads)
            josephForward2dKernel(const JosephRay* __restrict__ rays,
                                  const float2* __restrict__ checkpoints, int64_t nrays,
                                  VolumeShape vol, DetectorShape det, int depth, int nSlabs,
                                  int groups, int segments, const float* __restrict__ rows,
                                  const float* __restrict__ columns, float* __restrict__ y)
        {
            __shared__ float sums[kMaxForwardThreads];
            const int lane = threadIdx.x;
            const int perGroup = blockDim.y / groups;
            const int group = threadIdx.y / perGroup, member = threadIdx.y - group * perGroup;
            const int p = static_cast<int>(blockIdx.x / segments) * groups + group;
            const int u = static_cast<int>(blockIdx.x % segments) * 32 + lane;
            const bool valid = p < det.np && u < det.nu;
            const int64_t r = u + static_cast<int64_t>(det.nu) * p;
            JosephRay R{};
            if (valid)
                R = rays[r];
            const int g = R.meta & 3;
            const int dir = (R.meta & 4) ? -1 : 1;
            const int n = g == 0 ? vol.n[1] : vol.n[0], ng = g == 0 ? vol.n[0] : vol.n[1];
            const int pitch = linePitch(n);
            const float* lines = (g == 0 ? columns : rows) + kLinePad; // (Padded)
            float acc = 0.0f;
            for (int slab = member; slab < nSlabs; slab += perGroup) {
                int jLo, jHi;
                if (R.n == 0 || !sampleRange(R, slab * depth, (slab + 1) * depth - 1, jLo, jHi))
                    continue;
                int k = R.k0 + jLo * dir, count = jHi - jLo + 1;
                float pos = __ldg(checkpoints + (slab + 1) * nrays + r).x;
                // samples past the image's last line (a ray may start on its far face)
                for (; dir < 0 && k >= ng && count > 0; --k, --count)
                    pos = __fadd_rn(pos, R.sa);
                if (dir > 0)
                    count = min(count, ng - k);
                if (!Padded) {
                    const int lineStep = g == 0 ? 1 : vol.n[0], tapStep = g == 0 ? vol.n[0] : 1;
                    acc += imageSamples(rows + k * lineStep, dir * lineStep, tapStep, pos, R.sa,
                                        count, n);
                    continue;
                }
                // positions are monotone along the ray; a sample's line words are within the
                // padding unless the positions leave the image by several voxels
                const float end = pos + R.sa * static_cast<float>(count);
                const float far = static_cast<float>(n) + 4.0f;
                const bool inside = pos > -4.0f && pos < far && end > -4.0f && end < far;
                const float* q = lines + static_cast<int64_t>(k) * pitch;
                const int64_t step = static_cast<int64_t>(dir) * pitch;
                acc += inside ? lineSamples<false>(q, step, pos, R.sa, count, n)
                              : lineSamples<true>(q, step, pos, R.sa, count, n);
            }
            sums[threadIdx.y * 32 + lane] = acc;
            __syncthreads();
            if (member == 0 && valid) {
                for (int m = 1; m < perGroup; ++m)
                    acc += sums[(threadIdx.y + m) * 32 + lane];
                y[r] = R.len * acc;
            }
        }

        // Adjoint. A warp owns a TILE x TILE tile (with a one-pixel halo) in shared memory for
        // some views and splats 32 neighbouring rays at once, lane i delayed by i modulo m planes:
        // on any plane, the lanes that add at the same step are m rays apart, and rays m apart are
        // more than two pixels apart (the class check), so no two lanes touch one word and the
        // tile needs no atomics. Taps outside the tile belong to the neighbouring tile (halo words
        // are not written out). The NW warps of a block take views NW apart of the block's chunk;
        // their tiles are added in warp order, the chunks' partial images in chunk order.
        // Bound by the latency of the read-add-write chain of a step at 12 warps per SM (issue at
        // 58 %, 28 instructions per step of 32 rays). 512^2 / 720 views / 730 pixels: 0.54 ms;
        // eight warps sharing a tile, merging taps by shuffles and adding in phases, took 1.99.
        template <int TILE>
        struct Tile2d {
            static constexpr int kPitch = TILE + 3; // odd: lanes along either axis spread over banks
            static constexpr int kWords = kPitch * (TILE + 2);
        };

        template <int TILE, int G>
        __device__ __forceinline__ void tileRays(float* acc, const JosephRay* __restrict__ rays,
                                                 const float2* __restrict__ cps, int64_t nrays,
                                                 const float* __restrict__ y, int64_t viewBase,
                                                 int u, int u1, int m, int depth, int orgG, int orgA)
        {
            constexpr int kPitch = Tile2d<TILE>::kPitch;
            constexpr int strG = G == 0 ? 1 : kPitch, strA = G == 0 ? kPitch : 1;
            const int64_t r = viewBase + u;
            JosephRay R{};
            bool act = u <= u1;
            if (act)
                R = rays[r];
            int jLo = 0, jHi = -1;
            act = act && R.n > 0 && (R.meta & 3) == G &&
                  sampleRange(R, orgG, orgG + TILE - 1, jLo, jHi);
            const int dir = (R.meta & 4) ? -1 : 1;
            float pos = 0.0f, yl = 0.0f;
            int off = 0; // planes from the tile's first plane in ray direction
            if (act) {
                const int kFirst = R.k0 + jLo * dir;
                pos = __ldg(cps + (kFirst / depth + 1) * nrays + r).x;
                yl = __ldg(y + r) * R.len;
                off = dir > 0 ? kFirst - orgG : orgG + TILE - 1 - kFirst;
            }
            const int late = u % m;
            // rays towards higher and towards lower indices of a view cross planes in opposite
            // order: one direction at a time
            for (int d = 1; d >= -1; d -= 2) {
                const bool part = act && dir == d;
                if (!__any_sync(0xffffffffu, part))
                    continue;
                const int first = part ? off + late : 1 << 20;
                const int last = part ? first + jHi - jLo : -1;
                int t = __reduce_min_sync(0xffffffffu, first);
                const int tEnd = __reduce_max_sync(0xffffffffu, last);
                // byte address of the sample's left tap: base + column * 4 strA (the halo column
                // is -1), less the bias of the floor's bit pattern
                const int plane0 = (d > 0 ? t - late : TILE - 1 - (t - late)) + 1;
                unsigned base = static_cast<unsigned>(__cvta_generic_to_shared(acc)) +
                                4u * static_cast<unsigned>(plane0 * strG + (1 - orgA) * strA) -
                                0x4B400000u * 4u * strA;
                const unsigned bias = 0x4B400000u + static_cast<unsigned>(orgA) - 1u;
                const unsigned span = part ? static_cast<unsigned>(last - first) : 0u;
                for (; t <= tEnd; ++t) {
                    const float h = __fsub_rn(pos, 0.5f);
                    const float f = __fadd_rd(h, 12582912.0f); // floorSmall
                    const float cw = __fsub_rn(h, __fsub_rn(f, 12582912.0f));
                    const unsigned on =
                        part & (static_cast<unsigned>(t - first) <= span);
                    const unsigned in =
                        on & (__float_as_uint(f) - bias < static_cast<unsigned>(TILE + 1));
                    const unsigned q = base + __float_as_uint(f) * (4u * strA);
                    float a, b;
                    loadSharedIf(a, q, in);
                    loadSharedIf(b, q + 4u * strA, in);
                    storeSharedIf(__fmaf_rn(yl, __fsub_rn(1.0f, cw), a), q, in);
                    storeSharedIf(__fmaf_rn(yl, cw, b), q + 4u * strA, in);
                    pos = on ? __fadd_rn(pos, R.sa) : pos;
                    base += static_cast<unsigned>(4 * d * strG);
                    __syncwarp();
                }
            }
        }

        template <int TILE, int NW>
        __global__ void __launch_bounds__(NW * 32)
            josephAdjoint2dKernel(const JosephRay* __restrict__ rays,
                                  const float2* __restrict__ checkpoints, int64_t nrays,
                                  const float* __restrict__ y,
                                  const RayWindow* __restrict__ windows,
                                  const unsigned* __restrict__ viewAxes, VolumeShape vol,
                                  DetectorShape det, int m, int depth, int2 tiles,
                                  int viewsPerChunk, float* __restrict__ x)
        {
            // blockIdx.x: tile, blockIdx.y: view chunk (partial image x + chunk * nvox)
            extern __shared__ float smem[];
            constexpr int kWords = Tile2d<TILE>::kWords, kPitch = Tile2d<TILE>::kPitch;
            const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
            float* acc = smem + warp * kWords;
            const int org0 = (blockIdx.x % tiles.x) * TILE, org1 = (blockIdx.x / tiles.x) * TILE;
            for (int i = lane; i < kWords; i += 32)
                acc[i] = 0.0f;
            __syncwarp();
            const int pBegin = blockIdx.y * viewsPerChunk;
            const int pEnd = min(det.np, pBegin + viewsPerChunk);
            const int64_t nTiles = static_cast<int64_t>(tiles.x) * tiles.y;
            for (int p = pBegin + warp; p < pEnd; p += NW) {
                const RayWindow w = windows[p * nTiles + blockIdx.x];
                const unsigned axes = viewAxes[p];
                const int64_t viewBase = static_cast<int64_t>(det.nu) * p;
                for (int u = w.u0 + lane; u - lane <= w.u1; u += 32) {
                    if (axes & 1u)
                        tileRays<TILE, 0>(acc, rays, checkpoints, nrays, y, viewBase, u, w.u1, m,
                                          depth, org0, org1);
                    if (axes & 2u)
                        tileRays<TILE, 1>(acc, rays, checkpoints, nrays, y, viewBase, u, w.u1, m,
                                          depth, org1, org0);
                }
            }
            __syncthreads();
            float* out = x + blockIdx.y * (static_cast<int64_t>(vol.n[0]) * vol.n[1]);
            for (int i = threadIdx.x; i < TILE * TILE; i += NW * 32) {
                const int lx = i % TILE, ly = i / TILE;
                if (org0 + lx >= vol.n[0] || org1 + ly >= vol.n[1])
                    continue;
                const float* q = smem + (ly + 1) * kPitch + lx + 1;
                float s = q[0];
                for (int k = 1; k < NW; ++k)
                    s = s + q[k * kWords];
                out[org0 + lx + static_cast<int64_t>(vol.n[0]) * (org1 + ly)] = s;
            }
        }

        // x[v] = sum over chunks c = 0, 1, ... of partial[c][v], in chunk order
        __global__ void sumChunksKernel(const float* __restrict__ partial, int chunks,
                                        int64_t nvox, float* __restrict__ x)
        {
            const int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (v >= nvox)
                return;
            float s = partial[v];
            for (int c = 1; c < chunks; ++c)
                s = s + partial[c * nvox + v];
            x[v] = s;
        }

        // sumChunksKernel for many volumes: blockIdx.y selects (partials, count, nvox, out)
        struct SumChunksEntry {
            const float* partial;
            int chunks;
            int64_t nvox;
            float* x;
        };
        __global__ void sumChunksManyKernel(const SumChunksEntry* __restrict__ e)
        {
            const SumChunksEntry E = e[blockIdx.y];
            for (int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
                 v < E.nvox; v += static_cast<int64_t>(gridDim.x) * blockDim.x) {
                float s = E.chunks > 0 ? E.partial[v] : 0.0f;
                for (int c = 1; c < E.chunks; ++c)
                    s = s + E.partial[c * E.nvox + v];
                E.x[v] = s;
            }
        }

#ifndef ELSA_ADJ3D_WARPS_PER_SM
#define ELSA_ADJ3D_WARPS_PER_SM 22
#endif
        constexpr int kAdjoint3dWarpsPerSm = ELSA_ADJ3D_WARPS_PER_SM;
        constexpr int kMinAdjointChunks = 32;                // default floor of the view chunks
        constexpr int64_t kChunkMemory = int64_t(1) << 31;   // default partial-volume budget
        constexpr int64_t kBatchPartialMemory = int64_t(8) << 30; // batched adjoints: up to 8 GiB

        template <int TILE, int NW>
        struct Adjoint2dConfig {
            static constexpr size_t kShared = sizeof(float) * Tile2d<TILE>::kWords * NW;
            static constexpr int kBlocksPerSm = static_cast<int>((227 * 1024) / (kShared + 1024));
            // View chunks so that tiles x chunks is one wave of blocks, each warp with a view.
            static int chunks(int tiles, int np)
            {
                const int want = (kBlocksPerSm * 148 + tiles - 1) / tiles;
                return std::max(1, std::min(want, (np + NW - 1) / NW));
            }
            static void prepare()
            {
                ELSA_CUDA(cudaFuncSetAttribute(josephAdjoint2dKernel<TILE, NW>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(kShared)));
            }
            // nc view chunks; partial: scratch of nc images (unused with one chunk)
            static void launch(int2 tiles, int nc, int depth, cudaStream_t s, const JosephRay* rays,
                               const float2* cps, int64_t nrays, const float* y,
                               const RayWindow* win, const unsigned* axes, VolumeShape vol,
                               DetectorShape det, int m, float* x, float* partial)
            {
                const int per = (det.np + nc - 1) / nc;
                const int used = (det.np + per - 1) / per;
                const dim3 grid(static_cast<unsigned>(tiles.x * tiles.y),
                                static_cast<unsigned>(used));
                josephAdjoint2dKernel<TILE, NW><<<grid, NW * 32, kShared, s>>>(
                    rays, cps, nrays, y, win, axes, vol, det, m, depth, tiles, per,
                    used > 1 ? partial : x);
                if (used > 1)
                    launchSumChunks(partial, used,
                                    static_cast<int64_t>(vol.n[0]) * vol.n[1], x, s);
            }
        };

        // ---------------------------------------------------------------------------------------
        // 3D adjoint on axis bricks. The rays of one view all step along about the same axis G, so
        // the volume is cut, per driving axis present, into bricks that are TD planes deep along G
        // and TA x TB voxels across (a < b the other two axes). A ray crossing such a brick keeps
        // most of its TD samples inside it (a 16^3 brick loses half of the samples of oblique rays
        // to its sides), and the window of a brick, the pixels whose centres lie in the projection
        // of the brick grown by about half a voxel, holds few rays that miss it. One warp owns a
        // brick in shared memory for a chunk of views and splats the window's rays class by class:
        // rays of one class are more than two voxels apart, so no two lanes add to one word at
        // once and the brick needs no atomics. Taps outside the brick belong to the neighbouring
        // brick: those of rows are predicated off, those of columns fall into a halo column that
        // is not written out.
        // ---------------------------------------------------------------------------------------
        // Shared-memory brick of TD planes (along G) of TV rows x TW columns. Columns run along
        // the non-driving axis over which the rays of a detector row spread (the warp's lanes
        // spread along it, so stride 1 there keeps their taps in different banks), rows along the
        // other one. A halo column on either side takes the taps of samples that straddle the
        // brick's edge (they belong to the neighbouring brick and are not written out), so that
        // the four taps of a sample need two predicates, one per row, instead of four and a mask of
        // them carried along. 48 instructions per step of 32 rays instead of 62: 256^3 / 360 views /
        // 384^2 32.2 -> 28.2 ms, now bound by the shared-memory pipe (78 %; half of its wavefronts
        // are bank conflicts between the rows of a class). Rows of 35 words: 29.1 ms; 7 or 10 rows:
        // 28.6 / 30.2; 2 or 4 rays fetched per lane: 28.4 / 28.5; unrolled 1 or 4: 31.7 / 28.3.
        template <int TD, int TW, int TV>
        struct AxisBrick {
            static constexpr int kRow = TW + 2; // words per row
            static constexpr int kPlane = kRow * TV;
            static constexpr int kWords = kPlane * TD;
        };

        // Word of the voxel (a, b) of an axis brick's plane: a < b the non-driving axes of G; UB:
        // the columns run along b (else along a).
        template <int TD, bool UB, int TW, int TV>
        struct AxisRolesAB {
            using L = AxisBrick<TD, TW, TV>;
            static constexpr int SA = UB ? L::kRow : 1, SB = UB ? 1 : L::kRow;
            static constexpr int kOrigin = 1; // word of (a, b) = (0, 0)
        };

        // Samples jLo..jHi of ray R (position cp at sample jLo, on brick plane t0) into the brick.
        // (column, row) pairs run on the packed two-wide FP32 instructions with the reference's
        // roundings (JosephsMethod.cpp:37-52; the weight (p - floor) - 0.5 as (p - 0.5) - floor,
        // the same number for p >= 1). Software-pipelined: the footprint of sample j+1 (always on
        // another plane) is read before the sums of sample j are written back.
        template <int TD, bool UB, int TW, int TV>
        __device__ __forceinline__ void axisSplat(float* acc, const JosephRay& R, float yl,
                                                  float2 cp, int jLo, int jHi, int t0, int orgA,
                                                  int orgB)
        {
            using L = AxisBrick<TD, TW, TV>;
            constexpr int kRow = L::kRow;
            const float2 half = splat2(0.5f), one = splat2(1.0f), magic = splat2(12582912.0f);
            const float2 s2 = UB ? make_float2(R.sb, R.sa) : make_float2(R.sa, R.sb);
            float2 p2 = UB ? make_float2(cp.y, cp.x) : cp;
            // floor(p - 0.5) + 1 - origin of the columns (the halo column is 0), floor(p - 0.5) -
            // origin of the rows, from the bit patterns of the floors (floorSmall2)
            const unsigned biasC = 0x4B400000u + static_cast<unsigned>(UB ? orgB : orgA) - 1u;
            const unsigned biasR = 0x4B400000u + static_cast<unsigned>(UB ? orgA : orgB);
            const int dPlane = ((R.meta & 4) ? -1 : 1) * L::kPlane;
            int plane = t0 * L::kPlane;
            struct Tap {
                int o;      // word of the footprint's first tap
                bool r0, r1; // its rows lie in the brick
                float2 w, cw;
            };
            auto tap = [&]() {
                Tap t;
                const float2 h = sub2(p2, half);
                const float2 f = add2Down(h, magic);
                t.cw = sub2(h, sub2(f, magic));
                t.w = sub2(one, t.cw);
                const unsigned c = __float_as_uint(f.x) - biasC, r = __float_as_uint(f.y) - biasR;
                const bool in = c < static_cast<unsigned>(TW + 1);
                t.r0 = in && r < static_cast<unsigned>(TV);
                t.r1 = in && r + 1u < static_cast<unsigned>(TV);
                t.o = plane + static_cast<int>(r * kRow + c);
                return t;
            };
            Tap t = tap();
            float2 v0 = splat2(0.0f), v1 = splat2(0.0f);
            if (t.r0)
                v0 = make_float2(acc[t.o], acc[t.o + 1]);
            if (t.r1)
                v1 = make_float2(acc[t.o + kRow], acc[t.o + kRow + 1]);
            auto store = [&]() {
                const float ya = yl * t.w.x, yc = yl * t.cw.x;
                if (t.r0) {
                    acc[t.o] = __fmaf_rn(ya, t.w.y, v0.x);
                    acc[t.o + 1] = __fmaf_rn(yc, t.w.y, v0.y);
                }
                if (t.r1) {
                    acc[t.o + kRow] = __fmaf_rn(ya, t.cw.y, v1.x);
                    acc[t.o + kRow + 1] = __fmaf_rn(yc, t.cw.y, v1.y);
                }
            };
#pragma unroll kSplatUnroll
            for (int j = jLo; j < jHi; ++j) {
                plane += dPlane;
                p2 = add2(p2, s2);
                const Tap n = tap();
                float2 n0 = splat2(0.0f), n1 = splat2(0.0f);
                if (n.r0)
                    n0 = make_float2(acc[n.o], acc[n.o + 1]);
                if (n.r1)
                    n1 = make_float2(acc[n.o + kRow], acc[n.o + kRow + 1]);
                store();
                t = n, v0 = n0, v1 = n1;
            }
            store();
        }

        // One view for an axis brick of grid G: m x m ray classes separated by __syncwarp; lane i
        // takes class rays i, i + 32, ... (u fastest within the class grid).
        template <int G, int TD, bool UB, int TW, int TV, int CPD>
        __device__ __forceinline__ void axisView(float* acc, const RayWindow& w, int p, int m,
                                                 int cpdShift, const JosephRay* __restrict__ rays,
                                                 const float2* __restrict__ cps, int64_t nrays,
                                                 const float* __restrict__ y,
                                                 const DetectorShape& det, int orgG, int orgA,
                                                 int orgB)
        {
            // Checkpoint slabs of CPD planes, or of 2^cpdShift planes when CPD is 0 (the
            // deeper slabs that save memory). A brick that does not start at its ray's first
            // sample in the slab catches up from the checkpoint by exact additions.
            const int kLo = orgG, kHi = orgG + TD - 1;
            const int shift = CPD > 0 ? 0 : cpdShift;
            const int slabLo = CPD > 0 ? (orgG / CPD) * CPD : (orgG >> shift) << shift;
            const int slabHi = slabLo + (CPD > 0 ? CPD : 1 << shift) - 1;
            const bool catchUp = CPD > 0 ? TD < CPD : (1 << shift) > TD;
            const int64_t cpRow =
                static_cast<int64_t>((CPD > 0 ? orgG / CPD : orgG >> shift) + 1) * nrays;
            const int lane = threadIdx.x & 31;
            const int64_t viewBase = static_cast<int64_t>(det.nu) * det.nv * p;
            for (int ov = 0; ov < m; ++ov) {
                const int vStart = w.v0 + ov;
                const int nvc = vStart <= w.v1 ? (w.v1 - vStart) / m + 1 : 0;
                for (int ou = 0; ou < m; ++ou) {
                    const int uStart = w.u0 + ou;
                    const int nuc = uStart <= w.u1 ? (w.u1 - uStart) / m + 1 : 0;
                    const int total = nuc * nvc;
                    const float invNuc = nuc > 0 ? 1.0f / static_cast<float>(nuc) : 0.0f;
                    constexpr int kBatch = ELSA_ADJ_BATCH;
                    for (int base = lane; base < total; base += 32 * kBatch) {
                        JosephRay Rb[kBatch];
                        float2 cpb[kBatch];
                        float yb[kBatch];
#pragma unroll
                        for (int q = 0; q < kBatch; ++q) {
                            const int i = base + 32 * q;
                            Rb[q].n = 0;
                            if (i < total) {
                                // i / nuc by a float reciprocal: exact for i < 2^20, nuc < 2^11
                                const int iv =
                                    static_cast<int>((static_cast<float>(i) + 0.5f) * invNuc);
                                const int iu = i - iv * nuc;
                                const int64_t r = viewBase + (uStart + iu * m) +
                                                  static_cast<int64_t>(det.nu) * (vStart + iv * m);
                                Rb[q] = rays[r];
                                cpb[q] = __ldg(cps + cpRow + r);
                                yb[q] = __ldg(y + r);
                            }
                        }
#pragma unroll
                        for (int q = 0; q < kBatch; ++q) {
                            const JosephRay& R = Rb[q];
                            if (R.n == 0 || (R.meta & 3) != G)
                                continue;
                            int jLo, jHi;
                            if (!sampleRange(R, kLo, kHi, jLo, jHi))
                                continue;
                            // the checkpoint holds the position at the ray's first sample in
                            // the slab; a brick thinner than the slab advances it to its own
                            // planes
                            float2 cp = cpb[q];
                            if (catchUp) {
                                int jS0, jS1;
                                sampleRange(R, slabLo, slabHi, jS0, jS1);
                                for (int j = jS0; j < jLo; ++j) {
                                    cp.x = __fadd_rn(cp.x, R.sa);
                                    cp.y = __fadd_rn(cp.y, R.sb);
                                }
                            }
                            const int dir = (R.meta & 4) ? -1 : 1;
                            const int t0 = R.k0 + jLo * dir - orgG;
                            axisSplat<TD, UB, TW, TV>(acc, R, yb[q] * R.len, cp, jLo, jHi, t0,
                                                      orgA, orgB);
                        }
                    }
                    __syncwarp();
                }
            }
        }

        // Brick edges of grid G in volume axis order (x, y, z).
        template <int G, int TD, bool UB, int TW, int TV>
        __host__ __device__ constexpr int axisBrickEdge(int axis)
        {
            return axis == G ? TD : (axis == (G == 0 ? 1 : 0) ? (UB ? TV : TW) : (UB ? TW : TV));
        }

        // Shape of the axis bricks (depth along the driving axis, columns, rows) and the
        // checkpoint slab depth of the 3D operator.
        constexpr int kAxisTD = ELSA_AXIS_TD, kAxisTW = ELSA_AXIS_TW, kAxisTV = ELSA_AXIS_TV;
        constexpr int kAxisCheckpointDepth = 16; // the smallest checkpoint slab of the 3D adjoint
        static_assert(kAxisCheckpointDepth % kAxisTD == 0,
                      "axis bricks are a whole fraction of a checkpoint slab deep");

        // What one axis-brick adjoint launch works on: the operator's tables, the sinogram y,
        // the grid's windows and (chunk, partial volume) entries, and where partial volumes go.
        struct AxisJob {
            const JosephRay* rays;
            const float2* checkpoints;
            int64_t nrays;
            const float* y;
            const RayWindow* windows; // this grid's windows, [view][brick]
            const unsigned* viewAxes;
            const int2* chunks; // this grid's entries (chunk, partial volume)
            int entries;
            int viewsPerChunk;
            VolumeShape vol;
            DetectorShape det;
            int m;
            int cpdShift; // checkpoint slabs of 2^cpdShift planes
            int3 nBricks;
            float* out;       // partial volume k at out + k * nvox (x itself for one partial)
            int64_t itemBase; // batched launches: first block of this job
        };

        // One warp: brick bi of grid G, chunk entry e (views [chunks[e].x * per, ...)), written
        // to the entry's partial volume.
        template <int G, int TD, bool UB, int TW, int TV, int CPD>
        __device__ __forceinline__ void axisBrickWork(const AxisJob& J, int bi, int e, float* acc)
        {
            using L = AxisBrick<TD, TW, TV>;
            using AR = AxisRolesAB<TD, UB, TW, TV>;
            constexpr int EX = axisBrickEdge<G, TD, UB, TW, TV>(0);
            constexpr int EY = axisBrickEdge<G, TD, UB, TW, TV>(1);
            constexpr int EZ = axisBrickEdge<G, TD, UB, TW, TV>(2);
            const int lane = threadIdx.x;
            const int3 nBricks = J.nBricks;
            const int org[3] = {(bi % nBricks.x) * EX, ((bi / nBricks.x) % nBricks.y) * EY,
                                (bi / (nBricks.x * nBricks.y)) * EZ};
            int a, b;
            nonDrivingAxes(G, a, b);
            const int orgG = org[G], orgA = org[a], orgB = org[b];
            const int nb = nBricks.x * nBricks.y * nBricks.z;
            for (int i = lane; i < L::kWords; i += 32)
                acc[i] = 0.0f;
            __syncwarp();
            const int2 entry = J.chunks[e];
            const int pBegin = entry.x * J.viewsPerChunk;
            const int pEnd = min(J.det.np, pBegin + J.viewsPerChunk);
            for (int p = pBegin; p < pEnd; ++p) {
                if (!(J.viewAxes[p] & (1u << G)))
                    continue;
                const RayWindow w = J.windows[static_cast<int64_t>(p) * nb + bi];
                if (w.u0 > w.u1 || w.v0 > w.v1)
                    continue;
                axisView<G, TD, UB, TW, TV, CPD>(acc, w, p, J.m, J.cpdShift, J.rays,
                                                 J.checkpoints, J.nrays,
                                                 J.y, J.det, orgG, orgA, orgB);
            }
            __syncwarp();
            const VolumeShape& vol = J.vol;
            const int64_t nvox = static_cast<int64_t>(vol.n[0]) * vol.n[1] * vol.n[2];
            float* dst = J.out + static_cast<int64_t>(entry.y) * nvox;
            for (int i = lane; i < TD * TW * TV; i += 32) {
                // i runs x fastest over the brick's voxels
                const int lx = i % EX, ly = (i / EX) % EY, lz = i / (EX * EY);
                const int gx = org[0] + lx, gy = org[1] + ly, gz = org[2] + lz;
                if (gx < vol.n[0] && gy < vol.n[1] && gz < vol.n[2]) {
                    const int l[3] = {lx, ly, lz};
                    dst[gx + static_cast<int64_t>(vol.n[0]) *
                                 (gy + static_cast<int64_t>(vol.n[1]) * gz)] =
                        acc[AR::kOrigin + l[G] * L::kPlane + l[a] * AR::SA + l[b] * AR::SB];
                }
            }
        }

        // One warp per axis brick of grid G (blockIdx.x) and chunk entry (entryBase +
        // blockIdx.y); blockIdx.z: batch element (sinogram y + b yStride, partial volumes
        // out + b outStride).
        template <int G, int TD, bool UB, int TW, int TV, int CPD>
        __global__ void __launch_bounds__(32, ELSA_ADJ_MIN_BLOCKS)
            josephAdjointAxisKernel(AxisJob J, int entryBase, int64_t yStride, int64_t outStride)
        {
            __shared__ float acc[AxisBrick<TD, TW, TV>::kWords];
            J.y += blockIdx.z * yStride;
            J.out += blockIdx.z * outStride;
            axisBrickWork<G, TD, UB, TW, TV, CPD>(J, blockIdx.x, entryBase + blockIdx.y, acc);
        }

        // Many operators in one launch (batched solves): block k belongs to the job whose
        // [itemBase, itemBase + bricks x entries) holds k; within it, brick k % bricks and entry
        // k / bricks, exactly the work of that operator's own launch.
        template <int G, int TD, bool UB, int TW, int TV, int CPD>
        __global__ void __launch_bounds__(32, ELSA_ADJ_MIN_BLOCKS)
            josephAdjointAxisManyKernel(const AxisJob* __restrict__ jobs, int njobs)
        {
            __shared__ float acc[AxisBrick<TD, TW, TV>::kWords];
            const int64_t k = blockIdx.x;
            int lo = 0, hi = njobs - 1; // last job with itemBase <= k
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (jobs[mid].itemBase <= k)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            const AxisJob J = jobs[lo];
            const int nb = J.nBricks.x * J.nBricks.y * J.nBricks.z;
            const int64_t local = k - J.itemBase;
            axisBrickWork<G, TD, UB, TW, TV, CPD>(J, static_cast<int>(local % nb),
                                                  static_cast<int>(local / nb), acc);
        }

        // Tiles of 64 pixels for images that fill the GPU with them, of 32 for smaller ones (more
        // blocks; their rays start and end in more tiles).
        using Adjoint2dLarge = Adjoint2dConfig<64, 4>;
        using Adjoint2dSmall = Adjoint2dConfig<32, 8>;
        // pixels up to which the tiles are the small ones: a larger image fills the GPU with the large
        // ones, which need half the checkpoints (at 512^2 either takes the same, 0.504 ms and 0.514)
        constexpr int kSmallImage = 256 * 256;
        // Pixels, and pixels times views, up to which the forward reads the image itself. Padded /
        // direct in us, 1.45 pixels per column: 32^2 / 40 views 14.3 / 8.6; 80^2 / 180 (1.15e6)
        // 18.5 / 10.6; 96^2 / 180 (1.7e6) 20.5 / 25.2; 128^2 / 40 14.4 / 12.3, / 180 15.1 / 18.9.
        constexpr int kDirectImage = 128 * 128;
        constexpr int64_t kDirectWork = 1200000;

        class JosephProjector final : public Projector
        {
        public:
            // fast: elsa's unmatched `fast` adjoint (JosephsMethodCUDA.h:60-67) instead of the
            // matched one
            JosephProjector(const VolumeShape& vol, const DetectorShape& det,
                            const std::vector<PoseRecord>& poses, const CurvedDetector& curved,
                            bool fast)
                : Projector(0, vol, det, poses), curved_(vol.dim, det, curved), fast_(fast)
            {
                const int64_t nrays = rangeSize_;
                ELSA_CUDA(cudaMalloc(&dRays_, sizeof(JosephRay) * nrays));
                const int threads = 256;
                const unsigned blocks = static_cast<unsigned>((nrays + threads - 1) / threads);
                josephSetupKernel<<<blocks, threads>>>(dPoses_, vol_, det_, curved_.planar(),
                                                       dRays_);
                ELSA_LAUNCH_CHECK("josephSetupKernel");

                // per-view axis masks, then (at +np) the bad-spacing mask and a 64-bit counter
                const size_t axesWords = static_cast<size_t>(det_.np) + 4;
                ELSA_CUDA(cudaMalloc(&dViewAxes_, sizeof(unsigned) * axesWords));
                ELSA_CUDA(cudaMemset(dViewAxes_, 0, sizeof(unsigned) * axesWords));
                unsigned* dBad = dViewAxes_ + det_.np;
                auto* dCount = reinterpret_cast<unsigned long long*>(
                    dViewAxes_ + ((det_.np + 2) & ~1));
                josephClassCheckKernel<<<blocks, threads>>>(dRays_, det_, vol_.dim, dViewAxes_,
                                                            dBad, dCount);
                ELSA_LAUNCH_CHECK("josephClassCheckKernel");
                unsigned bad = 0;
                unsigned long long count = 0;
                ELSA_CUDA(cudaMemcpy(&bad, dBad, sizeof(unsigned), cudaMemcpyDeviceToHost));
                ELSA_CUDA(cudaMemcpy(&count, dCount, sizeof(count), cudaMemcpyDeviceToHost));
                sampleCount_ = static_cast<int64_t>(count);
                laneAxisBits();
                classSpacing_ = 0;
                for (int m = kMinClass; m <= kMaxClass; ++m)
                    if (!((bad >> m) & 1u)) {
                        classSpacing_ = m;
                        break;
                    }
                if (fast_)
                    buildFastAdjoint();
                if (vol_.dim == 2)
                    buildForward2d();
                if (fast_) {
                    if (vol_.dim == 3) {
                        std::vector<float> hp(poses_.size() * kPoseFloats);
                        std::memcpy(hp.data(), poses_.data(), sizeof(float) * hp.size());
                        tma_ = std::make_unique<JosephForwardTma>(vol_, det_, hp, dRays_);
                    }
                    ELSA_CUDA(cudaDeviceSynchronize());
                    curved_.release();
                    return;
                }
                if (classSpacing_ == 0)
                    throw Error(ELSA_ERROR_NOT_SUPPORTED,
                                "JosephsMethod: neighbouring detector rays pass within two voxels "
                                "of each other even eight pixels apart; the atomic-free adjoint "
                                "needs a coarser detector");

                if (vol_.dim == 3) {
                    buildCheckpoints(defaultCheckpointDepth());
                } else {
                    Adjoint2dLarge::prepare();
                    Adjoint2dSmall::prepare();
                }

                if (vol_.dim == 3) {
                    buildAxisGrids();
                } else {
                    nBricks_ = make_int3((vol_.n[0] + brick_.x - 1) / brick_.x,
                                         (vol_.n[1] + brick_.y - 1) / brick_.y,
                                         (vol_.n[2] + brick_.z - 1) / brick_.z);
                    const int64_t nwin =
                        static_cast<int64_t>(nBricks_.x) * nBricks_.y * nBricks_.z * det_.np;
                    ELSA_CUDA(cudaMalloc(&dWindows_, sizeof(RayWindow) * nwin));
                    josephWindowKernel<<<static_cast<unsigned>((nwin + 255) / 256), 256>>>(
                        dPoses_, vol_, det_, brick_, nBricks_, curved_.map(), windowGrow(vol_),
                        kWindowPixelMargin, dWindows_);
                    ELSA_LAUNCH_CHECK("josephWindowKernel");
                }
                setKnob(kKnobAdjointChunks, defaultChunks());
                if (vol_.dim == 3) {
                    std::vector<float> hp(poses_.size() * kPoseFloats);
                    std::memcpy(hp.data(), poses_.data(), sizeof(float) * hp.size());
                    tma_ = std::make_unique<JosephForwardTma>(vol_, det_, hp, dRays_);
                }
                ELSA_CUDA(cudaDeviceSynchronize());
                curved_.release(); // rays and windows are built
            }

            // 2D: checkpoints, one slab per tile of the matched adjoint, and the padded image copies.
            void buildForward2d()
            {
                if (domainSize_ > kDirectImage || domainSize_ * det_.np > kDirectWork) {
                    lines_ = std::make_unique<StreamScratch>(
                        sizeof(float) * (rowWords() + static_cast<size_t>(vol_.n[0]) *
                                                          linePitch(vol_.n[1])));
                    ELSA_CUDA(cudaMemset(lines_->initial(), 0, lines_->bytes()));
                }
                const int maxDim = std::max(vol_.n[0], vol_.n[1]);
                auto fits = [&](int cpd) { // the table in an eighth of the device's memory, as in 3D
                    const double bytes =
                        8.0 * static_cast<double>(rangeSize_) * (maxDim / cpd + 3);
                    if (bytes < 1e9)
                        return true; // (asking takes half a millisecond)
                    size_t freeBytes = 0, totalBytes = 0;
                    ELSA_CUDA(cudaMemGetInfo(&freeBytes, &totalBytes));
                    return bytes <= static_cast<double>(totalBytes) / 8.0;
                };
                const int tile = domainSize_ <= kSmallImage && fits(32) ? 32 : 64;
                brick_ = make_int3(tile, tile, 1);
                // The `fast` adjoint has no checkpoints: its forward takes deeper slabs (down to one,
                // 24 bytes per ray) where the table or the memory left is too small. (Samples past
                // the last line are at most one.)
                for (int cpd = tile;; cpd *= 2) {
                    const bool deepest = !fast_ || cpd > maxDim;
                    if (!deepest && !fits(cpd))
                        continue;
                    try {
                        buildCheckpoints(cpd);
                        break;
                    } catch (const Error&) {
                        if (deepest)
                            throw;
                        cudaGetLastError();
                    }
                }
            }

            // Per view and driving axis g: set bit 4+g of the view's axis word when neighbouring
            // pixels of a detector row spread along the second non-driving axis b on the planes
            // of g (centre pixel and its right neighbour).
            void laneAxisBits()
            {
                std::vector<unsigned> axes(det_.np);
                ELSA_CUDA(cudaMemcpy(axes.data(), dViewAxes_, sizeof(unsigned) * det_.np,
                                     cudaMemcpyDeviceToHost));
                for (int p = 0; p < det_.np; ++p) {
                    const float* P = poses_[p].v + kPoseOffPinv;
                    const int d = vol_.dim;
                    const float uc = det_.nu / 2 + 0.5f, vc = det_.nv / 2 + 0.5f;
                    float D[3] = {0, 0, 0}, E[3] = {0, 0, 0};
                    for (int i = 0; i < d; ++i) {
                        if (d == 3) {
                            D[i] = P[i * 3] * uc + P[i * 3 + 1] * vc + P[i * 3 + 2];
                            E[i] = P[i * 3] * (uc + 1.0f) + P[i * 3 + 1] * vc + P[i * 3 + 2];
                        } else {
                            D[i] = P[i * 2] * uc + P[i * 2 + 1];
                            E[i] = P[i * 2] * (uc + 1.0f) + P[i * 2 + 1];
                        }
                    }
                    if (d == 3) {
                        for (int g = 0; g < 3; ++g) {
                            int a, b;
                            nonDrivingAxes(g, a, b);
                            if (std::fabs(D[g]) == 0.0f || std::fabs(E[g]) == 0.0f)
                                continue;
                            const float da =
                                std::fabs(E[a] / std::fabs(E[g]) - D[a] / std::fabs(D[g]));
                            const float db =
                                std::fabs(E[b] / std::fabs(E[g]) - D[b] / std::fabs(D[g]));
                            if (db > da)
                                axes[p] |= 16u << g;
                        }
                    }
                }
                ELSA_CUDA(cudaMemcpy(dViewAxes_, axes.data(), sizeof(unsigned) * det_.np,
                                     cudaMemcpyHostToDevice));
            }

            // The fast adjoint's per-view table (leading block of P, column-major, and the ray
            // origin -Binv p4 as JosephsMethodCUDA.cpp:80-84 computes it, in float, k-sums in
            // order) and the layered sinogram array it reads through a texture.
            void buildFastAdjoint()
            {
                const int d = vol_.dim;
                const int kT = d == 3 ? 12 : 6;
                std::vector<float> table(static_cast<size_t>(kT) * det_.np);
                for (int p = 0; p < det_.np; ++p) {
                    const float* P = poses_[p].v;
                    const float* Pinv = poses_[p].v + kPoseOffPinv;
                    float* T = table.data() + static_cast<size_t>(kT) * p;
                    for (int c = 0; c < d; ++c)
                        for (int r = 0; r < d; ++r)
                            T[d * c + r] = P[(d + 1) * r + c];
                    for (int r = 0; r < d; ++r) {
                        float s = 0.0f;
                        for (int c = 0; c < d; ++c)
                            s += Pinv[d * r + c] * P[(d + 1) * c + d];
                        T[d * d + r] = -s;
                    }
                }
                // the kernel keeps the table in shared memory; the limit attribute only grows, as
                // for the brick-owner adjoints (shared by every projector of the process)
                const int need = static_cast<int>(sizeof(float) * table.size());
                if (need > 227 * 1024)
                    throw Error(ELSA_ERROR_NOT_SUPPORTED,
                                "JosephsMethodCUDA: too many poses for the fast adjoint");
                {
                    static std::mutex mu;
                    std::lock_guard<std::mutex> lock(mu);
                    cudaFuncAttributes attr{};
                    const void* fn = d == 3 ? reinterpret_cast<const void*>(
                                                  josephFastAdjointKernel<3>)
                                            : reinterpret_cast<const void*>(
                                                  josephFastAdjointKernel<2>);
                    ELSA_CUDA(cudaFuncGetAttributes(&attr, fn));
                    if (need > attr.maxDynamicSharedSizeBytes)
                        ELSA_CUDA(cudaFuncSetAttribute(
                            fn, cudaFuncAttributeMaxDynamicSharedMemorySize, need));
                }
                fastTable_ = std::make_unique<DeviceBuffer>(sizeof(float) * table.size());
                ELSA_CUDA(cudaMemcpy(fastTable_->as<float>(), table.data(),
                                     sizeof(float) * table.size(), cudaMemcpyHostToDevice));
                cudaDeviceProp prop{};
                ELSA_CUDA(cudaGetDeviceProperties(&prop, device_));
                const int* lim = d == 3 ? prop.maxTexture2DLayered : prop.maxTexture1DLayered;
                if (det_.nu > lim[0] || (d == 3 && det_.nv > lim[1]) || det_.np > lim[d - 1])
                    throw Error(ELSA_ERROR_NOT_SUPPORTED,
                                "JosephsMethodCUDA: the fast adjoint's layered texture cannot "
                                "hold this detector (size or number of poses)");
                const cudaChannelFormatDesc fd =
                    cudaCreateChannelDesc(32, 0, 0, 0, cudaChannelFormatKindFloat);
                const cudaExtent ext =
                    make_cudaExtent(det_.nu, d == 3 ? det_.nv : 0, det_.np);
                ELSA_CUDA(cudaMalloc3DArray(&fastArray_, &fd, ext, cudaArrayLayered));
                cudaResourceDesc res;
                std::memset(&res, 0, sizeof(res));
                res.resType = cudaResourceTypeArray;
                res.res.array.array = fastArray_;
                cudaTextureDesc tex;
                std::memset(&tex, 0, sizeof(tex));
                tex.addressMode[0] = tex.addressMode[1] = tex.addressMode[2] =
                    cudaAddressModeBorder;
                tex.filterMode = cudaFilterModeLinear;
                tex.readMode = cudaReadModeElementType;
                tex.normalizedCoords = 0;
                ELSA_CUDA(cudaCreateTextureObject(&fastTex_, &res, &tex, nullptr));
            }

            ~JosephProjector() override
            {
                if (fastTex_)
                    cudaDestroyTextureObject(fastTex_);
                if (fastArray_)
                    cudaFreeArray(fastArray_);
                cudaFree(dRays_);
                cudaFree(dViewAxes_);
                cudaFree(dWindows_);
                cudaFree(dCheckpoints_);
            }

            void doForward(const float* x, float* y, cudaStream_t s) override
            {
                if (tma_)
                    tma_->forward(x, y, s);
                else
                    forward2d(x, y, s);
            }

            size_t rowWords() const // words of the padded rows, a multiple of 4
            {
                return static_cast<size_t>(vol_.n[1]) * linePitch(vol_.n[0]);
            }

            void forward2d(const float* x, float* y, cudaStream_t s)
            {
                std::unique_ptr<StreamScratch::Lease> lines;
                const float *rows = x, *columns = nullptr; // (small images: the image itself)
                if (lines_) {
                    lines = std::make_unique<StreamScratch::Lease>(*lines_, s);
                    if (lines->fresh()) // the padding
                        ELSA_CUDA(cudaMemsetAsync(lines->as<void>(), 0, lines_->bytes(), s));
                    float* padded = lines->as<float>();
                    const dim3 blocks((vol_.n[0] + 31) / 32, (vol_.n[1] + 31) / 32);
                    padLinesKernel<<<blocks, dim3(32, 8), 0, s>>>(x, vol_.n[0], vol_.n[1], padded,
                                                                  padded + rowWords());
                    ELSA_LAUNCH_CHECK("padLinesKernel");
                    rows = padded, columns = padded + rowWords();
                }
                const int depth = 1 << cpdShift_;
                const int slabs = (std::max(vol_.n[0], vol_.n[1]) + depth - 1) / depth;
                const int segments = (det_.nu + 31) / 32;
                const int warps = forwardThreads_ / 32;
                // warps per view segment: as many as fill 32 warps per SM, at most its slabs
                int perGroup = 1;
                while (2 * perGroup <= std::min(warps, slabs) &&
                       static_cast<int64_t>(segments) * det_.np * perGroup < 148 * 32)
                    perGroup *= 2;
                const int groups = warps / perGroup;
                const int64_t grid =
                    static_cast<int64_t>(segments) * ((det_.np + groups - 1) / groups);
                auto* k = lines_ ? josephForward2dKernel<true> : josephForward2dKernel<false>;
                k<<<static_cast<unsigned>(grid), dim3(32, groups * perGroup), 0, s>>>(
                    dRays_, dCheckpoints_, rangeSize_, vol_, det_, depth, slabs, groups, segments,
                    rows, columns, y);
                ELSA_LAUNCH_CHECK("josephForward2dKernel");
            }

            void doAdjoint(const float* y, float* x, cudaStream_t s) override
            {
                if (fast_) {
                    // the sinogram into the layered array (JosephsMethodCUDA.cpp:234-240 copies
                    // the host data there on every call)
                    const int d = vol_.dim;
                    cudaMemcpy3DParms prm = {};
                    prm.srcPtr = make_cudaPitchedPtr(const_cast<float*>(y), sizeof(float) * det_.nu,
                                                     det_.nu, d == 3 ? det_.nv : 1);
                    prm.dstArray = fastArray_;
                    prm.extent = make_cudaExtent(det_.nu, d == 3 ? det_.nv : 1, det_.np);
                    prm.kind = cudaMemcpyDeviceToDevice;
                    ELSA_CUDA(cudaMemcpy3DAsync(&prm, s));
                    const int64_t rows =
                        static_cast<int64_t>(vol_.n[1]) * (d == 3 ? vol_.n[2] : 1);
                    const dim3 grid(static_cast<unsigned>((rows + kFastRows - 1) / kFastRows));
                    const dim3 block(32, kFastRows);
                    const size_t smem = sizeof(float) * (d == 3 ? 12 : 6) * det_.np;
                    if (d == 3)
                        josephFastAdjointKernel<3><<<grid, block, smem, s>>>(
                            fastTex_, fastTable_->as<float>(), det_.np, vol_, x);
                    else
                        josephFastAdjointKernel<2><<<grid, block, smem, s>>>(
                            fastTex_, fastTable_->as<float>(), det_.np, vol_, x);
                    ELSA_LAUNCH_CHECK("josephFastAdjointKernel");
                    return;
                }
                if (scatter_) {
                    const int64_t nrays = rangeSize_;
                    const unsigned blocks =
                        static_cast<unsigned>((nrays + kForwardThreads - 1) / kForwardThreads);
                    ELSA_CUDA(cudaMemsetAsync(x, 0, sizeof(float) * domainSize_, s));
                    if (vol_.dim == 3)
                        josephScatterKernel<3><<<blocks, kForwardThreads, 0, s>>>(dRays_, nrays, y,
                                                                                 vol_, x);
                    else
                        josephScatterKernel<2><<<blocks, kForwardThreads, 0, s>>>(dRays_, nrays, y,
                                                                                 vol_, x);
                    ELSA_LAUNCH_CHECK("josephScatterKernel");
                    return;
                }
                if (vol_.dim == 3) {
                    if (axisPartials_ == 0) { // no ray meets the volume: nothing else writes x
                        ELSA_CUDA(cudaMemsetAsync(x, 0, sizeof(float) * domainSize_, s));
                        return;
                    }
                    const int used = usedChunks();
                    float* out = axisPartials_ > 1 ? partial_->as<float>() : x;
                    launchAxisChunks(0, used, y, out, s);
                    if (axisPartials_ > 1)
                        launchSumChunks(partial_->as<float>(), axisPartials_, domainSize_, x, s);
                    return;
                }
                float* partial = partial_ ? partial_->as<float>() : nullptr;
                auto* launch = brick_.x == 64 ? Adjoint2dLarge::launch : Adjoint2dSmall::launch;
                launch(make_int2(nBricks_.x, nBricks_.y), adjointChunks_, 1 << cpdShift_, s, dRays_,
                       dCheckpoints_, rangeSize_, y, dWindows_, dViewAxes_, vol_, det_,
                       classSpacing_, x, partial);
                ELSA_LAUNCH_CHECK("josephAdjoint2dKernel");
            }

            // Batched applies (3D matched operator): one launch per kernel for all volumes,
            // sharing the ray tables; every batch element is computed exactly as by a single
            // apply (same kernels, chunks and summation order).
            void doForwardBatch(const float* x, int64_t xs, float* y, int64_t ys, int batch,
                                cudaStream_t s) override
            {
                if (!tma_) {
                    Projector::doForwardBatch(x, xs, y, ys, batch, s);
                    return;
                }
                tma_->forwardBatch(x, xs, y, ys, batch, s);
            }
            void doAdjointBatch(const float* y, int64_t ys, float* x, int64_t xs, int batch,
                                cudaStream_t s) override
            {
                if (batch <= 0)
                    return;
                if (fast_ || scatter_ || vol_.dim != 3 || axisPartials_ == 0) {
                    Projector::doAdjointBatch(y, ys, x, xs, batch, s);
                    return;
                }
                const int used = usedChunks();
                if (axisPartials_ <= 1) {
                    launchAxisChunks(0, used, y, x, s, batch, ys, xs);
                    return;
                }
                // partial volumes for as many batch elements as fit in kBatchPartialMemory
                const int64_t perElem = static_cast<int64_t>(axisPartials_) * domainSize_;
                const int fit = static_cast<int>(std::max<int64_t>(
                    1, std::min<int64_t>(batch, kBatchPartialMemory / (4 * perElem))));
                const size_t need = sizeof(float) * static_cast<size_t>(perElem) * fit;
                if (partial_->bytes() < need) {
                    ELSA_CUDA(cudaStreamSynchronize(s)); // no launch in flight reads the old one
                    ELSA_CUDA(cudaDeviceSynchronize());
                    partial_.reset();
                    partial_ = std::make_unique<DeviceBuffer>(need);
                }
                for (int b0 = 0; b0 < batch; b0 += fit) {
                    const int nb = std::min(fit, batch - b0);
                    launchAxisChunks(0, used, y + b0 * ys, partial_->as<float>(), s, nb, ys,
                                     perElem);
                    for (int b = 0; b < nb; ++b)
                        launchSumChunks(partial_->as<float>() + b * perElem, axisPartials_,
                                        domainSize_, x + (b0 + b) * xs, s);
                }
            }

            // Host-buffer pipelining: kHostGroups groups of views for the TMA forward; for the
            // chunked 3D brick-owner adjoint, groups of whole view chunks. Only the copy of the
            // forward's last group and of the adjoint's first group are not overlapped with a
            // kernel, so those groups are small: the forward's groups hold 30/30/30/10 % of
            // the views, the adjoint's first group one view chunk and the rest thirds.
            static constexpr int kHostGroups = 4;
            int forwardGroups() const override
            {
                return tma_ && det_.np >= 10 ? kHostGroups : 0;
            }
            std::pair<int, int> forwardGroupViews(int g, int G) const override
            {
                static constexpr int kEnd[kHostGroups + 1] = {0, 30, 60, 90, 100};
                (void)G;
                return {static_cast<int>(static_cast<int64_t>(det_.np) * kEnd[g] / 100),
                        static_cast<int>(static_cast<int64_t>(det_.np) * kEnd[g + 1] / 100)};
            }
            // first chunk of adjoint group g (g = 0 .. kHostGroups)
            int groupChunk(int g) const
            {
                const int used = usedChunks();
                if (g == 0)
                    return 0;
                return 1 + static_cast<int>(static_cast<int64_t>(used - 1) * (g - 1) /
                                            (kHostGroups - 1));
            }
            void prepareForward(const float* x, cudaStream_t s) override { tma_->prepare(x, s); }
            void forwardGroup(const float* x, float* y, int g, int G, cudaStream_t s) override
            {
                const auto v = forwardGroupViews(g, G);
                tma_->forwardViews(x, y, v.first, v.second, s);
            }
            int usedChunks() const
            {
                const int per = (det_.np + adjointChunks_ - 1) / adjointChunks_;
                return (det_.np + per - 1) / per;
            }
            int adjointGroups() const override
            {
                if (fast_ || scatter_ || vol_.dim != 3 || axisPartials_ <= 1)
                    return 0;
                return usedChunks() >= kHostGroups ? kHostGroups : 0;
            }
            std::pair<int, int> adjointGroupViews(int g, int G) const override
            {
                (void)G;
                const int per = (det_.np + adjointChunks_ - 1) / adjointChunks_;
                return {std::min(det_.np, groupChunk(g) * per),
                        std::min(det_.np, groupChunk(g + 1) * per)};
            }
            void adjointGroup(const float* y, int g, int G, cudaStream_t s) override
            {
                (void)G;
                launchAxisChunks(groupChunk(g), groupChunk(g + 1), y, partial_->as<float>(), s);
            }
            void adjointFinish(float* x, cudaStream_t s) override
            {
                launchSumChunks(partial_->as<float>(), axisPartials_, domainSize_, x, s);
            }

            std::vector<int> knobCandidates(int knob) const override
            {
                if (fast_ && knob != kKnobForwardThreads)
                    return {}; // the fast adjoint has no adjoint knobs
                if (knob == kKnobAdjointChunks) {
                    // partial volumes limited to 4 GiB
                    const int64_t byMemory =
                        std::max<int64_t>(1, (int64_t(1) << 32) / (4 * domainSize_));
                    const int limit = static_cast<int>(
                        std::min<int64_t>(std::min<int64_t>(det_.np, 256), byMemory));
                    return chunkCandidates(limit, std::min(limit, defaultChunks()));
                }
                if (knob == kKnobForwardThreads && !tma_)
                    return {64, 128, 256, 512};
                if (knob == kKnobAdjointScatter)
                    return {0, 1};
                if (knob == kKnobCheckpointDepth && vol_.dim == 3) {
                    // depths whose table takes at most an eighth of the device's memory, and
                    // the current one
                    size_t freeBytes = 0, totalBytes = 0;
                    ELSA_CUDA(cudaMemGetInfo(&freeBytes, &totalBytes));
                    const int maxDim = std::max(vol_.n[0], std::max(vol_.n[1], vol_.n[2]));
                    std::vector<int> c;
                    for (int cpd = kAxisCheckpointDepth; cpd <= 128; cpd *= 2)
                        if (cpd == (1 << cpdShift_) ||
                            8.0 * static_cast<double>(rangeSize_) * (maxDim / cpd + 3) <=
                                static_cast<double>(totalBytes) / 8.0)
                            c.push_back(cpd);
                    return c;
                }
                return {};
            }

            int knob(int knob) const override
            {
                if (knob == kKnobCheckpointDepth)
                    return vol_.dim == 3 && !fast_ ? 1 << cpdShift_ : -1;
                if (knob == kKnobAdjointChunks)
                    return adjointChunks_;
                if (knob == kKnobForwardThreads)
                    return tma_ ? -1 : forwardThreads_;
                if (knob == kKnobAdjointScatter)
                    return scatter_;
                return -1;
            }

            void setKnob(int knob, int value) override
            {
                const std::vector<int> c = knobCandidates(knob);
                if (knob == kKnobAdjointChunks && value == defaultChunks()) {
                    // the default is always allowed, also past the tuning limits
                } else if (std::find(c.begin(), c.end(), value) == c.end()) {
                    throw Error(ELSA_ERROR_INVALID_ARGUMENT,
                                "JosephsMethod: value " + std::to_string(value) +
                                    " is not a candidate of knob " + std::to_string(knob));
                }
                if (batchRefs_.load() > 0 && knob != kKnobForwardThreads)
                    throw Error(ELSA_ERROR_INVALID_ARGUMENT,
                                "JosephsMethod: a batched solver holds this operator's adjoint "
                                "tables; destroy it before changing an adjoint knob");
                if (knob == kKnobForwardThreads) {
                    forwardThreads_ = value;
                    return;
                }
                if (knob == kKnobAdjointScatter) {
                    scatter_ = value;
                    return;
                }
                if (knob == kKnobCheckpointDepth) {
                    buildCheckpoints(value);
                    return;
                }
                adjointChunks_ = value;
                const int volumes = vol_.dim == 3 ? buildAxisEntries() : value;
                const size_t need = sizeof(float) * static_cast<size_t>(domainSize_) *
                                    static_cast<size_t>(volumes);
                if (volumes <= 1)
                    partial_.reset();
                else if (!partial_ || partial_->bytes() < need) {
                    partial_.reset();
                    partial_ = std::make_unique<DeviceBuffer>(need);
                }
            }

            // Checkpoint slab depth of the 3D adjoint by default: the smallest of 16, 32, 64, 128
            // planes whose table (8 bytes per ray and slab) takes at most an eighth of the
            // device's memory (256^3 / 360 x 384^2: 16 planes, 8.1 GB; 512^3 / 720 x 768^2: 128
            // planes, 15 GB instead of 119 GB). Deeper slabs cost catch-up additions from the
            // slab's checkpoint to a brick's first plane; the results are the same.
            int defaultCheckpointDepth() const
            {
                size_t freeBytes = 0, totalBytes = 0;
                ELSA_CUDA(cudaMemGetInfo(&freeBytes, &totalBytes));
                const int maxDim = std::max(vol_.n[0], std::max(vol_.n[1], vol_.n[2]));
                int cpd = kAxisCheckpointDepth;
                while (cpd < 128 && 8.0 * static_cast<double>(rangeSize_) * (maxDim / cpd + 3) >
                                        static_cast<double>(totalBytes) / 8.0)
                    cpd *= 2;
                return cpd;
            }

            // (Re)builds the slab checkpoints for slabs of cpd planes.
            void buildCheckpoints(int cpd)
            {
                if (dCheckpoints_ != nullptr) {
                    ELSA_CUDA(cudaDeviceSynchronize()); // no adjoint may still read the table
                    ELSA_CUDA(cudaFree(dCheckpoints_));
                    dCheckpoints_ = nullptr;
                }
                int shift = 0;
                while ((1 << shift) < cpd)
                    ++shift;
                cpdShift_ = shift;
                const int maxDim = std::max(vol_.n[0], std::max(vol_.n[1], vol_.n[2]));
                const int64_t nrays = rangeSize_;
                cpStride_ = maxDim / cpd + 3;
                ELSA_CUDA(cudaMalloc(&dCheckpoints_, sizeof(float2) * nrays * cpStride_));
                const unsigned blocks = static_cast<unsigned>((nrays + 255) / 256);
                josephCheckpointKernel<<<blocks, 256>>>(dRays_, nrays, cpd, cpStride_,
                                                        dCheckpoints_);
                ELSA_LAUNCH_CHECK("josephCheckpointKernel");
            }

            bool setWaitTest(long long cycles, bool withhold) override
            {
                if (!tma_)
                    return false;
                tma_->setWaitTest(cycles, withhold);
                return true;
            }

            int64_t info(int key) const override
            {
                switch (key) {
                case 0:
                    return classSpacing_;
                case 1: // bricks of the matched adjoint (3D: over the axis grids)
                    if (vol_.dim == 3) {
                        int64_t n = 0;
                        for (const AxisGrid& g : grids_)
                            if (g.present)
                                n += static_cast<int64_t>(g.nb.x) * g.nb.y * g.nb.z;
                        return n;
                    }
                    return nBricks_.x * nBricks_.y * nBricks_.z;
                case 2:
                    return sampleCount_;
                case 3: // error word of the TMA forward (synchronizes)
                    return tma_ ? static_cast<int64_t>(tma_->errorWord()) : 0;
                case 4: // parts per million of detector tiles on the gather fallback
                    return tma_ ? static_cast<int64_t>(tma_->fallbackFraction() * 1e6) : -1;
                case 6: // kernel launches per forward call
                    return tma_ ? tma_->launchesPerForward() : (lines_ ? 2 : 1);
                case 7: // kernel launches per adjoint call (3D: one per axis grid; with
                        // several partial volumes: + the chunk sum)
                    if (fast_ || scatter_)
                        return 1;
                    if (vol_.dim == 3) {
                        int n = 0;
                        for (const AxisGrid& g : grids_)
                            n += g.present && g.entryEnd > g.entryBegin ? 1 : 0;
                        return n + (axisPartials_ > 1 ? 1 : 0);
                    }
                    return adjointChunks_ > 1 ? 2 : 1;
                case 8: // taps outside the windows of their bricks (test support; synchronizes)
                    return windowMisses();
                default:
                    return -1;
                }
            }

        private:
            int64_t windowMisses() const
            {
                if (fast_ || (vol_.dim == 2 && !dWindows_))
                    return -1;
                DeviceBuffer count(sizeof(unsigned long long));
                ELSA_CUDA(cudaMemset(count.as<unsigned long long>(), 0, sizeof(unsigned long long)));
                const int64_t nrays = rangeSize_;
                const unsigned blocks = static_cast<unsigned>((nrays + 255) / 256);
                if (vol_.dim == 3) {
                    for (int g = 0; g < 3; ++g)
                        if (grids_[g].present)
                            josephWindowCheckKernel<<<blocks, 256>>>(
                                dRays_, grids_[g].windows->as<RayWindow>(), vol_, det_,
                                grids_[g].edge, grids_[g].nb, g, count.as<unsigned long long>());
                } else {
                    josephWindowCheckKernel<<<blocks, 256>>>(dRays_, dWindows_, vol_, det_,
                                                             brick_, nBricks_, -1,
                                                             count.as<unsigned long long>());
                }
                ELSA_LAUNCH_CHECK("josephWindowCheckKernel");
                unsigned long long h = 0;
                ELSA_CUDA(cudaMemcpy(&h, count.as<unsigned long long>(), sizeof(h),
                                     cudaMemcpyDeviceToHost));
                return static_cast<int64_t>(h);
            }

            bool fast_ = false; // elsa's unmatched fast adjoint
            cudaArray_t fastArray_ = nullptr;
            cudaTextureObject_t fastTex_ = 0;
            std::unique_ptr<DeviceBuffer> fastTable_;
            int scatter_ = 0; // 1: atomic scatter adjoint (2D: 512^2 / 720 views 1.74 ms
                              // against 0.54; 3D 256^3 / 360 views 92 ms against 28.2)
            JosephRay* dRays_ = nullptr;
            unsigned* dViewAxes_ = nullptr;
            RayWindow* dWindows_ = nullptr;
            float2* dCheckpoints_ = nullptr;
            std::unique_ptr<StreamScratch> lines_; // 2D: the forward's padded image copies
            int cpStride_ = 0;
            int cpdShift_ = 4; // checkpoint slabs of 2^cpdShift_ planes (3D)

        public:
            // batched adjoint plans holding pointers into this operator's tables
            mutable std::atomic<int> batchRefs_{0};

        private:
            int classSpacing_ = 0;
            int64_t sampleCount_ = 0;
            std::unique_ptr<JosephForwardTma> tma_;
            CurvedTables curved_; // curved detector coordinates while the rays are set up
            std::unique_ptr<DeviceBuffer> partial_; // adjoint: per view-chunk partial volumes
            int adjointChunks_ = 1;                 // view chunks of the adjoint
            int forwardThreads_ = kForwardThreads;  // rays per block of the gather forward

            // View chunks of the adjoint: enough for bricks x chunks to fill the GPU (see the
            // launch configs) and at least kMinAdjointChunks, within kChunkMemory of partial
            // volumes. Finer chunks also balance bricks of uneven work: at 256^3 / 360 views
            // the adjoint takes 63.4 ms with 1 chunk, 55.5 with 8 and 54.8 with 16-32.
            int defaultChunks() const
            {
                int fill;
                if (vol_.dim == 2) {
                    fill = brick_.x == 64 ? Adjoint2dLarge::chunks(nBricks_.x * nBricks_.y, det_.np)
                                          : Adjoint2dSmall::chunks(nBricks_.x * nBricks_.y, det_.np);
                } else {
                    // bricks x chunks of the smallest present grid reach kAdjoint3dWarpsPerSm
                    // one-warp CTAs per SM (each grid sees about its share of the views)
                    int64_t nb = 0;
                    for (const AxisGrid& g : grids_)
                        if (g.present)
                            nb = std::max<int64_t>(nb, static_cast<int64_t>(g.nb.x) * g.nb.y *
                                                           g.nb.z);
                    const int64_t want = (kAdjoint3dWarpsPerSm * 148 + nb - 1) / std::max<int64_t>(nb, 1);
                    fill = static_cast<int>(std::min<int64_t>(det_.np, std::max<int64_t>(1, want)));
                }
                // partial volumes within kChunkMemory: the 3D adjoint writes one per (chunk,
                // axis grid) pair, so leave room for the chunks whose views drive along two axes
                const int64_t cap = std::max<int64_t>(1, kChunkMemory / (4 * domainSize_));
                const int64_t capChunks = vol_.dim == 3 ? std::max<int64_t>(1, cap * 7 / 8) : cap;
                const int least = vol_.dim == 3 ? kMinAdjointChunks : 1;
                return static_cast<int>(std::min<int64_t>(std::min<int64_t>(det_.np, capChunks),
                                                          std::max(fill, least)));
            }

            // ---- 3D matched adjoint on axis bricks ----

            struct AxisGrid {
                bool present = false;
                bool ub = false;   // columns (the wide, stride-1 edge) along b instead of a
                int3 edge{}, nb{}; // brick edges and brick counts in volume axis order
                std::unique_ptr<DeviceBuffer> windows; // [view][brick]
                int entryBegin = 0, entryEnd = 0;      // this grid's (chunk, partial) entries
            };
            AxisGrid grids_[3];
            std::vector<unsigned> viewAxesHost_;
            std::vector<int2> entries_;                 // (chunk, partial volume), grid-major
            std::unique_ptr<DeviceBuffer> dEntries_;
            int axisPartials_ = 0;                      // partial volumes of the 3D adjoint

            static int3 axisEdge(int g, bool ub)
            {
                int a, b;
                nonDrivingAxes(g, a, b);
                int e[3];
                e[g] = kAxisTD;
                e[a] = ub ? kAxisTV : kAxisTW;
                e[b] = ub ? kAxisTW : kAxisTV;
                return make_int3(e[0], e[1], e[2]);
            }

            // Brick grids and windows for every driving axis of the geometry.
            void buildAxisGrids()
            {
                viewAxesHost_.resize(det_.np);
                ELSA_CUDA(cudaMemcpy(viewAxesHost_.data(), dViewAxes_, sizeof(unsigned) * det_.np,
                                     cudaMemcpyDeviceToHost));
                for (int g = 0; g < 3; ++g) {
                    AxisGrid& G = grids_[g];
                    G.present = std::any_of(viewAxesHost_.begin(), viewAxesHost_.end(),
                                            [g](unsigned a) { return (a >> g) & 1u; });
                    if (!G.present)
                        continue;
                    // columns along the axis over which a detector row's rays spread, by a vote
                    // of the views driving along g (bit 4+g of a view's axis word: along b)
                    int alongB = 0, votes = 0;
                    for (unsigned w : viewAxesHost_)
                        if ((w >> g) & 1u) {
                            ++votes;
                            alongB += (w >> (4 + g)) & 1u;
                        }
                    G.ub = 2 * alongB > votes;
                    G.edge = axisEdge(g, G.ub);
                    G.nb = make_int3((vol_.n[0] + G.edge.x - 1) / G.edge.x,
                                     (vol_.n[1] + G.edge.y - 1) / G.edge.y,
                                     (vol_.n[2] + G.edge.z - 1) / G.edge.z);
                    const int64_t nwin = static_cast<int64_t>(G.nb.x) * G.nb.y * G.nb.z * det_.np;
                    G.windows = std::make_unique<DeviceBuffer>(sizeof(RayWindow) * nwin);
                    josephWindowKernel<<<static_cast<unsigned>((nwin + 255) / 256), 256>>>(
                        dPoses_, vol_, det_, G.edge, G.nb, curved_.map(), windowGrow(vol_),
                        kWindowPixelMargin, G.windows->as<RayWindow>());
                    ELSA_LAUNCH_CHECK("josephWindowKernel");
                }
            }

            // (chunk, partial volume) entries of every grid for adjointChunks_ view chunks: chunk
            // c covers views [c per, (c + 1) per); a grid takes the chunks holding a view that
            // drives along its axis. Partial volumes are numbered by (chunk, axis), the order in
            // which the chunk sum adds them. Returns the number of partial volumes.
            int buildAxisEntries()
            {
                const int per = (det_.np + adjointChunks_ - 1) / adjointChunks_;
                const int used = (det_.np + per - 1) / per;
                std::vector<std::vector<int2>> byGrid(3);
                int next = 0;
                for (int c = 0; c < used; ++c) {
                    for (int g = 0; g < 3; ++g) {
                        if (!grids_[g].present)
                            continue;
                        bool any = false;
                        for (int p = c * per; p < std::min(det_.np, (c + 1) * per) && !any; ++p)
                            any = (viewAxesHost_[p] >> g) & 1u;
                        if (any)
                            byGrid[g].push_back(make_int2(c, next++));
                    }
                }
                entries_.clear();
                for (int g = 0; g < 3; ++g) {
                    grids_[g].entryBegin = static_cast<int>(entries_.size());
                    entries_.insert(entries_.end(), byGrid[g].begin(), byGrid[g].end());
                    grids_[g].entryEnd = static_cast<int>(entries_.size());
                }
                if (next == 1) // one partial: the kernel writes x itself
                    for (auto& e : entries_)
                        e.y = 0;
                dEntries_ = std::make_unique<DeviceBuffer>(sizeof(int2) * std::max<size_t>(1, entries_.size()));
                if (!entries_.empty())
                    ELSA_CUDA(cudaMemcpy(dEntries_->as<int2>(), entries_.data(),
                                         sizeof(int2) * entries_.size(), cudaMemcpyHostToDevice));
                axisPartials_ = next;
                return next;
            }

        public:
            // This operator's share of a batched adjoint (planJosephAdjointMany): its axis-brick
            // jobs keyed by (grid, column axis), and its chunk sum (one partial volume: none; no
            // partial volume, as no ray meets the volume: a sum of none, which writes zeros).
            bool batchable() const
            {
                return vol_.dim == 3 && !fast_ && !scatter_ && dCheckpoints_ != nullptr;
            }
            void appendAxisJobs(const float* y, float* x, std::vector<AxisJob> (&jobs)[6],
                                std::vector<SumChunksEntry>& sums) const
            {
                float* out = axisPartials_ > 1 ? partial_->as<float>() : x;
                for (int g = 0; g < 3; ++g) {
                    const AxisGrid& G = grids_[g];
                    if (!G.present || G.entryEnd <= G.entryBegin)
                        continue;
                    jobs[2 * g + (G.ub ? 1 : 0)].push_back(axisJob(g, y, out));
                }
                if (axisPartials_ != 1)
                    sums.push_back(SumChunksEntry{axisPartials_ > 1 ? out : nullptr,
                                                  axisPartials_, domainSize_, x});
            }

        private:
            // The axis-brick job of grid g on sinogram y into out (entries indexed from the grid's
            // first entry; itemBase left to batched callers).
            AxisJob axisJob(int g, const float* y, float* out) const
            {
                const AxisGrid& G = grids_[g];
                AxisJob J{};
                J.rays = dRays_;
                J.checkpoints = dCheckpoints_;
                J.nrays = rangeSize_;
                J.y = y;
                J.windows = G.windows->as<RayWindow>();
                J.viewAxes = dViewAxes_;
                J.chunks = dEntries_->as<int2>() + G.entryBegin;
                J.entries = G.entryEnd - G.entryBegin;
                J.viewsPerChunk = (det_.np + adjointChunks_ - 1) / adjointChunks_;
                J.vol = vol_;
                J.det = det_;
                J.m = classSpacing_;
                J.cpdShift = cpdShift_;
                J.nBricks = G.nb;
                J.out = out;
                J.itemBase = 0;
                return J;
            }

            // The axis-brick kernels for view chunks [c0, c1), writing their partial volumes into
            // out (x itself when there is a single partial volume); `batch` sinograms
            // y + b yStride into out + b outStride.
            void launchAxisChunks(int c0, int c1, const float* y, float* out, cudaStream_t s,
                                  int batch = 1, int64_t yStride = 0, int64_t outStride = 0)
            {
                for (int g = 0; g < 3; ++g) {
                    const AxisGrid& G = grids_[g];
                    if (!G.present)
                        continue;
                    int e0 = G.entryBegin, e1 = G.entryBegin;
                    for (int e = G.entryBegin; e < G.entryEnd; ++e) {
                        if (entries_[e].x < c0)
                            e0 = e + 1;
                        if (entries_[e].x < c1)
                            e1 = e + 1;
                    }
                    if (e1 <= e0)
                        continue;
                    const dim3 grid(static_cast<unsigned>(G.nb.x * G.nb.y * G.nb.z),
                                    static_cast<unsigned>(e1 - e0), static_cast<unsigned>(batch));
                    const AxisJob J = axisJob(g, y, out);
                    // slabs of kAxisCheckpointDepth planes: the depth fixed at compile time;
                    // deeper ones (CPD 0): read from the job
                    const bool deep = (1 << cpdShift_) != kAxisCheckpointDepth;
#define ELSA_AXIS_LAUNCH(G_, UB_)                                                                \
    do {                                                                                         \
        if (deep)                                                                                \
            josephAdjointAxisKernel<G_, kAxisTD, UB_, kAxisTW, kAxisTV, 0>                       \
                <<<grid, 32, 0, s>>>(J, e0 - G.entryBegin, yStride, outStride);                  \
        else                                                                                     \
            josephAdjointAxisKernel<G_, kAxisTD, UB_, kAxisTW, kAxisTV, kAxisCheckpointDepth>     \
                <<<grid, 32, 0, s>>>(J, e0 - G.entryBegin, yStride, outStride);                  \
    } while (0)
                    if (g == 0) {
                        if (G.ub)
                            ELSA_AXIS_LAUNCH(0, true);
                        else
                            ELSA_AXIS_LAUNCH(0, false);
                    } else if (g == 1) {
                        if (G.ub)
                            ELSA_AXIS_LAUNCH(1, true);
                        else
                            ELSA_AXIS_LAUNCH(1, false);
                    } else {
                        if (G.ub)
                            ELSA_AXIS_LAUNCH(2, true);
                        else
                            ELSA_AXIS_LAUNCH(2, false);
                    }
#undef ELSA_AXIS_LAUNCH
                    ELSA_LAUNCH_CHECK("josephAdjointAxisKernel");
                }
            }

            int3 brick_{}, nBricks_{};
        };
    } // namespace

    void launchBrickWindows(const float* poses, const VolumeShape& vol, const DetectorShape& det,
                            int3 brick, int3 nBricks, RayWindow* out, cudaStream_t s,
                            CurvedMap cm, float grow, float pixMargin)
    {
        const int64_t nwin = static_cast<int64_t>(nBricks.x) * nBricks.y * nBricks.z * det.np;
        if (nwin == 0)
            return;
        josephWindowKernel<<<static_cast<unsigned>((nwin + 255) / 256), 256, 0, s>>>(
            poses, vol, det, brick, nBricks, cm, grow, pixMargin, out);
        ELSA_LAUNCH_CHECK("josephWindowKernel");
    }

    void launchSumChunks(const float* partial, int chunks, int64_t nvox, float* x,
                         cudaStream_t s)
    {
        if (nvox == 0)
            return;
        sumChunksKernel<<<static_cast<unsigned>((nvox + 255) / 256), 256, 0, s>>>(partial, chunks,
                                                                                  nvox, x);
        ELSA_LAUNCH_CHECK("sumChunksKernel");
    }

    class AdjointManyPlan
    {
    public:
        std::unique_ptr<DeviceBuffer> jobs[6]; // per (grid, column axis)
        int64_t items[6] = {0, 0, 0, 0, 0, 0};
        int counts[6] = {0, 0, 0, 0, 0, 0};
        std::unique_ptr<DeviceBuffer> sums;
        int sumCount = 0;
        int64_t maxVox = 0;
        bool deep = false; // some instance uses checkpoint slabs deeper than kAxisCheckpointDepth
        // operators whose tables the jobs point into: their adjoint knobs stay fixed meanwhile
        std::vector<const JosephProjector*> holds;
        ~AdjointManyPlan()
        {
            for (const JosephProjector* J : holds)
                --J->batchRefs_;
        }
    };

    std::shared_ptr<AdjointManyPlan> planJosephAdjointMany(const std::vector<Projector*>& ops,
                                                           const std::vector<const float*>& ys,
                                                           const std::vector<float*>& xs)
    {
        if (ops.size() != ys.size() || ops.size() != xs.size())
            throw Error(ELSA_ERROR_INVALID_ARGUMENT, "planJosephAdjointMany: size mismatch");
        std::vector<AxisJob> jobs[6];
        std::vector<SumChunksEntry> sums;
        auto plan = std::make_shared<AdjointManyPlan>();
        for (size_t i = 0; i < ops.size(); ++i) {
            const auto* J = dynamic_cast<const JosephProjector*>(ops[i]);
            if (!J || !J->batchable())
                throw Error(ELSA_ERROR_NOT_SUPPORTED,
                            "batched adjoints take 3D Joseph operators with the matched "
                            "brick-owner adjoint only");
            J->appendAxisJobs(ys[i], xs[i], jobs, sums);
            ++J->batchRefs_;
            plan->holds.push_back(J);
            plan->maxVox = std::max(plan->maxVox, J->domainSize());
            plan->deep = plan->deep || J->knob(kKnobCheckpointDepth) != kAxisCheckpointDepth;
        }
        for (int k = 0; k < 6; ++k) {
            int64_t base = 0;
            for (AxisJob& j : jobs[k]) {
                j.itemBase = base;
                base += static_cast<int64_t>(j.nBricks.x) * j.nBricks.y * j.nBricks.z * j.entries;
            }
            if (base >= (int64_t(1) << 31))
                throw Error(ELSA_ERROR_NOT_SUPPORTED, "planJosephAdjointMany: too many bricks");
            plan->items[k] = base;
            plan->counts[k] = static_cast<int>(jobs[k].size());
            if (!jobs[k].empty()) {
                plan->jobs[k] = std::make_unique<DeviceBuffer>(sizeof(AxisJob) * jobs[k].size());
                ELSA_CUDA(cudaMemcpy(plan->jobs[k]->as<AxisJob>(), jobs[k].data(),
                                     sizeof(AxisJob) * jobs[k].size(), cudaMemcpyHostToDevice));
            }
        }
        plan->sumCount = static_cast<int>(sums.size());
        if (!sums.empty()) {
            plan->sums = std::make_unique<DeviceBuffer>(sizeof(SumChunksEntry) * sums.size());
            ELSA_CUDA(cudaMemcpy(plan->sums->as<SumChunksEntry>(), sums.data(),
                                 sizeof(SumChunksEntry) * sums.size(), cudaMemcpyHostToDevice));
        }
        return plan;
    }

    void runJosephAdjointMany(const AdjointManyPlan& plan, cudaStream_t s)
    {
        constexpr int TD = kAxisTD, TW = kAxisTW, TV = kAxisTV, CPD = kAxisCheckpointDepth;
        for (int k = 0; k < 6; ++k) {
            if (plan.items[k] == 0)
                continue;
            const unsigned grid = static_cast<unsigned>(plan.items[k]);
            const AxisJob* jobs = plan.jobs[k]->as<AxisJob>();
            const int n = plan.counts[k];
#define ELSA_AXIS_MANY(G_, UB_)                                                                   \
    do {                                                                                         \
        if (plan.deep)                                                                           \
            josephAdjointAxisManyKernel<G_, TD, UB_, TW, TV, 0><<<grid, 32, 0, s>>>(jobs, n);    \
        else                                                                                     \
            josephAdjointAxisManyKernel<G_, TD, UB_, TW, TV, CPD><<<grid, 32, 0, s>>>(jobs, n);  \
    } while (0)
            switch (k) {
            case 0: ELSA_AXIS_MANY(0, false); break;
            case 1: ELSA_AXIS_MANY(0, true); break;
            case 2: ELSA_AXIS_MANY(1, false); break;
            case 3: ELSA_AXIS_MANY(1, true); break;
            case 4: ELSA_AXIS_MANY(2, false); break;
            default: ELSA_AXIS_MANY(2, true); break;
            }
#undef ELSA_AXIS_MANY
            ELSA_LAUNCH_CHECK("josephAdjointAxisManyKernel");
        }
        if (plan.sumCount > 0) {
            const int64_t blocks = std::min<int64_t>((plan.maxVox + 255) / 256, 148 * 8);
            sumChunksManyKernel<<<dim3(static_cast<unsigned>(blocks),
                                       static_cast<unsigned>(plan.sumCount)),
                                  256, 0, s>>>(plan.sums->as<SumChunksEntry>());
            ELSA_LAUNCH_CHECK("sumChunksManyKernel");
        }
    }

    std::unique_ptr<Projector> makeJosephProjector(const VolumeShape& vol,
                                                   const DetectorShape& det,
                                                   const std::vector<PoseRecord>& poses,
                                                   const CurvedDetector& curved, bool fast)
    {
        return std::make_unique<JosephProjector>(vol, det, poses, curved, fast);
    }
} // namespace elsa_b200
