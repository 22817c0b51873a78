// Per-ray traversal setup for the ray-driven projectors.
//
// This translation unit is compiled with --fmad=false: every multiply and add below must round
// separately so that the records are bit-identical to elsa's float CPU path:
//   ray:        core/Descriptors/DetectorDescriptor.cpp:90-128 (rd = normalize(Pinv [u+.5,v+.5,1]))
//   intersect:  projectors/Intersection.cpp:7-46 (slab test on [0, N])
//   traversal:  projectors/DrivingDirectionTraversal.cpp:6-57 (driving axis, .5-plane shift,
//               step count, intersection length)
//   Siddon:     projectors/TraverseAABB.cpp:6-40,104-166 (entry voxel, tDelta, first T)
//   LutProjector (ray-driven blob / B-spline): projectors/LutProjector.h:85-163 with
//               SliceTraversal.cpp:7-200, Intersection.cpp:47-119, CartesianIndices.cpp:341-356
#include "internal.cuh"
#include "raysetup.cuh"

#include <cfloat>
#include <type_traits>

namespace elsa_b200
{
    namespace
    {
        __device__ __forceinline__ float minNum(float x, float y)
        {
            return (y != y) ? x : (x < y ? x : y);
        }
        __device__ __forceinline__ float maxNum(float x, float y)
        {
            return (y != y) ? x : (x > y ? x : y);
        }

        // Ray through the centre of pixel (u, v) of a pose record, or, for a curved detector,
        // through the planar coordinate planar[u + nu * v] of that pixel centre
        // (CurvedDetectorDescriptor::computeRayFromDetectorCoord,
        // core/Descriptors/CurvedDetectorDescriptor.cpp:93-120).
        __device__ void pixelRay(const float* pose, int dim, int u, int v, const float2* planar,
                                 int nu, float* o, float* d)
        {
            const float* Pinv = pose + 12;
            float h0 = static_cast<float>(u) + 0.5f;
            float h1 = (dim == 3) ? static_cast<float>(v) + 0.5f : 1.0f;
            if (planar) {
                const float2 c = planar[u + static_cast<int64_t>(nu) * v];
                h0 = c.x;
                if (dim == 3)
                    h1 = c.y;
            }
            float dir[3];
            if (dim == 3) {
                for (int i = 0; i < 3; ++i) {
                    float s = 0.0f;
                    s = s + Pinv[i * 3 + 0] * h0;
                    s = s + Pinv[i * 3 + 1] * h1;
                    s = s + Pinv[i * 3 + 2] * 1.0f;
                    dir[i] = s;
                }
            } else {
                for (int i = 0; i < 2; ++i) {
                    float s = 0.0f;
                    s = s + Pinv[i * 2 + 0] * h0;
                    s = s + Pinv[i * 2 + 1] * 1.0f;
                    dir[i] = s;
                }
                dir[2] = 0.0f;
            }
            float z = dir[0] * dir[0];
            z = z + dir[1] * dir[1];
            if (dim == 3)
                z = z + dir[2] * dir[2];
            const float nrm = sqrtf(z);
            for (int i = 0; i < dim; ++i) {
                d[i] = z > 0.0f ? dir[i] / nrm : dir[i];
                o[i] = pose[24 + i];
            }
        }

        __device__ bool slabIntersect(const float* boxMax, int dim, const float* o, const float* d,
                                      float& tmin, float& tmax)
        {
            float inv = 1.0f / d[0];
            float t1 = (0.0f - o[0]) * inv;
            float t2 = (boxMax[0] - o[0]) * inv;
            tmin = inv >= 0.0f ? t1 : t2;
            tmax = inv >= 0.0f ? t2 : t1;
            for (int i = 1; i < dim; ++i) {
                inv = 1.0f / d[i];
                t1 = (0.0f - o[i]) * inv;
                t2 = (boxMax[i] - o[i]) * inv;
                tmin = maxNum(tmin, inv >= 0.0f ? t1 : t2);
                tmax = minNum(tmax, inv >= 0.0f ? t2 : t1);
            }
            if (tmax == 0.0f && tmin == 0.0f)
                return false;
            return tmax >= maxNum(tmin, 0.0f);
        }
    } // namespace

    __global__ void josephSetupKernel(const float* __restrict__ poses, VolumeShape vol,
                                      DetectorShape det, const float2* __restrict__ planar,
                                      JosephRay* __restrict__ rays)
    {
        const int64_t nrays = static_cast<int64_t>(det.nu) * det.nv * det.np;
        const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
        if (r >= nrays)
            return;
        const int dim = vol.dim;
        const int u = static_cast<int>(r % det.nu);
        const int v = static_cast<int>((r / det.nu) % det.nv);
        const int p = static_cast<int>(r / (static_cast<int64_t>(det.nu) * det.nv));
        float o[3] = {0, 0, 0}, d[3] = {0, 0, 0};
        pixelRay(poses + static_cast<int64_t>(p) * 40, dim, u, v, planar, det.nu, o, d);
        float boxMax[3] = {static_cast<float>(vol.n[0]), static_cast<float>(vol.n[1]),
                           static_cast<float>(vol.n[2])};
        float tmin, tmax;
        const bool hit = slabIntersect(boxMax, dim, o, d, tmin, tmax);
        int drv = 0;
        float best = fabsf(d[0]);
        for (int i = 1; i < dim; ++i)
            if (fabsf(d[i]) > best) {
                best = fabsf(d[i]);
                drv = i;
            }
        int a, b;
        nonDrivingAxes(drv, a, b);
        JosephRay rec;
        rec.pa = rec.pb = rec.sa = rec.sb = rec.len = 0.0f;
        rec.k0 = 0;
        rec.n = 0;
        rec.meta = drv;
        if (hit) {
            float pos[3] = {0, 0, 0}, ex[3] = {0, 0, 0}, step[3] = {0, 0, 0};
            for (int i = 0; i < dim; ++i) {
                pos[i] = o[i] + d[i] * tmin;
                ex[i] = o[i] + d[i] * tmax;
                pos[i] = pos[i] < 0.0f ? 0.0f : pos[i];
                pos[i] = pos[i] > boxMax[i] ? boxMax[i] : pos[i];
                ex[i] = ex[i] < 0.0f ? 0.0f : ex[i];
                ex[i] = ex[i] > boxMax[i] ? boxMax[i] : ex[i];
            }
            const float absd = fabsf(d[drv]);
            for (int i = 0; i < dim; ++i)
                step[i] = d[i] / absd;
            const float dist = pos[drv] - floorf(pos[drv]);
            const float sgn = step[drv] > 0.0f ? 1.0f : (step[drv] < 0.0f ? -1.0f : 0.0f);
            const float shift = 0.5f - dist;
            for (int i = 0; i < dim; ++i)
                pos[i] = pos[i] + (step[i] * shift) * sgn;
            pos[drv] = floorf(pos[drv]) + 0.5f;
            const float nsteps = ceilf(fabsf(ex[drv] - pos[drv]));
            float len;
            if (dim == 3)
                len = sqrtf(step[0] * step[0] + (step[1] * step[1] + step[2] * step[2]));
            else
                len = sqrtf(step[0] * step[0] + step[1] * step[1]);
            rec.pa = pos[a];
            rec.sa = step[a];
            if (dim == 3) {
                rec.pb = pos[b];
                rec.sb = step[b];
            }
            rec.len = len;
            rec.k0 = static_cast<int>(floorf(pos[drv] - 0.5f));
            rec.n = static_cast<int>(nsteps);
            rec.meta = drv | (sgn < 0.0f ? 4 : 0);
        }
        rays[r] = rec;
    }

    __global__ void siddonSetupKernel(const float* __restrict__ poses, VolumeShape vol,
                                      DetectorShape det, const float2* __restrict__ planar,
                                      SiddonRay* __restrict__ rays,
                                      SiddonLine* __restrict__ lines)
    {
        const int64_t nrays = static_cast<int64_t>(det.nu) * det.nv * det.np;
        const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
        if (r >= nrays)
            return;
        const int dim = vol.dim;
        const int u = static_cast<int>(r % det.nu);
        const int v = static_cast<int>((r / det.nu) % det.nv);
        const int p = static_cast<int>(r / (static_cast<int64_t>(det.nu) * det.nv));
        float o[3] = {0, 0, 0}, d[3] = {0, 0, 0};
        pixelRay(poses + static_cast<int64_t>(p) * 40, dim, u, v, planar, det.nu, o, d);
        float boxMax[3] = {static_cast<float>(vol.n[0]), static_cast<float>(vol.n[1]),
                           static_cast<float>(vol.n[2])};
        float tmin, tmax;
        bool inBox = slabIntersect(boxMax, dim, o, d, tmin, tmax);
        int g = 0;
        float best = fabsf(d[0]);
        for (int i = 1; i < dim; ++i)
            if (fabsf(d[i]) > best) {
                best = fabsf(d[i]);
                g = i;
            }
        int a, b;
        nonDrivingAxes(g, a, b);
        SiddonRay rec;
        for (int i = 0; i < 3; ++i) {
            rec.tDelta[i] = FLT_MAX;
            rec.T[i] = FLT_MAX;
        }
        rec.meta = g;
        rec.kFirst = rec.kLast = 0;
        rec.cur[0] = rec.cur[1] = 0;
        rec.crossings = 0;
        SiddonLine line{0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (inBox) {
            // entry point clamped to the box, TraverseAABB.cpp:13-20
            float entry[3] = {0, 0, 0}, cur[3] = {0, 0, 0};
            int stepDir[3] = {0, 0, 0};
            for (int i = 0; i < dim; ++i) {
                float e = o[i] + d[i] * tmin;
                e = e < 0.0f ? 0.0f : e;
                e = e > boxMax[i] ? boxMax[i] : e;
                entry[i] = e;
                stepDir[i] = d[i] > 0.0f ? 1 : (d[i] < 0.0f ? -1 : 0);
            }
            // entry voxel (one lower on a boundary when stepping down), :123-137
            for (int i = 0; i < dim; ++i) {
                float lc = floorf(entry[i]);
                if (lc == entry[i] && stepDir[i] < 0)
                    lc = lc - 1.0f;
                cur[i] = lc;
                if (cur[i] >= boxMax[i] || cur[i] < 0.0f)
                    inBox = false;
            }
            if (inBox) {
                for (int i = 0; i < dim; ++i) {
                    const bool moves = fabsf(d[i]) > FLT_EPSILON;
                    rec.tDelta[i] = moves ? static_cast<float>(stepDir[i]) / d[i] : FLT_MAX;
                    const float bound = d[i] > 0.0f ? cur[i] + 1.0f : cur[i];
                    rec.T[i] = moves ? (bound - entry[i]) / d[i] : FLT_MAX;
                    if (stepDir[i] < 0)
                        rec.meta |= 4 << i;
                    if (stepDir[i] == 0)
                        rec.meta |= 32 << i;
                }
                rec.meta |= 256;
                rec.kFirst = rec.kLast = static_cast<int>(cur[g]);
                rec.cur[0] = static_cast<int>(cur[a]);
                rec.cur[1] = dim == 3 ? static_cast<int>(cur[b]) : 0;
                line.g0 = entry[g];
                line.a0 = entry[a];
                line.sa = d[a] / d[g];
                if (dim == 3) {
                    line.b0 = entry[b];
                    line.sb = d[b] / d[g];
                }
            }
        }
        rays[r] = rec;
        if (lines)
            lines[r] = line;
    }

    // ---- ray-driven LUT projector -----------------------------------------------------------
    namespace
    {
        // Lut::operator() (projectors/Luts.hpp:61-80): linear interpolation of n samples on
        // [0, support], 0 outside, at two distances, with the reference's float operations
        // (distance / support * (n - 1), then t lut[ceil] + (1 - t) lut[floor]). The table is
        // staged as pairs (lut[i], lut[i + 1]), kLutCopies times: copy l % kLutCopies serves lane
        // l, so a half-warp reads 16 different bank pairs. At an integer index t is 0 and the
        // second entry of the pair has no effect.
        constexpr int kLutCopies = 16;
        __device__ __forceinline__ void stageLut(const float* __restrict__ lut, int n, float2* tab)
        {
            for (int i = threadIdx.x; i < n * kLutCopies; i += blockDim.x) {
                const int a = i / kLutCopies;
                tab[i] = make_float2(lut[a], lut[min(a + 1, n - 1)]);
            }
        }
        __device__ __forceinline__ float2 lutValue2(const float2* tab, int n, float support,
                                                    float exactInv, float2 distance,
                                                    float2 minusZero)
        {
            const float top = static_cast<float>(n - 1);
            float2 q;
            if (exactInv != 0.0f) { // support is a power of two
                q = mul2(distance, splat2(exactInv));
            } else if (midRange(support)) {
                const float2 b = splat2(support);
                q = quotient2(distance, b, refineRcp2(b, splat2(rcpApprox(support))));
            } else {
                q = make_float2(distance.x / support, distance.y / support);
            }
            const float2 index = fma2(q, splat2(top), minusZero);
            int a0, a1;
            const float2 inside = make_float2(fminf(index.x, top), fminf(index.y, top));
            const float2 af = floorSmall2(inside, a0, a1);
            const float2 e0 = tab[a0 * kLutCopies + threadIdx.x % kLutCopies];
            const float2 e1 = tab[a1 * kLutCopies + threadIdx.x % kLutCopies];
            const float2 t = sub2(index, af);
            const float2 v =
                add2(fma2(t, make_float2(e0.y, e1.y), minusZero),
                     fma2(sub2(splat2(1.0f), t), make_float2(e0.x, e1.x), minusZero));
            return make_float2(index.x > top ? 0.0f : v.x, index.y > top ? 0.0f : v.y);
        }

        struct SliceWalk {
            float start[3];
            float step[3];
            int count;
        };

        // SliceTraversal(box [lo, hi], ray) of the reference: the ray and box in traversal
        // coordinates (rotation R of the leading axis onto +x about the box centre hi / 2),
        // intersectXPlanes with its advance / retreat to voxel centres, then the slice walk along
        // the original ray. False when the ray misses.
        __device__ bool sliceWalk(int dim, const float* bmin, const float* bmax, const float* ro,
                                  const float* rd, const float* R, SliceWalk& w)
        {
            float centre[3] = {0.0f, 0.0f, 0.0f}, tcol[3] = {0.0f, 0.0f, 0.0f};
            for (int i = 0; i < dim; ++i)
                centre[i] = bmax[i] / 2.0f;
            for (int i = 0; i < dim; ++i) {
                float acc = 0.0f;
                for (int k = 0; k < dim; ++k)
                    acc = acc + R[i * 3 + k] * (-centre[k]);
                tcol[i] = acc + 0.0f;
            }
            float o[3], d[3], lo[3], hi[3];
            for (int i = 0; i < dim; ++i) {
                float ao = 0.0f, ad = 0.0f, al = 0.0f, ah = 0.0f;
                for (int k = 0; k < dim; ++k) {
                    ao = ao + R[i * 3 + k] * ro[k];
                    ad = ad + R[i * 3 + k] * rd[k];
                    al = al + R[i * 3 + k] * bmin[k];
                    ah = ah + R[i * 3 + k] * bmax[k];
                }
                o[i] = ao + tcol[i];
                d[i] = ad;
                lo[i] = al + tcol[i];
                hi[i] = ah + tcol[i];
                if (lo[i] > hi[i]) {
                    const float t = lo[i];
                    lo[i] = hi[i];
                    hi[i] = t;
                }
            }
            lo[0] = lo[0] + 0.5f;
            hi[0] = hi[0] - 0.5f;
            float inv = 1.0f / d[0];
            float t1 = (lo[0] - o[0]) * inv, t2 = (hi[0] - o[0]) * inv;
            float tmin = inv >= 0.0f ? t1 : t2, tmax = inv >= 0.0f ? t2 : t1;
            const float txmin = tmin, txmax = tmax;
            for (int i = 1; i < dim; ++i) {
                inv = 1.0f / d[i];
                t1 = (lo[i] - o[i]) * inv;
                t2 = (hi[i] - o[i]) * inv;
                tmin = maxNum(tmin, inv >= 0.0f ? t1 : t2);
                tmax = minNum(tmax, inv >= 0.0f ? t2 : t1);
            }
            const float xc = fabsf(lo[0] - static_cast<float>(static_cast<int>(roundf(lo[0]))));
            if (txmin < tmin) {
                const float e = o[0] + tmin * d[0];
                float ip;
                const float tmp = fabsf(modff(e - xc, &ip));
                const float frac = e < xc ? tmp : 1.0f - tmp;
                tmin = tmin + ((static_cast<double>(tmp) > 0.00001 &&
                                static_cast<double>(frac) > 0.00001)
                                   ? frac / d[0]
                                   : 0.0f);
            }
            if (txmax > tmax) {
                const float e = o[0] + tmax * d[0];
                float ip;
                const float tmp = fabsf(modff(e - xc, &ip));
                const float frac = e < xc ? 1.0f - tmp : tmp;
                tmax = tmax - ((static_cast<double>(tmp) > 0.00001 &&
                                static_cast<double>(frac) > 0.00001)
                                   ? frac / d[0]
                                   : 0.0f);
            }
            if (tmax == 0.0f && tmin == 0.0f)
                return false;
            if (!(static_cast<double>(tmax - maxNum(tmin, 0.0f)) > -0.000001))
                return false;
            const float first = o[0] + tmin * d[0], last = o[0] + tmax * d[0];
            w.count = max(1, static_cast<int>(ceilf(last - first + 0.5f)));
            const float tDelta = 1.0f / d[0];
            for (int i = 0; i < 3; ++i) {
                w.start[i] = i < dim ? ro[i] + tmin * rd[i] : 0.0f;
                w.step[i] = i < dim ? rd[i] * tDelta : 0.0f;
            }
            return true;
        }

        // Every (voxel, weight) of one ray with leading axis LEAD (LutProjector.h:85-163): the
        // slice walk over the volume box (forward) or the box grown by `support` off the leading
        // axis (backward), and per slice the voxels within `support` in the other axes, last axis
        // fastest, in pairs on the packed two-wide FP32 instructions (the reference's float
        // operations and order per voxel). f(word, two, weights): the voxels at `word` and, when
        // `two`, at the next one along the inner axis. stride: words per axis of the volume copy.
        template <int DIM, int LEAD, class F>
        __device__ __forceinline__ void lutRayAlong(const LutProjParams& lp, const float2* tab,
                                                    const int64_t* stride, const float* ro,
                                                    const float* rd, bool backward, F&& f)
        {
            // Products that an addition follows are written as fma with -0 from a kernel
            // argument: the assembler contracts a packed mul and add into one fma, which rounds
            // once where the reference rounds twice.
            const float2 zero = splat2(lp.minusZero);
            constexpr int I = DIM == 2 ? 1 - LEAD : (LEAD == 2 ? 1 : 2); // inner axis
            constexpr int O = DIM == 2 ? LEAD : 3 - LEAD - I;            // outer axis (3D)
            const int variant = LEAD * 2 + (rd[LEAD] >= 0.0f ? 0 : 1);
            float bmin[3] = {0.0f, 0.0f, 0.0f}, bmax[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int i = 0; i < DIM; ++i) {
                bmax[i] = static_cast<float>(lp.n[i]);
                if (backward && i != LEAD) {
                    bmin[i] = bmin[i] - static_cast<float>(lp.support);
                    bmax[i] = bmax[i] + static_cast<float>(lp.support);
                }
            }
            SliceWalk w;
            if (!sliceWalk(DIM, bmin, bmax, ro, rd, lp.rot[variant], w))
                return;
            float cur[3] = {w.start[0], w.start[1], w.start[2]};
            const int64_t sL = stride[LEAD], sO = DIM == 3 ? stride[O] : 0, sI = stride[I];
            for (int it = 0; it < w.count; ++it) {
                int from[3] = {0, 0, 0}, to[3] = {1, 1, 1};
#pragma unroll
                for (int i = 0; i < DIM; ++i) {
                    const int pos = static_cast<int>(cur[i]);
                    const int dist = i == LEAD ? 0 : lp.support;
                    from[i] = max(pos - dist, 0);
                    to[i] = min(pos + dist + 1, lp.n[i]);
                    if (to[i] == from[i])
                        from[i] -= 1;
                    cur[i] = cur[i] + w.step[i];
                }
                // (the leading axis has at most one voxel per slice)
                if (from[LEAD] < 0 || from[LEAD] >= to[LEAD])
                    continue;
                float2 diff[3];
                diff[LEAD] = splat2((static_cast<float>(from[LEAD]) + 0.5f) - ro[LEAD]);
                const int fromI = max(from[I], 0);
                for (int o = DIM == 3 ? max(from[O], 0) : 0; o < (DIM == 3 ? to[O] : 1); ++o) {
                    if (DIM == 3)
                        diff[O] = splat2((static_cast<float>(o) + 0.5f) - ro[O]);
                    int64_t word = from[LEAD] * sL + fromI * sI + (DIM == 3 ? o * sO : 0);
                    for (int i = fromI; i < to[I]; i += 2, word += 2 * sI) {
                        const float fi = static_cast<float>(i) + 0.5f;
                        diff[I] = sub2(make_float2(fi, fi + 1.0f), splat2(ro[I]));
                        float2 dot = fma2(splat2(rd[0]), diff[0], zero);
                        dot = add2(dot, fma2(splat2(rd[1]), diff[1], zero));
                        if (DIM == 3)
                            dot = add2(dot, fma2(splat2(rd[2]), diff[2], zero));
                        float2 sq = splat2(0.0f);
#pragma unroll
                        for (int k = 0; k < DIM; ++k) {
                            const float2 v = sub2(diff[k], fma2(dot, splat2(rd[k]), zero));
                            sq = k == 0 ? fma2(v, v, zero) : add2(sq, fma2(v, v, zero));
                        }
                        float2 dist;
                        // (a squared distance is below 2^40: volume edges are below 2^19)
                        if (fminf(sq.x, sq.y) >= 9.0949470e-13f)
                            dist = root2(sq);
                        else
                            dist = make_float2(sqrtf(sq.x), sqrtf(sq.y));
                        f(word, i + 1 < to[I],
                          lutValue2(tab, lp.lutN, lp.radius, lp.exactInv, dist, zero));
                    }
                }
            }
        }

        // body(<axis constant>) for the leading axis: largest |direction|, the first of equals.
        template <int DIM, class Body>
        __device__ __forceinline__ void withLead(const float* rd, Body&& body)
        {
            int lead = 0;
            float best = fabsf(rd[0]);
            for (int i = 1; i < DIM; ++i)
                if (fabsf(rd[i]) > best) {
                    best = fabsf(rd[i]);
                    lead = i;
                }
            if (lead == 0)
                body(std::integral_constant<int, 0>{});
            else if (DIM == 2 || lead == 1)
                body(std::integral_constant<int, 1>{});
            else
                body(std::integral_constant<int, DIM == 3 ? 2 : 1>{});
        }

        // Forward, one thread per ray. Bound by issue (about 50 instructions per voxel; 64^3 / 60
        // views / 96^2, forward and adjoint: 10.8 ms with one voxel at a time on the x-fastest
        // volume, now 4.20).
        template <int DIM>
        __global__ void __launch_bounds__(128)
            lutForwardKernel(const float* __restrict__ poses, DetectorShape det,
                             const __grid_constant__ LutProjParams lp,
                             const float* __restrict__ lutIn,
                             const __grid_constant__ LutLayouts layouts, float* __restrict__ y)
        {
            __shared__ float2 tab[kLutProjMaxSamples * kLutCopies];
            stageLut(lutIn, lp.lutN, tab);
            __syncthreads();
            const int64_t nrays = static_cast<int64_t>(det.nu) * det.nv * det.np;
            const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (r >= nrays)
                return;
            const int u = static_cast<int>(r % det.nu);
            const int v = static_cast<int>((r / det.nu) % det.nv);
            const int p = static_cast<int>(r / (static_cast<int64_t>(det.nu) * det.nv));
            float o[3] = {0, 0, 0}, d[3] = {0, 0, 0};
            pixelRay(poses + static_cast<int64_t>(p) * 40, DIM, u, v, nullptr, det.nu, o, d);
            float acc = 0.0f;
            withLead<DIM>(d, [&](auto lead) {
                constexpr int L = decltype(lead)::value;
                constexpr int I = DIM == 2 ? 1 - L : (L == 2 ? 1 : 2);
                const float* x = static_cast<const float*>(layouts.base[L]);
                const int64_t next = layouts.stride[L][I];
                lutRayAlong<DIM, L>(lp, tab, layouts.stride[L], o, d, false,
                                    [&](int64_t word, bool two, float2 w) {
                                        acc = acc + w.x * __ldg(x + word);
                                        if (two)
                                            acc = acc + w.y * __ldg(x + word + next);
                                    });
            });
            y[r] = acc;
        }

        // Backward in 64-bit fixed point: every contribution w * y is rounded once to a multiple
        // of 2^-k and the integer sums are exact, so the result does not depend on the order of
        // the atomic additions, nor on which of the two sums (layouts, added at the end) a ray
        // adds to. 2^k keeps any sum of up to 4 * nrays contributions of at most
        // max|y| * max|lut| below 2^62.
        template <int DIM>
        __global__ void __launch_bounds__(128)
            lutBackwardKernel(const float* __restrict__ poses, DetectorShape det,
                              const __grid_constant__ LutProjParams lp,
                              const float* __restrict__ lutIn, const float* __restrict__ y,
                              const unsigned* __restrict__ absMaxBits,
                              const __grid_constant__ LutLayouts layouts)
        {
            __shared__ float2 tab[kLutProjMaxSamples * kLutCopies];
            stageLut(lutIn, lp.lutN, tab);
            __syncthreads();
            const int64_t nrays = static_cast<int64_t>(det.nu) * det.nv * det.np;
            const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (r >= nrays)
                return;
            const double scale = lutFixedScale(__uint_as_float(*absMaxBits), lp.maxLut, nrays);
            const float yv = y[r];
            if (yv == 0.0f || scale == 0.0)
                return;
            const int u = static_cast<int>(r % det.nu);
            const int v = static_cast<int>((r / det.nu) % det.nv);
            const int p = static_cast<int>(r / (static_cast<int64_t>(det.nu) * det.nv));
            float o[3] = {0, 0, 0}, d[3] = {0, 0, 0};
            pixelRay(poses + static_cast<int64_t>(p) * 40, DIM, u, v, nullptr, det.nu, o, d);
            withLead<DIM>(d, [&](auto lead) {
                constexpr int L = decltype(lead)::value;
                constexpr int I = DIM == 2 ? 1 - L : (L == 2 ? 1 : 2);
                auto* acc = const_cast<unsigned long long*>(
                    static_cast<const unsigned long long*>(layouts.base[L]));
                const int64_t next = layouts.stride[L][I];
                // scale is a power of two: the product is exact in float too, where that holds it
                // (a result that is subnormal rounds to 0 either way)
                const float narrow =
                    scale > 1e-30 && scale < 1e30 ? static_cast<float>(scale) : 0.0f;
                auto add = [&](int64_t word, float c) {
                    const long long q = narrow != 0.0f
                                            ? __float2ll_rn(c * narrow)
                                            : __double2ll_rn(static_cast<double>(c) * scale);
                    if (q != 0)
                        atomicAdd(acc + word, static_cast<unsigned long long>(q));
                };
                lutRayAlong<DIM, L>(lp, tab, layouts.stride[L], o, d, true,
                                    [&](int64_t word, bool two, float2 w) {
                                        if (w.x != 0.0f)
                                            add(word, w.x * yv);
                                        if (two && w.y != 0.0f)
                                            add(word + next, w.y * yv);
                                    });
            });
        }

        __global__ void absMaxKernel(const float* __restrict__ y, int64_t n,
                                     unsigned* __restrict__ out)
        {
            unsigned m = 0;
            for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
                 i += static_cast<int64_t>(gridDim.x) * blockDim.x)
                m = max(m, __float_as_uint(fabsf(y[i])));
            for (int off = 16; off > 0; off >>= 1)
                m = max(m, __shfl_xor_sync(0xffffffffu, m, off));
            if ((threadIdx.x & 31) == 0 && m)
                atomicMax(out, m);
        }

        // second (may be null): the sums of the other layout, word c0 s.x + c1 s.y + c2 s.z
        __global__ void fixedToFloatKernel(const unsigned long long* __restrict__ acc,
                                           const unsigned long long* __restrict__ second,
                                           int3 shape, longlong3 stride, int64_t n,
                                           const unsigned* __restrict__ absMaxBits,
                                           float lutMax, int64_t nrays, float* __restrict__ x)
        {
            const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (i >= n)
                return;
            const double scale = lutFixedScale(__uint_as_float(*absMaxBits), lutMax, nrays);
            unsigned long long q = acc[i];
            if (second) {
                const int64_t row = i / shape.x;
                q += second[(i - row * shape.x) * stride.x + (row % shape.y) * stride.y +
                            (row / shape.y) * stride.z];
            }
            x[i] = scale == 0.0
                       ? 0.0f
                       : static_cast<float>(static_cast<double>(static_cast<long long>(q)) / scale);
        }
    } // namespace

    void launchLutForward(const float* poses, const DetectorShape& det, const LutProjParams& lp,
                          const float* lut, const LutLayouts& layouts, float* y, cudaStream_t s)
    {
        const int64_t nrays = static_cast<int64_t>(det.nu) * det.nv * det.np;
        if (nrays == 0)
            return;
        auto* k = lp.dim == 3 ? lutForwardKernel<3> : lutForwardKernel<2>;
        k<<<static_cast<unsigned>((nrays + 127) / 128), 128, 0, s>>>(poses, det, lp, lut, layouts,
                                                                     y);
    }

    void launchLutBackward(const float* poses, const DetectorShape& det, const LutProjParams& lp,
                           const float* lut, const float* y, unsigned* absMaxBits,
                           unsigned long long* acc, unsigned long long* second,
                           const LutLayouts& layouts, const int64_t (&secondStride)[3],
                           int64_t nvox, float* x, cudaStream_t s)
    {
        const int64_t nrays = static_cast<int64_t>(det.nu) * det.nv * det.np;
        const size_t bytes = sizeof(unsigned long long) * static_cast<size_t>(nvox);
        cudaMemsetAsync(absMaxBits, 0, sizeof(unsigned), s);
        cudaMemsetAsync(acc, 0, bytes, s);
        if (second)
            cudaMemsetAsync(second, 0, bytes, s);
        if (nrays > 0) {
            absMaxKernel<<<592, 256, 0, s>>>(y, nrays, absMaxBits);
            auto* k = lp.dim == 3 ? lutBackwardKernel<3> : lutBackwardKernel<2>;
            k<<<static_cast<unsigned>((nrays + 127) / 128), 128, 0, s>>>(poses, det, lp, lut, y,
                                                                         absMaxBits, layouts);
        }
        if (nvox > 0)
            fixedToFloatKernel<<<static_cast<unsigned>((nvox + 255) / 256), 256, 0, s>>>(
                acc, second, make_int3(lp.n[0], lp.n[1], lp.n[2]),
                make_longlong3(secondStride[0], secondStride[1], secondStride[2]), nvox,
                absMaxBits, lp.maxLut, nrays, x);
    }
} // namespace elsa_b200
