// Siddon's method (exact intersection lengths) for sm_100a.
//
// Reference semantics: projectors/SiddonsMethod.cpp:76-124 with projectors/TraverseAABB.cpp:6-184
// (elsa's CPU path, the parity target). A ray visits the voxels it crosses in order; each visit
// advances every axis whose next boundary parameter T is minimal, and the voxel's weight is the
// parameter difference tExit - tEntry:
//   forward  y[r] = sum_visits x[voxel] * (tExit - tEntry)
//   adjoint  x[v] = sum_r sum_{visits of v} y[r] * (tExit - tEntry)
// T advances by repeated float addition (T += tDelta), so both kernels replay the reference's
// float operations one by one (no contraction): the visited voxels and weights are bit-identical
// to the CPU traversal.
//
// Forward: one thread per ray, voxels gathered through the read-only cache.
//
// Adjoint, two kernels (launch knob kKnobAdjointScatter). The scatter kernel replays each ray
// like the forward, one thread per ray, and adds y * weight to every visited voxel with a
// fire-and-forget atomic: the reference's own scheme, with an addition order that varies from run
// to run. The brick-owner kernel is atomic-free and deterministic:
// on the brick-owner scheme of the Joseph adjoint. One
// warp owns a 16^3 brick in shared memory for all views. Rays are cut into slabs of 16 voxels
// along their axis g of largest |direction|; per (ray, slab) a checkpoint holds the traversal
// state (T of every axis, entry parameter, voxel) at the ray's first visit inside the slab,
// computed once per geometry. For each view the warp takes the rays of the brick's detector
// window class by class (pixel indices congruent modulo m, m validated per geometry so that
// same-class rays with the same g stay more than two voxels apart laterally on every slice);
// each lane replays one ray's visits inside the slab from its checkpoint and adds the weights of
// the visits that fall inside the brick. Same-class rays therefore never touch the same voxel,
// and every voxel sums its contributions in a fixed order.
#include "joseph_tma.cuh"
#include "projector.hpp"
#include "raysetup.cuh"
#include "solvers.hpp"

#include <algorithm>
#include <array>
#include <cfloat>
#include <climits>
#include <cstring>

namespace elsa_b200
{
    namespace
    {
        constexpr int kForwardThreads = 128;    // default rays per block of the forward
        constexpr int kScatterThreads = 256;    // rays per block of the scatter adjoint
        constexpr int kMaxForwardThreads = 512; // largest block the autotuner may choose
        constexpr int kAdjointWarpsPerSm = 22;  // view-chunk target of the warp-brick adjoint
        constexpr int kMinAdjointChunks = 32;   // default floor of the view chunks
        constexpr int64_t kChunkMemory = int64_t(1) << 31; // default partial-volume budget
        constexpr int kSlab = 16; // brick edge = checkpoint slab depth
        constexpr float kWindowSlack = 0.1f;       // voxels around a brick in its ray window
        constexpr float kWindowPixelMargin = 0.05f; // pixels around the projected brick
        constexpr int kMinClass = 2;
        constexpr int kMaxClass = 8;
        constexpr int kActive = 256;

        __device__ __forceinline__ int floorDiv(int a, int b)
        {
            const int q = a / b;
            return (a % b != 0 && ((a < 0) != (b < 0))) ? q - 1 : q;
        }

        __device__ __forceinline__ int axisStep(int meta, int i)
        {
            return ((meta >> (5 + i)) & 1) ? 0 : (((meta >> (2 + i)) & 1) ? -1 : 1);
        }

        // One visit: the parameter where the ray leaves the current voxel, and which axes cross
        // (TraverseAABB.cpp:55-100: all axes whose T is minimal advance together).
        template <int DIM>
        __device__ __forceinline__ float nextCrossing(float T0, float T1, float T2, bool& m0,
                                                      bool& m1, bool& m2)
        {
            // an axis crosses when its T is the minimum (T0 <= T1 && T0 <= T2 and so on: the T
            // are never NaN, FLT_MAX for an axis the ray does not cross)
            const float tm = DIM == 3 ? fminf(T0, fminf(T1, T2)) : fminf(T0, T1);
            m0 = T0 == tm;
            m1 = T1 == tm;
            m2 = DIM == 3 && T2 == tm;
            return tm;
        }

        // One axis of a visit: where its T is the crossing parameter, T, the word offset and the
        // steps left advance, all predicated (the compiler selects and adds instead: 37
        // instructions per visit of the forward against 29).
        __device__ __forceinline__ void crossIf(float tm, float& T, float tDelta, unsigned& idx,
                                                unsigned step, int& left, int one)
        {
            asm("{\n\t.reg .pred m;\n\tsetp.eq.f32 m, %0, %3;\n\t"
                "@m add.rn.f32 %0, %0, %4;\n\t@m add.u32 %1, %1, %5;\n\t"
                "@m sub.s32 %2, %2, %6;\n\t}"
                : "+f"(T), "+r"(idx), "+r"(left)
                : "f"(tm), "f"(tDelta), "r"(step), "r"(one));
        }
        __device__ __forceinline__ void crossIf(float tm, float& T, float tDelta, int64_t& idx,
                                                int64_t step, int& left, int one)
        {
            if (T == tm) {
                left -= one;
                idx += step;
                T = __fadd_rn(T, tDelta);
            }
        }

        __device__ __forceinline__ void crossIf(float tm, float& T, float tDelta, int& c, int step)
        {
            asm("{\n\t.reg .pred m;\n\tsetp.eq.f32 m, %0, %2;\n\t"
                "@m add.rn.f32 %0, %0, %3;\n\t@m add.s32 %1, %1, %4;\n\t}"
                : "+f"(T), "+r"(c)
                : "f"(tm), "f"(tDelta), "r"(step));
        }

        // Entry voxel in axis order from the record (g and the two other axes a < b).
        __device__ __forceinline__ void entryVoxel(int g, int kg, int ca, int cb, int& c0,
                                                   int& c1, int& c2)
        {
            c0 = g == 0 ? kg : ca;
            c1 = g == 1 ? kg : (g == 0 ? ca : cb);
            c2 = g == 2 ? kg : cb;
        }

        // Per driving axis of a ray, the copy of the volume it is read from (the volume itself, or
        // one with the axis contiguous along which neighbouring rays spread) and its strides.
        struct SiddonLayouts {
            const float* base[3];
            int64_t stride[3][3];
        };

        // 2D: one thread per ray on the image itself. A ray is a few hundred visits and a launch a few
        // warps per SM, so the time is the chain of a visit: the predicated form of the 3D kernel
        // below is slower here (256 x 231 / 300 views / 365 pixels: 81 us beside 5 of the image's copy,
        // this one 65), and a transposed image buys nothing while it stays in L1 and L2 (1000 x 900 /
        // 30 views: 320 us with it, 314 without).
        __global__ void __launch_bounds__(kMaxForwardThreads)
            siddonForward2dKernel(const SiddonRay* __restrict__ rays, int64_t nrays,
                                  const float* __restrict__ x, VolumeShape vol, int binary,
                                  float* __restrict__ y)
        {
            // binary: BinaryMethod (projectors/BinaryMethod.cpp:66-111), weight 1 per visit
            const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (r >= nrays)
                return;
            const SiddonRay R = rays[r];
            float acc = 0.0f;
            if (R.meta & kActive) {
                int c0, c1, c2;
                entryVoxel(R.meta & 3, R.kFirst, R.cur[0], R.cur[1], c0, c1, c2);
                const int s0 = axisStep(R.meta, 0), s1 = axisStep(R.meta, 1);
                const int nx = vol.n[0], ny = vol.n[1];
                const int64_t sy = nx;
                int64_t idx = c0 + sy * c1;
                float T0 = R.T[0], T1 = R.T[1];
                float tExit = 0.0f;
                const int maxVisits = nx + ny + 3;
                for (int it = 0; it < maxVisits; ++it) {
                    const float tEntry = tExit;
                    bool m0, m1, m2;
                    tExit = nextCrossing<2>(T0, T1, 0.0f, m0, m1, m2);
                    if (m0) {
                        c0 += s0;
                        T0 = __fadd_rn(T0, R.tDelta[0]);
                    }
                    if (m1) {
                        c1 += s1;
                        T1 = __fadd_rn(T1, R.tDelta[1]);
                    }
                    const float w = binary ? 1.0f : __fsub_rn(tExit, tEntry);
                    acc = __fadd_rn(acc, __fmul_rn(__ldg(x + idx), w));
                    if (static_cast<unsigned>(c0) >= static_cast<unsigned>(nx) ||
                        static_cast<unsigned>(c1) >= static_cast<unsigned>(ny))
                        break;
                    idx += (m0 ? s0 : 0) + (m1 ? s1 * sy : 0);
                }
            }
            y[r] = acc;
        }

        // 3D: one thread per ray, the reference's visits and float operations in order. Bound by issue
        // (29 instructions per visit) once neighbouring lanes read neighbouring words: with
        // every ray on the x-fastest volume, a warp whose rays drive along x read 32 sectors per
        // visit and the load pipe took the time (171 x 200 x 149 voxels, 240 views of
        // 250 x 231: 3.62 ms, now 2.69). The bounds test counts the steps left along each axis, so
        // a visit updates one word offset instead of three voxel indices and a 64-bit one. Offset:
        // unsigned below 2^32 words, else int64_t.
        template <typename Offset>
        __global__ void __launch_bounds__(kMaxForwardThreads)
            siddonForwardKernel(const SiddonRay* __restrict__ rays, int64_t nrays,
                                const __grid_constant__ SiddonLayouts layouts, VolumeShape vol,
                                int binary,
                                float* __restrict__ y)
        {
            // binary: weight 1 per visit, as above
            const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (r >= nrays)
                return;
            const SiddonRay R = rays[r];
            float acc = 0.0f;
            if (R.meta & kActive) {
                const int g = R.meta & 3;
                int c0, c1, c2;
                entryVoxel(g, R.kFirst, R.cur[0], R.cur[1], c0, c1, c2);
                const int s0 = axisStep(R.meta, 0), s1 = axisStep(R.meta, 1),
                          s2 = axisStep(R.meta, 2);
                const float* base = layouts.base[g];
                const Offset e0 = static_cast<Offset>(layouts.stride[g][0]),
                             e1 = static_cast<Offset>(layouts.stride[g][1]),
                             e2 = static_cast<Offset>(layouts.stride[g][2]);
                Offset idx = c0 * e0 + c1 * e1 + c2 * e2;
                const Offset i0 = s0 * e0, i1 = s1 * e1, i2 = s2 * e2;
                // steps left before the ray leaves the volume (the entry voxel is inside)
                int left0 = s0 > 0 ? vol.n[0] - 1 - c0 : c0;
                int left1 = s1 > 0 ? vol.n[1] - 1 - c1 : c1;
                int left2 = s2 > 0 ? vol.n[2] - 1 - c2 : c2;
                const int k0 = s0 != 0, k1 = s1 != 0, k2 = s2 != 0;
                float T0 = R.T[0], T1 = R.T[1], T2 = R.T[2];
                float tExit = 0.0f;
                const int maxVisits = vol.n[0] + vol.n[1] + vol.n[2] + 3;
                for (int it = 0; it < maxVisits; ++it) {
                    const float v = __ldg(base + idx);
                    const float tEntry = tExit;
                    tExit = fminf(T0, fminf(T1, T2));
                    crossIf(tExit, T0, R.tDelta[0], idx, i0, left0, k0);
                    crossIf(tExit, T1, R.tDelta[1], idx, i1, left1, k1);
                    crossIf(tExit, T2, R.tDelta[2], idx, i2, left2, k2);
                    const float w = binary ? 1.0f : __fsub_rn(tExit, tEntry);
                    acc = __fadd_rn(acc, __fmul_rn(v, w));
                    if ((left0 | left1 | left2) < 0)
                        break;
                }
            }
            y[r] = acc;
        }

        // Adjoint by atomic scatter: the forward's visit loop, adding y[r] * weight to each
        // visited voxel (x zeroed beforehand). The atomics' return values are unused, so they
        // compile to reductions that do not wait for the memory system.
        template <int DIM>
        __global__ void __launch_bounds__(kScatterThreads)
            siddonScatterKernel(const SiddonRay* __restrict__ rays, int64_t nrays,
                                const float* __restrict__ y, VolumeShape vol, int binary,
                                float* __restrict__ x)
        {
            const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (r >= nrays)
                return;
            const float yr = __ldg(y + r);
            const SiddonRay R = rays[r];
            if (!(R.meta & kActive) || yr == 0.0f)
                return;
            const int g = R.meta & 3;
            int c0, c1, c2;
            entryVoxel(g, R.kFirst, R.cur[0], R.cur[1], c0, c1, c2);
            const int s0 = axisStep(R.meta, 0), s1 = axisStep(R.meta, 1), s2 = axisStep(R.meta, 2);
            const int nx = vol.n[0], ny = vol.n[1], nz = vol.n[2];
            const int64_t sy = nx, sz = static_cast<int64_t>(nx) * ny;
            int64_t idx = c0 + sy * c1 + (DIM == 3 ? sz * c2 : 0);
            float T0 = R.T[0], T1 = R.T[1], T2 = R.T[2];
            float tExit = 0.0f;
            const int maxVisits = nx + ny + (DIM == 3 ? nz : 0) + 3;
            for (int it = 0; it < maxVisits; ++it) {
                const float tEntry = tExit;
                bool m0, m1, m2;
                tExit = nextCrossing<DIM>(T0, T1, T2, m0, m1, m2);
                if (m0) {
                    c0 += s0;
                    T0 = __fadd_rn(T0, R.tDelta[0]);
                }
                if (m1) {
                    c1 += s1;
                    T1 = __fadd_rn(T1, R.tDelta[1]);
                }
                if (m2) {
                    c2 += s2;
                    T2 = __fadd_rn(T2, R.tDelta[2]);
                }
                const bool inside = static_cast<unsigned>(c0) < static_cast<unsigned>(nx) &&
                                    static_cast<unsigned>(c1) < static_cast<unsigned>(ny) &&
                                    (DIM < 3 || static_cast<unsigned>(c2) < static_cast<unsigned>(nz));
                const float w = binary ? 1.0f : __fsub_rn(tExit, tEntry);
                atomicAdd(x + idx, __fmul_rn(yr, w));
                if (!inside)
                    break;
                idx += (m0 ? s0 : 0) + (m1 ? s1 * sy : 0) + (m2 ? s2 * sz : 0);
            }
        }

        // Replays every ray once: writes the traversal state at the ray's first visit in each
        // slab of kSlab voxels along g (slab-major, row floor(k/kSlab) + 1, column = ray; skipped
        // when cpState is null), the last visited index along g and the visit count
        // (SiddonsMethod's sample count; skipped when visits is null).
        template <int DIM>
        __global__ void siddonCheckpointKernel(SiddonRay* __restrict__ rays, int64_t nrays,
                                               VolumeShape vol, int slabRows,
                                               float4* __restrict__ cpState,
                                               unsigned* __restrict__ cpVoxel,
                                               unsigned long long* __restrict__ visits)
        {
            const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (r >= nrays)
                return;
            SiddonRay R = rays[r];
            if (!(R.meta & kActive))
                return;
            const int g = R.meta & 3;
            int a, b;
            nonDrivingAxes(g, a, b);
            int c0, c1, c2;
            entryVoxel(g, R.kFirst, R.cur[0], R.cur[1], c0, c1, c2);
            const int s0 = axisStep(R.meta, 0), s1 = axisStep(R.meta, 1), s2 = axisStep(R.meta, 2);
            const int nx = vol.n[0], ny = vol.n[1], nz = vol.n[2];
            float T0 = R.T[0], T1 = R.T[1], T2 = R.T[2];
            float tExit = 0.0f;
            int slab = INT_MIN, count = 0, kLast = R.kFirst;
            const int maxVisits = nx + ny + (DIM == 3 ? nz : 0) + 3;
            for (int it = 0; it < maxVisits; ++it) {
                const float tEntry = tExit;
                const int cg = g == 0 ? c0 : (g == 1 ? c1 : c2);
                const int s = floorDiv(cg, kSlab);
                if (s != slab) {
                    slab = s;
                    if (cpState != nullptr && s + 1 >= 0 && s + 1 < slabRows) {
                        const int ca = a == 0 ? c0 : c1;
                        const int cb = DIM == 3 ? (b == 1 ? c1 : c2) : 0;
                        const int64_t at = static_cast<int64_t>(s + 1) * nrays + r;
                        cpState[at] = make_float4(T0, T1, T2, tEntry);
                        cpVoxel[at] =
                            static_cast<unsigned>(ca) | (static_cast<unsigned>(cb) << 16);
                    }
                }
                kLast = cg;
                ++count;
                bool m0, m1, m2;
                tExit = nextCrossing<DIM>(T0, T1, T2, m0, m1, m2);
                if (m0) {
                    c0 += s0;
                    T0 = __fadd_rn(T0, R.tDelta[0]);
                }
                if (m1) {
                    c1 += s1;
                    T1 = __fadd_rn(T1, R.tDelta[1]);
                }
                if (m2) {
                    c2 += s2;
                    T2 = __fadd_rn(T2, R.tDelta[2]);
                }
                const bool inside =
                    static_cast<unsigned>(c0) < static_cast<unsigned>(nx) &&
                    static_cast<unsigned>(c1) < static_cast<unsigned>(ny) &&
                    (DIM < 3 || static_cast<unsigned>(c2) < static_cast<unsigned>(nz));
                if (!inside)
                    break;
            }
            R.kLast = kLast;
            R.crossings = count;
            rays[r] = R;
            if (visits != nullptr)
                atomicAdd(visits, static_cast<unsigned long long>(count));
        }

        // True when rays R and S (same axis g) stay more than two voxels apart in one lateral
        // coordinate over the slices of g that both visit.
        __device__ bool separated(const SiddonRay& R, const SiddonLine& LR, const SiddonRay& S,
                                  const SiddonLine& LS, int dim)
        {
            const int lo = max(min(R.kFirst, R.kLast), min(S.kFirst, S.kLast));
            const int hi = min(max(R.kFirst, R.kLast), max(S.kFirst, S.kLast));
            if (lo > hi)
                return true;
            const float margin = 2.05f;
            const float g0 = static_cast<float>(lo), g1 = static_cast<float>(hi + 1);
            const float da0 = fmaf(g0 - LR.g0, LR.sa, LR.a0) - fmaf(g0 - LS.g0, LS.sa, LS.a0);
            const float da1 = fmaf(g1 - LR.g0, LR.sa, LR.a0) - fmaf(g1 - LS.g0, LS.sa, LS.a0);
            if ((da0 > margin && da1 > margin) || (da0 < -margin && da1 < -margin))
                return true;
            if (dim == 3) {
                const float db0 = fmaf(g0 - LR.g0, LR.sb, LR.b0) - fmaf(g0 - LS.g0, LS.sb, LS.b0);
                const float db1 = fmaf(g1 - LR.g0, LR.sb, LR.b0) - fmaf(g1 - LS.g0, LS.sb, LS.b0);
                if ((db0 > margin && db1 > margin) || (db0 < -margin && db1 < -margin))
                    return true;
            }
            return false;
        }

        // Axes present per view and, per candidate class spacing m, whether two rays that the
        // adjoint may process concurrently could visit the same voxel. Neighbours checked: the
        // same detector row m pixels apart, and the next class row (m rows down) within +-32
        // pixels; rays further apart in a class are further apart on every slice (the pixel ->
        // slice-position map of a flat detector is monotone for rays sharing g).
        __global__ void siddonClassCheckKernel(const SiddonRay* __restrict__ rays,
                                               const SiddonLine* __restrict__ lines,
                                               DetectorShape det, int dim,
                                               unsigned* __restrict__ viewAxes,
                                               unsigned* __restrict__ badSpacing)
        {
            const int64_t nrays = static_cast<int64_t>(det.nu) * det.nv * det.np;
            const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (r >= nrays)
                return;
            const SiddonRay R = rays[r];
            if (!(R.meta & kActive))
                return;
            const SiddonLine LR = lines[r];
            const int u = static_cast<int>(r % det.nu);
            const int v = static_cast<int>((r / det.nu) % det.nv);
            const int p = static_cast<int>(r / (static_cast<int64_t>(det.nu) * det.nv));
            atomicOr(viewAxes + p, 1u << (R.meta & 3));
            unsigned bad = 0;
            for (int m = kMinClass; m <= kMaxClass; ++m) {
                const int noffs = dim == 3 ? 1 + 65 : 1;
                for (int o = 0; o < noffs; ++o) {
                    const int du = o == 0 ? m : o - 1 - 32;
                    const int dv = o == 0 ? 0 : m;
                    const int u2 = u + du, v2 = v + dv;
                    if (u2 < 0 || u2 >= det.nu || v2 < 0 || v2 >= det.nv)
                        continue;
                    const int64_t r2 =
                        u2 + static_cast<int64_t>(det.nu) * (v2 + static_cast<int64_t>(det.nv) * p);
                    const SiddonRay S = rays[r2];
                    if (!(S.meta & kActive) || (S.meta & 3) != (R.meta & 3))
                        continue;
                    if (!separated(R, LR, S, lines[r2], dim))
                        bad |= 1u << m;
                }
            }
            if (bad)
                atomicOr(badSpacing, bad);
        }

        // Shared-memory brick of one warp (x stride 1, row stride 17, plane stride = 1 mod 32).
        // Check of the brick windows (test support, elsa_projector_info key 8): every visited
        // voxel must lie in a brick whose window for the ray's view contains the ray. Counts the
        // visits that violate this.
        template <int DIM>
        __global__ void siddonWindowCheckKernel(const SiddonRay* __restrict__ rays,
                                                const RayWindow* __restrict__ windows,
                                                VolumeShape vol, DetectorShape det, int3 brick,
                                                int3 nBricks, int onlyAxis,
                                                unsigned long long* __restrict__ misses)
        {
            const int64_t nrays = static_cast<int64_t>(det.nu) * det.nv * det.np;
            const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (r >= nrays)
                return;
            const SiddonRay R = rays[r];
            if (!(R.meta & kActive) || (onlyAxis >= 0 && (R.meta & 3) != onlyAxis))
                return;
            const int u = static_cast<int>(r % det.nu);
            const int v = static_cast<int>((r / det.nu) % det.nv);
            const int p = static_cast<int>(r / (static_cast<int64_t>(det.nu) * det.nv));
            const int nb = nBricks.x * nBricks.y * nBricks.z;
            const int g = R.meta & 3;
            int c0, c1, c2;
            entryVoxel(g, R.kFirst, R.cur[0], R.cur[1], c0, c1, c2);
            const int s0 = axisStep(R.meta, 0), s1 = axisStep(R.meta, 1), s2 = axisStep(R.meta, 2);
            float T0 = R.T[0], T1 = R.T[1], T2 = R.T[2];
            const int maxVisits = vol.n[0] + vol.n[1] + (DIM == 3 ? vol.n[2] : 0) + 3;
            unsigned long long bad = 0;
            int lastBrick = -1;
            for (int it = 0; it < maxVisits; ++it) {
                const int o0 = c0, o1 = c1, o2 = DIM == 3 ? c2 : 0; // the voxel of this visit
                bool m0, m1, m2;
                nextCrossing<DIM>(T0, T1, T2, m0, m1, m2);
                if (m0) {
                    c0 += s0;
                    T0 = __fadd_rn(T0, R.tDelta[0]);
                }
                if (m1) {
                    c1 += s1;
                    T1 = __fadd_rn(T1, R.tDelta[1]);
                }
                if (m2) {
                    c2 += s2;
                    T2 = __fadd_rn(T2, R.tDelta[2]);
                }
                const int bi = o0 / brick.x + nBricks.x * (o1 / brick.y + nBricks.y * (o2 / brick.z));
                if (bi != lastBrick) {
                    const RayWindow w = windows[static_cast<int64_t>(p) * nb + bi];
                    if (u < w.u0 || u > w.u1 || v < w.v0 || v > w.v1)
                        ++bad;
                    else
                        lastBrick = bi;
                }
                const bool inside =
                    static_cast<unsigned>(c0) < static_cast<unsigned>(vol.n[0]) &&
                    static_cast<unsigned>(c1) < static_cast<unsigned>(vol.n[1]) &&
                    (DIM < 3 || static_cast<unsigned>(c2) < static_cast<unsigned>(vol.n[2]));
                if (!inside)
                    break;
            }
            if (bad)
                atomicAdd(misses, bad);
        }

        template <int DIM>
        struct SiddonBrick {
            static constexpr int kBz = DIM == 3 ? kSlab : 1;
            static constexpr int kRow = kSlab + 1;
            static constexpr int kPlaneMin = kRow * kSlab;
            static constexpr int kPlane = kPlaneMin + ((33 - kPlaneMin % 32) % 32);
            static constexpr int kWords = kPlane * kBz + 1; // + dummy word
        };

        // Replays the visits of one ray inside the slab [kLo, kLo + 15] along G from its
        // checkpoint and adds y * weight to the visited voxels of the brick (visits outside the
        // brick go to the dummy word).
        template <int DIM, int G>
        __device__ __forceinline__ void splatSegment(float* acc, float3 tDelta, int meta,
                                                     int kFirst, float4 cp, unsigned cpv, float yv,
                                                     int kLo, int org0, int org1, int org2,
                                                     const VolumeShape& vol, int binary)
        {
            using L = SiddonBrick<DIM>;
            const int dirG = ((meta >> (2 + G)) & 1) ? -1 : 1;
            const int kg = dirG > 0 ? max(kLo, kFirst) : min(kLo + kSlab - 1, kFirst);
            int c0, c1, c2;
            entryVoxel(G, kg, static_cast<int>(cpv & 0xffffu), static_cast<int>(cpv >> 16), c0,
                       c1, c2);
            const int s0 = axisStep(meta, 0), s1 = axisStep(meta, 1), s2 = axisStep(meta, 2);
            float T0 = cp.x, T1 = cp.y, T2 = cp.z;
            float tEntry = cp.w;
            float* dummy = acc + L::kWords - 1;
            for (int it = 0; it < 3 * kSlab + 3; ++it) {
                bool m0, m1, m2;
                const float tExit = nextCrossing<DIM>(T0, T1, T2, m0, m1, m2);
                const int l0 = c0 - org0, l1 = c1 - org1, l2 = DIM == 3 ? c2 - org2 : 0;
                const bool mine = static_cast<unsigned>(l0) < static_cast<unsigned>(kSlab) &&
                                  static_cast<unsigned>(l1) < static_cast<unsigned>(kSlab) &&
                                  static_cast<unsigned>(l2) < static_cast<unsigned>(L::kBz);
                float* adr = mine ? acc + l2 * L::kPlane + l1 * L::kRow + l0 : dummy;
                const float w = binary ? 1.0f : __fsub_rn(tExit, tEntry);
                *adr = __fadd_rn(*adr, __fmul_rn(yv, w));
                if (m0) {
                    c0 += s0;
                    T0 = __fadd_rn(T0, tDelta.x);
                }
                if (m1) {
                    c1 += s1;
                    T1 = __fadd_rn(T1, tDelta.y);
                }
                if (m2) {
                    c2 += s2;
                    T2 = __fadd_rn(T2, tDelta.z);
                }
                const bool inside =
                    static_cast<unsigned>(c0) < static_cast<unsigned>(vol.n[0]) &&
                    static_cast<unsigned>(c1) < static_cast<unsigned>(vol.n[1]) &&
                    (DIM < 3 || static_cast<unsigned>(c2) < static_cast<unsigned>(vol.n[2]));
                const int cg = G == 0 ? c0 : (G == 1 ? c1 : c2);
                if (!inside || cg < kLo || cg >= kLo + kSlab)
                    break;
                tEntry = tExit;
            }
        }

        // One (view, axis G) for a warp-owned brick: m x m ray classes separated by __syncwarp;
        // lane i takes class rays i, i + 32, ... (u fastest within the class grid).
        template <int DIM, int G>
        __device__ __forceinline__ void siddonView(float* acc, const RayWindow& w, int p, int m,
                                                   const SiddonRay* __restrict__ rays,
                                                   const float4* __restrict__ cpState,
                                                   const unsigned* __restrict__ cpVoxel,
                                                   int64_t nrays, const float* __restrict__ y,
                                                   const DetectorShape& det, int org0, int org1,
                                                   int org2, const VolumeShape& vol, int binary)
        {
            const int kLo = G == 0 ? org0 : (G == 1 ? org1 : org2);
            const int kHi = kLo + kSlab - 1;
            const int lane = threadIdx.x & 31;
            const int64_t viewBase = static_cast<int64_t>(det.nu) * det.nv * p;
            const int64_t cpRow = static_cast<int64_t>(kLo / kSlab + 1) * nrays;
            for (int ov = 0; ov < m; ++ov) {
                const int vStart = w.v0 + ov;
                const int nvc = vStart <= w.v1 ? (w.v1 - vStart) / m + 1 : 0;
                for (int ou = 0; ou < m; ++ou) {
                    const int uStart = w.u0 + ou;
                    const int nuc = uStart <= w.u1 ? (w.u1 - uStart) / m + 1 : 0;
                    const int total = nuc * nvc;
                    for (int i = lane; i < total; i += 32) {
                        const int iv = i / nuc;
                        const int iu = i - iv * nuc;
                        const int64_t r = viewBase + (uStart + iu * m) +
                                          static_cast<int64_t>(det.nu) * (vStart + iv * m);
                        const int4* rp = reinterpret_cast<const int4*>(rays + r);
                        const int4 q0 = __ldg(rp);     // tDelta[3], meta
                        const int4 q1 = __ldg(rp + 1); // kFirst, kLast, cur[2]
                        const int meta = q0.w;
                        if (!(meta & kActive) || (meta & 3) != G)
                            continue;
                        if (max(q1.x, q1.y) < kLo || min(q1.x, q1.y) > kHi)
                            continue;
                        const float3 td = make_float3(__int_as_float(q0.x), __int_as_float(q0.y),
                                                      __int_as_float(q0.z));
                        splatSegment<DIM, G>(acc, td, meta, q1.x, __ldg(cpState + cpRow + r),
                                             __ldg(cpVoxel + cpRow + r), __ldg(y + r), kLo, org0,
                                             org1, org2, vol, binary);
                    }
                    __syncwarp();
                }
            }
        }

        template <int DIM>
        __global__ void __launch_bounds__(32)
            siddonAdjointKernel(const SiddonRay* __restrict__ rays,
                                const float4* __restrict__ cpState,
                                const unsigned* __restrict__ cpVoxel, int64_t nrays,
                                const float* __restrict__ y,
                                const RayWindow* __restrict__ windows,
                                const unsigned* __restrict__ viewAxes, VolumeShape vol,
                                DetectorShape det, int m, int3 nBricks, int viewsPerChunk,
                                int binary, float* __restrict__ x)
        {
            // blockIdx.y selects a chunk of views; with several chunks the brick goes to
            // x + chunk * nvox and launchSumChunks adds the chunks in order
            using L = SiddonBrick<DIM>;
            __shared__ float acc[L::kWords];
            const int lane = threadIdx.x;
            const int bi = blockIdx.x;
            const int org0 = (bi % nBricks.x) * kSlab;
            const int org1 = ((bi / nBricks.x) % nBricks.y) * kSlab;
            const int org2 = (bi / (nBricks.x * nBricks.y)) * L::kBz;
            const int nb = nBricks.x * nBricks.y * nBricks.z;
            for (int i = lane; i < L::kWords; i += 32)
                acc[i] = 0.0f;
            __syncwarp();
            const int pBegin = blockIdx.y * viewsPerChunk;
            const int pEnd = min(det.np, pBegin + viewsPerChunk);
            for (int p = pBegin; p < pEnd; ++p) {
                const RayWindow w = windows[static_cast<int64_t>(p) * nb + bi];
                if (w.u0 > w.u1 || w.v0 > w.v1)
                    continue;
                const unsigned ax = viewAxes[p];
                if (ax & 1u)
                    siddonView<DIM, 0>(acc, w, p, m, rays, cpState, cpVoxel, nrays, y, det, org0,
                                       org1, org2, vol, binary);
                if (ax & 2u)
                    siddonView<DIM, 1>(acc, w, p, m, rays, cpState, cpVoxel, nrays, y, det, org0,
                                       org1, org2, vol, binary);
                if (DIM == 3 && (ax & 4u))
                    siddonView<DIM, DIM == 3 ? 2 : 0>(acc, w, p, m, rays, cpState, cpVoxel, nrays,
                                                      y, det, org0, org1, org2, vol, binary);
            }
            __syncwarp();
            const int64_t nvox = static_cast<int64_t>(vol.n[0]) * vol.n[1] * vol.n[2];
            float* out = x + blockIdx.y * nvox;
            for (int i = lane; i < kSlab * kSlab * L::kBz; i += 32) {
                const int lx = i % kSlab, ly = (i / kSlab) % kSlab, lz = i / (kSlab * kSlab);
                const int gx = org0 + lx, gy = org1 + ly, gz = org2 + lz;
                if (gx < vol.n[0] && gy < vol.n[1] && gz < vol.n[2])
                    out[gx + static_cast<int64_t>(vol.n[0]) *
                                 (gy + static_cast<int64_t>(vol.n[1]) * gz)] =
                        acc[lz * L::kPlane + ly * L::kRow + lx];
            }
        }

        // ---------------------------------------------------------------------------------------
        // 3D brick-owner adjoint on axis bricks: per driving axis G present, bricks one checkpoint
        // slab (kSlab planes) deep along G, kAxisTW voxels along the non-driving axis over which
        // the rays of a detector row spread (the columns: stride 1 in shared memory, the lanes
        // spread along it) and kAxisTV along the other. A ray crossing a brick keeps most of its
        // visits inside it, and a warp's taps fall into different banks. Visits outside the brick
        // across the rays are predicated off. As the 16^3 kernel: one warp per (brick, chunk
        // entry), the window's rays class by class, each lane replaying one ray's visits of the
        // slab from its checkpoint.
        // ---------------------------------------------------------------------------------------
        constexpr int kAxisTW = 32, kAxisTV = 8; // columns and rows of a brick

        struct SiddonAxisBrick {
            static constexpr int kRow = kAxisTW + 1; // columns (+1: rows land in other banks)
            // unpadded planes keep the brick at 16.9 KB (12 resident per SM instead of 11)
            static constexpr int kPlane = kRow * kAxisTV;
            static constexpr int kWords = kPlane * kSlab;
        };

        // Brick edges of grid G (UB: columns along b) in volume axis order.
        template <int G, bool UB>
        __host__ __device__ constexpr int siddonAxisEdge(int axis)
        {
            return axis == G ? kSlab
                             : (axis == (G == 0 ? 1 : 0) ? (UB ? kAxisTV : kAxisTW)
                                                         : (UB ? kAxisTW : kAxisTV));
        }

        struct SiddonAxisJob {
            const SiddonRay* rays;
            const float4* cpState;
            const unsigned* cpVoxel;
            int64_t nrays;
            const float* y;
            const RayWindow* windows;
            const unsigned* viewAxes;
            const int2* chunks;
            int viewsPerChunk;
            VolumeShape vol;
            DetectorShape det;
            int m;
            int3 nBricks;
            int binary;
            float* out;
        };

        // Replays the visits of one ray inside the slab [kLo, kLo + kSlab) along G from its
        // checkpoint and adds y * weight to the visits inside the axis brick.
        template <int G, bool UB>
        __device__ __forceinline__ void splatAxisSegment(float* acc, float3 tDelta, int meta,
                                                         int kFirst, float4 cp, unsigned cpv,
                                                         float yv, int kLo, int orgA, int orgB,
                                                         const VolumeShape& vol, int binary)
        {
            using L = SiddonAxisBrick;
            constexpr int EA = UB ? kAxisTV : kAxisTW, EB = UB ? kAxisTW : kAxisTV;
            constexpr int SA = UB ? L::kRow : 1, SB = UB ? 1 : L::kRow;
            int a, b;
            nonDrivingAxes(G, a, b);
            const int dirG = ((meta >> (2 + G)) & 1) ? -1 : 1;
            const int kg = dirG > 0 ? max(kLo, kFirst) : min(kLo + kSlab - 1, kFirst);
            int c[3]; // voxel from the brick's first voxel
            entryVoxel(G, kg, static_cast<int>(cpv & 0xffffu), static_cast<int>(cpv >> 16), c[0],
                       c[1], c[2]);
            c[G] -= kLo, c[a] -= orgA, c[b] -= orgB;
            const int s0 = axisStep(meta, 0), s1 = axisStep(meta, 1), s2 = axisStep(meta, 2);
            float T0 = cp.x, T1 = cp.y, T2 = cp.z;
            float tEntry = cp.w;
            // the walk stays inside the volume and the slab: along G the two tests are one,
            // kLo <= cg < min(kLo + kSlab, n_G)
            const unsigned nA =
                static_cast<unsigned>(a == 0 ? vol.n[0] : (a == 1 ? vol.n[1] : vol.n[2]));
            const unsigned nB = static_cast<unsigned>(b == 1 ? vol.n[1] : vol.n[2]);
            const int nG = G == 0 ? vol.n[0] : (G == 1 ? vol.n[1] : vol.n[2]);
            const unsigned spanG = static_cast<unsigned>(min(kLo + kSlab, nG) - kLo);
            const unsigned base = static_cast<unsigned>(__cvta_generic_to_shared(acc));
            // software-pipelined: the word of a visit is read before the sum of the previous
            // visit (always another voxel) is written back
            unsigned prevAt = 0, prevIn = 0;
            float prevVal = 0.0f, prevW = 0.0f;
            for (int it = 0; it < 3 * kSlab + 3; ++it) {
                const float tExit = fminf(T0, fminf(T1, T2));
                const unsigned in = (static_cast<unsigned>(c[a]) < static_cast<unsigned>(EA)) &
                                    (static_cast<unsigned>(c[b]) < static_cast<unsigned>(EB));
                const unsigned at =
                    base + 4u * static_cast<unsigned>(c[G] * L::kPlane + c[a] * SA + c[b] * SB);
                float val;
                loadSharedIf(val, at, in);
                storeSharedIf(__fadd_rn(prevVal, __fmul_rn(yv, prevW)), prevAt, prevIn);
                prevAt = at, prevVal = val, prevIn = in;
                prevW = binary ? 1.0f : __fsub_rn(tExit, tEntry);
                crossIf(tExit, T0, tDelta.x, c[0], s0);
                crossIf(tExit, T1, tDelta.y, c[1], s1);
                crossIf(tExit, T2, tDelta.z, c[2], s2);
                if ((static_cast<unsigned>(c[a] + orgA) >= nA) |
                    (static_cast<unsigned>(c[b] + orgB) >= nB) |
                    (static_cast<unsigned>(c[G]) >= spanG))
                    break;
                tEntry = tExit;
            }
            storeSharedIf(__fadd_rn(prevVal, __fmul_rn(yv, prevW)), prevAt, prevIn);
        }

        template <int G, bool UB>
        __global__ void __launch_bounds__(32)
            siddonAxisKernel(SiddonAxisJob J, int entryBase)
        {
            using L = SiddonAxisBrick;
            __shared__ float acc[L::kWords];
            constexpr int EX = siddonAxisEdge<G, UB>(0), EY = siddonAxisEdge<G, UB>(1),
                          EZ = siddonAxisEdge<G, UB>(2);
            constexpr int SA = UB ? L::kRow : 1, SB = UB ? 1 : L::kRow;
            const int lane = threadIdx.x;
            const int bi = blockIdx.x;
            const int3 nb3 = J.nBricks;
            const int org[3] = {(bi % nb3.x) * EX, ((bi / nb3.x) % nb3.y) * EY,
                                (bi / (nb3.x * nb3.y)) * EZ};
            int a, b;
            nonDrivingAxes(G, a, b);
            const int kLo = org[G], kHi = kLo + kSlab - 1;
            const int nb = nb3.x * nb3.y * nb3.z;
            for (int i = lane; i < L::kWords; i += 32)
                acc[i] = 0.0f;
            __syncwarp();
            const int2 entry = J.chunks[entryBase + blockIdx.y];
            const int pBegin = entry.x * J.viewsPerChunk;
            const int pEnd = min(J.det.np, pBegin + J.viewsPerChunk);
            const int64_t cpRow = static_cast<int64_t>(kLo / kSlab + 1) * J.nrays;
            const int m = J.m;
            for (int p = pBegin; p < pEnd; ++p) {
                if (!(J.viewAxes[p] & (1u << G)))
                    continue;
                const RayWindow w = J.windows[static_cast<int64_t>(p) * nb + bi];
                if (w.u0 > w.u1 || w.v0 > w.v1)
                    continue;
                const int64_t viewBase = static_cast<int64_t>(J.det.nu) * J.det.nv * p;
                // rounds of 32 class rays, class by class; the records of a round are loaded while
                // the rays of the round before are walked (171 x 200 x 149 / 240 views of 250 x
                // 231: 7.48 -> 6.77 ms)
                struct Record {
                    int4 q0, q1; // tDelta[3], meta; kFirst, kLast, cur[2]
                    float4 cp;
                    unsigned cpv;
                    float y;
                };
                int ov = 0, ou = -1, uStart = 0, vStart = 0, nuc = 0, total = 0, base = 0;
                float invNuc = 0.0f;
                auto nextRound = [&](bool& newClass) { // false: the view is done
                    base += 32;
                    while (base >= total) {
                        if (++ou == m) {
                            ou = 0;
                            if (++ov == m)
                                return false;
                        }
                        uStart = w.u0 + ou, vStart = w.v0 + ov;
                        const int nvc = vStart <= w.v1 ? (w.v1 - vStart) / m + 1 : 0;
                        nuc = uStart <= w.u1 ? (w.u1 - uStart) / m + 1 : 0;
                        total = nuc * nvc;
                        invNuc = nuc > 0 ? 1.0f / static_cast<float>(nuc) : 0.0f;
                        base = 0;
                        newClass = true;
                    }
                    return true;
                };
                auto load = [&](Record& rec) {
                    const int i = base + lane;
                    rec.q0.w = 0;
                    if (i < total) {
                        // i / nuc by a float reciprocal: exact for i < 2^20, nuc < 2^11
                        const int iv = static_cast<int>((static_cast<float>(i) + 0.5f) * invNuc);
                        const int iu = i - iv * nuc;
                        const int64_t r = viewBase + (uStart + iu * m) +
                                          static_cast<int64_t>(J.det.nu) * (vStart + iv * m);
                        const int4* rp = reinterpret_cast<const int4*>(J.rays + r);
                        rec.q0 = __ldg(rp);
                        rec.q1 = __ldg(rp + 1);
                        rec.cp = __ldg(J.cpState + cpRow + r);
                        rec.cpv = __ldg(J.cpVoxel + cpRow + r);
                        rec.y = __ldg(J.y + r);
                    }
                };
                bool newClass = false;
                bool more = nextRound(newClass);
                Record ahead;
                if (more)
                    load(ahead);
                while (more) {
                    const Record rec = ahead;
                    const bool separate = newClass;
                    newClass = false;
                    more = nextRound(newClass);
                    if (more)
                        load(ahead);
                    if (separate)
                        __syncwarp();
                    const int meta = rec.q0.w;
                    if (!(meta & kActive) || (meta & 3) != G)
                        continue;
                    if (max(rec.q1.x, rec.q1.y) < kLo || min(rec.q1.x, rec.q1.y) > kHi)
                        continue;
                    const float3 td = make_float3(__int_as_float(rec.q0.x),
                                                  __int_as_float(rec.q0.y),
                                                  __int_as_float(rec.q0.z));
                    splatAxisSegment<G, UB>(acc, td, meta, rec.q1.x, rec.cp, rec.cpv, rec.y, kLo,
                                            org[a], org[b], J.vol, J.binary);
                }
            }
            __syncwarp();
            const VolumeShape& vol = J.vol;
            const int64_t nvox = static_cast<int64_t>(vol.n[0]) * vol.n[1] * vol.n[2];
            float* dst = J.out + static_cast<int64_t>(entry.y) * nvox;
            for (int i = lane; i < EX * EY * EZ; i += 32) {
                const int lx = i % EX, ly = (i / EX) % EY, lz = i / (EX * EY);
                const int gx = org[0] + lx, gy = org[1] + ly, gz = org[2] + lz;
                if (gx < vol.n[0] && gy < vol.n[1] && gz < vol.n[2]) {
                    const int l[3] = {lx, ly, lz};
                    dst[gx + static_cast<int64_t>(vol.n[0]) *
                                 (gy + static_cast<int64_t>(vol.n[1]) * gz)] =
                        acc[l[G] * L::kPlane + l[a] * SA + l[b] * SB];
                }
            }
        }

        class SiddonProjector final : public Projector
        {
        public:
            // binary: BinaryMethod (kind 6), the same visits with weight 1
            SiddonProjector(const VolumeShape& vol, const DetectorShape& det,
                            const std::vector<PoseRecord>& poses, bool binary,
                            const CurvedDetector& curved)
                : Projector(binary ? 6 : 1, vol, det, poses), binary_(binary ? 1 : 0),
                  curved_(curved)
            {
                CurvedTables tables(vol.dim, det, curved); // used while setting up
                const int maxDim = std::max(vol_.n[0], std::max(vol_.n[1], vol_.n[2]));
                if (maxDim >= 65536)
                    throw Error(ELSA_ERROR_NOT_SUPPORTED,
                                "SiddonsMethod: volume edges must be below 65536 voxels");
                const int64_t nrays = rangeSize_;
                const int threads = 256;
                const unsigned blocks = static_cast<unsigned>((nrays + threads - 1) / threads);
                rays_ = std::make_unique<DeviceBuffer>(sizeof(SiddonRay) * nrays);
                DeviceBuffer lines(sizeof(SiddonLine) * nrays);
                siddonSetupKernel<<<blocks, threads>>>(dPoses_, vol_, det_, tables.planar(),
                                                       rays_->as<SiddonRay>(),
                                                       lines.as<SiddonLine>());
                ELSA_LAUNCH_CHECK("siddonSetupKernel");

                cpRows_ = maxDim / kSlab + 3;
                // per-view axis masks, the bad-spacing mask and a 64-bit visit counter
                const size_t words = static_cast<size_t>(det_.np) + 4;
                viewAxes_ = std::make_unique<DeviceBuffer>(sizeof(unsigned) * words);
                unsigned* dAxes = viewAxes_->as<unsigned>();
                ELSA_CUDA(cudaMemset(dAxes, 0, sizeof(unsigned) * words));
                unsigned* dBad = dAxes + det_.np;
                auto* dCount =
                    reinterpret_cast<unsigned long long*>(dAxes + ((det_.np + 2) & ~1));
                // last visited slice and visit count of every ray; the checkpoints themselves are
                // written once the brick-owner adjoint is selected (buildOwner)
                if (vol_.dim == 3)
                    siddonCheckpointKernel<3><<<blocks, threads>>>(
                        rays_->as<SiddonRay>(), nrays, vol_, cpRows_, nullptr, nullptr, dCount);
                else
                    siddonCheckpointKernel<2><<<blocks, threads>>>(
                        rays_->as<SiddonRay>(), nrays, vol_, cpRows_, nullptr, nullptr, dCount);
                ELSA_LAUNCH_CHECK("siddonCheckpointKernel");
                siddonClassCheckKernel<<<blocks, threads>>>(rays_->as<SiddonRay>(),
                                                            lines.as<SiddonLine>(), det_,
                                                            vol_.dim, dAxes, dBad);
                ELSA_LAUNCH_CHECK("siddonClassCheckKernel");
                unsigned bad = 0;
                unsigned long long count = 0;
                ELSA_CUDA(cudaMemcpy(&bad, dBad, sizeof(unsigned), cudaMemcpyDeviceToHost));
                ELSA_CUDA(cudaMemcpy(&count, dCount, sizeof(count), cudaMemcpyDeviceToHost));
                visits_ = static_cast<int64_t>(count);
                // class spacing of the brick-owner adjoint; 0 when neighbouring detector rays pass
                // within two voxels of each other even eight pixels apart (only the scatter
                // adjoint is available then)
                for (int m = kMinClass; m <= kMaxClass; ++m)
                    if (!((bad >> m) & 1u)) {
                        classSpacing_ = m;
                        break;
                    }
                const int bz = vol_.dim == 3 ? kSlab : 1;
                nBricks_ = make_int3((vol_.n[0] + kSlab - 1) / kSlab,
                                     (vol_.n[1] + kSlab - 1) / kSlab, (vol_.n[2] + bz - 1) / bz);
                adjointChunks_ = defaultChunks();
                // The deterministic brick-owner adjoint is the default wherever it exists (a
                // valid class spacing) and its per-(ray, slab) checkpoints (20 B each: about
                // 20 GB at 256^3 / 360 x 384^2) take at most a quarter of the device's memory and
                // half of what is free; otherwise the atomic scatter.
                if (classSpacing_ > 0) {
                    size_t freeBytes = 0, totalBytes = 0;
                    ELSA_CUDA(cudaMemGetInfo(&freeBytes, &totalBytes));
                    const double need = 20.0 * static_cast<double>(nrays) * cpRows_;
                    if (need <= 0.25 * static_cast<double>(totalBytes) &&
                        need <= 0.5 * static_cast<double>(freeBytes))
                        setKnob(kKnobAdjointScatter, 0);
                }
                // last, since the volume itself serves where there is no room for the copies: they
                // must not turn the adjoint to the scatter, nor take its partial volumes' memory
                if (vol_.dim == 3)
                    chooseLayouts();
                ELSA_CUDA(cudaDeviceSynchronize());
            }

            // 3D: the axis that is contiguous in the volume each driving axis is read from, and the
            // copies' buffers (for the driving axes that occur). A copy costs about 8 us and 5 ps per
            // voxel on every call; per visit of a view that reads it, it saves about 0.9 ps, and 3
            // where the volume is larger than L2. It is made where that is 1.5 times the cost.
            // Copy / none: 128^3 / 192^2, 30 views 199 / 221 us, 8 views 88 / 78, 8 views that all
            // drive along x 70 / 84; 64^3 / 90 views 87 / 95; 32^3 / 40 views 18.5 / 13.3; 500^3 /
            // 8 views, 600^2 2732 / 3482, 200^2 810 / 381.
            void chooseLayouts()
            {
                std::vector<unsigned> axes(static_cast<size_t>(det_.np));
                ELSA_CUDA(cudaMemcpy(axes.data(), viewAxes_->as<unsigned>(),
                                     sizeof(unsigned) * axes.size(), cudaMemcpyDeviceToHost));
                std::vector<float> hp(poses_.size() * kPoseFloats);
                std::memcpy(hp.data(), poses_.data(), sizeof(float) * hp.size());
                const std::array<int, 3> fast = fastAxes(hp, det_);
                constexpr double kL2Bytes = 1e8; // (126 MB, shared with the sinogram and the rays)
                const double perVoxel = 4.0 * domainSize_ > kL2Bytes ? 2.8 : 8.3;
                const double least = 1.3e7 + perVoxel * static_cast<double>(domainSize_);
                for (int f = 1; f < 3; ++f) {
                    unsigned readers = 0; // driving axes that would read this copy
                    for (int g = 0; g < 3; ++g)
                        if (fast[g] == f)
                            readers |= 1u << g;
                    const auto views = std::count_if(axes.begin(), axes.end(),
                                                     [&](unsigned a) { return a & readers; });
                    if (static_cast<double>(visits_) * views <= least * det_.np)
                        continue;
                    try {
                        copies_[f] = std::make_unique<StreamScratch>(
                            sizeof(float) * static_cast<size_t>(domainSize_));
                    } catch (const Error&) { // no room: the volume itself serves
                        cudaGetLastError();
                        continue;
                    }
                    for (int g = 0; g < 3; ++g)
                        if (fast[g] == f)
                            fast_[g] = f;
                }
            }

            void doForward(const float* x, float* y, cudaStream_t s) override
            {
                const int64_t nrays = rangeSize_;
                const unsigned blocks =
                    static_cast<unsigned>((nrays + forwardThreads_ - 1) / forwardThreads_);
                if (vol_.dim == 2) {
                    siddonForward2dKernel<<<blocks, forwardThreads_, 0, s>>>(
                        rays_->as<SiddonRay>(), nrays, x, vol_, binary_, y);
                    ELSA_LAUNCH_CHECK("siddonForward2dKernel");
                    return;
                }
                SiddonLayouts layouts;
                const int64_t plane = static_cast<int64_t>(vol_.n[0]) * vol_.n[1];
                for (int g = 0; g < 3; ++g) {
                    layouts.base[g] = x;
                    layouts.stride[g][0] = 1, layouts.stride[g][1] = vol_.n[0];
                    layouts.stride[g][2] = plane;
                }
                std::unique_ptr<StreamScratch::Lease> copies[3];
                for (int f = 1; f < 3; ++f) {
                    if (!copies_[f])
                        continue;
                    copies[f] = std::make_unique<StreamScratch::Lease>(*copies_[f], s, true);
                    if (!copies[f]->as<float>()) // no room: the volume itself serves
                        continue;
                    // axis f contiguous, then x, then the third axis
                    const int64_t nf = vol_.n[f];
                    int64_t stride[3];
                    stride[f] = 1, stride[0] = nf, stride[3 - f] = nf * vol_.n[0];
                    launchLayoutCopy(x, vol_, f, stride, copies[f]->as<float>(), s);
                    for (int g = 0; g < 3; ++g)
                        if (fast_[g] == f) {
                            layouts.base[g] = copies[f]->as<float>();
                            std::copy(stride, stride + 3, layouts.stride[g]);
                        }
                }
                auto* k = domainSize_ < (int64_t(1) << 32) ? siddonForwardKernel<unsigned>
                                                           : siddonForwardKernel<int64_t>;
                k<<<blocks, forwardThreads_, 0, s>>>(rays_->as<SiddonRay>(), nrays, layouts, vol_,
                                                     binary_, y);
                ELSA_LAUNCH_CHECK("siddonForwardKernel");
            }

            void doAdjoint(const float* y, float* x, cudaStream_t s) override
            {
                if (scatter_) {
                    const int64_t nrays = rangeSize_;
                    const unsigned blocks =
                        static_cast<unsigned>((nrays + kScatterThreads - 1) / kScatterThreads);
                    ELSA_CUDA(cudaMemsetAsync(x, 0, sizeof(float) * domainSize_, s));
                    if (vol_.dim == 3)
                        siddonScatterKernel<3><<<blocks, kScatterThreads, 0, s>>>(
                            rays_->as<SiddonRay>(), nrays, y, vol_, binary_, x);
                    else
                        siddonScatterKernel<2><<<blocks, kScatterThreads, 0, s>>>(
                            rays_->as<SiddonRay>(), nrays, y, vol_, binary_, x);
                    ELSA_LAUNCH_CHECK("siddonScatterKernel");
                    return;
                }
                if (!cpState_)
                    throw Error(ELSA_ERROR_LOGIC, "SiddonsMethod: brick-owner adjoint not built");
                if (vol_.dim == 3) {
                    if (axisPartials_ == 0) { // no ray meets the volume: nothing else writes x
                        ELSA_CUDA(cudaMemsetAsync(x, 0, sizeof(float) * domainSize_, s));
                        return;
                    }
                    float* out = axisPartials_ > 1 ? partial_->as<float>() : x;
                    const int per = (det_.np + adjointChunks_ - 1) / adjointChunks_;
                    for (int g = 0; g < 3; ++g) {
                        const SiddonGrid& G = grids_[g];
                        if (!G.present || G.entryEnd <= G.entryBegin)
                            continue;
                        SiddonAxisJob J{};
                        J.rays = rays_->as<SiddonRay>();
                        J.cpState = cpState_->as<float4>();
                        J.cpVoxel = cpVoxel_->as<unsigned>();
                        J.nrays = rangeSize_;
                        J.y = y;
                        J.windows = G.windows->as<RayWindow>();
                        J.viewAxes = viewAxes_->as<unsigned>();
                        J.chunks = dEntries_->as<int2>() + G.entryBegin;
                        J.viewsPerChunk = per;
                        J.vol = vol_;
                        J.det = det_;
                        J.m = classSpacing_;
                        J.nBricks = G.nb;
                        J.binary = binary_;
                        J.out = out;
                        const dim3 grid(static_cast<unsigned>(G.nb.x * G.nb.y * G.nb.z),
                                        static_cast<unsigned>(G.entryEnd - G.entryBegin));
#define ELSA_SIDDON_AXIS(G_, UB_) siddonAxisKernel<G_, UB_><<<grid, 32, 0, s>>>(J, 0)
                        if (g == 0) {
                            if (G.ub)
                                ELSA_SIDDON_AXIS(0, true);
                            else
                                ELSA_SIDDON_AXIS(0, false);
                        } else if (g == 1) {
                            if (G.ub)
                                ELSA_SIDDON_AXIS(1, true);
                            else
                                ELSA_SIDDON_AXIS(1, false);
                        } else {
                            if (G.ub)
                                ELSA_SIDDON_AXIS(2, true);
                            else
                                ELSA_SIDDON_AXIS(2, false);
                        }
#undef ELSA_SIDDON_AXIS
                        ELSA_LAUNCH_CHECK("siddonAxisKernel");
                    }
                    if (axisPartials_ > 1)
                        launchSumChunks(partial_->as<float>(), axisPartials_, domainSize_, x, s);
                    return;
                }
                const int nb = nBricks_.x * nBricks_.y * nBricks_.z;
                const int per = (det_.np + adjointChunks_ - 1) / adjointChunks_;
                const int used = (det_.np + per - 1) / per;
                const dim3 grid(static_cast<unsigned>(nb), static_cast<unsigned>(used));
                float* out = used > 1 ? partial_->as<float>() : x;
                // 2D: square bricks (3D volumes take the axis bricks above)
                siddonAdjointKernel<2><<<grid, 32, 0, s>>>(
                    rays_->as<SiddonRay>(), cpState_->as<float4>(), cpVoxel_->as<unsigned>(),
                    rangeSize_, y, windows_->as<RayWindow>(), viewAxes_->as<unsigned>(), vol_,
                    det_, classSpacing_, nBricks_, per, binary_, out);
                ELSA_LAUNCH_CHECK("siddonAdjointKernel");
                if (used > 1)
                    launchSumChunks(partial_->as<float>(), used, domainSize_, x, s);
            }

            int64_t info(int key) const override
            {
                switch (key) {
                case 0:
                    return classSpacing_;
                case 1: // bricks of the brick-owner adjoint (3D: over the axis grids)
                    if (vol_.dim == 3) {
                        int64_t n = 0;
                        for (const SiddonGrid& g : grids_)
                            if (g.present)
                                n += static_cast<int64_t>(g.nb.x) * g.nb.y * g.nb.z;
                        return n;
                    }
                    return static_cast<int64_t>(nBricks_.x) * nBricks_.y * nBricks_.z;
                case 2:
                    return visits_;
                case 3:
                    return 0;
                case 6: // kernel launches per forward call: the layout copies and the rays
                    return 1 + (copies_[1] ? 1 : 0) + (copies_[2] ? 1 : 0);
                case 7: // kernel launches per adjoint call (brick owner in 3D: one per axis
                        // grid; with several partial volumes: + the chunk sum)
                    if (scatter_)
                        return 1;
                    if (vol_.dim == 3) {
                        int n = 0;
                        for (const SiddonGrid& g : grids_)
                            n += g.present && g.entryEnd > g.entryBegin ? 1 : 0;
                        return n + (axisPartials_ > 1 ? 1 : 0);
                    }
                    return adjointChunks_ > 1 ? 2 : 1;
                case 8: // visits outside the windows of their bricks (brick-owner adjoint only;
                        // test support; synchronizes)
                    return windowMisses();
                default:
                    return -1;
                }
            }

            int64_t windowMisses() const
            {
                if (!cpState_)
                    return -1;
                DeviceBuffer count(sizeof(unsigned long long));
                ELSA_CUDA(cudaMemset(count.as<unsigned long long>(), 0, sizeof(unsigned long long)));
                const int64_t nrays = rangeSize_;
                const unsigned blocks = static_cast<unsigned>((nrays + 255) / 256);
                const int bz = vol_.dim == 3 ? kSlab : 1;
                if (vol_.dim == 3)
                    for (int g = 0; g < 3; ++g) {
                        if (!grids_[g].present)
                            continue;
                        siddonWindowCheckKernel<3><<<blocks, 256>>>(
                            rays_->as<SiddonRay>(), grids_[g].windows->as<RayWindow>(), vol_,
                            det_, grids_[g].edge, grids_[g].nb, g,
                            count.as<unsigned long long>());
                    }
                else
                    siddonWindowCheckKernel<2><<<blocks, 256>>>(
                        rays_->as<SiddonRay>(), windows_->as<RayWindow>(), vol_, det_,
                        make_int3(kSlab, kSlab, bz), nBricks_, -1,
                        count.as<unsigned long long>());
                ELSA_LAUNCH_CHECK("siddonWindowCheckKernel");
                unsigned long long h = 0;
                ELSA_CUDA(cudaMemcpy(&h, count.as<unsigned long long>(), sizeof(h),
                                     cudaMemcpyDeviceToHost));
                return static_cast<int64_t>(h);
            }

            std::vector<int> knobCandidates(int knob) const override
            {
                if (knob == kKnobAdjointChunks) {
                    if (scatter_)
                        return {}; // chunks only exist in the brick-owner adjoint
                    // partial volumes limited to 4 GiB
                    const int64_t byMemory =
                        std::max<int64_t>(1, (int64_t(1) << 32) / (4 * domainSize_));
                    const int limit = static_cast<int>(
                        std::min<int64_t>(std::min<int64_t>(det_.np, 256), byMemory));
                    return chunkCandidates(limit, std::min(limit, defaultChunks()));
                }
                if (knob == kKnobForwardThreads)
                    return {64, 128, 256, 512};
                if (knob == kKnobAdjointScatter)
                    return classSpacing_ > 0 ? std::vector<int>{0, 1} : std::vector<int>{1};
                return {};
            }

            int knob(int knob) const override
            {
                if (knob == kKnobAdjointChunks)
                    return adjointChunks_;
                if (knob == kKnobForwardThreads)
                    return forwardThreads_;
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
                                "SiddonsMethod: value " + std::to_string(value) +
                                    " is not a candidate of knob " + std::to_string(knob));
                }
                if (knob == kKnobForwardThreads) {
                    forwardThreads_ = value;
                    return;
                }
                if (knob == kKnobAdjointScatter) {
                    if (value == 0)
                        buildOwner();
                    else
                        releaseOwner();
                    scatter_ = value;
                } else {
                    adjointChunks_ = value;
                }
                // the partial volumes exist only while the brick-owner adjoint uses chunks (3D:
                // one per (chunk, axis grid) pair)
                int volumes = adjointChunks_;
                if (!scatter_ && vol_.dim == 3)
                    volumes = buildAxisEntries();
                const size_t need = sizeof(float) * static_cast<size_t>(domainSize_) *
                                    static_cast<size_t>(volumes);
                if (scatter_ || volumes <= 1)
                    partial_.reset();
                else if (!partial_ || partial_->bytes() < need) {
                    partial_.reset();
                    partial_ = std::make_unique<DeviceBuffer>(need);
                }
            }

        private:
            // Per-(ray, slab) checkpoints (16 + 4 bytes per ray and slab: about 20 GB at
            // 256^3 / 360 x 384^2) and per-(brick, view) ray windows of the brick-owner adjoint,
            // built when that adjoint is selected and released when the scatter adjoint is.
            void buildOwner()
            {
                if (cpState_)
                    return;
                const int64_t nrays = rangeSize_;
                const int threads = 256;
                const unsigned blocks = static_cast<unsigned>((nrays + threads - 1) / threads);
                cpState_ = std::make_unique<DeviceBuffer>(sizeof(float4) * nrays * cpRows_);
                cpVoxel_ = std::make_unique<DeviceBuffer>(sizeof(unsigned) * nrays * cpRows_);
                if (vol_.dim == 3)
                    siddonCheckpointKernel<3><<<blocks, threads>>>(
                        rays_->as<SiddonRay>(), nrays, vol_, cpRows_, cpState_->as<float4>(),
                        cpVoxel_->as<unsigned>(), nullptr);
                else
                    siddonCheckpointKernel<2><<<blocks, threads>>>(
                        rays_->as<SiddonRay>(), nrays, vol_, cpRows_, cpState_->as<float4>(),
                        cpVoxel_->as<unsigned>(), nullptr);
                ELSA_LAUNCH_CHECK("siddonCheckpointKernel");
                CurvedTables tables(vol_.dim, det_, curved_);
                if (vol_.dim == 3) {
                    buildAxisGrids(tables.map());
                    ELSA_CUDA(cudaDeviceSynchronize());
                    return;
                }
                const int bz = vol_.dim == 3 ? kSlab : 1;
                const int64_t nwin =
                    static_cast<int64_t>(nBricks_.x) * nBricks_.y * nBricks_.z * det_.np;
                windows_ = std::make_unique<DeviceBuffer>(sizeof(RayWindow) * nwin);
                // Siddon visits exactly the voxels a ray crosses: the window is the projection
                // of the brick itself, grown by kWindowSlack for the rounding of the float rays
                launchBrickWindows(dPoses_, vol_, det_, make_int3(kSlab, kSlab, bz), nBricks_,
                                   windows_->as<RayWindow>(), nullptr, tables.map(),
                                   kWindowSlack, kWindowPixelMargin);
                ELSA_CUDA(cudaDeviceSynchronize());
            }

            void releaseOwner()
            {
                ELSA_CUDA(cudaDeviceSynchronize());
                cpState_.reset();
                cpVoxel_.reset();
                windows_.reset();
                for (SiddonGrid& g : grids_)
                    g = SiddonGrid{};
                dEntries_.reset();
                axisPartials_ = 0;
            }

            // ---- 3D brick-owner adjoint on axis bricks ----
            struct SiddonGrid {
                bool present = false;
                bool ub = false; // columns along b instead of a
                int3 edge{}, nb{};
                std::unique_ptr<DeviceBuffer> windows;
                int entryBegin = 0, entryEnd = 0;
            };
            SiddonGrid grids_[3];
            std::vector<unsigned> viewAxesHost_;
            std::vector<int2> entries_;
            std::unique_ptr<DeviceBuffer> dEntries_;
            int axisPartials_ = 0;

            // Per view and driving axis g: true when neighbouring pixels of the centre detector
            // row spread more along b than along a on the planes of g.
            bool rowAlongB(int p, int g) const
            {
                const float* P = poses_[p].v + kPoseOffPinv;
                const float uc = det_.nu / 2 + 0.5f, vc = det_.nv / 2 + 0.5f;
                float D[3], E[3];
                for (int i = 0; i < 3; ++i) {
                    D[i] = P[i * 3] * uc + P[i * 3 + 1] * vc + P[i * 3 + 2];
                    E[i] = P[i * 3] * (uc + 1.0f) + P[i * 3 + 1] * vc + P[i * 3 + 2];
                }
                int a, b;
                nonDrivingAxes(g, a, b);
                if (std::fabs(D[g]) == 0.0f || std::fabs(E[g]) == 0.0f)
                    return false;
                const float da = std::fabs(E[a] / std::fabs(E[g]) - D[a] / std::fabs(D[g]));
                const float db = std::fabs(E[b] / std::fabs(E[g]) - D[b] / std::fabs(D[g]));
                return db > da;
            }

            void buildAxisGrids(CurvedMap cm)
            {
                viewAxesHost_.resize(det_.np);
                ELSA_CUDA(cudaMemcpy(viewAxesHost_.data(), viewAxes_->as<unsigned>(),
                                     sizeof(unsigned) * det_.np, cudaMemcpyDeviceToHost));
                for (int g = 0; g < 3; ++g) {
                    SiddonGrid& G = grids_[g];
                    int votes = 0, alongB = 0;
                    for (int p = 0; p < det_.np; ++p)
                        if ((viewAxesHost_[p] >> g) & 1u) {
                            ++votes;
                            alongB += rowAlongB(p, g) ? 1 : 0;
                        }
                    G.present = votes > 0;
                    if (!G.present)
                        continue;
                    G.ub = 2 * alongB > votes;
                    int a, b;
                    nonDrivingAxes(g, a, b);
                    int e[3];
                    e[g] = kSlab;
                    e[a] = G.ub ? kAxisTV : kAxisTW;
                    e[b] = G.ub ? kAxisTW : kAxisTV;
                    G.edge = make_int3(e[0], e[1], e[2]);
                    G.nb = make_int3((vol_.n[0] + e[0] - 1) / e[0], (vol_.n[1] + e[1] - 1) / e[1],
                                     (vol_.n[2] + e[2] - 1) / e[2]);
                    const int64_t nwin = static_cast<int64_t>(G.nb.x) * G.nb.y * G.nb.z * det_.np;
                    G.windows = std::make_unique<DeviceBuffer>(sizeof(RayWindow) * nwin);
                    launchBrickWindows(dPoses_, vol_, det_, G.edge, G.nb,
                                       G.windows->as<RayWindow>(), nullptr, cm, kWindowSlack,
                                       kWindowPixelMargin);
                }
            }

            // (chunk, partial volume) entries per grid for adjointChunks_ view chunks (the
            // chunks holding a view that drives along the grid's axis), partial volumes numbered
            // by (chunk, axis); returns their number.
            int buildAxisEntries()
            {
                const int per = (det_.np + adjointChunks_ - 1) / adjointChunks_;
                const int used = (det_.np + per - 1) / per;
                std::vector<std::vector<int2>> byGrid(3);
                int next = 0;
                for (int c = 0; c < used; ++c)
                    for (int g = 0; g < 3; ++g) {
                        if (!grids_[g].present)
                            continue;
                        bool any = false;
                        for (int p = c * per; p < std::min(det_.np, (c + 1) * per) && !any; ++p)
                            any = (viewAxesHost_[p] >> g) & 1u;
                        if (any)
                            byGrid[g].push_back(make_int2(c, next++));
                    }
                entries_.clear();
                for (int g = 0; g < 3; ++g) {
                    grids_[g].entryBegin = static_cast<int>(entries_.size());
                    entries_.insert(entries_.end(), byGrid[g].begin(), byGrid[g].end());
                    grids_[g].entryEnd = static_cast<int>(entries_.size());
                }
                if (next == 1)
                    for (auto& e : entries_)
                        e.y = 0;
                dEntries_ = std::make_unique<DeviceBuffer>(sizeof(int2) *
                                                           std::max<size_t>(1, entries_.size()));
                if (!entries_.empty())
                    ELSA_CUDA(cudaMemcpy(dEntries_->as<int2>(), entries_.data(),
                                         sizeof(int2) * entries_.size(), cudaMemcpyHostToDevice));
                axisPartials_ = next;
                return next;
            }

            // View chunks: enough for bricks x chunks to reach kAdjointWarpsPerSm one-warp CTAs
            // per SM and at least kMinAdjointChunks, within kChunkMemory of partial volumes
            // (256^3 / 360 views: 103.8 ms with 1 chunk, 85.5 with 32).
            int defaultChunks() const
            {
                const int nb = nBricks_.x * nBricks_.y * nBricks_.z;
                const int want = std::max((kAdjointWarpsPerSm * 148 + nb - 1) / nb,
                                          kMinAdjointChunks);
                const int64_t cap = std::max<int64_t>(1, kChunkMemory / (4 * domainSize_));
                return static_cast<int>(
                    std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(want, det_.np), cap)));
            }

            std::unique_ptr<DeviceBuffer> partial_; // adjoint: per view-chunk partial volumes
            int adjointChunks_ = 1;
            int scatter_ = 1; // until the constructor selects the brick owner (see there)
            int forwardThreads_ = kForwardThreads;
            int binary_ = 0;
            CurvedDetector curved_;
            std::unique_ptr<DeviceBuffer> rays_, cpState_, cpVoxel_, viewAxes_, windows_;
            std::array<int, 3> fast_{{0, 0, 0}};     // contiguous axis per driving axis (forward)
            std::unique_ptr<StreamScratch> copies_[3]; // volume copies with axis 1 or 2 contiguous
            int cpRows_ = 0;
            int classSpacing_ = 0;
            int64_t visits_ = 0;
            int3 nBricks_{};
        };
    } // namespace

    std::unique_ptr<Projector> makeSiddonProjector(const VolumeShape& vol,
                                                   const DetectorShape& det,
                                                   const std::vector<PoseRecord>& poses,
                                                   bool binary, const CurvedDetector& curved)
    {
        return std::make_unique<SiddonProjector>(vol, det, poses, binary, curved);
    }
} // namespace elsa_b200
