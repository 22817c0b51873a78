// TMA-staged, plane-synchronous forward projection for 3D Joseph on sm_100a.
//
// A CTA owns a kTileU x kTileV tile of detector pixels of one view; thread = ray. When every ray
// of the tile has the same driving axis g and direction, the tile's rays cross the planes of g in
// lockstep. The volume is read from a copy laid out [g][slow][fast], where `fast` is the
// non-driving axis along which neighbouring pixels of a detector row spread, so a warp (32
// neighbouring rays) reads consecutive words. Chunks of kBoxD planes are staged into shared
// memory by one cp.async.bulk.tensor.3d per chunk (kStages-deep mbarrier pipeline); taps outside
// the volume read the TMA zero fill, which matches the reference's masked taps
// (projectors/JosephsMethod.cpp:60-97). Box origins per (tile, chunk) are computed once per
// geometry from the same accumulated sample positions the kernel uses, so every tap is inside its
// box; tiles whose rays disagree on axis or direction, or do not fit the box, use the per-ray
// gather.
//
// All waits on mbarriers are bounded (about one second of clock cycles by default); on timeout the
// CTA records bit 0 of the error word, waits (bounded again) for the copies it has issued and
// not yet consumed, and returns. For tests of that path, setWaitTest() shortens the limit and can
// withhold the copies (the barriers then expect bytes that never arrive), so the waits run out
// without any fault.
#include "joseph_tma.cuh"

#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstring>

namespace elsa_b200
{
    namespace
    {
        constexpr int TU = JosephForwardTma::kTileU, TV = JosephForwardTma::kTileV;
        constexpr int BW = JosephForwardTma::kBoxW, BH = JosephForwardTma::kBoxH;
        constexpr int BD = JosephForwardTma::kBoxD, NS = JosephForwardTma::kStages;
        constexpr int NT = JosephForwardTma::kThreads;
        constexpr int kStageFloats = BW * BH * BD;
        constexpr unsigned kStageBytes = kStageFloats * sizeof(float);
        constexpr int kFlagFallback = 8;

        __device__ __forceinline__ int floorDivI(int a, int b)
        {
            return a >= 0 ? a / b : -((-a + b - 1) / b);
        }

        __device__ __forceinline__ uint32_t smemAddr(const void* p)
        {
            return static_cast<uint32_t>(__cvta_generic_to_shared(p));
        }

        __device__ __forceinline__ void mbarInit(uint64_t* bar, unsigned count)
        {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smemAddr(bar)),
                         "r"(count)
                         : "memory");
        }

        __device__ __forceinline__ void mbarExpectTx(uint64_t* bar, unsigned bytes)
        {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                             smemAddr(bar)),
                         "r"(bytes)
                         : "memory");
        }

        __device__ __forceinline__ bool mbarTryWait(uint64_t* bar, unsigned parity)
        {
            unsigned ok;
            asm volatile("{\n\t.reg .pred p;\n\t"
                         "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                         "selp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(ok)
                         : "r"(smemAddr(bar)), "r"(parity)
                         : "memory");
            return ok != 0;
        }

        // Bounded wait of at most `limit` clock cycles; false on timeout.
        __device__ __forceinline__ bool mbarWait(uint64_t* bar, unsigned parity, long long limit)
        {
            if (mbarTryWait(bar, parity))
                return true;
            const long long t0 = clock64();
            while (!mbarTryWait(bar, parity)) {
                if (clock64() - t0 > limit)
                    return false;
            }
            return true;
        }

        // Box (c0, c1, c2) of batch element c3 of the permuted copies (a 4D tensor map whose
        // slowest dimension is the batch element; the box is one element deep there).
        __device__ __forceinline__ void tmaLoad4d(float* dst, const CUtensorMap* map, int c0,
                                                  int c1, int c2, int c3, uint64_t* bar)
        {
            asm volatile(
                "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smemAddr(dst)),
                "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3),
                "r"(smemAddr(bar))
                : "memory");
        }

        // A volume with another axis contiguous: out[sum of coordinate * outStride] = x. fast: the
        // axis that is contiguous in out (outStride 1). 32 x 8 threads per 32 x 32 block of the
        // (x, fast) plane, staged in shared memory so that reads and writes are both coalesced
        // (256^3 forward: 10.51 ms reading along `fast` directly, 10.41 so); fast == x is a
        // strided copy of rows. blockIdx.z counts the planes (and batch elements) in turn.
        struct LayoutCopy {
            int nx, nf, no, batch;
            int64_t strF, strO;          // words of x per step along fast and the third axis
            int64_t outX, outF, outO;    // words of out per step along x, fast and the third axis
            int64_t xBatch, outBatch;
        };

        __global__ void __launch_bounds__(256)
            layoutCopyKernel(const float* __restrict__ x, LayoutCopy c, float* __restrict__ out)
        {
            __shared__ float t[32][33];
            const int x0 = blockIdx.x * 32, f0 = blockIdx.y * 32;
            const int planes = c.no * c.batch;
            for (int plane = blockIdx.z; plane < planes; plane += gridDim.z) {
                const int b = plane / c.no, o = plane - b * c.no;
                const float* src = x + b * c.xBatch + o * c.strO;
                float* dst = out + b * c.outBatch + o * c.outO;
                const int ix = x0 + threadIdx.x;
                for (int j = threadIdx.y; j < 32; j += 8) {
                    const int f = f0 + j;
                    if (ix < c.nx && f < c.nf) {
                        const float v = __ldg(src + ix + f * c.strF);
                        if (c.outX == 1)
                            dst[ix + f * c.outF] = v;
                        else
                            t[j][threadIdx.x] = v;
                    }
                }
                if (c.outX == 1)
                    continue;
                __syncthreads();
                const int f = f0 + threadIdx.x;
                for (int j = threadIdx.y; j < 32; j += 8)
                    if (x0 + j < c.nx && f < c.nf)
                        dst[(x0 + j) * c.outX + f * c.outF] = t[threadIdx.x][j];
                __syncthreads();
            }
        }

        struct RayCursor {
            float pf, ps, sf, ss; // fast/slow position and step
            int t0, n;            // first plane index of the ray in tile order, sample count
        };

        __device__ __forceinline__ RayCursor cursorOf(const JosephRay& R, int fastIsA, int kStart,
                                                      int dir)
        {
            RayCursor c;
            c.pf = fastIsA ? R.pa : R.pb;
            c.ps = fastIsA ? R.pb : R.pa;
            c.sf = fastIsA ? R.sa : R.sb;
            c.ss = fastIsA ? R.sb : R.sa;
            c.t0 = (R.k0 - kStart) * dir;
            c.n = R.n;
            return c;
        }

        // Per tile: uniformity of axis/direction, plane range, and the box origin of every chunk
        // from the exact accumulated sample positions (min/max over the tile's samples).
        __global__ void __launch_bounds__(NT)
            tileSetupKernel(const JosephRay* __restrict__ rays, DetectorShape det, int tilesU,
                            int tilesV, int3 fastAxis, int maxChunks,
                            ForwardTile* __restrict__ tiles, int2* __restrict__ origins,
                            unsigned* __restrict__ fallbackCount)
        {
            constexpr int kMaxChunksSmem = 128;
            __shared__ int axisMask, dirMask, kMin, kMax, tEnd;
            __shared__ int minF[kMaxChunksSmem], maxF[kMaxChunksSmem], minS[kMaxChunksSmem],
                maxS[kMaxChunksSmem];
            __shared__ int bad;
            const int tile = blockIdx.x;
            const int p = tile / (tilesU * tilesV);
            const int tu = tile % tilesU, tv = (tile / tilesU) % tilesV;
            const int u = tu * TU + threadIdx.x % TU, v = tv * TV + threadIdx.x / TU;
            const bool valid = u < det.nu && v < det.nv;
            JosephRay R{};
            if (valid)
                R = rays[u + static_cast<int64_t>(det.nu) * (v + static_cast<int64_t>(det.nv) * p)];
            const bool live = valid && R.n > 0;
            if (threadIdx.x == 0) {
                axisMask = 0, dirMask = 0, kMin = 1 << 30, kMax = -(1 << 30), tEnd = 0, bad = 0;
            }
            for (int i = threadIdx.x; i < kMaxChunksSmem; i += NT) {
                minF[i] = 1 << 30, maxF[i] = -(1 << 30), minS[i] = 1 << 30, maxS[i] = -(1 << 30);
            }
            __syncthreads();
            if (live) {
                atomicOr(&axisMask, 1 << (R.meta & 3));
                atomicOr(&dirMask, (R.meta & 4) ? 2 : 1);
                atomicMin(&kMin, R.k0);
                atomicMax(&kMax, R.k0);
            }
            __syncthreads();
            const int g = axisMask == 4 ? 2 : (axisMask == 2 ? 1 : 0);
            const bool uniform = (axisMask == 1 || axisMask == 2 || axisMask == 4) &&
                                 (dirMask == 1 || dirMask == 2);
            const int dir = dirMask == 2 ? -1 : 1;
            const int kStart = dir > 0 ? kMin : kMax;
            int a, b;
            nonDrivingAxes(g, a, b);
            const int fast = g == 0 ? fastAxis.x : (g == 1 ? fastAxis.y : fastAxis.z);
            const bool fastIsA = fast == a;
            RayCursor c{};
            if (live && uniform) {
                c = cursorOf(R, fastIsA, kStart, dir);
                atomicMax(&tEnd, c.t0 + c.n);
            }
            __syncthreads();
            const int nChunks = (tEnd + BD - 1) / BD;
            const bool chunksOk = uniform && nChunks <= kMaxChunksSmem && nChunks <= maxChunks;
            if (live && chunksOk) {
                float pf = c.pf, ps = c.ps;
                for (int j = 0; j < c.n; ++j) {
                    const int ch = (c.t0 + j) / BD;
                    const int fi = static_cast<int>(floorf(__fsub_rn(pf, 0.5f)));
                    const int si = static_cast<int>(floorf(__fsub_rn(ps, 0.5f)));
                    atomicMin(&minF[ch], fi);
                    atomicMax(&maxF[ch], fi + 1);
                    atomicMin(&minS[ch], si);
                    atomicMax(&maxS[ch], si + 1);
                    pf = __fadd_rn(pf, c.sf);
                    ps = __fadd_rn(ps, c.ss);
                }
            }
            __syncthreads();
            if (chunksOk) {
                for (int ch = threadIdx.x; ch < nChunks; ch += NT) {
                    int2 o = make_int2(0, 0);
                    if (minF[ch] <= maxF[ch]) {
                        o.x = floorDivI(minF[ch], 4) * 4;
                        o.y = minS[ch];
                        if (maxF[ch] - o.x > BW - 1 || maxS[ch] - o.y > BH - 1)
                            atomicOr(&bad, 1);
                    }
                    origins[static_cast<int64_t>(tile) * maxChunks + ch] = o;
                }
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                ForwardTile t;
                t.kStart = kStart;
                t.nChunks = nChunks;
                const bool fallback = !chunksOk || bad || axisMask == 0;
                t.flags = g | (dir < 0 ? 4 : 0) | (fallback ? kFlagFallback : 0);
                t.pad = 0;
                tiles[tile] = t;
                if (fallback && axisMask != 0)
                    atomicAdd(fallbackCount, 1u);
            }
        }

        // The per-ray gather (fallback tiles).
        __device__ float gatherRay(const JosephRay& R, const float* __restrict__ x,
                                   const VolumeShape& vol)
        {
            const int g = R.meta & 3;
            const int dir = (R.meta & 4) ? -1 : 1;
            int a, b;
            nonDrivingAxes(g, a, b);
            const int64_t plane = static_cast<int64_t>(vol.n[0]) * vol.n[1];
            const int64_t sg = g == 0 ? 1 : (g == 1 ? vol.n[0] : plane);
            const int64_t sa = a == 0 ? 1 : (a == 1 ? vol.n[0] : plane);
            const int ng = g == 0 ? vol.n[0] : (g == 1 ? vol.n[1] : vol.n[2]);
            const int na = a == 0 ? vol.n[0] : (a == 1 ? vol.n[1] : vol.n[2]);
            const int64_t sb = b == 1 ? vol.n[0] : plane;
            const int nb = b == 1 ? vol.n[1] : vol.n[2];
            float acc = 0.0f;
            float pa = R.pa, pb = R.pb;
            int k = R.k0;
            for (int j = 0; j < R.n; ++j, k += dir, pa = __fadd_rn(pa, R.sa),
                     pb = __fadd_rn(pb, R.sb)) {
                if (static_cast<unsigned>(k) >= static_cast<unsigned>(ng))
                    continue;
                const float fa = floorf(__fsub_rn(pa, 0.5f)), fb = floorf(__fsub_rn(pb, 0.5f));
                const float cwa = __fsub_rn(__fsub_rn(pa, fa), 0.5f);
                const float cwb = __fsub_rn(__fsub_rn(pb, fb), 0.5f);
                const float wa = __fsub_rn(1.0f, cwa), wb = __fsub_rn(1.0f, cwb);
                const int ia = static_cast<int>(fa), ib = static_cast<int>(fb);
                const bool a0 = static_cast<unsigned>(ia) < static_cast<unsigned>(na);
                const bool a1 = static_cast<unsigned>(ia + 1) < static_cast<unsigned>(na);
                const bool b0 = static_cast<unsigned>(ib) < static_cast<unsigned>(nb);
                const bool b1 = static_cast<unsigned>(ib + 1) < static_cast<unsigned>(nb);
                const float* p0 = x + k * sg + ia * sa + ib * sb;
                const float v00 = (a0 && b0) ? __ldg(p0) : 0.0f;
                const float v10 = (a1 && b0) ? __ldg(p0 + sa) : 0.0f;
                const float v01 = (a0 && b1) ? __ldg(p0 + sb) : 0.0f;
                const float v11 = (a1 && b1) ? __ldg(p0 + sa + sb) : 0.0f;
                acc += wb * (wa * v00 + cwa * v10) + cwb * (wa * v01 + cwa * v11);
            }
            return R.len * acc;
        }

        // v = the shared word at byte address p where cond != 0, else v as it is (ordered with the
        // barrier waits, as every volatile asm).
        __device__ __forceinline__ void readSharedIf(float& v, unsigned p, unsigned cond)
        {
            asm volatile("{\n\t.reg .pred t;\n\tsetp.ne.u32 t, %2, 0;\n\t"
                         "@t ld.shared.f32 %0, [%1];\n\t}"
                         : "+f"(v)
                         : "r"(p), "r"(cond));
        }

        // Samples of one chunk of a ray: p2 the (fast, slow) position of its next sample, acc the
        // sums of the two footprint rows (their interpolation along fast; the one along slow is
        // the weights w.y and cw.y). DIR: the ray's direction, so that a sample's plane is an
        // immediate offset. Full: all BD samples; otherwise those with 0 <= jBase + kk < n.
        // origin: word of the chunk's stage buffer less the box origin and the bias of the two
        // floors' bit patterns (floorSmall2). The box origins of every (tile, chunk) come from the
        // same accumulated positions (tileSetupKernel: identical float operations, and a tile
        // whose samples do not fit its boxes takes the per-ray gather), so every tap lies in its
        // box and no index is clamped.
        // Bound by issue: 31 instructions per sample (position, floors and weights packed
        // two-wide). 256^3 / 360 views / 384^2: 10.41 -> 9.40 ms.
        template <int DIR, bool Full>
        __device__ __forceinline__ void chunkSamples(const float* stage, unsigned origin,
                                                     float2& p2, float2 s2, float2& acc, int jBase,
                                                     int n)
        {
            const float2 magic = make_float2(12582912.0f, 12582912.0f); // 1.5 * 2^23
            const float2 half = make_float2(0.5f, 0.5f), one = make_float2(1.0f, 1.0f);
#pragma unroll
            for (int kk = 0; kk < BD; ++kk) {
                const float2 h = sub2(p2, half);
                const float2 t = add2Down(h, magic);
                const float2 cw = sub2(h, sub2(t, magic));
                const float2 w = sub2(one, cw);
                const int word = static_cast<int>(__float_as_uint(t.y) * BW +
                                                  __float_as_uint(t.x) + origin);
                const int plane = (DIR > 0 ? kk : BD - 1 - kk) * (BW * BH);
                if (Full) {
                    const float* q = stage + word + plane;
                    acc.x = __fmaf_rn(w.y, __fmaf_rn(cw.x, q[1], w.x * q[0]), acc.x);
                    acc.y = __fmaf_rn(cw.y, __fmaf_rn(cw.x, q[BW + 1], w.x * q[BW]), acc.y);
                    p2 = add2(p2, s2);
                } else {
                    // predicated, not branched around: half of the warps would diverge
                    const unsigned on = static_cast<unsigned>(jBase + kk) <
                                        static_cast<unsigned>(n);
                    const unsigned q = static_cast<unsigned>(__cvta_generic_to_shared(stage)) +
                                       4u * static_cast<unsigned>(word + plane);
                    float v00 = 0.0f, v10 = 0.0f, v01 = 0.0f, v11 = 0.0f;
                    readSharedIf(v00, q, on);
                    readSharedIf(v10, q + 4, on);
                    readSharedIf(v01, q + 4 * BW, on);
                    readSharedIf(v11, q + 4 * BW + 4, on);
                    acc.x = __fmaf_rn(w.y, __fmaf_rn(cw.x, v10, w.x * v00), acc.x);
                    acc.y = __fmaf_rn(cw.y, __fmaf_rn(cw.x, v11, w.x * v01), acc.y);
                    const float2 next = add2(p2, s2);
                    p2 = on ? next : p2;
                }
            }
        }

        __global__ void __launch_bounds__(NT)
            forwardTmaKernel(const __grid_constant__ CUtensorMap map0,
                             const __grid_constant__ CUtensorMap map1,
                             const __grid_constant__ CUtensorMap map2,
                             const JosephRay* __restrict__ rays,
                             const ForwardTile* __restrict__ tiles,
                             const int2* __restrict__ origins, int maxChunks,
                             const float* __restrict__ x, VolumeShape vol, DetectorShape det,
                             int tilesU, int tilesV, int3 fastAxis, float* __restrict__ y,
                             unsigned* __restrict__ error, int tileBase, long long waitCycles,
                             int withhold, int64_t xStride, int64_t yStride)
        {
            // blockIdx.y: batch element (volume x + b xStride, sinogram y + b yStride)
            const int batch = static_cast<int>(blockIdx.y);
            x += batch * xStride;
            y += batch * yStride;
            extern __shared__ __align__(128) float stage[];
            __shared__ __align__(8) uint64_t full[NS];
            __shared__ int abortFlag;
            const int tile = tileBase + blockIdx.x; // tiles are view-major
            const int p = tile / (tilesU * tilesV);
            const int tu = tile % tilesU, tv = (tile / tilesU) % tilesV;
            const int u = tu * TU + threadIdx.x % TU, v = tv * TV + threadIdx.x / TU;
            const bool valid = u < det.nu && v < det.nv;
            const int64_t r = u + static_cast<int64_t>(det.nu) * (v + static_cast<int64_t>(det.nv) * p);
            JosephRay R{};
            if (valid)
                R = rays[r];
            const ForwardTile T = tiles[tile];
            if (T.flags & kFlagFallback) {
                if (valid)
                    y[r] = R.n > 0 ? gatherRay(R, x, vol) : 0.0f;
                return;
            }
            const int g = T.flags & 3;
            const int dir = (T.flags & 4) ? -1 : 1;
            const CUtensorMap* map = g == 0 ? &map0 : (g == 1 ? &map1 : &map2);
            int a, b;
            nonDrivingAxes(g, a, b);
            const int fast = g == 0 ? fastAxis.x : (g == 1 ? fastAxis.y : fastAxis.z);
            RayCursor c = cursorOf(R, fast == a, T.kStart, dir);
            if (!valid)
                c.n = 0;
            const int2* org = origins + static_cast<int64_t>(tile) * maxChunks;
            if (threadIdx.x == 0) {
                abortFlag = 0;
                for (int i = 0; i < NS; ++i)
                    mbarInit(&full[i], 1);
                asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            }
            __syncthreads();
            // box origin along g of chunk ch: planes kStart + dir * (ch*BD .. ch*BD + BD-1)
            auto issue = [&](int ch) {
                const int s = ch % NS;
                const int2 o = org[ch];
                const int gOrg = dir > 0 ? T.kStart + ch * BD : T.kStart - ch * BD - (BD - 1);
                mbarExpectTx(&full[s], kStageBytes);
                if (!withhold) // test mode: the barrier waits for bytes that never come
                    tmaLoad4d(stage + s * kStageFloats, map, o.x, o.y, gOrg, batch, &full[s]);
            };
            if (threadIdx.x == 0)
                for (int ch = 0; ch < NS && ch < T.nChunks; ++ch)
                    issue(ch);
            float2 acc = make_float2(0.0f, 0.0f); // the two footprint rows' sums
            float2 p2 = make_float2(c.pf, c.ps);  // (fast, slow) position
            const float2 s2 = make_float2(c.sf, c.ss);
            int failed = -1; // chunk whose wait timed out
            int2 ahead = T.nChunks > 0 ? org[0] : make_int2(0, 0); // next chunk's box origin
            for (int ch = 0; ch < T.nChunks; ++ch) {
                const int s = ch % NS;
                const bool ready = mbarWait(&full[s], (ch / NS) & 1, waitCycles);
                if (!ready) {
                    atomicOr(error, 1u);
                    abortFlag = 1;
                }
                const int2 o = ahead;
                if (ch + 1 < T.nChunks)
                    ahead = org[ch + 1];
                const unsigned origin = static_cast<unsigned>(s * kStageFloats) -
                                        (0x4B400000u + static_cast<unsigned>(o.x)) -
                                        (0x4B400000u + static_cast<unsigned>(o.y)) * BW;
                const int jBase = ch * BD - c.t0;
                // chunks in which every ray of the warp has all BD samples: no per-sample test
                const bool full = __all_sync(0xffffffffu, ready && jBase >= 0 && jBase + BD <= c.n);
                const int n = ready ? c.n : 0;
                if (dir > 0) {
                    if (full)
                        chunkSamples<1, true>(stage, origin, p2, s2, acc, jBase, n);
                    else
                        chunkSamples<1, false>(stage, origin, p2, s2, acc, jBase, n);
                } else {
                    if (full)
                        chunkSamples<-1, true>(stage, origin, p2, s2, acc, jBase, n);
                    else
                        chunkSamples<-1, false>(stage, origin, p2, s2, acc, jBase, n);
                }
                __syncthreads();
                if (abortFlag) { // a copy never completed: issue no more
                    failed = ch;
                    break;
                }
                if (threadIdx.x == 0 && ch + NS < T.nChunks)
                    issue(ch + NS);
            }
            if (failed >= 0) {
                // chunks failed .. failed + NS - 1 were issued and not consumed: give their
                // copies a bounded time to land before the CTA's shared memory goes away
                if (threadIdx.x == 0)
                    for (int ch = failed; ch < failed + NS && ch < T.nChunks; ++ch)
                        mbarWait(&full[ch % NS], (ch / NS) & 1, waitCycles);
                __syncthreads();
            }
            if (valid)
                y[r] = c.n > 0 ? R.len * (acc.x + acc.y) : 0.0f;
        }
    } // namespace

    namespace
    {
        PFN_cuTensorMapEncodeTiled_v12000 tensorMapEncoder()
        {
            static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
            if (!fn) {
                void* p = nullptr;
                cudaDriverEntryPointQueryResult q{};
                ELSA_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault,
                                                  &q));
                if (!p || q != cudaDriverEntryPointSuccess)
                    throw Error(ELSA_ERROR_CUDA, "cuTensorMapEncodeTiled is not available");
                fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
            }
            return fn;
        }

    } // namespace

    void launchLayoutCopy(const float* x, const VolumeShape& vol, int fast,
                          const int64_t (&outStride)[3], float* out, cudaStream_t s, int batch,
                          int64_t xStride, int64_t outBatchStride)
    {
        // with fast == x, the second axis takes the place of `fast` in the (x, fast) plane
        const int f = fast == 0 ? 1 : fast, o = 3 - f;
        const int64_t str[3] = {1, vol.n[0], static_cast<int64_t>(vol.n[0]) * vol.n[1]};
        LayoutCopy c;
        c.nx = vol.n[0], c.nf = vol.n[f], c.no = vol.n[o], c.batch = batch;
        c.strF = str[f], c.strO = str[o];
        c.outX = outStride[0], c.outF = outStride[f], c.outO = outStride[o];
        c.xBatch = xStride, c.outBatch = outBatchStride;
        const int64_t planes = static_cast<int64_t>(c.no) * batch;
        const dim3 grid((c.nx + 31) / 32, (c.nf + 31) / 32,
                        static_cast<unsigned>(std::min<int64_t>(planes, 65535)));
        layoutCopyKernel<<<grid, dim3(32, 8), 0, s>>>(x, c, out);
        ELSA_LAUNCH_CHECK("layoutCopyKernel");
    }

    // centre pixel and its right neighbour of every view
    std::array<int, 3> fastAxes(const std::vector<float>& poses, const DetectorShape& det)
    {
        {
            int votes[3][3] = {};
            for (int p = 0; p < det.np; ++p) {
                const float* Pinv = poses.data() + static_cast<size_t>(p) * 40 + 12;
                const float uc = det.nu / 2 + 0.5f, vc = det.nv / 2 + 0.5f;
                float D[3], E[3];
                for (int i = 0; i < 3; ++i) {
                    D[i] = Pinv[i * 3] * uc + Pinv[i * 3 + 1] * vc + Pinv[i * 3 + 2];
                    E[i] = Pinv[i * 3] * (uc + 1.0f) + Pinv[i * 3 + 1] * vc + Pinv[i * 3 + 2];
                }
                int g = 0;
                for (int i = 1; i < 3; ++i)
                    if (std::fabs(D[i]) > std::fabs(D[g]))
                        g = i;
                int a, b;
                nonDrivingAxes(g, a, b);
                const float da = std::fabs(E[a] / std::fabs(E[g]) - D[a] / std::fabs(D[g]));
                const float db = std::fabs(E[b] / std::fabs(E[g]) - D[b] / std::fabs(D[g]));
                votes[g][da >= db ? a : b] += 1;
            }
            std::array<int, 3> fast{};
            for (int g = 0; g < 3; ++g) {
                int a, b;
                nonDrivingAxes(g, a, b);
                fast[g] = votes[g][b] > votes[g][a] ? b : a;
            }
            return fast;
        }
    }

    JosephForwardTma::JosephForwardTma(const VolumeShape& vol, const DetectorShape& det,
                                       const std::vector<float>& poses, const JosephRay* dRays)
        : vol_(vol), det_(det), dRays_(dRays)
    {
        fast_ = fastAxes(poses, det);
        for (int g = 0; g < 3; ++g) {
            int a, b;
            nonDrivingAxes(g, a, b);
            slow_[g] = fast_[g] == a ? b : a;
        }
        tilesU_ = (det.nu + TU - 1) / TU;
        tilesV_ = (det.nv + TV - 1) / TV;
        nTiles_ = static_cast<int64_t>(tilesU_) * tilesV_ * det.np;
        const int maxN = std::max(vol.n[0], std::max(vol.n[1], vol.n[2]));
        maxChunks_ = (maxN + 2 + BD - 1) / BD + 1;
        ELSA_CUDA(cudaMalloc(&dTiles_, sizeof(ForwardTile) * nTiles_));
        ELSA_CUDA(cudaMalloc(&dChunkOrigins_, sizeof(int2) * nTiles_ * maxChunks_));
        ELSA_CUDA(cudaMalloc(&dError_, sizeof(unsigned) * 2));
        ELSA_CUDA(cudaMemset(dError_, 0, sizeof(unsigned) * 2));
        const int3 fa = make_int3(fast_[0], fast_[1], fast_[2]);
        tileSetupKernel<<<static_cast<unsigned>(nTiles_), NT>>>(
            dRays_, det_, tilesU_, tilesV_, fa, maxChunks_, dTiles_, dChunkOrigins_, dError_ + 1);
        ELSA_LAUNCH_CHECK("tileSetupKernel");
        std::vector<ForwardTile> tiles(static_cast<size_t>(nTiles_));
        ELSA_CUDA(cudaMemcpy(tiles.data(), dTiles_, sizeof(ForwardTile) * nTiles_,
                             cudaMemcpyDeviceToHost));
        int64_t fallback = 0, live = 0;
        for (const auto& t : tiles) {
            if (t.flags & kFlagFallback) {
                fallback += t.nChunks > 0 ? 1 : 0;
            } else {
                present_[t.flags & 3] = true;
                ++live;
            }
        }
        fallbackFraction_ = live + fallback ? double(fallback) / double(live + fallback) : 0.0;
        for (int g = 0; g < 3; ++g)
            if (present_[g])
                padFast_[g] = (vol.n[fast_[g]] + 3) / 4 * 4;
        ensureBatch(1);
        ELSA_CUDA(cudaFuncSetAttribute(forwardTmaKernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(NS * kStageBytes)));
    }

    // Permuted copies for `batch` volumes and their tensor maps (4D: fast, slow, driving axis,
    // batch element). Grows only; growing waits for the device, since launches in flight read
    // the old copies.
    void JosephForwardTma::ensureBatch(int batch)
    {
        if (batch <= batchCap_)
            return;
        if (batchCap_ > 0)
            ELSA_CUDA(cudaDeviceSynchronize());
        auto encode = tensorMapEncoder();
        for (int g = 0; g < 3; ++g) {
            if (!present_[g])
                continue;
            const int nf = vol_.n[fast_[g]], ns = vol_.n[slow_[g]], ng = vol_.n[g];
            if (dLayouts_[g])
                ELSA_CUDA(cudaFree(dLayouts_[g]));
            dLayouts_[g] = nullptr;
            ELSA_CUDA(cudaMalloc(&dLayouts_[g],
                                 sizeof(float) * padFast_[g] * ns * ng * static_cast<size_t>(batch)));
            const cuuint64_t dims[4] = {static_cast<cuuint64_t>(nf), static_cast<cuuint64_t>(ns),
                                        static_cast<cuuint64_t>(ng),
                                        static_cast<cuuint64_t>(batch)};
            const cuuint64_t strides[3] = {static_cast<cuuint64_t>(padFast_[g]) * 4,
                                           static_cast<cuuint64_t>(padFast_[g]) * ns * 4,
                                           static_cast<cuuint64_t>(padFast_[g]) * ns * ng * 4};
            const cuuint32_t box[4] = {BW, BH, BD, 1};
            const cuuint32_t estr[4] = {1, 1, 1, 1};
            const CUresult rc = encode(&maps_[g], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
                                       dLayouts_[g], dims, strides, box, estr,
                                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                       CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (rc != CUDA_SUCCESS)
                throw Error(ELSA_ERROR_CUDA, "cuTensorMapEncodeTiled failed");
        }
        batchCap_ = batch;
    }

    JosephForwardTma::~JosephForwardTma()
    {
        cudaFree(dTiles_);
        cudaFree(dChunkOrigins_);
        cudaFree(dError_);
        for (auto p : dLayouts_)
            if (p)
                cudaFree(p);
    }

    void JosephForwardTma::forward(const float* x, float* y, cudaStream_t s)
    {
        prepare(x, s);
        forwardViews(x, y, 0, det_.np, s);
    }

    void JosephForwardTma::forwardBatch(const float* x, int64_t xStride, float* y,
                                        int64_t yStride, int batch, cudaStream_t s)
    {
        if (batch <= 0)
            return;
        ensureBatch(batch);
        prepare(x, s, batch, xStride);
        forwardViews(x, y, 0, det_.np, s, batch, xStride, yStride);
    }

    void JosephForwardTma::prepare(const float* x, cudaStream_t s, int batch, int64_t xStride)
    {
        for (int g = 0; g < 3; ++g) {
            if (!present_[g])
                continue;
            // [g][slow][fast], rows padded to 16 bytes (the padding is outside the tensor map)
            int64_t stride[3];
            stride[fast_[g]] = 1;
            stride[slow_[g]] = padFast_[g];
            stride[g] = static_cast<int64_t>(padFast_[g]) * vol_.n[slow_[g]];
            launchLayoutCopy(x, vol_, fast_[g], stride, dLayouts_[g], s, batch, xStride,
                             stride[g] * vol_.n[g]);
        }
    }

    void JosephForwardTma::forwardViews(const float* x, float* y, int p0, int p1, cudaStream_t s,
                                        int batch, int64_t xStride, int64_t yStride)
    {
        const int64_t perView = static_cast<int64_t>(tilesU_) * tilesV_;
        const int64_t count = perView * (p1 - p0);
        if (count <= 0)
            return;
        forwardTmaKernel<<<dim3(static_cast<unsigned>(count), static_cast<unsigned>(batch)), NT,
                           NS * kStageBytes, s>>>(
            maps_[0], maps_[1], maps_[2], dRays_, dTiles_, dChunkOrigins_, maxChunks_, x, vol_,
            det_, tilesU_, tilesV_, make_int3(fast_[0], fast_[1], fast_[2]), y, dError_,
            static_cast<int>(perView * p0), waitCycles_, withhold_ ? 1 : 0, xStride, yStride);
        ELSA_LAUNCH_CHECK("forwardTmaKernel");
    }

    void JosephForwardTma::setWaitTest(long long cycles, bool withhold)
    {
        ELSA_CUDA(cudaDeviceSynchronize()); // no launch of the old setting in flight
        waitCycles_ = cycles > 0 ? cycles : kDefaultWaitCycles;
        withhold_ = withhold;
        ELSA_CUDA(cudaMemset(dError_, 0, sizeof(unsigned)));
    }

    unsigned JosephForwardTma::errorWord() const
    {
        unsigned e = 0;
        ELSA_CUDA(cudaMemcpy(&e, dError_, sizeof(unsigned), cudaMemcpyDeviceToHost));
        return e;
    }
} // namespace elsa_b200
