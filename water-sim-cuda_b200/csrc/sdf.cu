// Signed distance field of the obstacle triangles on the simulation grid
// (makeSDF, kernels.cu:282-300; Engine::initSDF, engine.cu:105-114).
//
// Each node at integer coordinates gets the distance to the closest triangle
// (closest point by Voronoi regions, Ericson, "Real-Time Collision Detection"
// 5.1.5), negative where its winding number (the sum of the triangles' signed
// solid angles, Van Oosterom & Strackee, 1983, over 4 * 3.1415, the
// reference's constant, kernels.cu:298) exceeds 0.5.  Evaluating both for
// every node-triangle pair is bound by issue: 30.9 ms on 128^3 nodes and
// 2,304 triangles.  Two launches instead:
//
//  1. sdf_distance_kernel: a warp per brick of 4 x 4 x 2 nodes.  Triangles are
//     sorted by the Morton code of their centroids in groups of 32 with
//     bounding boxes.  The warp looks up the vertex nearest to the brick's
//     centre and evaluates its triangle for all 32 nodes; from then on a
//     triangle whose box lies farther from the brick than the largest of the
//     nodes' distances so far cannot be the nearest one of any of them.  Lanes
//     test 32 boxes at a time, then the nodes evaluate the few triangles left,
//     so the minimum is over the same per-pair values as a pass over every
//     triangle.
//  2. the sign.  On a closed mesh (every directed edge is matched by an
//     opposite one; sdf_prepare_host) the winding number is a whole number
//     that is constant wherever the mesh is not crossed, and a ball of a
//     node's distance around it is not crossed: sdf_sign_kernel gives a CTA
//     8 x 8 x 8 nodes, sums the solid angles for the node of the largest
//     distance, spreads its sign through overlapping balls, and repeats for
//     the nodes left.  Nodes within kSdfOnMesh of the mesh, where the sum
//     itself decides, get the sum over every triangle in the order given.
//     Other meshes, and small ones on small grids (kSumPairs):
//     sdf_winding_kernel takes that sum for every node.
//     Both stream triangles through shared memory in tiles of 512: one thread
//     issues a bulk async copy (cp.async.bulk, the 1-D TMA path) of the next
//     tile into the second buffer while the CTA evaluates the current one,
//     completion tracked by an mbarrier.
//
// Measured (distance + sign): 128^3 nodes and 2,304 triangles 30.9 -> 0.52 +
// 0.36 ms, 256^3 and 3,276 triangles 330 -> 2.96 + 1.81 ms; with an open mesh,
// whose sign takes the sum at every node, 31.1 -> 27.3 and 330 -> 301 ms.  The
// distance kernel is bound by issue (81 % of issue slots, about 130 box tests
// and 30 triangles a brick), the sign kernel by the chain of sums of the few
// bricks that the mesh crosses.
//
// Each wait gives up after a fixed time, records kStatusTimeout and drains
// the copies still in flight before the CTA returns, so a lost completion
// cannot hang the device.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <utility>
#include <vector>

#include "kernels.h"
#include "launch.cuh"

namespace mpm {
namespace {

constexpr int kSdfThreads = 256;
constexpr int kTriTile = 512;                 // triangles per stage
constexpr int kTriFloats = 9;
constexpr unsigned long long kWaitNs = 2000000000ull;  // 2 s per wait
constexpr unsigned long long kSdfTestWaitNs = 20000000ull;  // the test hook's expiring wait: 20 ms
// Test hooks (the engine's wait test, the values of kWaitTest* in
// corrector_tc.cuh), acted on at the first tile after its copy has landed.
constexpr uint32_t kSdfTestGiveUp = 1u, kSdfTestExpire = 2u;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

__device__ __forceinline__ void proxy_fence_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
}

__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits for phase `parity` of `bar`; false after limit_ns.
__device__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, unsigned long long limit_ns = kWaitNs) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = globaltimer_ns();
    while (!mbar_try_wait(bar, parity)) {
        if (globaltimer_ns() - t0 > limit_ns) return false;
    }
    return true;
}

__device__ __forceinline__ float dot3(float ax, float ay, float az, float bx, float by, float bz) {
    return ax * bx + ay * by + az * bz;
}

// Signed solid angle of triangle (a, b, c) seen from the origin, the vertices
// already relative to the node (calculateSolidAngle, common.cuh:310-323).
__device__ __forceinline__ float solid_angle(float ax, float ay, float az, float bx, float by, float bz, float cx,
                                             float cy, float cz) {
    const float la = norm3df(ax, ay, az), lb = norm3df(bx, by, bz), lc = norm3df(cx, cy, cz);
    const float det = ax * (by * cz - bz * cy) + ay * (bz * cx - bx * cz) + az * (bx * cy - by * cx);
    const float div = la * lb * lc + dot3(ax, ay, az, bx, by, bz) * lc + dot3(ax, ay, az, cx, cy, cz) * lb +
                      dot3(bx, by, bz, cx, cy, cz) * la;
    return 2.0f * atan2f(det, div);
}

// Squared distance from P to triangle (a, b, c) (pointTriangleDistanceSq,
// common.cuh:325-378).
__device__ __forceinline__ float tri_dist2(float px, float py, float pz, const float* t) {
    const float ax = t[0], ay = t[1], az = t[2];
    const float abx = t[3] - ax, aby = t[4] - ay, abz = t[5] - az;
    const float acx = t[6] - ax, acy = t[7] - ay, acz = t[8] - az;
    const float apx = px - ax, apy = py - ay, apz = pz - az;
    const float d1 = dot3(abx, aby, abz, apx, apy, apz), d2 = dot3(acx, acy, acz, apx, apy, apz);
    if (d1 <= 0.0f && d2 <= 0.0f) return dot3(apx, apy, apz, apx, apy, apz);
    const float bpx = px - t[3], bpy = py - t[4], bpz = pz - t[5];
    const float d3 = dot3(abx, aby, abz, bpx, bpy, bpz), d4 = dot3(acx, acy, acz, bpx, bpy, bpz);
    if (d3 >= 0.0f && d4 <= d3) return dot3(bpx, bpy, bpz, bpx, bpy, bpz);
    const float vc = d1 * d4 - d3 * d2;
    if (vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f) {
        const float v = d1 / (d1 - d3);
        const float qx = px - (ax + v * abx), qy = py - (ay + v * aby), qz = pz - (az + v * abz);
        return dot3(qx, qy, qz, qx, qy, qz);
    }
    const float cpx = px - t[6], cpy = py - t[7], cpz = pz - t[8];
    const float d5 = dot3(abx, aby, abz, cpx, cpy, cpz), d6 = dot3(acx, acy, acz, cpx, cpy, cpz);
    if (d6 >= 0.0f && d5 <= d6) return dot3(cpx, cpy, cpz, cpx, cpy, cpz);
    const float vb = d5 * d2 - d1 * d6;
    if (vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f) {
        const float w = d2 / (d2 - d6);
        const float qx = px - (ax + w * acx), qy = py - (ay + w * acy), qz = pz - (az + w * acz);
        return dot3(qx, qy, qz, qx, qy, qz);
    }
    const float va = d3 * d6 - d5 * d4;
    if (va <= 0.0f && (d4 - d3) >= 0.0f && (d5 - d6) >= 0.0f) {
        const float w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
        const float qx = px - (t[3] + w * (t[6] - t[3])), qy = py - (t[4] + w * (t[7] - t[4])),
                    qz = pz - (t[5] + w * (t[8] - t[5]));
        return dot3(qx, qy, qz, qx, qy, qz);
    }
    const float denom = 1.0f / (va + vb + vc);
    const float v = vb * denom, w = vc * denom;
    const float qx = px - (ax + abx * v + acx * w), qy = py - (ay + aby * v + acy * w),
                qz = pz - (az + abz * v + acz * w);
    return dot3(qx, qy, qz, qx, qy, qz);
}

// The triangle list streamed tile by tile through two shared buffers.  Every
// thread of the CTA calls the members; `fresh` is false once the first tile's
// wait has been seen (the test hooks act on that one).
struct TileStream {
    float (*tri)[kTriTile * kTriFloats];
    uint64_t* bar;
    const float* src;
    int count, tiles;
    uint32_t wait_test;
    uint32_t* status;
    int issued = 0, taken = 0;  // tiles over all passes: tile i uses buffer i & 1

    __device__ __forceinline__ TileStream(float (*s_tri)[kTriTile * kTriFloats], uint64_t* s_bar, const float* t, int n,
                                          uint32_t hooks, uint32_t* st)
        : tri(s_tri), bar(s_bar), src(t), count(n), tiles((n + kTriTile - 1) / kTriTile), wait_test(hooks), status(st) {
        if (threadIdx.x == 0) {
            mbar_init(&bar[0], 1);
            mbar_init(&bar[1], 1);
            mbar_init_fence();
        }
        __syncthreads();
    }
    __device__ __forceinline__ int size(int tile) const { return min(kTriTile, count - tile * kTriTile); }
    __device__ __forceinline__ void issue(int tile) {
        if (threadIdx.x == 0) {
            const uint32_t bytes = (uint32_t)((size(tile) * kTriFloats * 4 + 15) & ~15);
            uint64_t* b = &bar[issued & 1];
            proxy_fence_shared();
            mbar_expect_tx(b, bytes);
            bulk_copy_g2s(tri[issued & 1], src + (size_t)tile * kTriTile * kTriFloats, bytes, b);
        }
        ++issued;
    }
    // Waits for the oldest tile in flight: its buffer, or null when the wait
    // gave up (every copy in flight drained; the CTA returns).
    __device__ __forceinline__ const float* take() {
        const int b = taken & 1;
        const uint32_t phase = (uint32_t)((taken >> 1) & 1);
        bool ok = mbar_wait_bounded(&bar[b], phase);
        if (ok && taken == 0 && wait_test) {
            // Test hooks, with the first copy landed: report a give-up, or
            // wait for the barrier's next phase, which no copy completes yet
            // (the buffer is refilled only after this tile), until the short
            // limit runs out.
            if (wait_test & kSdfTestGiveUp) ok = false;
            else if (wait_test & kSdfTestExpire) ok = mbar_wait_bounded(&bar[b], 1u, kSdfTestWaitNs);
        }
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0) {
                atomicOr(status, kStatusTimeout);
                for (int i = taken; i < issued; ++i) mbar_wait_bounded(&bar[i & 1], (uint32_t)((i >> 1) & 1));
            }
            __syncthreads();
            return nullptr;
        }
        ++taken;
        return tri[b];
    }
};

// The winding number of every node by the sum over every triangle in the
// order given; the sign goes to the distance that sdf holds.  A thread per
// node, a CTA per brick of 8 x 8 x 4.
constexpr int kBrickX = 8, kBrickY = 8, kBrickZ = 4;  // kSdfThreads nodes per CTA
static_assert(kBrickX * kBrickY * kBrickZ == kSdfThreads, "one node per thread");

__global__ void __launch_bounds__(kSdfThreads) sdf_winding_kernel(SimParams p, const float* __restrict__ tris,
                                                                  int t_count, float* __restrict__ sdf,
                                                                  uint32_t* __restrict__ status, uint32_t wait_test) {
    pdl_wait();
    __shared__ __align__(128) float s_tri[2][kTriTile * kTriFloats];
    __shared__ __align__(8) uint64_t s_bar[2];
    const int nbx = (p.sx + kBrickX - 1) / kBrickX, nby = (p.sy + kBrickY - 1) / kBrickY;
    const int bxi = blockIdx.x % nbx, byi = (blockIdx.x / nbx) % nby, bzi = blockIdx.x / (nbx * nby);
    const int t = threadIdx.x;
    const int x = bxi * kBrickX + t % kBrickX, y = byi * kBrickY + (t / kBrickX) % kBrickY,
              z = bzi * kBrickZ + t / (kBrickX * kBrickY);
    const float px = x * 1.0f, py = y * 1.0f, pz = z * 1.0f;
    TileStream ts(s_tri, s_bar, tris, t_count, wait_test, status);
    float wsum = 0.0f;
    if (ts.tiles > 0) ts.issue(0);
    for (int tile = 0; tile < ts.tiles; ++tile) {
        if (tile + 1 < ts.tiles) ts.issue(tile + 1);
        const float* st = ts.take();
        if (!st) return;
        const int cnt = ts.size(tile);
        for (int k = 0; k < cnt; ++k) {
            const float* tr = st + k * kTriFloats;
            wsum += solid_angle(tr[0] - px, tr[1] - py, tr[2] - pz, tr[3] - px, tr[4] - py, tr[5] - pz, tr[6] - px,
                                tr[7] - py, tr[8] - pz);
        }
        __syncthreads();
    }
    if (x < p.sx && y < p.sy && z < p.sz && wsum / (4.0f * 3.1415f) > 0.5f) {
        float* d = sdf + node_index(p, x, y, z);
        *d = -*d;
    }
}

// Squared distance from c to the nearest (lo) and farthest (hi) point of a
// box given by centre and half extents.
__device__ __forceinline__ float2 box_dist2(float cx, float cy, float cz, float4 b0, float4 b1) {
    const float ax = fabsf(cx - b0.x), ay = fabsf(cy - b0.y), az = fabsf(cz - b0.z);
    const float lx = fmaxf(ax - b0.w, 0.f), ly = fmaxf(ay - b1.x, 0.f), lz = fmaxf(az - b1.y, 0.f);
    const float hx = ax + b0.w, hy = ay + b1.x, hz = az + b1.y;
    return make_float2(lx * lx + ly * ly + lz * lz, hx * hx + hy * hy + hz * hz);
}
__device__ __forceinline__ float len2(float x, float y, float z) { return x * x + y * y + z * z; }
// Smallest of the lanes' non-negative floats (their bits order like the values).
__device__ __forceinline__ float warp_min_nonneg(float v) {
    return __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(v)));
}

constexpr int kGroup = 32;  // triangles per group of the sorted list
constexpr float kFar2 = 1e30f;

// tri: the sorted triangles, three float4 each (9 coordinates, 3 unused);
// tbox / gbox: boxes of triangles / groups, two float4 each (centre, half x;
// half y, half z).
__global__ void __launch_bounds__(256) sdf_distance_kernel(SimParams p, const float4* __restrict__ tri,
                                                           const float4* __restrict__ tbox,
                                                           const float4* __restrict__ gbox, int t_count,
                                                           float* __restrict__ sdf) {
    const int nbx = (p.sx + 3) / 4, nby = (p.sy + 3) / 4, nbz = (p.sz + 1) / 2;
    const long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    if (w >= (long long)nbx * nby * nbz) return;
    const int lane = threadIdx.x & 31;
    const int x0 = (int)(w % nbx) * 4, y0 = (int)(w / nbx % nby) * 4, z0 = (int)(w / ((long long)nbx * nby)) * 2;
    const int x = x0 + (lane & 3), y = y0 + ((lane >> 2) & 3), z = z0 + (lane >> 4);
    const float px = x * 1.0f, py = y * 1.0f, pz = z * 1.0f;
    const float cx = x0 + 1.5f, cy = y0 + 1.5f, cz = z0 + 0.5f;
    const int groups = (t_count + kGroup - 1) / kGroup;

    // The vertex nearest to c, in the groups that can hold it: those nearer
    // than the farthest corner of the nearest box, then than the best so far.
    float ub2 = kFar2;
    for (int g = lane; g < groups; g += 32) ub2 = fminf(ub2, box_dist2(cx, cy, cz, __ldg(gbox + 2 * g), __ldg(gbox + 2 * g + 1)).y);
    ub2 = warp_min_nonneg(ub2);
    int near = 0;  // the triangle of the nearest vertex
    for (int g0 = 0; g0 < groups; g0 += 32) {
        const int g = g0 + lane;
        const float lo2 = g < groups ? box_dist2(cx, cy, cz, __ldg(gbox + 2 * g), __ldg(gbox + 2 * g + 1)).x : 2.0f * kFar2;
        for (uint32_t m = __ballot_sync(0xffffffffu, lo2 <= ub2); m; m &= m - 1) {
            const int k = __ffs(m) - 1;
            if (__shfl_sync(0xffffffffu, lo2, k) > ub2) continue;  // the bound has moved
            const int i = (g0 + k) * kGroup + lane;
            float v2 = kFar2;
            if (i < t_count) {
                const float4 a = __ldg(tri + 3 * (size_t)i), b = __ldg(tri + 3 * (size_t)i + 1), c = __ldg(tri + 3 * (size_t)i + 2);
                v2 = fminf(v2, fminf(len2(a.x - cx, a.y - cy, a.z - cz),
                                     fminf(len2(a.w - cx, b.x - cy, b.y - cz), len2(b.z - cx, b.w - cy, c.x - cz))));
            }
            const float best = warp_min_nonneg(v2);
            if (best < ub2) {
                ub2 = best;
                near = (g0 + k) * kGroup + __ffs(__ballot_sync(0xffffffffu, v2 == best)) - 1;
            }
        }
    }

    // The minimum over the triangles that can be nearest to some node.
    float dmin2 = kFar2;
    auto evaluate = [&](int i) {
        const float4 a = __ldg(tri + 3 * (size_t)i), b = __ldg(tri + 3 * (size_t)i + 1), c = __ldg(tri + 3 * (size_t)i + 2);
        const float t[9] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x};
        const float d2 = tri_dist2(px, py, pz, t);
        if (d2 < dmin2) dmin2 = d2;
    };
    evaluate(near);
    // The largest of the nodes' distances so far, squared, with a margin for
    // the rounding of the values and the boxes: a box farther than that from
    // the brick (half extents 1.5, 1.5, 0.5) holds no node's nearest triangle.
    auto reach = [&] { return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(dmin2))) * 1.001f + 1e-6f; };
    auto from_brick = [&](const float4* box) {
        const float4 b0 = __ldg(box), b1 = __ldg(box + 1);
        return len2(fmaxf(fabsf(cx - b0.x) - b0.w - 1.5f, 0.f), fmaxf(fabsf(cy - b0.y) - b1.x - 1.5f, 0.f),
                    fmaxf(fabsf(cz - b0.z) - b1.y - 0.5f, 0.f));
    };
    float reach2 = reach();
    for (int g0 = 0; g0 < groups; g0 += 32) {
        const int g = g0 + lane;
        const float gd2 = g < groups ? from_brick(gbox + 2 * (size_t)g) : 2.0f * kFar2;
        for (uint32_t m = __ballot_sync(0xffffffffu, gd2 <= reach2); m; m &= m - 1) {
            const int k = __ffs(m) - 1;
            if (__shfl_sync(0xffffffffu, gd2, k) > reach2) continue;  // the reach has shrunk
            const int base = (g0 + k) * kGroup, i = base + lane;
            const bool can = i < t_count && from_brick(tbox + 2 * (size_t)i) <= reach2;
            for (uint32_t q = __ballot_sync(0xffffffffu, can); q; q &= q - 1) {
                const int j = base + __ffs(q) - 1;
                // a node skips a triangle whose box lies farther than its
                // distance so far
                const float lo2 = box_dist2(px, py, pz, __ldg(tbox + 2 * (size_t)j), __ldg(tbox + 2 * (size_t)j + 1)).x;
                if (lo2 * 0.999f <= dmin2) evaluate(j);
            }
            reach2 = reach();
        }
    }
    if (x < p.sx && y < p.sy && z < p.sz) sdf[node_index(p, x, y, z)] = sqrtf(dmin2);
}

// The sign on a closed mesh (file comment); sdf holds the distances.  A CTA
// per brick of 8 x 8 x 8 nodes and the nodes around it: a node of the brick
// close to the mesh is mostly reached through a neighbour farther from it,
// which can lie outside the brick (without that rim such nodes each need a
// sum of their own).  The nodes left over, next to the mesh, are summed a node
// per warp: starting a CTA-wide sum for each of them took 1.11 ms on 128^3
// nodes and 2,304 triangles, against 0.36.
constexpr int kSignCore = 8, kSignEdge = kSignCore + 2, kSignNodes = kSignEdge * kSignEdge * kSignEdge;
constexpr float kSdfOnMesh = 0.01f;
constexpr float kSignSpread = 1.0f;  // nodes farther from the mesh than this start a spread
enum : uint8_t { kSignOpen = 0, kSignOut = 1, kSignIn = 2, kSignSum = 3 };

__global__ void __launch_bounds__(kSdfThreads) sdf_sign_kernel(SimParams p, const float* __restrict__ tris, int t_count,
                                                               float* __restrict__ sdf, uint32_t* __restrict__ status,
                                                               uint32_t wait_test) {
    pdl_wait();
    __shared__ __align__(128) float s_tri[2][kTriTile * kTriFloats];
    __shared__ __align__(8) uint64_t s_bar[2];
    __shared__ float s_d[kSignNodes];
    __shared__ uint8_t s_sign[kSignNodes];
    __shared__ uint16_t s_left[kSignCore * kSignCore * kSignCore];
    __shared__ int s_nleft;
    __shared__ unsigned long long s_best[kSdfThreads / 32];
    __shared__ float s_part[kSdfThreads / 32];
    __shared__ float s_angle[kSdfThreads / 32][32];
    const int nbx = (p.sx + kSignCore - 1) / kSignCore, nby = (p.sy + kSignCore - 1) / kSignCore;
    // Node 0 of the region: one before the brick's first on every axis.
    const int x0 = (int)(blockIdx.x % nbx) * kSignCore - 1, y0 = (int)(blockIdx.x / nbx % nby) * kSignCore - 1,
              z0 = (int)(blockIdx.x / (nbx * nby)) * kSignCore - 1;
    auto in_core = [](int k) {
        const int kx = k % kSignEdge, ky = k / kSignEdge % kSignEdge, kz = k / (kSignEdge * kSignEdge);
        return (unsigned)(kx - 1) < kSignCore && (unsigned)(ky - 1) < kSignCore && (unsigned)(kz - 1) < kSignCore;
    };
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) s_nleft = 0;
    TileStream ts(s_tri, s_bar, tris, t_count, wait_test, status);  // its barrier publishes s_nleft
    for (int k = t; k < kSignNodes; k += kSdfThreads) {
        const int x = x0 + k % kSignEdge, y = y0 + k / kSignEdge % kSignEdge, z = z0 + k / (kSignEdge * kSignEdge);
        const bool in = node_in_grid(p, x, y, z);
        const float d = in ? fabsf(sdf[node_index(p, x, y, z)]) : 0.f;  // a rim node may have its sign already
        s_d[k] = d;
        s_sign[k] = !in ? kSignOut : (d < kSdfOnMesh ? kSignSum : kSignOpen);
    }
    __syncthreads();
    for (;;) {
        // The open node of the largest distance, while the brick has an open
        // node and that ball is wide enough to reach others.
        unsigned long long best = 0ull;
        bool open = false;
        for (int k = t; k < kSignNodes; k += kSdfThreads)
            if (s_sign[k] == kSignOpen) {
                open = open || in_core(k);
                if (s_d[k] < kSignSpread) continue;
                const unsigned long long key = ((unsigned long long)__float_as_uint(s_d[k]) << 32) | (unsigned)(k + 1);
                best = key > best ? key : best;
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
            best = other > best ? other : best;
        }
        if (lane == 0) s_best[warp] = best;
        if (!__syncthreads_or(open)) break;
#pragma unroll
        for (int q = 0; q < kSdfThreads / 32; ++q) best = s_best[q] > best ? s_best[q] : best;
        if (best == 0ull) break;
        const int a = (int)(unsigned)best - 1;
        const float px = x0 + a % kSignEdge, py = y0 + a / kSignEdge % kSignEdge, pz = z0 + a / (kSignEdge * kSignEdge);
        // Its winding number, two triangles per thread and tile.
        float wsum = 0.f;
        ts.issue(0);
        for (int tile = 0; tile < ts.tiles; ++tile) {
            if (tile + 1 < ts.tiles) ts.issue(tile + 1);
            const float* st = ts.take();
            if (!st) return;
            for (int i = t; i < ts.size(tile); i += kSdfThreads) {
                const float* tr = st + i * kTriFloats;
                wsum += solid_angle(tr[0] - px, tr[1] - py, tr[2] - pz, tr[3] - px, tr[4] - py, tr[5] - pz,
                                    tr[6] - px, tr[7] - py, tr[8] - pz);
            }
            __syncthreads();
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
        if (lane == 0) s_part[warp] = wsum;
        __syncthreads();
        wsum = 0.f;
#pragma unroll
        for (int q = 0; q < kSdfThreads / 32; ++q) wsum += s_part[q];
        const uint8_t sign = wsum / (4.0f * 3.1415f) > 0.5f ? kSignIn : kSignOut;
        // The nodes inside its ball, then on from neighbour to neighbour: two
        // balls that together cover the way between their nodes (a little
        // less, for the rounding of the distances) hold one sign.
        const float ra = s_d[a] * 0.999f;
        for (int k = t; k < kSignNodes; k += kSdfThreads) {
            const float dx = x0 + k % kSignEdge - px, dy = y0 + k / kSignEdge % kSignEdge - py,
                        dz = z0 + k / (kSignEdge * kSignEdge) - pz;
            if (s_sign[k] == kSignOpen && (k == a || len2(dx, dy, dz) < ra * ra)) s_sign[k] = sign;
        }
        __syncthreads();
        for (;;) {
            bool changed = false;
            for (int k = t; k < kSignNodes; k += kSdfThreads) {
                if (s_sign[k] != kSignOpen) continue;
                const int kx = k % kSignEdge, ky = k / kSignEdge % kSignEdge, kz = k / (kSignEdge * kSignEdge);
                uint8_t got = kSignOpen;
                for (int o = 0; o < 27; ++o) {
                    const int ox = o % 3 - 1, oy = o / 3 % 3 - 1, oz = o / 9 - 1;
                    const int nx = kx + ox, ny = ky + oy, nz = kz + oz;
                    if ((unsigned)nx >= kSignEdge || (unsigned)ny >= kSignEdge || (unsigned)nz >= kSignEdge) continue;
                    const int q = (nz * kSignEdge + ny) * kSignEdge + nx;
                    const uint8_t sq = s_sign[q];
                    const float r = 0.999f * (s_d[k] + s_d[q]);
                    if ((sq == kSignIn || sq == kSignOut) && s_d[q] > 0.f && (float)(ox * ox + oy * oy + oz * oz) < r * r)
                        got = sq;
                }
                if (got != kSignOpen) {
                    s_sign[k] = got;
                    changed = true;
                }
            }
            if (!__syncthreads_or(changed)) break;
        }
    }
    // The nodes left (close to the mesh), a node per warp and a triangle per
    // lane; for those on the mesh lane 0 adds the 32 values in the order given.
    for (int k = t; k < kSignNodes; k += kSdfThreads)
        if (in_core(k) && (s_sign[k] == kSignOpen || s_sign[k] == kSignSum)) s_left[atomicAdd(&s_nleft, 1)] = (uint16_t)k;
    __syncthreads();
    for (int j = warp; j < s_nleft; j += kSdfThreads / 32) {
        const int k = s_left[j];
        const bool ordered = s_sign[k] == kSignSum;
        const float px = x0 + k % kSignEdge, py = y0 + k / kSignEdge % kSignEdge, pz = z0 + k / (kSignEdge * kSignEdge);
        auto angle = [&](int i) {
            const float* tr = tris + (size_t)i * kTriFloats;
            return solid_angle(__ldg(tr) - px, __ldg(tr + 1) - py, __ldg(tr + 2) - pz, __ldg(tr + 3) - px,
                               __ldg(tr + 4) - py, __ldg(tr + 5) - pz, __ldg(tr + 6) - px, __ldg(tr + 7) - py,
                               __ldg(tr + 8) - pz);
        };
        float wsum = 0.f;
        if (!ordered) {
#pragma unroll 4
            for (int i = lane; i < t_count; i += 32) wsum += angle(i);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
        } else {
            for (int i0 = 0; i0 < t_count; i0 += 32) {
                if (i0 + lane < t_count) s_angle[warp][lane] = angle(i0 + lane);
                __syncwarp();
                if (lane == 0)
                    for (int q = 0; q < min(32, t_count - i0); ++q) wsum += s_angle[warp][q];
                __syncwarp();
            }
        }
        if (lane == 0) s_sign[k] = wsum / (4.0f * 3.1415f) > 0.5f ? kSignIn : kSignOut;
    }
    __syncthreads();
    for (int k = t; k < kSignNodes; k += kSdfThreads) {
        const int x = x0 + k % kSignEdge, y = y0 + k / kSignEdge % kSignEdge, z = z0 + k / (kSignEdge * kSignEdge);
        if (s_sign[k] == kSignIn && in_core(k) && x < p.sx && y < p.sy && z < p.sz)
            sdf[node_index(p, x, y, z)] = -s_d[k];
    }
}

}  // namespace

// Morton code of a point in [0, 1)^3, 10 bits per axis.
static uint32_t morton10(float x, float y, float z) {
    auto q = [](float f) { return (uint32_t)std::min(1023.0f, std::max(0.0f, f * 1024.0f)); };
    return (spread_bits3(q(z)) << 2) | (spread_bits3(q(y)) << 1) | spread_bits3(q(x));
}

// Whether the winding number is a whole number off the mesh and the kernels
// may rely on the distances: every edge is run through as often one way as the
// other (vertices compared by value), and FP32 distances exceed the true ones
// by less than half of the 0.001 by which the sign kernel's balls fall short of
// them (a distance that is too small costs a spread, never a sign).  A closest
// point errs by a few units in the last place of the coordinates, hence
// kSpreadCoord, and within the triangle's plane by the cancellation in its
// barycentric coordinates, d = about 5e-8 L (L / h)^2 with the longest edge L and
// the height h, which lengthens a distance D by d^2 / 2D: most at the smallest
// that takes part in the spread (kSdfOnMesh; nodes nearer get a sum of their
// own), hence kSpreadSliver.  Measured against 64 bits, with and without
// contraction, over 1e9 pairs of a triangle and a point at 0.01 or more from
// it: at most 1.8e-4 within both limits together, 3e-5 within kSpreadSliver
// alone at coordinates of 64 (1.2e-4 at twice the limit, 5e-4 at five times).
// The edges are matched by adding up a 128-bit hash
// of each, with the sign of its direction: the sums vanish when every edge
// cancels, and else with a probability of 2^-128.
constexpr float kSpreadCoord = 1024.0f;
constexpr double kSpreadSliver = 2e4;
static bool closed_mesh(const float* tris, int t) {
    auto mix = [](uint64_t v) {  // the finaliser of MurmurHash3 (public domain)
        v ^= v >> 33;
        v *= 0xff51afd7ed558ccdull;
        v ^= v >> 33;
        v *= 0xc4ceb9fe1a85ec53ull;
        return v ^ (v >> 33);
    };
    uint64_t sum[2] = {0, 0};
    for (int i = 0; i < t; ++i) {
        const float* v = tris + (size_t)i * 9;
        uint64_t h[3][2];
        for (int k = 0; k < 3; ++k) {
            uint32_t b[3];
            for (int a = 0; a < 3; ++a) {
                const float f = v[3 * k + a] + 0.0f;  // -0 becomes 0
                if (!(std::fabs(f) <= kSpreadCoord)) return false;
                std::memcpy(&b[a], &f, 4);
            }
            const uint64_t xy = ((uint64_t)b[0] << 32) | b[1];
            h[k][0] = mix(mix(xy + 0x9e3779b97f4a7c15ull) + b[2]);
            h[k][1] = mix(mix(xy ^ 0x2545f4914f6cdd1dull) ^ ((uint64_t)b[2] << 16));
        }
        double e[3][3], longest = 0.0;
        for (int k = 0; k < 3; ++k) {
            const float *a = v + 3 * k, *b = v + 3 * ((k + 1) % 3);
            double l2 = 0.0;
            for (int c = 0; c < 3; ++c) {
                e[k][c] = (double)b[c] - a[c];
                l2 += e[k][c] * e[k][c];
            }
            longest = std::max(longest, l2);
        }
        const double nx = e[0][1] * e[1][2] - e[0][2] * e[1][1], ny = e[0][2] * e[1][0] - e[0][0] * e[1][2],
                     nz = e[0][0] * e[1][1] - e[0][1] * e[1][0];
        // L (L / h)^2 = L^5 / |n|^2, n the cross product of two edges
        if (!(longest * longest * std::sqrt(longest) < kSpreadSliver * (nx * nx + ny * ny + nz * nz))) return false;
        for (int k = 0; k < 3; ++k)
            for (int w = 0; w < 2; ++w) {
                const uint64_t a = h[k][w], b = h[(k + 1) % 3][w];
                const uint64_t edge = mix(std::min(a, b) + mix(std::max(a, b) + 0x9e3779b97f4a7c15ull));
                if (a != b) sum[w] += a < b ? edge : (uint64_t)0 - edge;
            }
    }
    return sum[0] == 0 && sum[1] == 0;
}

// aux: the sorted triangles (12 floats each), their boxes and the groups'
// boxes (8 floats each).
constexpr int kAuxTri = 12, kAuxBox = 8;
size_t sdf_aux_floats(int t) {
    const size_t groups = (size_t)(t + kGroup - 1) / kGroup;
    return (size_t)t * (kAuxTri + kAuxBox) + groups * kAuxBox;
}

// Sums over every triangle for every node (sdf_winding_kernel) below this many
// pairs, a grid counting for at least kSumNodes nodes (what fills the GPU): the
// sign kernel's chain of sums takes 150 to 370 us on any mesh.  Sign / sums:
// 12 triangles at 128^3 262 / 160 us, 48 at 64^3 319 / 80 and at 128^3 306 / 585,
// 192 at 64^3 349 / 307, 480 at 32^3 193 / 181, 960 at 32^3 196 / 357.
constexpr long long kSumPairs = 50000000, kSumNodes = 65536;

bool sdf_prepare_host(const float* tris, int t, long long nodes, float* aux) {
    float lo[3] = {1e30f, 1e30f, 1e30f}, hi[3] = {-1e30f, -1e30f, -1e30f};
    for (int i = 0; i < t; ++i)
        for (int k = 0; k < 9; ++k) {
            lo[k % 3] = std::min(lo[k % 3], tris[i * 9 + k]);
            hi[k % 3] = std::max(hi[k % 3], tris[i * 9 + k]);
        }
    std::vector<std::pair<uint32_t, int>> key((size_t)t);
    for (int i = 0; i < t; ++i) {
        float c[3];
        for (int a = 0; a < 3; ++a) {
            const float mid = (tris[i * 9 + a] + tris[i * 9 + 3 + a] + tris[i * 9 + 6 + a]) / 3.0f;
            const float ext = hi[a] - lo[a];
            c[a] = ext > 0.0f ? (mid - lo[a]) / ext : 0.0f;
        }
        key[i] = {morton10(c[0], c[1], c[2]), i};
    }
    std::sort(key.begin(), key.end());
    float* sorted = aux;
    float* tbox = aux + (size_t)t * kAuxTri;
    float* gbox = tbox + (size_t)t * kAuxBox;
    // Centre and half extents of [lo, hi], the latter enlarged to cover it with
    // room for the rounding of the kernel's differences with centre and extents.
    auto box = [](const float* l, const float* h, float* out) {
        float half[3];
        for (int a = 0; a < 3; ++a) {
            out[a] = 0.5f * l[a] + 0.5f * h[a];
            half[a] = std::max(h[a] - out[a], out[a] - l[a]);
            half[a] = std::nextafter(half[a] + 5e-7f * (std::fabs(out[a]) + half[a]), INFINITY);
        }
        out[3] = half[0], out[4] = half[1], out[5] = half[2], out[6] = out[7] = 0.0f;
    };
    float gl[3] = {}, gh[3] = {};
    for (int i = 0; i < t; ++i) {
        const float* v = tris + (size_t)key[i].second * 9;
        std::copy(v, v + 9, sorted + (size_t)i * kAuxTri);
        float l[3], h[3];
        for (int a = 0; a < 3; ++a) {
            l[a] = std::min(v[a], std::min(v[3 + a], v[6 + a]));
            h[a] = std::max(v[a], std::max(v[3 + a], v[6 + a]));
            gl[a] = i % kGroup ? std::min(gl[a], l[a]) : l[a];
            gh[a] = i % kGroup ? std::max(gh[a], h[a]) : h[a];
        }
        box(l, h, tbox + (size_t)i * kAuxBox);
        if (i % kGroup == kGroup - 1 || i == t - 1) box(gl, gh, gbox + (size_t)(i / kGroup) * kAuxBox);
    }
    return t * std::max(nodes, kSumNodes) > kSumPairs && closed_mesh(tris, t);
}

int launch_sdf_build(const SimParams& p, const float* tris, const float* aux, int t, bool spread, float* sdf,
                     uint32_t* status, cudaStream_t st, uint32_t wait_test) {
    if (p.g <= 0 || t <= 0) return 0;
    auto bricks = [&](int ex, int ey, int ez) {
        return (long long)((p.sx + ex - 1) / ex) * ((p.sy + ey - 1) / ey) * ((p.sz + ez - 1) / ez);
    };
    const float4* tri = reinterpret_cast<const float4*>(aux);
    const float4* tbox = reinterpret_cast<const float4*>(aux + (size_t)t * kAuxTri);
    const float4* gbox = reinterpret_cast<const float4*>(aux + (size_t)t * (kAuxTri + kAuxBox));
    sdf_distance_kernel<<<(unsigned)((bricks(4, 4, 2) + 7) / 8), 256, 0, st>>>(p, tri, tbox, gbox, t, sdf);
    if (spread)
        launch_dep(sdf_sign_kernel, (unsigned)bricks(kSignCore, kSignCore, kSignCore), kSdfThreads, 0, st, p, tris, t, sdf,
                   status, wait_test);
    else
        launch_dep(sdf_winding_kernel, (unsigned)bricks(kBrickX, kBrickY, kBrickZ), kSdfThreads, 0, st, p, tris, t, sdf,
                   status, wait_test);
    return 2;
}

}  // namespace mpm
