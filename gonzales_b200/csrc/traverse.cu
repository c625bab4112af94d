// traverse.cu - closest-hit and any-hit traversal kernels for sm_100a.
//
// k_wide: 8-wide quantised nodes (layout in gzg_internal.h).  One ray per
//   thread.  The current "node group" (child base, 8-bit hit mask in
//   front-to-back key order, interior mask) lives in registers; groups still to
//   visit go to a short per-thread stack in shared memory laid out
//   [depth][blockDim] so consecutive threads hit consecutive banks.  Node
//   records are fetched as five 128-bit read-only loads; child planes are
//   8-bit offsets turned into floats with a byte permute.  Leaf triangles are
//   tested as soon as their node is opened, in leaf order.
// k_wide_persistent, k_wide_instanced (two levels): the same steps in warps that
//   stay resident and refill idle lanes.
// k_wide_queued, k_wide_instanced_queued: those with a warp's triangle tests
//   gathered in shared memory, one pair of ray and triangle per lane; the default
//   but for launches of very many rays per node (lane_tests).  All wide kernels
//   give a ray the same hit.
// k_bvh2: the host's BVH2 traversed exactly as the reference's
//   traverse_bvh2_core (kernel.mojo:223-364), one thread per ray, with the
//   reference's slab arithmetic (kernel.mojo:171-206) in _rn intrinsics.
//
// All kernels are bounded: a step cap equal to the node count (each node is
// visited at most once per ray in a tree) and a stack-depth check set a bit in
// the scene's error word and end the ray instead of trapping.
#include "device.cuh"
#include "kernels.h"

namespace gzg {

// A persistent warp fetches new rays once at least this many of its lanes are
// idle (or all are): batching the divergent refill beats refilling every idle
// lane at once (ray-cast closest hit: 3,917 Mrays/s at 1, 4,011 at 4, 3,969
// at 8, 3,664 at 16).
constexpr int kRefillMin = 4;

// Fetch statistics of the persistent kernels (instrumented launches only,
// s.counters set): adds the lanes that reach the call to counter `which`
// (0 nodes opened, 1 triangles tested, 2 rays finished), one atomic per
// converged group.  Uninstrumented launches pay one uniform branch and keep no
// per-thread tallies (three registers under the 72-register cap).
__device__ __forceinline__ void count_lanes(const DevScene &s, int which) {
        if (s.counters == nullptr) return;
        const unsigned m = __activemask();
        if ((threadIdx.x & 31u) == (unsigned)(__ffs(m) - 1)) atomicAdd(s.counters + which, (unsigned long long)__popc(m));
}

// Chunk schedule of the persistent kernels.  Rays go out in 32-ray chunks;
// warp w of W starts with chunk w.  A warp that has used up its chunk pulls
// the next from the launch's pull counter (s.sched, cleared by launch_trace
// before the launch; one atomicAdd per 32 rays gives chunk W + the old value),
// or, without a counter, takes w + W,
// w + 2W, ...  Chunks differ in cost by the depth of their rays' traversals;
// the static sequence left the warps that drew costly chunks running alone at
// the launch's tail (ray-cast workload, closest hit: incoherent half 2,884 ->
// 3,148 Mrays/s, coherent half 7,097 -> 8,401 with the pull counter).
// 32-bit indices: launch_trace splits launches above kMaxLaunchRays.  (A
// reset of the word by the launch's last warp, instead of a clear before the
// launch, kept one more value live and spilled at the 72-register cap.)
struct ChunkCursor {
        uint32_t chunk, cursor, end;
};

__device__ __forceinline__ uint32_t grid_warps() { return (gridDim.x * blockDim.x) >> 5; }

__device__ __forceinline__ void chunk_first(ChunkCursor &c, uint32_t n) {
        c.chunk = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        c.cursor = c.chunk * 32u;
        c.end = c.cursor + 32u < n ? c.cursor + 32u : n;
}

// Warp-uniform: moves the warp to its next chunk; false when none is left.
// A warp stops pulling once a pull lands past n, so the counter ends below
// n / 32 + 2W and every index stays below 2^32.
__device__ __forceinline__ bool chunk_next(ChunkCursor &c, uint32_t *sched, uint32_t n) {
        if (sched) {
                uint32_t k = 0u;
                if ((threadIdx.x & 31u) == 0u) k = atomicAdd(sched, 1u);
                c.chunk = grid_warps() + __shfl_sync(0xFFFFFFFFu, k, 0);
        } else {
                c.chunk += grid_warps();
        }
        c.cursor = c.chunk * 32u;
        c.end = c.cursor + 32u < n ? c.cursor + 32u : n;
        return c.cursor < n;
}

// 1/d for the wide kernels' slab tests, kept finite: beyond +-limit (2^64 unless
// the scene is huge; zero included) it is +-limit with d's sign.  Finite
// reciprocals keep every plane distance free of 0 * inf = NaN, which lets the
// slab test compare float bits as integers (below).  A plane then appears at
// distance |dx| * limit instead of beyond it, still far past any hit distance
// of a scene with coordinates below about 1e12, so the test stays conservative.
// The approximate reciprocal is within an ulp; the far planes' slack covers it
// (an IEEE division costs ten instructions and a branch for each of the three
// components, at every ray and, on two levels, at every instance entered and
// left: 8M camera rays 992 -> 919 us, 8M incoherent rays 2,251 -> 2,117, 4M
// any-hit rays 915 -> 892, 2M rays through 4096 instances 1,380 -> 1,358).
__device__ __forceinline__ float wide_rcp(float d, float limit) {
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
        return copysignf(fminf(fabsf(r), limit), d);
}

// Packed FP32 pairs (sm_100a f32x2): each element rounds exactly as the
// scalar fadd / fmaf would, two elements per instruction.
struct F2 {
        float x, y;
};
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
        F2 d;
        asm("{.reg .b64 ra, rb, rc, rd;\n\t"
            "mov.b64 ra, {%2, %3};\n\t"
            "mov.b64 rb, {%4, %5};\n\t"
            "mov.b64 rc, {%6, %7};\n\t"
            "fma.rn.f32x2 rd, ra, rb, rc;\n\t"
            "mov.b64 {%0, %1}, rd;}"
            : "=f"(d.x), "=f"(d.y)
            : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
        return d;
}
// Two quantised planes as 2^15 + q floats: byte 1 of 0x470000 00 is worth q.
__device__ __forceinline__ F2 qbytes(uint32_t wa, uint32_t wb, uint32_t sel) {
        return F2{__uint_as_float(__byte_perm(wa, 0x47000000u, sel)), __uint_as_float(__byte_perm(wb, 0x47000000u, sel))};
}

struct WideRay {
        float ox, oy, oz, dx, dy, dz;
        float rdx, rdy, rdz;
        uint32_t oct;  // sign bits of the inverse direction; queued kernels: and kAlone
};

// A ray whose triangles are tested as soon as their node is opened (k_wide_queued).
constexpr uint32_t kAlone = 8u;

// What a ray hits in a wide node.
struct NodeHits {
        uint32_t nodes;       // interior children, bit key = slot ^ oct
        uint32_t imask;       // the node's interior mask, by slot
        uint32_t child_base;
        uint32_t tris;        // triangles of the leaf children hit, as bits of tri_bits
        uint32_t tri_base, tri_bits;
};
// Record of triangle bit b of a node.
__device__ __forceinline__ uint32_t tri_record(uint32_t tri_base, uint32_t tri_bits, uint32_t b) {
        return tri_base + __popc(tri_bits & ((1u << b) - 1u));
}

// Tests the 8 child boxes of a wide node against [0, thit].
// The kernels are bound by instruction issue (73 % of the slots, 14 of 32 lanes
// active on incoherent rays), and this is most of it, so it is laid out for few
// instructions per child:
// - A plane's byte q goes to byte 1 of a float worth 2^15 + q, and the 2^15 is
//   folded into the per-node constant (a - 2^15 s) instead of subtracted per
//   plane.  Rounding that constant is off by at most 2^-9 of a grid step, which
//   the boxes' margin covers (2^-15 of the extent, twice as much), or by
//   2^-23 of the distance, which the far planes' slack covers.
// - The six planes of a child are three packed pairs (near x, y; far x, y; near
//   z, far z), one f32x2 fma each.
// - A hit child sets one constant bit per slot order (hit) and its four
//   triangle bits (tris); interior and leaf children part after the loop, with
//   imask_perm and tri_bits, once per node and not per child.
// Against a subtract per plane and a per-child branch on a meta byte (us per
// launch): 8M incoherent rays on 1,310,720 triangles 2,581 -> 2,266, 8M camera
// rays 1,041 -> 951, 4M any-hit rays 1,036 -> 907, 2M rays through 4096
// instances 1,572 -> 1,384.
__device__ __forceinline__ NodeHits open_node(const uint4 *__restrict__ node, const WideRay &r, float thit) {
        const uint4 n0 = __ldg(node + 0);
        const uint4 n1 = __ldg(node + 1);
        const uint4 n2 = __ldg(node + 2);
        const uint4 n3 = __ldg(node + 3);
        const uint4 n4 = __ldg(node + 4);
        const float px = __uint_as_float(n0.x), py = __uint_as_float(n0.y), pz = __uint_as_float(n0.z);
        const uint32_t ew = n0.w;
        // step * rdir (exact power-of-two scaling) and the grid origin in t.
        const float sx = __uint_as_float((ew & 0xFFu) << 23) * r.rdx;
        const float sy = __uint_as_float(((ew >> 8) & 0xFFu) << 23) * r.rdy;
        const float sz = __uint_as_float(((ew >> 16) & 0xFFu) << 23) * r.rdz;
        const float ax = (px - r.ox) * r.rdx;
        const float ay = (py - r.oy) * r.rdy;
        const float az = (pz - r.oz) * r.rdz;
        // Far planes carry a relative slack (the reference's tFar has 1.0000003,
        // kernel.mojo:204) in their per-node constants instead of one multiply
        // per child; thit is scaled the same way once.  A plane's distance is
        // off by at most 3.5 x 2^-23 of itself (reciprocal 1, difference 0.5,
        // product 0.5, folded constant 1, fma 0.5), a near and a far plane
        // together by 7; the slack is 9.
        const float kSlack = 1.0000011f;
        const float fsx = sx * kSlack, fsy = sy * kSlack, fsz = sz * kSlack;
        const float fax = ax * kSlack, fay = ay * kSlack, faz = az * kSlack;
        const int thit_far = __float_as_int(thit * kSlack);
        const F2 bias{-32768.0f, -32768.0f};
        const F2 s_nxy{sx, sy}, s_fxy{fsx, fsy}, s_z{sz, fsz};
        const F2 a_nxy = fma2(bias, s_nxy, F2{ax, ay}), a_fxy = fma2(bias, s_fxy, F2{fax, fay}),
                 a_z = fma2(bias, s_z, F2{az, faz});
        // near/far plane words by ray sign (lo planes are near for rdir >= 0)
        const bool nx = r.oct & 1u, ny = r.oct & 2u, nz = r.oct & 4u;
        const uint32_t lx0 = n2.x, lx1 = n2.y, ly0 = n2.z, ly1 = n2.w, lz0 = n3.x, lz1 = n3.y;
        const uint32_t hx0 = n3.z, hx1 = n3.w, hy0 = n4.x, hy1 = n4.y, hz0 = n4.z, hz1 = n4.w;
        const uint32_t nearx[2] = {nx ? hx0 : lx0, nx ? hx1 : lx1};
        const uint32_t farx[2] = {nx ? lx0 : hx0, nx ? lx1 : hx1};
        const uint32_t neary[2] = {ny ? hy0 : ly0, ny ? hy1 : ly1};
        const uint32_t fary[2] = {ny ? ly0 : hy0, ny ? ly1 : hy1};
        const uint32_t nearz[2] = {nz ? hz0 : lz0, nz ? hz1 : lz1};
        const uint32_t farz[2] = {nz ? lz0 : hz0, nz ? lz1 : hz1};
        uint32_t hit = 0, tris = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
                const int w = k >> 2;
                const uint32_t sel = 0x7404u | ((uint32_t)(k & 3) << 4);
                const F2 tn = fma2(qbytes(nearx[w], neary[w], sel), s_nxy, a_nxy);
                const F2 tf = fma2(qbytes(farx[w], fary[w], sel), s_fxy, a_fxy);
                const F2 tz = fma2(qbytes(nearz[w], farz[w], sel), s_z, a_z);
                // max(0, tn*) and min(tf*, thit) on the float bits as signed
                // integers: order-preserving for non-negative floats; tnear is
                // never negative, and a negative tfar (a negative integer)
                // rejects the box either way.  No NaN occurs (finite rdir).
                const int tnear = __vimax3_s32_relu(__float_as_int(tn.x), __float_as_int(tn.y), __float_as_int(tz.x));
                const int tfar = __vimin3_s32(__float_as_int(tf.x), __float_as_int(tf.y),
                                              min(__float_as_int(tz.y), thit_far));
                if (tnear <= tfar) {
                        hit |= (1u << k) | (1u << (8 + (k ^ 1))) | (1u << (16 + (k ^ 2))) | (1u << (24 + (k ^ 3)));
                        tris |= 15u << (4 * k);
                }
        }
        NodeHits h;
        // the byte of the octant's low two bits, then its nibbles swapped for
        // the third
        const uint32_t key = ((hit & n1.z) >> ((r.oct & 3u) * 8u)) & 0xFFu;
        h.nodes = ((key * 0x101u) >> (r.oct & 4u)) & 0xFFu;
        h.imask = n1.z & 0xFFu;
        h.child_base = n1.x;
        h.tris = tris & n1.w;
        h.tri_base = n1.y;
        h.tri_bits = n1.w;
        return h;
}

template <int RAYFMT, int OUTFMT, bool ANY, int STACK, int LEAF>
__global__ void __launch_bounds__(256) k_wide(DevScene s, const void *__restrict__ rays, const float *__restrict__ tmaxs,
                                              int64_t n, void *__restrict__ out) {
        extern __shared__ uint2 smem_stack[];
        const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
        n = ray_count(s, n);
        if (i >= n) return;
        const RayIn in = load_ray<RAYFMT>(rays, tmaxs, i);
        WideRay r;
        r.ox = in.ox;
        r.oy = in.oy;
        r.oz = in.oz;
        r.dx = in.dx;
        r.dy = in.dy;
        r.dz = in.dz;
        r.rdx = wide_rcp(in.dx, s.rcp_max);
        r.rdy = wide_rcp(in.dy, s.rcp_max);
        r.rdz = wide_rcp(in.dz, s.rcp_max);
        r.oct = (__float_as_uint(r.rdx) >> 31) | ((__float_as_uint(r.rdy) >> 31) << 1) |
                ((__float_as_uint(r.rdz) >> 31) << 2);

        uint2 *stack = smem_stack + threadIdx.x;
        const int stride = blockDim.x;
        int sp = 0;
        float thit = in.tmax, bu = 0.0f, bv = 0.0f;
        int prim = -1;
        uint32_t steps = 0, n_nodes = 0, n_tris = 0;
        // The root is key 0 of a virtual parent whose only interior slot is oct.
        uint2 group = make_uint2(s.per_ray_root ? in.root : 0u, (1u << 24) | (1u << r.oct));
        for (;;) {
                uint32_t tri_hits = 0, tri_base = 0, tri_bits = 0;
                uint32_t hits = group.y >> 24;
                if (hits) {
                        const uint32_t key = __ffs(hits) - 1;
                        hits &= hits - 1;
                        const uint32_t im = group.y & 0xFFu;
                        const uint32_t slot = key ^ r.oct;
                        const uint32_t node = group.x + __popc(im & ((1u << slot) - 1u));
                        if (hits) {
                                if (sp >= STACK) {
                                        atomicOr(s.err, kErrStackOverflow);
                                        break;
                                }
                                stack[sp * stride] = make_uint2(group.x, (hits << 24) | im);
                                ++sp;
                        }
                        if (++steps > s.wide_count) {
                                atomicOr(s.err, kErrStepCap);
                                break;
                        }
                        const NodeHits h = open_node(s.wide + 5 * (size_t)node, r, thit);
                        ++n_nodes;
                        group = make_uint2(h.child_base, (h.nodes << 24) | h.imask);
                        tri_hits = h.tris;
                        tri_base = h.tri_base;
                        tri_bits = h.tri_bits;
                }
                bool done = false;
                while (tri_hits) {
                        const uint32_t b = __ffs(tri_hits) - 1;
                        tri_hits &= tri_hits - 1;
                        const uint32_t ti = tri_record(tri_base, tri_bits, b);
                        ++n_tris;
                        const float4 a = __ldg(s.tv0 + ti);
                        const float4 bb = __ldg(s.tv1 + ti);
                        const float4 c = __ldg(s.tv2 + ti);
                        float t, u, v;
                        if (leaf_test<LEAF>(r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, a, bb, c, thit, t, u, v)) {
                                thit = t;
                                bu = u;
                                bv = v;
                                prim = __float_as_int(a.w);
                                if (ANY) {
                                        done = true;
                                        break;
                                }
                        }
                }
                if (done) break;
                if ((group.y >> 24) == 0) {
                        if (sp == 0) break;
                        --sp;
                        group = stack[sp * stride];
                }
        }
        if (prim < 0) {
                thit = in.tmax;
                bu = 0.0f;
                bv = 0.0f;
        }
        store_hit<OUTFMT>(s, out, i, prim, thit, bu, bv);
        add_counters(s, n_nodes, n_tris, 1u);
}

// Persistent variant of k_wide.  The grid is sized to the resident capacity
// (SM count x blocks per SM); each warp takes 32-ray chunks by the chunk
// schedule above (the pull counter when the launch has one) and hands out the
// rays of its current chunk in order.  A lane whose ray finishes takes the
// next ray at the top of the next iteration, so lanes are not left idle while
// the slowest ray of a fixed 32-ray batch finishes.  Each iteration opens one
// node and tests its triangles.  A miss reads its tMax again at the end
// instead of keeping it in a register.
// Capped at 64 registers (8 blocks of 128 per SM; closest hit spills 8 bytes).
// With the pull counter the extra warps pay (figures of a build that spilled 28):
// ray-cast halves against 7 blocks (72 registers, no spills), incoherent 3,170 -> 3,261
// Mrays/s closest and 3,827 -> 4,148 any hit, coherent 8,362 -> 8,456 closest
// and 9,692 -> 10,197 any hit.  9 blocks (56 registers, 84 bytes of spills)
// was slower than 7.  On the static schedule 8 blocks was slower than 7.
template <int RAYFMT, int OUTFMT, bool ANY, int STACK, int LEAF>
__global__ void __launch_bounds__(128, 8) k_wide_persistent(DevScene s, const void *__restrict__ rays,
                                                         const float *__restrict__ tmaxs, int64_t n,
                                                         void *__restrict__ out) {
        extern __shared__ uint2 smem_stack[];
        const unsigned FULL = 0xFFFFFFFFu;
        const uint32_t nr = (uint32_t)ray_count(s, n);
        const unsigned lane = threadIdx.x & 31u;
        const unsigned lt_mask = (1u << lane) - 1u;
        ChunkCursor cc;
        chunk_first(cc, nr);

        uint2 *stack = smem_stack + threadIdx.x;
        const int stride = blockDim.x;
        int ray_i = -1;
        WideRay r;
        float thit = 0.0f, bu = 0.0f, bv = 0.0f;
        int prim = -1, sp = 0;
        uint2 group = make_uint2(0u, 0u);
        uint32_t steps = 0;

        for (;;) {
                // ---- refill idle lanes from this warp's chunk sequence (warp-uniform cursor)
                unsigned need = __ballot_sync(FULL, ray_i < 0);
                if (__popc(need) < kRefillMin && need != FULL) need = 0u;
                while (need != 0u && cc.cursor < nr) {
                        if (cc.cursor >= cc.end && !chunk_next(cc, s.sched, nr)) break;
                        const int avail = (int)(cc.end - cc.cursor);
                        const int rank = __popc(need & lt_mask);
                        if (ray_i < 0 && rank < avail) {
                                ray_i = (int)(cc.cursor + (uint32_t)rank);
                                const RayIn in = load_ray<RAYFMT>(rays, tmaxs, ray_i);
                                r.ox = in.ox;
                                r.oy = in.oy;
                                r.oz = in.oz;
                                r.dx = in.dx;
                                r.dy = in.dy;
                                r.dz = in.dz;
                                r.rdx = wide_rcp(in.dx, s.rcp_max);
                                r.rdy = wide_rcp(in.dy, s.rcp_max);
                                r.rdz = wide_rcp(in.dz, s.rcp_max);
                                r.oct = (__float_as_uint(r.rdx) >> 31) | ((__float_as_uint(r.rdy) >> 31) << 1) |
                                        ((__float_as_uint(r.rdz) >> 31) << 2);
                                thit = in.tmax;
                                bu = bv = 0.0f;
                                prim = -1;
                                sp = 0;
                                steps = 0;
                                group = make_uint2(s.per_ray_root ? in.root : 0u, (1u << 24) | (1u << r.oct));
                        }
                        const int npop = __popc(need);
                        cc.cursor += (uint32_t)(npop < avail ? npop : avail);
                        need = __ballot_sync(FULL, ray_i < 0);
                }
                if (__all_sync(FULL, ray_i < 0)) break;
                if (ray_i < 0) continue;

                // ---- one traversal step: open one node, test its triangles
                bool finished = false;
                uint32_t tri_hits = 0, tri_base = 0, tri_bits = 0;
                uint32_t hits = group.y >> 24;
                if (hits) {
                        const uint32_t key = __ffs(hits) - 1;
                        hits &= hits - 1;
                        const uint32_t im = group.y & 0xFFu;
                        const uint32_t slot = key ^ r.oct;
                        const uint32_t node = group.x + __popc(im & ((1u << slot) - 1u));
                        bool fault = false;
                        if (hits) {
                                if (sp >= STACK) {
                                        atomicOr(s.err, kErrStackOverflow);
                                        fault = true;
                                } else {
                                        stack[sp * stride] = make_uint2(group.x, (hits << 24) | im);
                                        ++sp;
                                }
                        }
                        if (++steps > s.wide_count) {
                                atomicOr(s.err, kErrStepCap);
                                fault = true;
                        }
                        if (fault) {
                                group.y = 0u;
                                sp = 0;
                        } else {
                                const NodeHits h = open_node(s.wide + 5 * (size_t)node, r, thit);
                                count_lanes(s, 0);
                                group = make_uint2(h.child_base, (h.nodes << 24) | h.imask);
                                tri_hits = h.tris;
                                tri_base = h.tri_base;
                                tri_bits = h.tri_bits;
                        }
                }
                while (tri_hits) {
                        const uint32_t b = __ffs(tri_hits) - 1;
                        tri_hits &= tri_hits - 1;
                        const uint32_t ti = tri_record(tri_base, tri_bits, b);
                        count_lanes(s, 1);
                        const float4 a = __ldg(s.tv0 + ti);
                        const float4 bb = __ldg(s.tv1 + ti);
                        const float4 c = __ldg(s.tv2 + ti);
                        float t, u, v;
                        if (leaf_test<LEAF>(r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, a, bb, c, thit, t, u, v)) {
                                thit = t;
                                bu = u;
                                bv = v;
                                prim = __float_as_int(a.w);
                                if (ANY) {
                                        finished = true;
                                        break;
                                }
                        }
                }
                if (!finished && (group.y >> 24) == 0) {
                        if (sp == 0)
                                finished = true;
                        else {
                                --sp;
                                group = stack[sp * stride];
                        }
                }
                if (finished) {
                        if (prim < 0) {
                                // a miss reports the ray's tMax, read again
                                // rather than kept in a register
                                thit = load_ray<RAYFMT>(rays, tmaxs, ray_i).tmax;
                                bu = 0.0f;
                                bv = 0.0f;
                        }
                        store_hit<OUTFMT>(s, out, ray_i, prim, thit, bu, bv);
                        ray_i = -1;
                        count_lanes(s, 2);
                }
        }
}

// Triangle queue of a warp (k_wide_queued, k_wide_instanced_queued): up to 32
// (record, owner lane) pairs, and the tests' results by queue position.
struct TriQueue {
        float4 result[32];  // t, u, v, prim bits; written where the test passed
        uint2 pair[32];
};

// The two-level kernel has no registers left for what only the end of a ray reads
// (2M rays through 4096 instances 1,298 us with it in registers, 1,219 here; the
// one-level kernel is 2 % faster with registers).
struct InstQueue : TriQueue {
        float2 uv[32];  // u, v of each lane's nearest hit
        int inst[32];   // its instance
};

// Adds the triangles `tris` (bits of tri_bits) of every lane to the queue of
// `queued` pairs, in lane order, as far as there is room; `have` = the lanes
// that have some, and a lane adds `most` at a time.  The positions a lane's
// triangles get are added to `mine`.  Returns the new length.
__device__ __forceinline__ uint32_t queue_append(TriQueue &queue, uint32_t queued, unsigned have, uint32_t &tris,
                                                 uint32_t tri_base, uint32_t tri_bits, uint32_t &mine, int most) {
        const unsigned FULL = 0xFFFFFFFFu;
        const unsigned lane = threadIdx.x & 31u;
        const unsigned lt_mask = (1u << lane) - 1u;
        uint32_t added;
        if (__any_sync(FULL, (tris & (tris - 1u)) != 0u)) {
                // up to 7 a lane at once, counted by three ballots; the rest is
                // left to the next call
                const uint32_t count = min(__popc(tris), most);
                const unsigned c0 = __ballot_sync(FULL, count & 1u), c1 = __ballot_sync(FULL, count & 2u),
                               c2 = __ballot_sync(FULL, count & 4u);
                uint32_t at = queued + __popc(c0 & lt_mask) + 2u * __popc(c1 & lt_mask) + 4u * __popc(c2 & lt_mask);
                added = __popc(c0) + 2u * __popc(c1) + 4u * __popc(c2);
                for (const uint32_t last = min(at + count, 32u); at < last; ++at) {
                        const uint32_t b = __ffs(tris) - 1;
                        tris &= tris - 1;
                        queue.pair[at] = make_uint2(tri_record(tri_base, tri_bits, b), lane);
                        mine |= 1u << at;
                }
        } else {
                const uint32_t at = queued + __popc(have & lt_mask);
                added = __popc(have);
                if (tris != 0u && at < 32u) {
                        queue.pair[at] = make_uint2(tri_record(tri_base, tri_bits, (uint32_t)(__ffs(tris) - 1)), lane);
                        mine |= 1u << at;
                        tris = 0u;
                }
        }
        return min(queued + added, 32u);
}

// Tests the queue's pairs, one per lane, each against its owner's ray and
// nearest hit so far; the results of the tests that passed (the bits returned)
// are in queue.result.
template <int LEAF>
__device__ __forceinline__ unsigned queue_test(const DevScene &s, TriQueue &queue, uint32_t queued, const WideRay &r,
                                               float thit) {
        const unsigned FULL = 0xFFFFFFFFu;
        const unsigned lane = threadIdx.x & 31u;
        __syncwarp();
        const bool test = lane < queued;
        const uint2 pair = queue.pair[test ? lane : 0u];
        const int owner = (int)pair.y;
        const float ox = __shfl_sync(FULL, r.ox, owner), oy = __shfl_sync(FULL, r.oy, owner),
                    oz = __shfl_sync(FULL, r.oz, owner), dx = __shfl_sync(FULL, r.dx, owner),
                    dy = __shfl_sync(FULL, r.dy, owner), dz = __shfl_sync(FULL, r.dz, owner);
        const float limit = __shfl_sync(FULL, thit, owner);
        bool ok = false;
        if (test) {
                count_lanes(s, 1);
                const float4 a = __ldg(s.tv0 + pair.x);
                const float4 b = __ldg(s.tv1 + pair.x);
                const float4 c = __ldg(s.tv2 + pair.x);
                float t, u, v;
                ok = leaf_test<LEAF>(ox, oy, oz, dx, dy, dz, a, b, c, limit, t, u, v);
                if (ok) queue.result[lane] = make_float4(t, u, v, a.w);
        }
        const unsigned passed = __ballot_sync(FULL, ok);
        __syncwarp();
        return passed;
}

// Whether a ray that prunes at once would test triangle ti too, which the queue
// accepted at t, at most the nearest hit before it: every box above the triangle
// is entered before t.  Those boxes hold the triangle's own bounds with a margin
// of 2^-18 of the coordinates; half of it is used here, half is left to rounding.
// A box's distance and the one here come from the same reciprocals and differ by
// at most 3.5 x 2^-23 of themselves, 4.2 x 2^-23 is forgiven here, and open_node
// forgives 9.
__device__ __forceinline__ float tri_entry_axis(float o, float rd, float a, float b, float c) {
        const float lo = fminf(a, fminf(b, c)), hi = fmaxf(a, fmaxf(b, c));
        const float margin = fmaxf(fabsf(lo), fabsf(hi)) * 1.9073486e-6f;  // 2^-19
        return ((rd < 0.0f ? hi + margin : lo - margin) - o) * rd;
}

__device__ __forceinline__ bool box_before(const DevScene &s, const WideRay &r, uint32_t ti, float t) {
        const float4 a = __ldg(s.tv0 + ti), b = __ldg(s.tv1 + ti), c = __ldg(s.tv2 + ti);
        const float entry = fmaxf(tri_entry_axis(r.ox, r.rdx, a.x, b.x, c.x),
                                  fmaxf(tri_entry_axis(r.oy, r.rdy, a.y, b.y, c.y),
                                        tri_entry_axis(r.oz, r.rdz, a.z, b.z, c.z)));
        return entry <= t * 1.0000005f;
}

// Pairs that make a warp test its queue, and rays that only wait for it.  More
// pairs fill the tests' lanes better but prune later: of 8 to 32 pairs and 2 to
// 8 rays these were the best over camera, incoherent and any-hit rays (8M
// incoherent rays 1,769 us at 20 pairs and 1,833 at 8 or 32, 8M camera rays 960
// at 32).
constexpr int kQueueTests = 12, kQueueWaiting = 3;

// k_wide_persistent with its triangle tests gathered over the warp.  An
// incoherent warp opens nodes on 29 lanes but finds about six triangles a step,
// two or three on one lane: testing them lane by lane ran the 90 instructions
// of a test two or three times a step on two or three lanes.  Here the pairs
// queue up in shared memory and are tested one per lane, with the owner's ray
// by shuffle; a ray goes on opening nodes meanwhile, against the nearest hit it
// knows.  The hits are those of k_wide_persistent: a triangle is accepted at
// t <= the nearest t of those before it, and pairs are taken in the order of the
// nodes.  Nodes opened before a hit in the queue is known add triangles that
// k_wide_persistent would not test; one of them can only be accepted if its
// computed t falls before its own boxes (slivers, rays along a surface), if a t
// is NaN, or if the watertight test's rounded limit let a t above the limit in.
// Such a ray starts over with its triangles tested one by one as their node is
// opened (kAlone), so its hit depends on the ray alone and not on its warp
// (2 to 3 % of a launch: 8M incoherent rays 1,802 -> 1,849 us, 8M camera rays
// 870 -> 894).
// Against k_wide_persistent: 8M incoherent rays on 1,310,720 triangles 2,116 ->
// 1,849 us, 4M any-hit rays 892 -> 830, 8M camera rays 918 -> 894, 64 x 64 camera
// rays on 20,480 triangles 41.1 -> 35.9.  launch_trace says where k_wide_persistent stays.
template <int RAYFMT, int OUTFMT, bool ANY, int STACK, int LEAF>
__global__ void __launch_bounds__(128, 8) k_wide_queued(DevScene s, const void *__restrict__ rays,
                                                        const float *__restrict__ tmaxs, int64_t n,
                                                        void *__restrict__ out) {
        extern __shared__ __align__(16) uint2 smem_stack[];
        const unsigned FULL = 0xFFFFFFFFu;
        const uint32_t nr = (uint32_t)ray_count(s, n);
        const unsigned lane = threadIdx.x & 31u;
        const unsigned lt_mask = (1u << lane) - 1u;
        ChunkCursor cc;
        chunk_first(cc, nr);

        uint2 *stack = smem_stack + threadIdx.x;
        const int stride = blockDim.x;
        TriQueue &queue = reinterpret_cast<TriQueue *>(smem_stack + STACK * blockDim.x)[threadIdx.x >> 5];
        uint32_t queued = 0;  // pairs in the queue (warp-uniform)
        uint32_t mine = 0;    // queue positions of this lane's ray
        int ray_i = -1;
        WideRay r;
        float thit = 0.0f, bu = 0.0f, bv = 0.0f;
        int prim = -1, sp = 0;
        uint2 group = make_uint2(0u, 0u);
        uint32_t steps = 0;

        for (;;) {
                // ---- refill idle lanes from this warp's chunk sequence (warp-uniform cursor)
                unsigned need = __ballot_sync(FULL, ray_i < 0);
                if (__popc(need) < kRefillMin && need != FULL) need = 0u;
                while (need != 0u && cc.cursor < nr) {
                        if (cc.cursor >= cc.end && !chunk_next(cc, s.sched, nr)) break;
                        const int avail = (int)(cc.end - cc.cursor);
                        const int rank = __popc(need & lt_mask);
                        if (ray_i < 0 && rank < avail) {
                                ray_i = (int)(cc.cursor + (uint32_t)rank);
                                const RayIn in = load_ray<RAYFMT>(rays, tmaxs, ray_i);
                                r.ox = in.ox;
                                r.oy = in.oy;
                                r.oz = in.oz;
                                r.dx = in.dx;
                                r.dy = in.dy;
                                r.dz = in.dz;
                                r.rdx = wide_rcp(in.dx, s.rcp_max);
                                r.rdy = wide_rcp(in.dy, s.rcp_max);
                                r.rdz = wide_rcp(in.dz, s.rcp_max);
                                r.oct = (__float_as_uint(r.rdx) >> 31) | ((__float_as_uint(r.rdy) >> 31) << 1) |
                                        ((__float_as_uint(r.rdz) >> 31) << 2);
                                thit = in.tmax;
                                bu = bv = 0.0f;
                                prim = -1;
                                sp = 0;
                                steps = 0;
                                group = make_uint2(s.per_ray_root ? in.root : 0u, (1u << 24) | (1u << r.oct));
                        }
                        const int npop = __popc(need);
                        cc.cursor += (uint32_t)(npop < avail ? npop : avail);
                        need = __ballot_sync(FULL, ray_i < 0);
                }
                if (__all_sync(FULL, ray_i < 0)) break;

                // ---- open one node of every ray that has one left; a ray without
                // hits left in its group takes the next from its stack at once
                uint32_t tris = 0, tri_base = 0, tri_bits = 0;
                uint32_t hits = group.y >> 24;
                if (hits) {
                        const uint32_t key = __ffs(hits) - 1;
                        hits &= hits - 1;
                        const uint32_t im = group.y & 0xFFu;
                        const uint32_t slot = (key ^ r.oct) & 7u;
                        const uint32_t node = group.x + __popc(im & ((1u << slot) - 1u));
                        bool fault = false;
                        if (hits) {
                                if (sp >= STACK) {
                                        atomicOr(s.err, kErrStackOverflow);
                                        fault = true;
                                } else {
                                        stack[sp * stride] = make_uint2(group.x, (hits << 24) | im);
                                        ++sp;
                                }
                        }
                        if (++steps > s.wide_count) {
                                atomicOr(s.err, kErrStepCap);
                                fault = true;
                        }
                        group.y = 0u;
                        if (fault) {
                                sp = 0;
                        } else {
                                const NodeHits h = open_node(s.wide + 5 * (size_t)node, r, thit);
                                count_lanes(s, 0);
                                group = make_uint2(h.child_base, (h.nodes << 24) | h.imask);
                                tris = h.tris;
                                tri_base = h.tri_base;
                                tri_bits = h.tri_bits;
                        }
                        if ((group.y >> 24) == 0 && sp > 0) {
                                --sp;
                                group = stack[sp * stride];
                        }
                }
                __syncwarp();

                // ---- queue the triangles of the leaves hit; test the queue when it
                // is full enough, or rays only wait for it
                unsigned have = __ballot_sync(FULL, tris != 0u);
                while ((have | queued) != 0u) {
                        if (have != 0u) {
                                queued = queue_append(queue, queued, have, tris, tri_base, tri_bits, mine,
                                                      !ANY && (r.oct & kAlone) ? 1 : 7);
                                have = __ballot_sync(FULL, tris != 0u);  // what found no room
                        }
                        if (have == 0u && queued < kQueueTests &&
                            (ANY || !__any_sync(FULL, (r.oct & kAlone) && mine != 0u))) {
                                const unsigned busy = __ballot_sync(FULL, (group.y >> 24) != 0u);
                                const unsigned waiting = __ballot_sync(FULL, (group.y >> 24) == 0u && mine != 0u);
                                if (busy != 0u && __popc(waiting) < kQueueWaiting) break;
                        }
                        bool again = false;
                        uint32_t passed = queue_test<LEAF>(s, queue, queued, r, thit) & mine;
                        // in queue order, a later triangle at the same t wins
                        while (passed) {
                                const uint32_t b = __ffs(passed) - 1;
                                passed &= passed - 1;
                                float4 h = queue.result[b];
                                const uint32_t ti = queue.pair[b].x;
                                if (LEAF == GZG_LEAF_WATERTIGHT) {
                                        // its limit is rounded with the triangle's
                                        // determinant: tested again against the
                                        // hits before it
                                        if (!leaf_test<LEAF>(r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, __ldg(s.tv0 + ti),
                                                             __ldg(s.tv1 + ti), __ldg(s.tv2 + ti), thit, h.x, h.y, h.z))
                                                continue;
                                } else if (h.x > thit) {  // as mt_test: a NaN limit or distance accepts
                                        continue;
                                }
                                if (!ANY && !(h.x <= thit && (prim < 0 || box_before(s, r, ti, h.x))) &&
                                    !(r.oct & kAlone)) {
                                        again = true;
                                        break;
                                }
                                thit = h.x;
                                bu = h.y;
                                bv = h.z;
                                prim = __float_as_int(h.w);
                                if (ANY) {
                                        tris = 0u;
                                        break;  // the first one, whatever was tested with it
                                }
                        }
                        __syncwarp();
                        mine = 0u;
                        queued = 0u;
                        if (again) {
                                const RayIn in = load_ray<RAYFMT>(rays, tmaxs, ray_i);
                                thit = in.tmax;
                                prim = -1;
                                sp = 0;
                                steps = 0;
                                group = make_uint2(s.per_ray_root ? in.root : 0u, (1u << 24) | (1u << r.oct));
                                r.oct |= kAlone;
                                tris = 0u;
                        }
                        have = __ballot_sync(FULL, tris != 0u);
                }
                if (ray_i >= 0 && mine == 0u && (ANY ? prim >= 0 || (group.y >> 24) == 0u : (group.y >> 24) == 0u)) {
                        if (prim < 0) {
                                // a miss reports the ray's tMax, read again
                                // rather than kept in a register
                                thit = load_ray<RAYFMT>(rays, tmaxs, ray_i).tmax;
                                bu = 0.0f;
                                bv = 0.0f;
                        }
                        store_hit<OUTFMT>(s, out, ray_i, prim, thit, bu, bv);
                        ray_i = -1;
                        group.y = 0u;
                        sp = 0;
                        count_lanes(s, 2);
                }
        }
}

__device__ __forceinline__ void set_ray_dirs(WideRay &r, float limit) {
        r.rdx = wide_rcp(r.dx, limit);
        r.rdy = wide_rcp(r.dy, limit);
        r.rdz = wide_rcp(r.dz, limit);
        r.oct = (__float_as_uint(r.rdx) >> 31) | ((__float_as_uint(r.rdy) >> 31) << 1) |
                ((__float_as_uint(r.rdz) >> 31) << 2);
}

// The world-space ray of device-ray slot i, read again from the ray array (the
// two-level kernel keeps it out of registers: it is needed only when a ray
// enters or leaves an instance).
__device__ __forceinline__ void world_ray(const void *rays, int i, WideRay &r) {
        const float4 *p = reinterpret_cast<const float4 *>(rays) + 2 * (size_t)i;
        const float4 a = __ldg(p), b = __ldg(p + 1);
        r.ox = a.x;
        r.oy = a.y;
        r.oz = a.z;
        r.dx = b.x;
        r.dy = b.y;
        r.dz = b.z;
}

// Transform*Point / Transform*Vector of Geometry/Transform.swift:31-65 with a
// 3x4 affine matrix (w = 1, so the division is exact and omitted), each product
// and sum rounded separately in the reference's order.
__device__ __forceinline__ float xf_point(const float4 &row, float x, float y, float z) {
        return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(row.x, x), __fmul_rn(row.y, y)), __fmul_rn(row.z, z)), row.w);
}
__device__ __forceinline__ float xf_vector(const float4 &row, float x, float y, float z) {
        return __fadd_rn(__fadd_rn(__fmul_rn(row.x, x), __fmul_rn(row.y, y)), __fmul_rn(row.z, z));
}

// Two-level persistent traversal (TransformedPrimitive.intersect,
// Primitive/TransformedPrimitive.swift:5-22).  The top-level tree's leaf
// records are instances (v0.w = -(instance + 1)); reaching one pushes, in this
// order, the rest of the current node's children, the rest of its leaf
// records (0x80000000 | base, mask) and a return marker (0xFFFFFFFF), moves the
// ray to object space and descends into the bottom-level root.  Popping the
// marker restores the world ray.  Bottom-level trees are ordinary wide trees
// stored after the top-level nodes in the same arrays.
// The world ray is not kept in registers: it is read again from the ray
// array when a ray enters or leaves an instance.  Bounded to 128-thread
// blocks, 8 resident per SM (64 registers, 12-36 bytes of spills): the
// unbounded build's 99 registers left 4 blocks per SM; 6 blocks (80 registers)
// gave 1.6x its camera-ray rate and 7 another 2 % on the two-level frame
// (1,187 -> 1,162 ms); with the pull counter and the world ray out of
// registers, 8 blocks another 1.3 % (16-spp frame 265.5 -> 262.0 ms).
template <int OUTFMT, bool ANY, int STACK>
__global__ void __launch_bounds__(128, 8) k_wide_instanced(DevScene s, const void *__restrict__ rays,
                                                        const float *__restrict__ tmaxs, int64_t n,
                                                        void *__restrict__ out) {
        extern __shared__ uint2 smem_stack[];
        const unsigned FULL = 0xFFFFFFFFu;
        const uint32_t nr = (uint32_t)ray_count(s, n);
        const unsigned lane = threadIdx.x & 31u;
        const unsigned lt_mask = (1u << lane) - 1u;
        ChunkCursor cc;
        chunk_first(cc, nr);

        uint2 *stack = smem_stack + threadIdx.x;
        const int stride = blockDim.x;
        int ray_i = -1;
        WideRay r;
        float thit = 0.0f, bu = 0.0f, bv = 0.0f;
        int prim = -1, hit_inst = -1, cur_inst = -1, sp = 0;
        uint2 group = make_uint2(0u, 0u);
        uint32_t steps = 0;

        for (;;) {
                unsigned need = __ballot_sync(FULL, ray_i < 0);
                if (__popc(need) < kRefillMin && need != FULL) need = 0u;
                while (need != 0u && cc.cursor < nr) {
                        if (cc.cursor >= cc.end && !chunk_next(cc, s.sched, nr)) break;
                        const int avail = (int)(cc.end - cc.cursor);
                        const int rank = __popc(need & lt_mask);
                        if (ray_i < 0 && rank < avail) {
                                ray_i = (int)(cc.cursor + (uint32_t)rank);
                                const RayIn in = load_ray<kRayDevice>(rays, tmaxs, ray_i);
                                r.ox = in.ox;
                                r.oy = in.oy;
                                r.oz = in.oz;
                                r.dx = in.dx;
                                r.dy = in.dy;
                                r.dz = in.dz;
                                set_ray_dirs(r, s.rcp_max);
                                thit = in.tmax;
                                bu = bv = 0.0f;
                                prim = hit_inst = cur_inst = -1;
                                sp = 0;
                                steps = 0;
                                group = make_uint2(0u, (1u << 24) | (1u << r.oct));
                        }
                        const int npop = __popc(need);
                        cc.cursor += (uint32_t)(npop < avail ? npop : avail);
                        need = __ballot_sync(FULL, ray_i < 0);
                }
                if (__all_sync(FULL, ray_i < 0)) break;
                if (ray_i < 0) continue;

                bool finished = false, fault = false;
                // leaf records to look at in this step: bits pend_mask of pend_bits
                uint32_t pend_base = 0, pend_bits = 0, pend_mask = 0;
                // pop until there is work: a world-ray marker restores the world
                // ray and pops again in the same step
                while ((group.y >> 24) == 0 && sp > 0) {
                        --sp;
                        const uint2 e = stack[sp * stride];
                        if (e.x == 0xFFFFFFFFu) {
                                world_ray(rays, ray_i, r);
                                set_ray_dirs(r, s.rcp_max);
                                cur_inst = -1;
                        } else if (e.x & 0x80000000u) {
                                pend_base = e.x & 0x7FFFFFFFu;
                                pend_mask = e.y;
                                pend_bits = 0xFFFFFFFFu;
                                break;
                        } else {
                                group = e;
                        }
                }
                uint32_t hits = group.y >> 24;
                if (pend_mask == 0 && hits) {
                        const uint32_t key = __ffs(hits) - 1;
                        hits &= hits - 1;
                        const uint32_t im = group.y & 0xFFu;
                        const uint32_t slot = key ^ r.oct;
                        const uint32_t node = group.x + __popc(im & ((1u << slot) - 1u));
                        if (hits) {
                                if (sp >= STACK) {
                                        atomicOr(s.err, kErrStackOverflow);
                                        fault = true;
                                } else {
                                        stack[sp * stride] = make_uint2(group.x, (hits << 24) | im);
                                        ++sp;
                                }
                        }
                        if (++steps > s.wide_count) {
                                atomicOr(s.err, kErrStepCap);
                                fault = true;
                        }
                        if (!fault) {
                                const NodeHits h = open_node(s.wide + 5 * (size_t)node, r, thit);
                                count_lanes(s, 0);
                                group = make_uint2(h.child_base, (h.nodes << 24) | h.imask);
                                pend_mask = h.tris;
                                pend_base = h.tri_base;
                                pend_bits = h.tri_bits;
                        }
                }
                while (!fault && pend_mask) {
                        const uint32_t b = __ffs(pend_mask) - 1;
                        pend_mask &= pend_mask - 1;
                        const uint32_t ti = tri_record(pend_base, pend_bits, b);
                        const float4 a = __ldg(s.tv0 + ti);
                        const int tag = __float_as_int(a.w);
                        if (tag < 0) {
                                // instance record: save the resume state and descend
                                const int inst = -tag - 1;
                                const int need_slots = ((group.y >> 24) ? 1 : 0) + (pend_mask ? 1 : 0) + 1;
                                if (sp + need_slots > STACK || inst >= (int)s.instance_count) {
                                        atomicOr(s.err, inst >= (int)s.instance_count ? kErrBadIndex : kErrStackOverflow);
                                        fault = true;
                                        break;
                                }
                                if (group.y >> 24) {
                                        stack[sp * stride] = group;
                                        ++sp;
                                        group.y = 0u;
                                }
                                if (pend_mask) {
                                        // the records left, as plain offsets from pend_base
                                        uint32_t left = 0;
                                        while (pend_mask) {
                                                const uint32_t q = __ffs(pend_mask) - 1;
                                                pend_mask &= pend_mask - 1;
                                                left |= 1u << __popc(pend_bits & ((1u << q) - 1u));
                                        }
                                        stack[sp * stride] = make_uint2(0x80000000u | pend_base, left);
                                        ++sp;
                                }
                                stack[sp * stride] = make_uint2(0xFFFFFFFFu, 0u);
                                ++sp;
                                const float4 m0 = __ldg(s.instances + 4 * inst), m1 = __ldg(s.instances + 4 * inst + 1),
                                             m2 = __ldg(s.instances + 4 * inst + 2), m3 = __ldg(s.instances + 4 * inst + 3);
                                WideRay w;
                                world_ray(rays, ray_i, w);
                                r.ox = xf_point(m0, w.ox, w.oy, w.oz);
                                r.oy = xf_point(m1, w.ox, w.oy, w.oz);
                                r.oz = xf_point(m2, w.ox, w.oy, w.oz);
                                r.dx = xf_vector(m0, w.dx, w.dy, w.dz);
                                r.dy = xf_vector(m1, w.dx, w.dy, w.dz);
                                r.dz = xf_vector(m2, w.dx, w.dy, w.dz);
                                set_ray_dirs(r, s.rcp_max);
                                cur_inst = inst;
                                group = make_uint2((uint32_t)__float_as_int(m3.x), (1u << 24) | (1u << r.oct));
                                break;
                        }
                        count_lanes(s, 1);
                        const float4 bb = __ldg(s.tv1 + ti);
                        const float4 c = __ldg(s.tv2 + ti);
                        float t, u, v;
                        if (mt_test(r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, a, bb, c, thit, t, u, v)) {
                                thit = t;
                                bu = u;
                                bv = v;
                                prim = tag;
                                hit_inst = cur_inst;
                                if (ANY) {
                                        finished = true;
                                        break;
                                }
                        }
                }
                if (fault || (!finished && pend_mask == 0 && (group.y >> 24) == 0 && sp == 0)) finished = true;
                if (finished) {
                        if (prim < 0) {
                                thit = load_ray<kRayDevice>(rays, tmaxs, ray_i).tmax;
                                bu = 0.0f;
                                bv = 0.0f;
                                hit_inst = -1;
                        }
                        store_hit<OUTFMT>(s, out, ray_i, prim, thit, bu, bv);
                        if (s.inst_out) s.inst_out[ray_i] = hit_inst;
                        ray_i = -1;
                        count_lanes(s, 2);
                }
        }
}

constexpr int kQueueTestsInst = 12, kQueueWaitingInst = 4;

// k_wide_instanced with the triangle queue of k_wide_queued.  The top level's
// leaves hold instances only and the bottom levels' triangles only, so an
// instance is entered where its record is met and triangles are queued; a ray
// whose triangles are still queued waits before it leaves its instance, because
// they are tested with its object-space ray (so top-level nodes are always opened
// with the nearest hit known, and starting over is decided by the instance's own
// boxes).  2M rays through 4096 instances
// 1,359 -> 1,219 us, two-level frame 26.2 -> 24.6 ms.
template <int OUTFMT, bool ANY, int STACK>
__global__ void __launch_bounds__(128, 8) k_wide_instanced_queued(DevScene s, const void *__restrict__ rays,
                                                                  const float *__restrict__ tmaxs, int64_t n,
                                                                  void *__restrict__ out) {
        extern __shared__ __align__(16) uint2 smem_stack[];
        const unsigned FULL = 0xFFFFFFFFu;
        const uint32_t nr = (uint32_t)ray_count(s, n);
        const unsigned lane = threadIdx.x & 31u;
        const unsigned lt_mask = (1u << lane) - 1u;
        ChunkCursor cc;
        chunk_first(cc, nr);

        uint2 *stack = smem_stack + threadIdx.x;
        const int stride = blockDim.x;
        InstQueue &queue = reinterpret_cast<InstQueue *>(smem_stack + STACK * blockDim.x)[threadIdx.x >> 5];
        uint32_t queued = 0;  // pairs in the queue (warp-uniform)
        uint32_t mine = 0;    // queue positions of this lane's ray
        int ray_i = -1;
        WideRay r;
        float thit = 0.0f;
        int prim = -1, cur_inst = -1, sp = 0;
        uint2 group = make_uint2(0u, 0u);
        uint32_t steps = 0;

        for (;;) {
                unsigned need = __ballot_sync(FULL, ray_i < 0);
                if (__popc(need) < kRefillMin && need != FULL) need = 0u;
                while (need != 0u && cc.cursor < nr) {
                        if (cc.cursor >= cc.end && !chunk_next(cc, s.sched, nr)) break;
                        const int avail = (int)(cc.end - cc.cursor);
                        const int rank = __popc(need & lt_mask);
                        if (ray_i < 0 && rank < avail) {
                                ray_i = (int)(cc.cursor + (uint32_t)rank);
                                const RayIn in = load_ray<kRayDevice>(rays, tmaxs, ray_i);
                                r.ox = in.ox;
                                r.oy = in.oy;
                                r.oz = in.oz;
                                r.dx = in.dx;
                                r.dy = in.dy;
                                r.dz = in.dz;
                                set_ray_dirs(r, s.rcp_max);
                                thit = in.tmax;
                                prim = cur_inst = -1;
                                sp = 0;
                                steps = 0;
                                group = make_uint2(0u, (1u << 24) | (1u << r.oct));
                        }
                        const int npop = __popc(need);
                        cc.cursor += (uint32_t)(npop < avail ? npop : avail);
                        need = __ballot_sync(FULL, ray_i < 0);
                }
                if (__all_sync(FULL, ray_i < 0)) break;

                // top-level leaf records to enter: bits pend_mask of pend_bits
                uint32_t pend_base = 0, pend_bits = 0, pend_mask = 0;
                // bottom-level triangles to queue
                uint32_t tris = 0, tri_base = 0, tri_bits = 0;
                bool fault = false, waits = false;
                // pop until there is work: a world-ray marker restores the world
                // ray and pops again in the same step, unless the queue still
                // holds triangles of the instance
                while ((group.y >> 24) == 0 && sp > 0) {
                        const uint2 e = stack[(sp - 1) * stride];
                        if (e.x == 0xFFFFFFFFu) {
                                if (mine != 0u) {
                                        waits = true;
                                        break;
                                }
                                --sp;
                                world_ray(rays, ray_i, r);
                                const uint32_t alone = r.oct & kAlone;
                                set_ray_dirs(r, s.rcp_max);
                                r.oct |= alone;
                                cur_inst = -1;
                        } else {
                                --sp;
                                if (e.x & 0x80000000u) {
                                        pend_base = e.x & 0x7FFFFFFFu;
                                        pend_mask = e.y;
                                        pend_bits = 0xFFFFFFFFu;
                                        break;
                                }
                                group = e;
                        }
                }
                uint32_t hits = group.y >> 24;
                if (pend_mask == 0 && hits) {
                        const uint32_t key = __ffs(hits) - 1;
                        hits &= hits - 1;
                        const uint32_t im = group.y & 0xFFu;
                        const uint32_t slot = (key ^ r.oct) & 7u;
                        const uint32_t node = group.x + __popc(im & ((1u << slot) - 1u));
                        if (hits) {
                                if (sp >= STACK) {
                                        atomicOr(s.err, kErrStackOverflow);
                                        fault = true;
                                } else {
                                        stack[sp * stride] = make_uint2(group.x, (hits << 24) | im);
                                        ++sp;
                                }
                        }
                        if (++steps > s.wide_count) {
                                atomicOr(s.err, kErrStepCap);
                                fault = true;
                        }
                        if (!fault) {
                                const NodeHits h = open_node(s.wide + 5 * (size_t)node, r, thit);
                                count_lanes(s, 0);
                                group = make_uint2(h.child_base, (h.nodes << 24) | h.imask);
                                if (cur_inst < 0) {
                                        // the top level's leaves hold instances,
                                        // the bottom levels' triangles
                                        pend_mask = h.tris;
                                        pend_base = h.tri_base;
                                        pend_bits = h.tri_bits;
                                } else {
                                        tris = h.tris;
                                        tri_base = h.tri_base;
                                        tri_bits = h.tri_bits;
                                }
                        }
                }
                if (pend_mask && !fault) {
                        // instance record: save the resume state and descend
                        const uint32_t b = __ffs(pend_mask) - 1;
                        pend_mask &= pend_mask - 1;
                        const int inst = -__float_as_int(__ldg(&s.tv0[tri_record(pend_base, pend_bits, b)].w)) - 1;
                        const int need_slots = ((group.y >> 24) ? 1 : 0) + (pend_mask ? 1 : 0) + 1;
                        if (sp + need_slots > STACK || (uint32_t)inst >= (uint32_t)s.instance_count) {
                                atomicOr(s.err, (uint32_t)inst >= (uint32_t)s.instance_count ? kErrBadIndex : kErrStackOverflow);
                                fault = true;
                        } else {
                                if (group.y >> 24) {
                                        stack[sp * stride] = group;
                                        ++sp;
                                }
                                if (pend_mask) {
                                        // the records left, as plain offsets from pend_base
                                        uint32_t left = 0;
                                        while (pend_mask) {
                                                const uint32_t q = __ffs(pend_mask) - 1;
                                                pend_mask &= pend_mask - 1;
                                                left |= 1u << __popc(pend_bits & ((1u << q) - 1u));
                                        }
                                        stack[sp * stride] = make_uint2(0x80000000u | pend_base, left);
                                        ++sp;
                                }
                                stack[sp * stride] = make_uint2(0xFFFFFFFFu, 0u);
                                ++sp;
                                const float4 m0 = __ldg(s.instances + 4 * inst), m1 = __ldg(s.instances + 4 * inst + 1),
                                             m2 = __ldg(s.instances + 4 * inst + 2), m3 = __ldg(s.instances + 4 * inst + 3);
                                WideRay w;
                                world_ray(rays, ray_i, w);
                                r.ox = xf_point(m0, w.ox, w.oy, w.oz);
                                r.oy = xf_point(m1, w.ox, w.oy, w.oz);
                                r.oz = xf_point(m2, w.ox, w.oy, w.oz);
                                r.dx = xf_vector(m0, w.dx, w.dy, w.dz);
                                r.dy = xf_vector(m1, w.dx, w.dy, w.dz);
                                r.dz = xf_vector(m2, w.dx, w.dy, w.dz);
                                const uint32_t alone = r.oct & kAlone;
                                set_ray_dirs(r, s.rcp_max);
                                cur_inst = inst;
                                group = make_uint2((uint32_t)__float_as_int(m3.x), (1u << 24) | (1u << r.oct));
                                r.oct |= alone;
                        }
                }
                if (fault) {
                        group.y = 0u;
                        sp = 0;
                        tris = 0u;
                }
                waits = waits || (ray_i >= 0 && (group.y >> 24) == 0u && sp == 0 && (mine | tris) != 0u);
                __syncwarp();
                // queue the triangles; test the queue when it is full enough, or
                // rays wait for it
                unsigned have = __ballot_sync(FULL, tris != 0u);
                while ((have | queued) != 0u) {
                        if (have != 0u) {
                                queued = queue_append(queue, queued, have, tris, tri_base, tri_bits, mine,
                                                      !ANY && (r.oct & kAlone) ? 1 : 7);
                                have = __ballot_sync(FULL, tris != 0u);  // what found no room
                        }
                        if (have == 0u && queued < kQueueTestsInst &&
                            (ANY || !__any_sync(FULL, (r.oct & kAlone) && mine != 0u))) {
                                const unsigned waiting = __ballot_sync(FULL, waits);
                                const unsigned busy = __ballot_sync(FULL, ray_i >= 0 && !waits);
                                if (busy != 0u && __popc(waiting) < kQueueWaitingInst) break;
                        }
                        bool again = false;
                        uint32_t passed = queue_test<GZG_LEAF_MOLLER_TRUMBORE>(s, queue, queued, r, thit) & mine;
                        while (passed) {
                                const uint32_t b = __ffs(passed) - 1;
                                passed &= passed - 1;
                                const float4 h = queue.result[b];
                                if (h.x > thit) continue;  // as mt_test: a NaN limit or distance accepts
                                if (!ANY && !(h.x <= thit && (prim < 0 || box_before(s, r, queue.pair[b].x, h.x))) &&
                                    !(r.oct & kAlone)) {
                                        again = true;
                                        break;
                                }
                                thit = h.x;
                                queue.uv[lane] = make_float2(h.y, h.z);
                                prim = __float_as_int(h.w);
                                queue.inst[lane] = cur_inst;
                                if (ANY) {
                                        tris = 0u;
                                        break;
                                }
                        }
                        __syncwarp();
                        mine = 0u;
                        queued = 0u;
                        if (again) {
                                thit = load_ray<kRayDevice>(rays, tmaxs, ray_i).tmax;
                                world_ray(rays, ray_i, r);
                                set_ray_dirs(r, s.rcp_max);
                                prim = cur_inst = -1;
                                sp = 0;
                                steps = 0;
                                group = make_uint2(0u, (1u << 24) | (1u << r.oct));
                                r.oct |= kAlone;
                                tris = 0u;
                                waits = false;
                        }
                        have = __ballot_sync(FULL, tris != 0u);
                }
                if (ray_i >= 0 && mine == 0u && ((ANY && prim >= 0) || ((group.y >> 24) == 0u && sp == 0))) {
                        if (prim < 0) {
                                thit = load_ray<kRayDevice>(rays, tmaxs, ray_i).tmax;
                        }
                        const float2 uv = prim < 0 ? make_float2(0.0f, 0.0f) : queue.uv[lane];
                        store_hit<OUTFMT>(s, out, ray_i, prim, thit, uv.x, uv.y);
                        if (s.inst_out) s.inst_out[ray_i] = prim < 0 ? -1 : queue.inst[lane];
                        ray_i = -1;
                        group.y = 0u;
                        sp = 0;
                        count_lanes(s, 2);
                }
        }
}

// The reference's slab test (kernel.mojo:171-206), separately rounded.
__device__ __forceinline__ bool ref_aabb(const float4 &lo, const float4 &hi, const float rd[3], const float ord[3],
                                         const bool nm[3], float tmax, float &tnear_out) {
        const float mn[3] = {lo.x, lo.y, lo.z};
        const float mx[3] = {lo.w, hi.x, hi.y};
        float tn[3], tf[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
                const float nr = nm[k] ? mn[k] : mx[k];
                const float fr = nm[k] ? mx[k] : mn[k];
                tn[k] = __fsub_rn(__fmul_rn(nr, rd[k]), ord[k]);
                tf[k] = __fsub_rn(__fmul_rn(fr, rd[k]), ord[k]);
        }
        float tnear = tn[0] > tn[1] ? tn[0] : tn[1];
        tnear = tn[2] > tnear ? tn[2] : tnear;
        tnear = 0.0f > tnear ? 0.0f : tnear;
        float tfar = tf[0] < tf[1] ? tf[0] : tf[1];
        tfar = tf[2] < tfar ? tf[2] : tfar;
        tfar = tmax < tfar ? tmax : tfar;
        tfar = __fmul_rn(tfar, 1.0000003f);
        tnear_out = tnear;
        return tnear <= tfar;
}

template <int RAYFMT, int OUTFMT, bool ANY, int LEAF>
__global__ void __launch_bounds__(128) k_bvh2(DevScene s, const void *__restrict__ rays, const float *__restrict__ tmaxs,
                                              int64_t n, void *__restrict__ out) {
        const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
        n = ray_count(s, n);
        if (i >= n) return;
        const RayIn in = load_ray<RAYFMT>(rays, tmaxs, i);
        const float rd[3] = {__fdiv_rn(1.0f, in.dx), __fdiv_rn(1.0f, in.dy), __fdiv_rn(1.0f, in.dz)};
        const float ord[3] = {__fmul_rn(in.ox, rd[0]), __fmul_rn(in.oy, rd[1]), __fmul_rn(in.oz, rd[2])};
        const bool nm[3] = {rd[0] >= 0.0f, rd[1] >= 0.0f, rd[2] >= 0.0f};
        int stack[64];
        int to_visit = 0;
        int64_t current = 0;
        int hit_index = -1;
        float thit = in.tmax, bu = 0.0f, bv = 0.0f;
        int64_t steps = 0;
        uint32_t n_nodes = 0, n_tris = 0;
        for (;;) {
                if (++steps > s.bvh2_count) {
                        atomicOr(s.err, kErrStepCap);
                        break;
                }
                const float4 *nd = s.bvh2 + 2 * current;
                const float4 hi = __ldg(nd + 1);
                const int count = __float_as_int(hi.w);
                ++n_nodes;
                if (count > 0) {
                        const int off = __float_as_int(hi.z);
                        for (int j = 0; j < count; ++j) {
                                const int k = off + j;
                                const float4 a = __ldg(s.pv0 + k);
                                if (__float_as_int(a.w) == 0) continue;  // id2 == -1 / not a triangle
                                const float4 b = __ldg(s.pv1 + k);
                                const float4 c = __ldg(s.pv2 + k);
                                ++n_tris;
                                float t, u, v;
                                if (leaf_test<LEAF>(in.ox, in.oy, in.oz, in.dx, in.dy, in.dz, a, b, c, thit, t, u, v)) {
                                        thit = t;
                                        bu = u;
                                        bv = v;
                                        hit_index = k;
                                }
                        }
                        if (ANY && hit_index >= 0) break;
                        if (to_visit == 0) break;
                        current = stack[--to_visit];
                } else {
                        const int64_t li = current + 1, ri = __float_as_int(hi.z);
                        const float4 l0 = __ldg(s.bvh2 + 2 * li), l1 = __ldg(s.bvh2 + 2 * li + 1);
                        const float4 r0 = __ldg(s.bvh2 + 2 * ri), r1 = __ldg(s.bvh2 + 2 * ri + 1);
                        n_nodes += 2;
                        float lt, rt;
                        const bool lh = ref_aabb(l0, l1, rd, ord, nm, thit, lt);
                        const bool rh = ref_aabb(r0, r1, rd, ord, nm, thit, rt);
                        if (lh && rh) {
                                if (to_visit >= 64) {
                                        atomicOr(s.err, kErrStackOverflow);
                                        break;
                                }
                                if (lt <= rt) {
                                        current = li;
                                        stack[to_visit] = (int)ri;
                                } else {
                                        current = ri;
                                        stack[to_visit] = (int)li;
                                }
                                ++to_visit;
                        } else if (lh) {
                                current = li;
                        } else if (rh) {
                                current = ri;
                        } else {
                                if (to_visit == 0) break;
                                current = stack[--to_visit];
                        }
                }
        }
        if (hit_index < 0) {
                thit = in.tmax;
                bu = 0.0f;
                bv = 0.0f;
        }
        store_hit<OUTFMT>(s, out, i, hit_index, thit, bu, bv);
        add_counters(s, n_nodes, n_tris, 1u);
}

__global__ void k_hits_to_isect(DevScene s, const float4 *__restrict__ hits, int64_t n, void *__restrict__ out) {
        const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
        if (i >= n) return;
        const float4 h = __ldcs(hits + i);
        const int prim = __float_as_int(h.w);
        if (prim >= (int)s.prim_count) {
                atomicOr(s.err, kErrBadIndex);
                store_hit<kOutIntersection>(s, out, i, -1, h.x, 0.0f, 0.0f);
                return;
        }
        store_hit<kOutIntersection>(s, out, i, prim, h.x, h.y, h.z);
}

// ------------------------------------------------------------ launchers

namespace {

using TraceKernel = void (*)(DevScene, const void *, const float *, int64_t, void *);

// Launches a wide-node kernel with a STACK-deep shared-memory stack.  The
// persistent kernel gets one wave of resident blocks (SM count x blocks per
// SM, from the occupancy calculator unless blocks_per_sm is given), capped at
// the blocks the ray count needs; the one-ray-per-thread kernel one thread per
// ray.
cudaError_t launch_wide_kernel(TraceKernel k, int stack, bool persistent, bool queued, const LaunchParams &p, const DevScene &s,
                               const void *rays, const float *tmax, int64_t n, void *out, cudaStream_t st) {
        // The persistent kernel is compiled for blocks of at most 128 threads
        // (measured faster for any-hit queries than a 256-thread bound).
        const int block = (p.block_size == 64 || (p.block_size == 256 && !persistent)) ? p.block_size : 128;
        const int blocks_per_sm = p.blocks_per_sm;
        const size_t smem = (size_t)stack * block * sizeof(uint2) + (queued ? (size_t)(block / 32) * (s.instances ? sizeof(InstQueue) : sizeof(TriQueue)) : 0);
        if (smem > 48 * 1024) {
                cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
                if (e != cudaSuccess) return e;
        }
        // L1 / shared split: explicit percent, or the driver's choice (-1).
        {
                const int carve = p.l1_carveout > 0 ? (p.l1_carveout > 100 ? 100 : p.l1_carveout) : -1;
                cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, carve);
                if (e != cudaSuccess) return e;
        }
        int64_t grid = (n + block - 1) / block;
        if (persistent) {
                int dev = 0, sms = 0, per_sm = blocks_per_sm;
                cudaGetDevice(&dev);
                cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
                if (per_sm <= 0) {
                        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, block, smem);
                        if (e != cudaSuccess) return e;
                        if (per_sm <= 0) per_sm = 1;
                }
                const int64_t wave = (int64_t)sms * per_sm;
                if (wave < grid) grid = wave;
                // The pull counter pays off once some warp has a second chunk
                // (with one chunk per warp both schedules are the same); it
                // starts every launch at zero.
                if (s.sched != nullptr) {
                        if (s.n_dev == nullptr && n <= grid * block) {
                                DevScene ws = s;
                                ws.sched = nullptr;
                                k<<<(unsigned)grid, block, smem, st>>>(ws, rays, tmax, n, out);
                                return cudaGetLastError();
                        }
                        const cudaError_t e = p.sched_zeroed ? cudaSuccess : cudaMemsetAsync(s.sched, 0, sizeof(uint32_t), st);
                        if (e != cudaSuccess) return e;
                }
        }
        k<<<(unsigned)grid, block, smem, st>>>(s, rays, tmax, n, out);
        return cudaGetLastError();
}

// Whether a launch of n rays over a wide tree of `nodes` nodes tests triangles
// lane by lane (k_wide_persistent, k_wide_instanced) instead of through the
// warp's queue.  Where many rays meet each triangle, neighbouring rays meet it
// in the same step and the lanes are full as they are: pinhole rays are slower
// with the queue from about 150 rays a node on, by 2 to 3 % at 250 to 500 (4.2M
// rays on 20,480 triangles 525 -> 547 us, on 81,920 618 -> 625) and by 10 % above
// 2,000, and faster below (0.5M rays on 81,920 triangles 113 -> 107, 8.4M on
// 1,310,720 894 -> 876).  Incoherent rays are 5 to 12 % faster with it at every
// size, but a launch does not know its rays: the line lies where pinhole rays
// would lose more than 3 %.  A launch that reads its ray count on the device (a
// renderer's queues) goes by its capacity.
bool lane_tests(int64_t n, uint32_t nodes) { return n > 400 * (int64_t)nodes; }

template <int RAYFMT, int OUTFMT, bool ANY, int STACK, int LEAF>
cudaError_t launch_wide_stack(const DevScene &s, const LaunchParams &p, const void *rays, const float *tmax, int64_t n,
                              void *out, cudaStream_t st) {
        if constexpr (OUTFMT != kOutShadow)  // (launch_trace takes shadow queues in the persistent kernels only)
                if (p.traversal != GZG_TRAVERSAL_WIDE)
                        return launch_wide_kernel(k_wide<RAYFMT, OUTFMT, ANY, STACK, LEAF>, STACK, false, false, p, s, rays, tmax,
                                                  n, out, st);
        // (the caller may ask for more entries than the tree needs, so every size has both)
        if (lane_tests(n, s.wide_nodes))
                return launch_wide_kernel(k_wide_persistent<RAYFMT, OUTFMT, ANY, STACK, LEAF>, STACK, true, false, p, s, rays,
                                          tmax, n, out, st);
        return launch_wide_kernel(k_wide_queued<RAYFMT, OUTFMT, ANY, STACK, LEAF>, STACK, true, true, p, s, rays, tmax, n, out, st);
}

template <int RAYFMT, int OUTFMT, bool ANY, int LEAF>
cudaError_t launch_wide_depth(const DevScene &s, const LaunchParams &p, const void *rays, const float *tmax, int64_t n,
                              void *out, cudaStream_t st) {
        // A ray pushes at most one group (the rest of a node's interior hits)
        // per level whose nodes have interior children, so the stack holds at
        // most depth - 1 groups; a requested depth below that is raised so no
        // ray can overflow it (an overflow would set kErrStackOverflow).
        const int need = p.wide_depth > 2 ? p.wide_depth - 1 : 1;
        const int want = p.stack_depth > need ? p.stack_depth : need;
        if (want <= 8) return launch_wide_stack<RAYFMT, OUTFMT, ANY, 8, LEAF>(s, p, rays, tmax, n, out, st);
        if (want <= 16) return launch_wide_stack<RAYFMT, OUTFMT, ANY, 16, LEAF>(s, p, rays, tmax, n, out, st);
        if (want <= 32) return launch_wide_stack<RAYFMT, OUTFMT, ANY, 32, LEAF>(s, p, rays, tmax, n, out, st);
        return launch_wide_stack<RAYFMT, OUTFMT, ANY, 64, LEAF>(s, p, rays, tmax, n, out, st);
}

template <int STACK>
cudaError_t launch_instanced_stack(const DevScene &s, const LaunchParams &p, int out_fmt, const void *rays, int64_t n,
                                   void *out, cudaStream_t st) {
        const bool lanes = lane_tests(n, s.wide_nodes);
        const TraceKernel k =
            out_fmt == kOutHit    ? (lanes ? k_wide_instanced<kOutHit, false, STACK> : k_wide_instanced_queued<kOutHit, false, STACK>)
            : out_fmt == kOutShadow ? (lanes ? k_wide_instanced<kOutShadow, true, STACK> : k_wide_instanced_queued<kOutShadow, true, STACK>)
                                    : (lanes ? k_wide_instanced<kOutAnyPrim, true, STACK> : k_wide_instanced_queued<kOutAnyPrim, true, STACK>);
        return launch_wide_kernel(k, STACK, true, !lanes, p, s, rays, nullptr, n, out, st);
}

template <int RAYFMT, int OUTFMT, bool ANY>
cudaError_t launch_fmt(const DevScene &s, const LaunchParams &p, const void *rays, const float *tmax, int64_t n,
                       void *out, cudaStream_t st) {
        const int block = 128;
        if (p.traversal == GZG_TRAVERSAL_BVH2) {
                if (!s.bvh2) return cudaErrorInvalidValue;  // a device-built scene has no reference BVH2
                const int64_t grid = (n + block - 1) / block;
                if (p.leaf_test == GZG_LEAF_WATERTIGHT)
                        k_bvh2<RAYFMT, OUTFMT, ANY, GZG_LEAF_WATERTIGHT><<<(unsigned)grid, block, 0, st>>>(s, rays, tmax, n, out);
                else
                        k_bvh2<RAYFMT, OUTFMT, ANY, GZG_LEAF_MOLLER_TRUMBORE><<<(unsigned)grid, block, 0, st>>>(s, rays, tmax, n, out);
                return cudaGetLastError();
        }
        if (p.leaf_test == GZG_LEAF_WATERTIGHT)
                return launch_wide_depth<RAYFMT, OUTFMT, ANY, GZG_LEAF_WATERTIGHT>(s, p, rays, tmax, n, out, st);
        return launch_wide_depth<RAYFMT, OUTFMT, ANY, GZG_LEAF_MOLLER_TRUMBORE>(s, p, rays, tmax, n, out, st);
}

}  // namespace

cudaError_t launch_trace(const DevScene &scene, const LaunchParams &p, int ray_fmt, int out_fmt, const void *rays,
                         const float *tmax, int64_t n, void *out, cudaStream_t st) {
        if (n <= 0) return cudaSuccess;
        if (n > kMaxLaunchRays) {
                // consecutive launches over slices of the arrays
                if (p.n_dev) return cudaErrorInvalidValue;
                const size_t ray_bytes = ray_fmt == kRayDevice ? 32 : 24;
                const size_t out_bytes = out_fmt == kOutHit ? 16 : out_fmt == kOutIntersection ? 48 : out_fmt == kOutAnyPrim ? 4 : 1;
                LaunchParams q = p;
                for (int64_t off = 0; off < n; off += kMaxLaunchRays) {
                        const int64_t m = n - off < kMaxLaunchRays ? n - off : kMaxLaunchRays;
                        q.inst_out = p.inst_out ? p.inst_out + off : nullptr;
                        const cudaError_t e = launch_trace(scene, q, ray_fmt, out_fmt,
                                                           reinterpret_cast<const char *>(rays) + off * ray_bytes,
                                                           tmax ? tmax + off : nullptr, m,
                                                           reinterpret_cast<char *>(out) + off * out_bytes, st);
                        if (e != cudaSuccess) return e;
                }
                return cudaSuccess;
        }
        DevScene s = scene;
        s.counters = p.counters;
        s.n_dev = p.n_dev;
        s.inst_out = p.inst_out;
        s.sched = p.sched;
        if (s.instances) {
                // two-level scenes: persistent wide traversal only
                if (ray_fmt != kRayDevice || (out_fmt != kOutHit && out_fmt != kOutAnyPrim && out_fmt != kOutShadow))
                        return cudaErrorNotSupported;
                const int need = p.wide_depth > 1 ? p.wide_depth : 1;
                const int want = p.stack_depth > need ? p.stack_depth : need;
                LaunchParams q = p;
                q.traversal = GZG_TRAVERSAL_WIDE;
                if (want <= 16) return launch_instanced_stack<16>(s, q, out_fmt, rays, n, out, st);
                if (want <= 32) return launch_instanced_stack<32>(s, q, out_fmt, rays, n, out, st);
                return launch_instanced_stack<64>(s, q, out_fmt, rays, n, out, st);
        }
        if (out_fmt == kOutShadow) {
                // a renderer's shadow queue: one traversal, one leaf test
                if (ray_fmt != kRayDevice || p.traversal != GZG_TRAVERSAL_WIDE) return cudaErrorNotSupported;
                return launch_wide_depth<kRayDevice, kOutShadow, true, GZG_LEAF_MOLLER_TRUMBORE>(s, p, rays, tmax, n, out, st);
        }
        if (ray_fmt == kRayDevice) {
                switch (out_fmt) {
                case kOutHit: return launch_fmt<kRayDevice, kOutHit, false>(s, p, rays, tmax, n, out, st);
                case kOutIntersection: return launch_fmt<kRayDevice, kOutIntersection, false>(s, p, rays, tmax, n, out, st);
                case kOutAnyPrim: return launch_fmt<kRayDevice, kOutAnyPrim, true>(s, p, rays, tmax, n, out, st);
                default: return launch_fmt<kRayDevice, kOutOccluded, true>(s, p, rays, tmax, n, out, st);
                }
        }
        switch (out_fmt) {
        case kOutHit: return launch_fmt<kRayReference, kOutHit, false>(s, p, rays, tmax, n, out, st);
        case kOutIntersection: return launch_fmt<kRayReference, kOutIntersection, false>(s, p, rays, tmax, n, out, st);
        case kOutAnyPrim: return launch_fmt<kRayReference, kOutAnyPrim, true>(s, p, rays, tmax, n, out, st);
        default: return launch_fmt<kRayReference, kOutOccluded, true>(s, p, rays, tmax, n, out, st);
        }
}

cudaError_t launch_shadow(const DevScene &scene, const LaunchParams &p, const void *rays, int64_t n,
                          const ShadowSink &sink, cudaStream_t st) {
        if (n > kMaxLaunchRays) return cudaErrorInvalidValue;
        DevScene s = scene;
        s.shadow_path = sink.path;
        s.shadow_contrib = sink.contrib;
        s.shadow_radiance = sink.radiance;
        return launch_trace(s, p, kRayDevice, kOutShadow, rays, nullptr, n, nullptr, st);
}

cudaError_t launch_hits_to_isect(const DevScene &s, const void *hits, int64_t n, void *out, cudaStream_t st) {
        if (n <= 0) return cudaSuccess;
        const int block = 256;
        k_hits_to_isect<<<(unsigned)((n + block - 1) / block), block, 0, st>>>(s, reinterpret_cast<const float4 *>(hits), n, out);
        return cudaGetLastError();
}

}  // namespace gzg
