// force_device.cuh -- the Barnes-Hut force walk of one warp group, shared
// by the single-system kernel (k_force.cu) and the batched one (k_batch.cu).
// (calculate_force_local, kernels/calculate_forces.cl:4-185.)
//
// One warp owns 32 consecutive bodies of the in-order sort (spatial
// neighbours) and keeps one shared stack of cells still to open.  A cell is
// accepted when EVERY body of the group accepts it (d^2 >= dq[level], the
// reference's work_group_all at :121, over a real 32-lane warp), otherwise it
// is pushed.  The lanes change roles between finding interactions and summing
// them:
//
//   classify  a round pops up to kBatch = 8 cells; lane L holds child slot
//             L%8 of popped cells L/8 and 4 + L/8 (coalesced 128-byte lines).
//             Each lane decides its two children against the group's
//             bounding box: the distance to the box, formed with the same
//             operations as a body's d^2, is a lower bound of every body's d^2
//             also after rounding (rounding is monotonic), so box d^2 >= dq
//             accepts exactly; the d^2 of one of two sample bodies below dq
//             rejects exactly.  What is left (one cell in seven) is listed
//             and voted on by all 32 bodies, eight cells at a time.
//   sum       accepted cells and child bodies wait in lists; eight of them
//             make a tile.  Lane L sums the pair of sources L%4 over the four
//             bodies 4 (L/4) .. + 3, whose positions and sums stay in its
//             registers for the whole walk: one shared-memory load per operand
//             for 8 x 32 interactions, no vote, no branch, and two
//             interactions per FP32 instruction (f32x2).  At the end the four
//             lanes of a body add their sums in a fixed tree.
//
// The children of the next round's cells are on their way to shared memory
// (cp.async) while a round is summed.
//
// What bounds it: the FP32 arithmetic with its register reads.  A packed
// instruction of three different register pairs takes three issue cycles, of
// two pairs two, so the 30-operation quadrupole term costs about 38 cycles a
// warp interaction (32 bodies) in every form tried: two sources x four
// bodies packed 38.1, one source x eight bodies scalar 37.2, lane = body with
// broadcast sources 43 (that kernel's vote, branch and loads came on top:
// 64 in all).  Measured on a GB300, force kernel, lane = body walk against
// this one: 4,194,304 flat, quadrupoles, compensated 13.62 -> 11.78 ms;
// 262,144 ball, monopoles 0.449 -> 0.367 ms; 100,003, quadrupoles 0.205 ->
// 0.161 ms; 6,007 0.117 -> 0.067 ms.  At 1M: 3.18e9 -> 1.93e9 warp
// instructions, FMA pipe 52 -> 60 % busy.  Sixteen warps an SM (128
// registers); 20 (96 registers) and 14 are equal within 2 %.
//
// Softened gravity F = m rsqrt(d^2)^3 (MUFU rsqrt), d^2 = |d|^2 + eps^2 as
// FMAs; accepted cells optionally add their traceless quadrupole.
//
// Stack bound: kBatch cells are popped only while the stack holds at most `room`
// entries, so a batch leaves at most room - 8 + 8*kBatch entries and 7 more that
// wait for their vote (= room - 1 + 8*kBatch together); beyond that the walk pops
// one cell at a time (depth first) and votes at once, which adds at most 7 pending
// siblings per level of the tree and one more.  So room = kStack - 8*kBatch - 7 *
// levels - 1: 255 for a tree of 63 levels, the most there are, and 549 for one of
// 21.  Entries pack (level << 26) | node.
//
// The integrator writes the next position buffer, so every force of the step
// sees step-start positions (the reference integrates in place while other
// work-items still read positions, :159-180).
#pragma once
#include "integrate.cuh"
#include "packed.cuh"

namespace nbgb {

constexpr int kForceWarps = 2;
constexpr int kForceThreads = kForceWarps * 32;
constexpr int kStack = 768;
constexpr int kBatch = 8;
static_assert(kBatch == 8, "lane L holds child slot L%8 of popped cells L/8 and 4 + L/8");
// A single pop costs a whole round: with batches up to 128 entries only, the walks
// of long stacks (the reference's opening rule, which opens every cell within
// sqrt(eps)) took longer than the walk with a vote a cell did (ms, that walk / up
// to 128 / now: cusps, 6,869 bodies 0.51 / 0.75 / 0.32, 60,000 6.01 / 12.4 / 3.49; 4M in
// the reference's boxes, theta 1.5, 4.88 / 6.20 / 5.08).
__device__ __forceinline__ int stack_room(int levels) {
    return kStack - 8 * kBatch - 7 * min(levels, kMaxDepth - 1) - 1;
}
constexpr int kNodeBits = 26;
constexpr int kNodeMask = (1 << kNodeBits) - 1;

// TwoSum (Knuth): hi + t = s + e exactly; e goes to the low word.
__device__ __forceinline__ void two_sum_add(float &hi, float &lo, float t) {
    const float s = __fadd_rn(hi, t);
    const float bp = __fsub_rn(s, hi);
    const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(t, bp));
    hi = s;
    lo = __fadd_rn(lo, e);
}

// Shared-memory lists of one warp.  Sources lie in pairs (entry k is half k%2
// of pair k/2): the operands of the packed instructions, loaded as they are.
constexpr int kTile8 = 8;                  // sources per tile: a pair for each of four lanes
constexpr int kListU = 8 * kBatch + kTile8;      // 64 new entries a round and at most 7 carried over
constexpr int kListC = 8 * kBatch + 2 * kTile8;  // the same, and at most 7 voted in from earlier rounds
template <bool kQuad>
struct WarpLists {
    int stack[kStack];  // packed cell entries still to open
    // bodies, and accepted cells without quadrupoles: {x0,x1,y0,y1}, {z0,z1,-m0,-m1}
    float4 src[2][kListC / 2];
    // accepted cells: the same, then their quadrupoles {xx0,xx1,yy0,yy1}, {zz,xy}, {xz,yz}
    float4 cell[5][kQuad ? kListC / 2 : 1];
    float4 upm[kListU];  // cells the group still has to vote on {x,y,z,m}
    int2 ument[kListU];  // {packed entry, place of the cell in its parent's packed line}
    // the children of the popped cells, on their way from memory (two per lane)
    float4 in_pm[64], in_qa[kQuad ? 64 : 1];
    float2 in_qb[kQuad ? 64 : 1];
    int in_ch[64];
    // values of the whole walk that the sums leave no registers for: the
    // group's box and two sample bodies {lo, hi x | hi yz, s0 xy | s0 z, s1},
    // and each body's running TwoSum
    float4 box[3];
    float run[6][32];
};

template <int kBytes>
__device__ __forceinline__ void cp_async(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(kBytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// entry k's place is float 4 (k/2) + k%2 of the first row; the others follow
// every kListC / 2 float4
__device__ __forceinline__ void put_source(float *at, const float4 q) {
    at[0] = q.x;
    at[2] = q.y;
    at[2 * kListC] = q.z;
    at[2 * kListC + 2] = -q.w;
}
__device__ __forceinline__ void put_moments(float *at, const float4 Q, const float2 R) {
    at[4 * kListC] = Q.x;
    at[4 * kListC + 2] = Q.y;
    at[6 * kListC] = Q.z;
    at[6 * kListC + 2] = Q.w;
    at[8 * kListC] = R.x;
    at[8 * kListC + 2] = R.y;
}

// A lane's four bodies: minus the positions, each twice, and minus the sums
// over the even and over the odd sources.  Packed FP32 instructions (add / mul /
// fma.rn.f32x2) round each half as the scalar ones do.
struct LaneBodies {
    float2 nx[4], ny[4], nz[4];
    float2 ax[4], ay[4], az[4];
};

// One tile of monopole sources: the lane's pair over its four bodies.
template <bool kEpsZero>
__device__ __forceinline__ void sum_tile(const float4 xy, const float4 zm, float2 eps2, LaneBodies &B) {
    const float2 qx = lo2(xy), qy = hi2(xy), qz = lo2(zm), m = hi2(zm);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 dx = __fadd2_rn(qx, B.nx[k]), dy = __fadd2_rn(qy, B.ny[k]), dz = __fadd2_rn(qz, B.nz[k]);
        const float2 d2 = pair_dist2(dx, dy, dz, eps2);
        const float2 r = make_float2(rsqrt_fast(d2.x), rsqrt_fast(d2.y));
        float2 F = __fmul2_rn(m, __fmul2_rn(r, __fmul2_rn(r, r)));
        if constexpr (kEpsZero) {
            F.x = d2.x > 0.0f ? F.x : 0.0f;
            F.y = d2.y > 0.0f ? F.y : 0.0f;
        }
        B.ax[k] = __ffma2_rn(dx, F, B.ax[k]);
        B.ay[k] = __ffma2_rn(dy, F, B.ay[k]);
        B.az[k] = __ffma2_rn(dz, F, B.az[k]);
    }
}

// One tile of cells with their quadrupoles Q (xx yy zz xy | xz yz):
//   m d / r^3 + 2.5 (d.Q.d) d / r^7 - Q d / r^5
//   = (d (m d^2 + 2.5 (d.Q.d) / r^2) - Q d) / r^5, with r^-2 = d^2.
// The sources carry -m and the sums are kept with the opposite sign, so that
// no packed operand needs a sign.
__device__ __forceinline__ void sum_tile_quad(const float4 (&v)[5], float2 eps2, LaneBodies &B) {
    const float2 qx = lo2(v[0]), qy = hi2(v[0]), qz = lo2(v[1]), m = hi2(v[1]);
    const float2 xx = lo2(v[2]), yy = hi2(v[2]), zz = lo2(v[3]), xy = hi2(v[3]), xz = lo2(v[4]), yz = hi2(v[4]);
    const float2 c = dup(-2.5f);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 dx = __fadd2_rn(qx, B.nx[k]), dy = __fadd2_rn(qy, B.ny[k]), dz = __fadd2_rn(qz, B.nz[k]);
        const float2 d2 = pair_dist2(dx, dy, dz, eps2);
        const float2 r = make_float2(rsqrt_fast(d2.x), rsqrt_fast(d2.y));
        const float2 r2 = __fmul2_rn(r, r);
        const float2 ux = __ffma2_rn(xz, dz, __ffma2_rn(xy, dy, __fmul2_rn(xx, dx)));
        const float2 uy = __ffma2_rn(yz, dz, __ffma2_rn(yy, dy, __fmul2_rn(xy, dx)));
        const float2 uz = __ffma2_rn(zz, dz, __ffma2_rn(yz, dy, __fmul2_rn(xz, dx)));
        const float2 sq = __ffma2_rn(dz, uz, __ffma2_rn(dy, uy, __fmul2_rn(dx, ux)));
        const float2 r5 = __fmul2_rn(r, __fmul2_rn(r2, r2));
        const float2 t = __ffma2_rn(__fmul2_rn(c, sq), r2, __fmul2_rn(m, d2));
        B.ax[k] = __ffma2_rn(__ffma2_rn(dx, t, ux), r5, B.ax[k]);
        B.ay[k] = __ffma2_rn(__ffma2_rn(dy, t, uy), r5, B.ay[k]);
        B.az[k] = __ffma2_rn(__ffma2_rn(dz, t, uz), r5, B.az[k]);
    }
}

// Sum over the four lanes and two halves of each body, in a fixed tree: lane
// L gets the sum of body L (body k of a lane is body 4 (L/4) + k).
__device__ __forceinline__ float tile_reduce(const float2 (&a)[4], int lane) {
    float u[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float s0 = a[k].x + a[k].y, s1 = a[k + 2].x + a[k + 2].y;
        const float give = (lane & 2) ? s0 : s1, keep = (lane & 2) ? s1 : s0;
        u[k] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
    }
    const float give = (lane & 1) ? u[0] : u[1], keep = (lane & 1) ? u[1] : u[0];
    return keep + __shfl_xor_sync(0xffffffffu, give, 1);
}

// Entry k of a list of cnt is a lane's first half: halves beyond the list
// take the list's last source (loaded in the first half of the last pair when
// cnt is odd) without its mass and moments, so that they add exactly nothing.
template <int kVec>
__device__ __forceinline__ void drop_beyond(float4 (&v)[kVec], int k, int cnt) {
    if (k + 1 >= cnt) {
        if (cnt & 1) {  // the last pair's second half is empty
            v[0].y = v[0].x;
            v[0].w = v[0].z;
            v[1].y = v[1].x;
        }
        v[1].w = 0.0f;
        for (int i = 2; i < kVec; ++i) v[i].y = v[i].w = 0.0f;
        if (k >= cnt) {
            v[1].z = 0.0f;
            for (int i = 2; i < kVec; ++i) v[i].x = v[i].z = 0.0f;
        }
    }
}

__device__ __forceinline__ float dist2(const float4 q, float x, float y, float z, float eps2) {
    const float dx = q.x - x, dy = q.y - y, dz = q.z - z;
    return fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, eps2)));
}

// max(a, b, 0), not a number where a or b is not: a cell without mass has no
// centre, and no distance accepts it
__device__ __forceinline__ float outside(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, 0f00000000;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

__device__ __forceinline__ float warp_min(float v) { return key2f(__reduce_min_sync(0xffffffffu, f2key(v))); }
__device__ __forceinline__ float warp_max(float v) { return key2f(__reduce_max_sync(0xffffffffu, f2key(v))); }

// Compensated sums: the lanes' sums go into the running TwoSum after at most
// kFlushTiles + 16 tiles, i.e. after at most 40 terms in a row per lane and
// half, and the three additions across them.
constexpr int kFlushTiles = 24;

// Walk of warp group g of system s (dq: its 64 thresholds, room: its tree's
// stack_room), with the fused integrator.  All 32 lanes call it together.
template <int kMethod, bool kComp, bool kEpsZero, bool kQuad>
__device__ __forceinline__ void force_group(const DevSim &s, const StepParams &p, const float *dq, int room, int g,
                                            int lane, WarpLists<kQuad> &ws) {
    Ctrl *ctrl = s.ctrl;
    const int n = s.n, root = n + s.cap;
    const float eps2 = __fmul_rn(p.eps, p.eps);
    const int cidx = lane >> 3, slot = lane & 7, col = lane & 3;
    const unsigned below = (1u << lane) - 1u;
    const int sidx = g * 32 + lane;
    const bool valid = sidx < n;
    // a lane past the end takes lane 0's body: its votes copy lane 0's,
    // so the warp vote needs no validity test; its result is discarded
    LaneBodies B;
    {
        const float4 P = s.body_cur[s.sorted[valid ? sidx : g * 32]];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int l = (lane & 28) | k;
            B.nx[k] = dup(-__shfl_sync(0xffffffffu, P.x, l));
            B.ny[k] = dup(-__shfl_sync(0xffffffffu, P.y, l));
            B.nz[k] = dup(-__shfl_sync(0xffffffffu, P.z, l));
            B.ax[k] = B.ay[k] = B.az[k] = make_float2(0.0f, 0.0f);
        }
        const float lox = warp_min(P.x), loy = warp_min(P.y), loz = warp_min(P.z);
        const float hix = warp_max(P.x), hiy = warp_max(P.y), hiz = warp_max(P.z);
        if (lane == 0) ws.box[0] = make_float4(lox, loy, loz, hix);
        if (lane == 8) {
            ws.box[1] = make_float4(hiy, hiz, P.x, P.y);
            ws.box[2].x = P.z;
        }
        if (lane == 24) {
            ws.box[2].y = P.x;
            ws.box[2].z = P.y;
            ws.box[2].w = P.z;
        }
        if constexpr (kComp)
            for (int k = 0; k < 6; ++k) ws.run[k][lane] = 0.0f;
    }
    const float2 eps2p = dup(eps2);
    unsigned n_body = 0, n_open = 0;
    int sp = 0, nb = 0, nc = 0, nu = 0, tiles_b = 0, tiles_c = 0, flushed = 0;
    int np = 1;                // cells popped for the next round
    int e[2] = {root, 0};      // the popped cells whose child slot this lane holds; level 0
    // the loads of child slot L%8 of popped cells L/8 and 4 + L/8: independent
    // of one another (the packed line of a cell is whole; empty slots hold
    // zeros or stale values)
    auto fetch = [&]() {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (cidx + 4 * h < np) {
                const int ref = ((e[h] & kNodeMask) - n) * 8 + slot, at = lane + 32 * h;
                cp_async<4>(&ws.in_ch[at], &s.wchild[ref]);
                cp_async<16>(&ws.in_pm[at], &s.wpm[ref]);
                if constexpr (kQuad) {
                    cp_async<16>(&ws.in_qa[at], &s.wqa[ref]);
                    cp_async<8>(&ws.in_qb[at], &s.wqb[ref]);
                }
            }
        }
    };
    fetch();
    n_open = 1;
    __syncwarp();
    while (true) {
        cp_async_wait();
        const float4 b0 = ws.box[0], b1 = ws.box[1], b2 = ws.box[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int at = lane + 32 * h;
            int ch = -1;
            float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (cidx + 4 * h < np) {
                ch = ws.in_ch[at];
                q = ws.in_pm[at];
            }
            const int lv = (int)((unsigned)e[h] >> kNodeBits);
            const float thr = dq[lv];
            const bool isb = ch >= 0 && ch < n, isc = ch >= n;
            const float ex = outside(b0.x - q.x, q.x - b0.w);
            const float ey = outside(b0.y - q.y, q.y - b1.x);
            const float ez = outside(b0.z - q.z, q.z - b1.y);
            const float lower = fmaf(ez, ez, fmaf(ey, ey, fmaf(ex, ex, eps2)));
            const bool acc = isc && lower >= thr;
            const bool rej = isc && !acc && (dist2(q, b1.z, b1.w, b2.x, eps2) < thr || dist2(q, b2.y, b2.z, b2.w, eps2) < thr);
            const bool uns = isc && !acc && !rej;
            const unsigned mr = __ballot_sync(0xffffffffu, rej), mu = __ballot_sync(0xffffffffu, uns);
            const unsigned mb = __ballot_sync(0xffffffffu, isb), ma = __ballot_sync(0xffffffffu, acc);
            const int entry = ((lv + 1) << kNodeBits) | ch;
            if (isb || acc) {
                const bool to_cells = kQuad && acc;
                const int k = to_cells ? nc + __popc(ma & below) : nb + __popc((kQuad ? mb : mb | ma) & below);
                float *at4 = (to_cells ? &ws.cell[0][0].x : &ws.src[0][0].x) + ((k >> 1) * 4 + (k & 1));
                put_source(at4, q);
                if (to_cells) put_moments(at4, ws.in_qa[at], ws.in_qb[at]);
            }
            if constexpr (kQuad) {
                nc += __popc(ma);
                nb += __popc(mb);
            } else {
                nb += __popc(mb | ma);
                n_body += __popc(mb);
            }
            if (uns) {
                const int k = nu + __popc(mu & below);
                ws.upm[k] = q;
                ws.ument[k] = make_int2(entry, ((e[h] & kNodeMask) - n) * 8 + slot);
            }
            nu += __popc(mu);
            if (rej) {
                const int k = sp + __popc(mr & below);
                if (k < kStack) ws.stack[k] = entry;
                else set_status(ctrl, kStDepth, kStack);  // outside the stack bound: never overrun shared memory
            }
            sp = min(sp + __popc(mr), kStack);
        }
        __syncwarp();
        // the undecided cells: every body of the group votes, eight cells at a
        // time (a lane tests cells L%4 and 4 + L%4 against its four bodies)
        while (nu >= kTile8 || (nu > 0 && (sp == 0 || sp > room))) {
            const int cnt = min(nu, kTile8);
            nu -= cnt;
            const int i0 = nu + min(col, cnt - 1), i1 = nu + min(col + 4, cnt - 1);
            const float4 q0 = ws.upm[i0], q1 = ws.upm[i1];
            const float t0 = dq[((unsigned)ws.ument[i0].x >> kNodeBits) - 1];
            const float t1 = dq[((unsigned)ws.ument[i1].x >> kNodeBits) - 1];
            const float2 qx = make_float2(q0.x, q1.x), qy = make_float2(q0.y, q1.y), qz = make_float2(q0.z, q1.z);
            bool ok0 = true, ok1 = true;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 d2 = pair_dist2(__fadd2_rn(qx, B.nx[k]), __fadd2_rn(qy, B.ny[k]),
                                             __fadd2_rn(qz, B.nz[k]), eps2p);
                ok0 = ok0 && d2.x >= t0;
                ok1 = ok1 && d2.y >= t1;
            }
            unsigned m0 = __ballot_sync(0xffffffffu, ok0), m1 = __ballot_sync(0xffffffffu, ok1);
            m0 &= m0 >> 16;
            m1 &= m1 >> 16;
            m0 &= m0 >> 8;
            m1 &= m1 >> 8;
            const unsigned m = (m0 & (m0 >> 4) & 15u) | ((m1 & (m1 >> 4) & 15u) << 4);
            const unsigned all = (1u << cnt) - 1u;
            const unsigned ma = m & all, mr = ~m & all;
            if (lane < cnt) {
                const int2 me = ws.ument[nu + lane];
                if ((ma >> lane) & 1u) {
                    const int k = (kQuad ? nc : nb) + __popc(ma & below);
                    float *at4 = (kQuad ? &ws.cell[0][0].x : &ws.src[0][0].x) + ((k >> 1) * 4 + (k & 1));
                    put_source(at4, ws.upm[nu + lane]);
                    if constexpr (kQuad) put_moments(at4, s.wqa[me.y], s.wqb[me.y]);
                } else {
                    const int k = sp + __popc(mr & below);
                    if (k < kStack) ws.stack[k] = me.x;
                    else set_status(ctrl, kStDepth, kStack);
                }
            }
            if constexpr (kQuad) nc += __popc(ma);
            else nb += __popc(ma);
            sp = min(sp + __popc(mr), kStack);
            __syncwarp();
        }
        // the next round's cells are popped and fetched before this round's
        // sums, which outlast the fetch
        np = sp > room ? min(sp, 1) : min(sp, kBatch);
        sp -= np;
        n_open += np;
        e[0] = cidx < np ? ws.stack[sp + cidx] : 0;
        e[1] = cidx + 4 < np ? ws.stack[sp + cidx + 4] : 0;
        fetch();
        const bool last = np == 0;
        // whole tiles from the (even) ends of the lists; at the end of the walk
        // also the rest, filled up with its last source without mass and moments
        if constexpr (kQuad) {
            const int even = nc & ~1;
            int k = even >> 1;  // in pairs
            for (; k >= 4; k -= 4) {
                const int i = k - 4 + col;
                const float4 v[5] = {ws.cell[0][i], ws.cell[1][i], ws.cell[2][i], ws.cell[3][i], ws.cell[4][i]};
                sum_tile_quad(v, eps2p, B);
                ++tiles_c;
            }
            if (k < (even >> 1)) {
                if (nc > even) {  // the odd one closes up
                    __syncwarp();
                    if (lane < 10)
                        reinterpret_cast<float *>(&ws.cell[lane >> 1][k])[2 * (lane & 1)] =
                            reinterpret_cast<const float *>(&ws.cell[lane >> 1][even >> 1])[2 * (lane & 1)];
                    __syncwarp();
                }
                nc = 2 * k + (nc - even);
            }
            if (last && nc > 0) {
                const int i = min(col, (nc - 1) >> 1);
                float4 v[5] = {ws.cell[0][i], ws.cell[1][i], ws.cell[2][i], ws.cell[3][i], ws.cell[4][i]};
                drop_beyond(v, 2 * col, nc);
                sum_tile_quad(v, eps2p, B);
            }
        }
        {
            const int even = nb & ~1;
            int k = even >> 1;
            for (; k >= 4; k -= 4) {
                sum_tile<kEpsZero>(ws.src[0][k - 4 + col], ws.src[1][k - 4 + col], eps2p, B);
                ++tiles_b;
            }
            if (k < (even >> 1)) {
                if (nb > even) {
                    __syncwarp();
                    if (lane < 4)
                        reinterpret_cast<float *>(&ws.src[lane >> 1][k])[2 * (lane & 1)] =
                            reinterpret_cast<const float *>(&ws.src[lane >> 1][even >> 1])[2 * (lane & 1)];
                    __syncwarp();
                }
                nb = 2 * k + (nb - even);
            }
            if (last && nb > 0) {
                const int i = min(col, (nb - 1) >> 1);
                float4 v[2] = {ws.src[0][i], ws.src[1][i]};
                drop_beyond(v, 2 * col, nb);
                sum_tile<kEpsZero>(v[0], v[1], eps2p, B);
            }
        }
        if (kComp && (tiles_b + tiles_c - flushed >= kFlushTiles || last)) {
            const float t[3] = {-tile_reduce(B.ax, lane), -tile_reduce(B.ay, lane), -tile_reduce(B.az, lane)};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                float hi = ws.run[k][lane], lo = ws.run[3 + k][lane];
                two_sum_add(hi, lo, t[k]);
                ws.run[k][lane] = hi;
                ws.run[3 + k][lane] = lo;
            }
            flushed = tiles_b + tiles_c;
#pragma unroll
            for (int k = 0; k < 4; ++k) B.ax[k] = B.ay[k] = B.az[k] = make_float2(0.0f, 0.0f);
        }
        if (last) break;
        __syncwarp();  // the lists and the stack are read before the next round adds to them
    }
    // nb and nc sources were left for the last, partial tiles
    const unsigned n_src = 8u * tiles_b + nb, n_cell = kQuad ? 8u * tiles_c + nc : n_src - n_body;
    if (kQuad) n_body = n_src;
    if (lane == 0) {
        const unsigned lanes = (unsigned)min(32, n - g * 32);
        atomicAdd(&ctrl->interactions, (unsigned long long)(n_body + n_cell) * lanes);
        atomicAdd(&ctrl->cell_interactions, (unsigned long long)n_cell * lanes);
        atomicAdd(&ctrl->opened, (unsigned long long)n_open);
    }
    float hx, hy, hz;
    if constexpr (kComp) {
        hx = ws.run[0][lane] + ws.run[3][lane];
        hy = ws.run[1][lane] + ws.run[4][lane];
        hz = ws.run[2][lane] + ws.run[5][lane];
    } else {
        hx = -tile_reduce(B.ax, lane);
        hy = -tile_reduce(B.ay, lane);
        hz = -tile_reduce(B.az, lane);
    }
    if (valid) {
        const int b = s.sorted[sidx];
        integrate_body<kMethod>(s, p, b, s.body_cur[b], hx * p.G, hy * p.G, hz * p.G);
    }
    __syncwarp();  // the next group's box goes where this one's was read
}

}  // namespace nbgb
