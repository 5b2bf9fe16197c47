// Barnes-Hut potential on the centre-of-mass octree.
//
// Reference: NewGalFinder/ost.c:226-251 (treeplumpotential) with the cell
// term CELLPLUMPOTENT (:144-176) and the particle term PARTICLEPLUMPOTENT
// (:178-193), opening test treeopen (:72-83): a node is opened when
// |p - com|^2 < dist2/theta2.  The cell term is
//     -M/r + trQ/(2 r^3) - 3 (d.Q.d)/(2 r^5)
// which the reference reads from linearly interpolated tables of -1/x,
// 1/(2x^3) and -3/(2x^5) (force_spline.mod3.c:81-138); here it is evaluated
// directly.  The drivers Self_Halo_Potent / External_Halo_Potent
// (subhaloden.mod6.c:1477-1621) use a direct sum below 100 members (self) or
// 1000 targets (external), then scale by potentfact and add the NFW
// background term of the halo mass (GetBGpotent, :1093-1101).
//
// A warp serves 32 targets, neighbours in tree order, one per lane.  The tree
// is expanded for all of them together and every accepted cell and opened
// leaf particle is evaluated by all lanes at once, so that no lane walks:
//   * nodes to visit, each with the mask of the lanes that opened its parent,
//     wait on a per-warp stack in shared memory; a step pops up to 32 and
//     tests one per lane against the bounding box of the targets.  Four out
//     of five are accepted (or opened) by every possible target in the box;
//     the others are tested target by target, all lanes on one node.
//     Opening decisions are those of an FP64 walk of the same tree: FP32
//     distances decide only outside a margin above their rounding error, and
//     what falls inside it is decided by the reference's FP64 test;
//   * accepted cells and the loose particles of opened nodes are gathered in
//     lists, each entry with its lane mask, and 32 entries are evaluated at
//     once: lane = entry, its fields in registers, against all 32 targets,
//     two per instruction (packed FP32 pairs; a 16-byte load of one coordinate
//     serves four targets), inactive targets by a zero 1/r.  Every lane has
//     32 partial sums; each kFlush tiles they go through shared memory to the
//     targets' lanes, which add them up with Kahan compensation.
// The terms are FP32 evaluated from position differences with two roundings
// (the node centre is held as the sum of two floats).  Against an FP64 walk of
// the same tree phi has 2.63e-8 to 2.81e-8 rms (1.4e5 to 1e6 particles), as
// with one Kahan sum per target; without the Kahan step, or with eight tiles
// between two additions, up to 2.9e-8.
//
// What bounds it: issue slots (62 % used, 29 k instructions per warp) and, at 5
// blocks per SM (96 registers, of which 32 are sums and 26 a cell's fields),
// the latency of the expansion's loads and shuffles; the FP32 pipe is 44 %
// busy.  A 131072-particle NFW halo at theta2 = 0.5 has, per warp, 937 cells
// (23 of 32 lanes) and 1268 particles (12 of 32).  With lane = target and the
// entries in shared memory, 13 floats of every cell were loaded by all lanes:
// 70 % of the shared-memory cycles, 35 k instructions.
// Measured, a lockstep walk (every lane at its own next node, the warp at the
// smallest) -> lane = target -> lane = entry: 4096 halos (6.1 M particles)
// 13.3 -> 9.2 -> 8.7 ms, 300,007 particles at theta2 = 0.25 1.93 -> 1.27 ->
// 1.07 ms, 256 halos (247 k) 0.60 -> 0.42 -> 0.39, 131,072 at 0.5 0.46 -> 0.30
// -> 0.32 ms, 64 small halos 0.31 -> 0.085 -> 0.095 ms (the last tiles of a
// warp are partly filled and cost as much as full ones).  4 blocks per SM: 9.3
// ms, 6 (80 registers, spilled): 10.6; a stack of 320 entries lets fewer nodes
// be popped at once: 9.0 ms; 64 threads per block: 8.7, but 64 small halos
// 0.136 ms.
#include <float.h>
#include <limits.h>
#include <math.h>

#include <algorithm>

#include "gf_tree.cuh"

namespace gf {

namespace {

struct Kahan {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float v) {
        const float y = v - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ float value() const { return s + (-c); }
};

// GetBGpotent, subhaloden.mod6.c:1059-1101
__device__ double bg_potent_dev(double mvir, const PotentialParams &pp) {
    const double G = 6.672E-8, RHOC = 2.7755E11;
    const double redshift = (double)(pp.amax / pp.a) - 1.0;
    const double c = 14.5 * pow(mvir / 1.3E13, -0.15) / (1.0 + redshift);
    const double gc = 1. / (log(1.0 + c) - c / (1.0 + c));
    const double om = pp.omep;
    const double vv = 18.0 * M_PI * M_PI + 82.0 * (om - 1.0) - 39.0 * pow(om - 1.0, 2.0);
    const double rvir = pow(3. * mvir / (4.0 * M_PI * vv * RHOC), 0.3333333333333);
    const double vc2 = G * mvir / rvir * pp.potentfact;
    return vc2 * (1 - gc * log(1 + c));
}

// ---- packed pairs of floats (two FP32 operations per instruction, each
// rounded as the scalar one)
using f2 = unsigned long long;
__device__ __forceinline__ f2 f2_pack(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_unpack(f2 v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// ---- per-warp shared memory of bh_kernel
constexpr int kStack = 416;  // (node, lanes) still to visit
constexpr int kDeal = 4;     // nodes per part before they are dealt out
constexpr int kFlush = 4;    // tiles between two additions to the targets' sums
struct __align__(16) BhWarp {
    float target[3][32];  // positions of the warp's targets
    uint2 cells[64];      // accepted (node, lanes) waiting for a tile
    uint2 leaf[64];       // loose (particle, lanes) waiting for a tile
    uint2 stack[kStack];
    float sums[32][36];   // a lane's terms of every target, 16 bytes beside the banks of the next lane's
};

// Two Kahan sums side by side; nc is the negated compensation.
struct Kahan2 {
    f2 s, nc;
    __device__ __forceinline__ void add(f2 t, f2 minus1) {
        const f2 y = f2_add(t, nc);
        const f2 n = f2_add(s, y);
        nc = f2_add(y, f2_fma(n, minus1, s));  // y - (n - s)
        s = n;
    }
};

// The walk one node at a time over the preorder nodes [i, end): every lane at
// its own next node, the warp at the smallest of them (taking part: lanes
// with `on`).  Serves what the tiles do not: subtrees that no longer fit the
// stack, and targets whose tiled sum is not finite (a squared distance below
// the normal floats, where this walk's rsqrtf is still exact to its 2 ulp).
__device__ __noinline__ float lockstep_walk(int i, int end, bool on, bool always_open, float4 P,
                                            const float4 *__restrict__ spos, const BhNode *__restrict__ nodes) {
    const double px = P.x, py = P.y, pz = P.z;
    Kahan acc;
    int my = on ? i : INT_MAX;
    while (i < end) {
        bool open = false;
        const int4 links = __ldg(reinterpret_cast<const int4 *>(nodes + i) + 4);  // skip, lstart, lcount, count
        if (my <= i) {
            const BhNode &nd = nodes[i];
            const double dx = px - nd.com[0], dy = py - nd.com[1], dz = pz - nd.com[2];
            // separately rounded, as the reference's treeopen (ost.c:79)
            const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
            open = always_open || d2 < nd.open_r2;
            if (open) {
                for (int j = links.y; j < links.y + links.z; j++) {
                    const float4 S = spos[j];
                    const float fx = P.x - S.x, fy = P.y - S.y, fz = P.z - S.z;
                    const float r2 = fx * fx + fy * fy + fz * fz;
                    if (r2 > 0.f) acc.add(-S.w * rsqrtf(r2));
                }
            } else {
                const float fx = (float)dx, fy = (float)dy, fz = (float)dz;
                const float r2 = fx * fx + fy * fy + fz * fz;
                const float inv = rsqrtf(r2), inv2 = inv * inv, inv3 = inv * inv2;
                const float qxy = nd.q[0] * fx * fx + nd.q[1] * fy * fy + nd.q[2] * fz * fz +
                                  2.f * (nd.q[3] * fx * fy + nd.q[4] * fx * fz + nd.q[5] * fy * fz);
                acc.add(-nd.mass * inv + 0.5f * nd.trq * inv3 - 1.5f * qxy * inv3 * inv2);
                my = links.x;
            }
        }
        // a lane that accepted an ancestor waits at or past this node's skip
        i = __any_sync(0xffffffffu, open) ? i + 1 : links.x;
    }
    return acc.value();
}

// COUNT: interaction counters (bench and tests); off in the stage's walk.
template <bool COUNT>
__global__ void __launch_bounds__(GF_BH_BLOCK, GF_BH_MINB)
bh_kernel(int64_t ntarget, const float4 *__restrict__ tpos, const int32_t *__restrict__ thalo,
          const int32_t *__restrict__ tout, const float4 *__restrict__ spos,
          const int32_t *__restrict__ root, const int32_t *__restrict__ rend,
          const BhNode *__restrict__ nodes, const WalkNode *__restrict__ wnodes,
          const int32_t *__restrict__ direct, const double *__restrict__ bg, PotentialParams pp,
          float *__restrict__ out, float *__restrict__ raw, unsigned long long *__restrict__ counters,
          unsigned long long *__restrict__ work, bool together) {
    extern __shared__ __align__(16) unsigned char bh_smem[];
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    BhWarp &W = reinterpret_cast<BhWarp *>(bh_smem)[threadIdx.x >> 5];
    // `together`: the warps of a block share 32 targets and divide the nodes
    // among them; warp 0 adds up and writes (one pass per launch)
    const int split = together ? (int)blockDim.x >> 5 : 1;
    const int part = together ? threadIdx.x >> 5 : 0;
    const int64_t warp0 = (((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) / split) * 32;
    const int64_t wstride = (int64_t)gridDim.x * blockDim.x / split;
    const f2 minus1 = f2_pack(-1.f, -1.f);
    unsigned long long npp = 0, npc = 0;
    // the warp's next 32 targets: from the work counter, or grid-stride
    auto next = [&](int64_t stride_base) -> int64_t {
        if (!GF_BH_DYN || !work) return stride_base;
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(work, 32ull);
        return (int64_t)__shfl_sync(0xffffffffu, b, 0);
    };
    for (int64_t base = next(warp0); base < ntarget; base = next(base + wstride)) {
        const int64_t t = base + lane;
        const bool valid = t < ntarget;
        int h = -1;
        float4 P = make_float4(0.f, 0.f, 0.f, 0.f);
        if (valid) {
            h = thalo[t];
            P = tpos[t];
        }
        W.target[0][lane] = P.x;
        W.target[1][lane] = P.y;
        W.target[2][lane] = P.z;
        __syncwarp();
        f2 acc[16];  // this lane's terms of the targets 2i, 2i + 1
#pragma unroll
        for (int i = 0; i < 16; i++) acc[i] = 0ull;
        Kahan2 total{0ull, 0ull};  // of this lane's target
        float aside = 0.f;   // subtrees walked one node at a time
        int cn = 0, ln = 0;  // waiting cells and particles (warp-uniform)
        int tiles = 0;
        auto flush = [&]() {
#pragma unroll
            for (int g = 0; g < 8; g++) {
                *reinterpret_cast<ulonglong2 *>(&W.sums[lane][4 * g]) = make_ulonglong2(acc[2 * g], acc[2 * g + 1]);
                acc[2 * g] = acc[2 * g + 1] = 0ull;
            }
            __syncwarp();
#pragma unroll
            for (int r = 0; r < 32; r += 2) total.add(f2_pack(W.sums[r][lane], W.sums[r + 1][lane]), minus1);
            __syncwarp();
            tiles = 0;
        };
        auto quad = [&](int a, int g) { return *reinterpret_cast<const ulonglong2 *>(&W.target[a][4 * g]); };

        // a tile of up to 32 cells, taken from the end of the waiting list: a lane each
        auto eval_cells = [&](int n) {
            cn -= n;
            const uint2 c = lane < n ? W.cells[cn + lane] : make_uint2(0u, 0u);
            const unsigned on = c.y;
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a, m = a, q = a;
            if (lane < n) {
                const float4 *w = reinterpret_cast<const float4 *>(wnodes + c.x);
                a = __ldg(w);
                b = __ldg(w + 2);
                m = __ldg(w + 3);
                q = __ldg(w + 4);
            }
            auto dup = [](float v) { return f2_pack(v, v); };
            const f2 hx = dup(-a.x), hy = dup(-a.y), hz = dup(-a.z), lx = dup(-b.x), ly = dup(-b.y), lz = dup(-b.z);
            const f2 mass = dup(b.w), txx = dup(m.x), tyy = dup(m.y), tzz = dup(m.z), txy = dup(m.w);
            const f2 txz = dup(q.x), tyz = dup(q.y);
#pragma unroll
            for (int g = 0; g < 8; g++) {
                const ulonglong2 X = quad(0, g), Y = quad(1, g), Z = quad(2, g);
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const f2 dx = f2_add(f2_add(u ? X.y : X.x, hx), lx);
                    const f2 dy = f2_add(f2_add(u ? Y.y : Y.x, hy), ly);
                    const f2 dz = f2_add(f2_add(u ? Z.y : Z.x, hz), lz);
                    const f2 r2 = f2_fma(dx, dx, f2_fma(dy, dy, f2_mul(dz, dz)));
                    float ra, rb;
                    f2_unpack(r2, ra, rb);
                    ra = (on & (1u << (4 * g + 2 * u))) ? rsqrt_ftz(ra) : 0.f;
                    rb = (on & (2u << (4 * g + 2 * u))) ? rsqrt_ftz(rb) : 0.f;
                    const f2 inv = f2_pack(ra, rb), inv2 = f2_mul(inv, inv), inv4 = f2_mul(inv2, inv2);
                    // d.Q.d over the upper triangle (off-diagonals doubled)
                    const f2 q1 = f2_fma(txx, dx, f2_fma(txy, dy, f2_mul(txz, dz)));
                    const f2 q2 = f2_fma(tyy, dy, f2_mul(tyz, dz));
                    const f2 qd = f2_fma(dx, q1, f2_fma(dy, q2, f2_mul(f2_mul(tzz, dz), dz)));
                    acc[2 * g + u] = f2_fma(f2_fma(qd, inv4, mass), inv, acc[2 * g + u]);
                }
            }
            __syncwarp();  // the list is read
            if (++tiles == kFlush) flush();
        };
        // up to 32 particles from the end of the waiting list
        auto eval_leaf = [&](int n) {
            ln -= n;
            const uint2 c = lane < n ? W.leaf[ln + lane] : make_uint2(0u, 0u);
            const unsigned on = c.y;
            float4 S = make_float4(0.f, 0.f, 0.f, 0.f);
            if (lane < n) S = __ldg(spos + c.x);
            const f2 sx = f2_pack(-S.x, -S.x), sy = f2_pack(-S.y, -S.y), sz = f2_pack(-S.z, -S.z);
            const f2 mass = f2_pack(S.w, S.w);
            const unsigned any = __reduce_or_sync(0xffffffffu, on);
#pragma unroll
            for (int g = 0; g < 8; g++) {
                if (!(any & (15u << (4 * g)))) continue;  // four targets that opened none of these leaves
                const ulonglong2 X = quad(0, g), Y = quad(1, g), Z = quad(2, g);
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const f2 dx = f2_add(u ? X.y : X.x, sx), dy = f2_add(u ? Y.y : Y.x, sy);
                    const f2 dz = f2_add(u ? Z.y : Z.x, sz);
                    const f2 r2 = f2_fma(dx, dx, f2_fma(dy, dy, f2_mul(dz, dz)));
                    float ra, rb;
                    f2_unpack(r2, ra, rb);
                    // ost.c:186-191: particle terms with r > 0
                    ra = (on & (1u << (4 * g + 2 * u))) && ra > 0.f ? rsqrt_ftz(ra) : 0.f;
                    rb = (on & (2u << (4 * g + 2 * u))) && rb > 0.f ? rsqrt_ftz(rb) : 0.f;
                    acc[2 * g + u] = f2_fma(mass, f2_pack(ra, rb), acc[2 * g + u]);
                }
            }
            __syncwarp();
            if (++tiles == kFlush) flush();
        };

        // ---- one halo of the warp's targets at a time (nearly always one)
        for (unsigned todo = __ballot_sync(0xffffffffu, valid); todo;) {
            const int hl = __shfl_sync(0xffffffffu, h, __ffs(todo) - 1);
            const unsigned grp = __ballot_sync(0xffffffffu, valid && h == hl);
            todo &= ~grp;
            if (root[hl] >= rend[hl]) continue;
            const bool all_open = direct && direct[hl];
            float blo[3], bhi[3];  // the box of this halo's targets
            {
                const bool in = (grp >> lane) & 1u;
                const float c[3] = {P.x, P.y, P.z};
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    float lo = in ? c[a] : FLT_MAX, hi = in ? c[a] : -FLT_MAX;
#pragma unroll
                    for (int o = 16; o; o >>= 1) {
                        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
                    }
                    blo[a] = lo;
                    bhi[a] = hi;
                }
            }
            if (lane == 0) W.stack[0] = make_uint2((unsigned)hl, grp);  // the root of halo h is walk node h
            __syncwarp();
            int top = 1;
            // every part expands the first nodes, part 0 keeps their cells
            // and particles; once there are a few nodes for each part, they
            // are dealt out
            bool shared = together;
            while (top > 0) {
                if (shared && top >= kDeal * split) {
                    shared = false;
                    const int mine = (top - part + split - 1) / split;
                    for (int i = 0; i < mine; i += 32) {
                        uint2 v = make_uint2(0u, 0u);
                        if (i + lane < mine) v = W.stack[part + split * (i + lane)];
                        __syncwarp();
                        if (i + lane < mine) W.stack[i + lane] = v;
                        __syncwarp();
                    }
                    top = mine;
                    continue;
                }
                // as many as leave room for eight children each
                int take = min(min(32, top), (kStack - top) / 7);
                const bool full = take < 1;
                take = max(take, 1);
                top -= take;
                int node = 0;
                unsigned m = 0u;
                if (lane < take) {
                    const uint2 v = W.stack[top + lane];
                    node = (int)v.x;
                    m = v.y;
                }
                __syncwarp();
                if (full) {  // no room for this node's children
                    const int nd = __shfl_sync(0xffffffffu, node, 0);
                    const unsigned mm = __shfl_sync(0xffffffffu, m, 0);
                    const int pre = wnodes[nd].pre;
                    const float v = lockstep_walk(pre, nodes[pre].skip, (mm >> lane) & 1u, all_open, P, spos, nodes);
                    if (!(shared && part)) aside += v;
                    continue;
                }
                const WalkNode *w = wnodes + node;
                int4 lk = make_int4(0, 0, 0, 0);  // first, nchild, lstart, lcount
                unsigned am = 0u, om = m;         // lanes that accept, that open
                bool mixed = false;
                if (lane < take) {
                    const float4 a = __ldg(reinterpret_cast<const float4 *>(w));
                    lk = __ldg(reinterpret_cast<const int4 *>(w) + 1);
                    // nearest and farthest distance from the node's centre to
                    // the box, widened by the rounding of a coordinate
                    const float c[3] = {a.x, a.y, a.z};
                    float mn = 0.f, mx = 0.f;
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        const float g0 = blo[i] - c[i], g1 = c[i] - bhi[i];
                        const float e = fabsf(c[i]) * 1.2e-7f;
                        const float g = fmaxf(fmaxf(g0, g1) - e, 0.f), f = fmaxf(fabsf(g0), fabsf(g1)) + e;
                        mn += g * g;
                        mx += f * f;
                    }
                    if (!all_open) {
                        if (mn > walk_open_hi(a.w) * (1.f + 2e-6f)) {
                            am = m;
                            om = 0u;
                        } else {
                            mixed = !(mx * (1.f + 2e-6f) < a.w);
                        }
                    }
                }
                // nodes that the box does not settle, target by target
                for (unsigned mb = __ballot_sync(0xffffffffu, mixed); mb; mb &= mb - 1) {
                    const int src = __ffs(mb) - 1;
                    const int nd = __shfl_sync(0xffffffffu, node, src);
                    const unsigned ms = __shfl_sync(0xffffffffu, m, src);
                    const float4 a = __ldg(reinterpret_cast<const float4 *>(wnodes + nd));
                    const float4 b = __ldg(reinterpret_cast<const float4 *>(wnodes + nd) + 2);
                    const float dx = (P.x - a.x) - b.x, dy = (P.y - a.y) - b.y, dz = (P.z - a.z) - b.z;
                    const float r2 = dx * dx + dy * dy + dz * dz;
                    bool open = r2 < a.w;
                    if (!open && !(r2 > walk_open_hi(a.w)) && ((ms >> lane) & 1u)) {
                        // within the margin: the reference's treeopen in FP64,
                        // separately rounded (ost.c:79)
                        const BhNode &n = nodes[wnodes[nd].pre];
                        const double ex = (double)P.x - n.com[0], ey = (double)P.y - n.com[1], ez = (double)P.z - n.com[2];
                        open = __dadd_rn(__dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)), __dmul_rn(ez, ez)) < n.open_r2;
                    }
                    const unsigned ob = __ballot_sync(0xffffffffu, open);
                    if (lane == src) {
                        am = m & ~ob;
                        om = m & ob;
                    }
                }
                // ---- children of the opened nodes onto the stack
                const int nch = om ? lk.y : 0;
                int at = nch;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, at, o);
                    if (lane >= o) at += v;
                }
                const int nall = __shfl_sync(0xffffffffu, at, 31);
                for (int c = 0, s0 = top + at - nch; c < nch; c++) W.stack[s0 + c] = make_uint2((unsigned)(lk.x + c), om);
                top += nall;
                if (shared && part) {  // part 0 has these
                    am = 0u;
                    lk.w = 0;
                }
                if (COUNT) {
                    npc += __popc(am);
                    npp += (unsigned long long)lk.w * __popc(om);
                }
                // ---- accepted cells
                const unsigned ab = __ballot_sync(0xffffffffu, am != 0u);
                if (am) W.cells[cn + __popc(ab & lt)] = make_uint2((unsigned)node, am);
                cn += __popc(ab);
                __syncwarp();
                while (cn >= 32 || (top == 0 && cn > 0)) eval_cells(min(cn, 32));
                // ---- loose particles of the opened nodes
                int o = 0;
                for (unsigned lb = __ballot_sync(0xffffffffu, om != 0u && lk.w > 0);;) {
                    if (ln >= 32 || (!lb && top == 0 && ln > 0)) {
                        eval_leaf(min(ln, 32));
                        continue;
                    }
                    if (!lb) break;
                    const int src = __ffs(lb) - 1;
                    const int l0 = __shfl_sync(0xffffffffu, lk.z, src), lc = __shfl_sync(0xffffffffu, lk.w, src);
                    const unsigned lm = __shfl_sync(0xffffffffu, om, src);
                    const int k = min(32, lc - o);
                    if (lane < k) W.leaf[ln + lane] = make_uint2((unsigned)(l0 + o + lane), lm);
                    ln += k;
                    o += 32;
                    if (o >= lc) {
                        lb &= lb - 1;
                        o = 0;
                    }
                    __syncwarp();
                }
            }
        }
        flush();
        float s0, s1, c0, c1;  // the two sums and their compensations
        f2_unpack(total.s, s0, s1);
        f2_unpack(total.nc, c0, c1);
        double sum = (double)aside - (((double)s0 + (double)s1) + ((double)c0 + (double)c1));
        if (together) {
            double *red = reinterpret_cast<double *>(W.stack);  // 32 of each part, done with its stack
            __syncwarp();
            red[lane] = sum;
            __syncthreads();
            if (part) continue;
            for (int q = 1; q < split; q++) sum += reinterpret_cast<const double *>((&W + q)->stack)[lane];
        }
        float phi = (float)(0.0 + sum);
        bool redo = valid && !(fabsf(phi) <= FLT_MAX);
        for (unsigned rb = __ballot_sync(0xffffffffu, redo); rb;) {
            const int hl = __shfl_sync(0xffffffffu, h, __ffs(rb) - 1);
            const bool on = redo && h == hl;
            const float v = lockstep_walk(root[hl], rend[hl], on, direct && direct[hl], P, spos, nodes);
            if (on) phi = v;
            rb &= ~__ballot_sync(0xffffffffu, on);
        }
        if (valid) {
            const int64_t o = tout ? tout[t] : t;
            if (raw) raw[o] = phi;
            if (out) {
                double e = pp.potentfact != 0.0 ? (double)phi * pp.potentfact : (double)phi;
                if (pp.add_bg && bg) e += bg[h];
                out[o] = (float)e;  // penergy = potent*potentfact + halobgpotent
            }
        }
    }
    if (COUNT && counters) {
        for (int off = 16; off; off >>= 1) {
            npp += __shfl_xor_sync(0xffffffffu, npp, off);
            npc += __shfl_xor_sync(0xffffffffu, npc, off);
        }
        if (lane == 0) {
            atomicAdd(counters + 0, npp);
            atomicAdd(counters + 1, npc);
        }
    }
}

// The walk over ntarget targets on a grid of one resident wave.  With
// GF_BH_DYN each warp takes its next 32 targets from a counter in device
// memory, so warps that drew cheap targets keep drawing and the launch ends
// when the work does (with a static grid-stride split, the warps holding the
// costliest targets finish last, alone).
int launch_bh(gf_ctx *ctx, int64_t ntarget, const float4 *tpos, const int32_t *thalo,
              const int32_t *tout, const TreeView &t, const int32_t *direct, const double *bg,
              const PotentialParams &pp, float *out, float *raw, unsigned long long *counters) {
    const int block = GF_BH_BLOCK;
    const size_t shmem = (size_t)(block / 32) * sizeof(BhWarp);
    unsigned long long *work = nullptr;
    auto kern = counters ? bh_kernel<true> : bh_kernel<false>;
    int per_sm = 0;
    GF_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shmem));
    GF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, shmem));
    const int64_t wave = (int64_t)sm_count() * std::max(per_sm, 1);  // resident blocks
    const int64_t groups = (ntarget + 31) / 32, warps = block / 32;
    // few targets: a block's warps divide the nodes of 32 targets among them
    // instead of leaving most of the SMs' warps without work.  Above half of
    // the resident warps the dealing costs more than it fills (more steps
    // with less than 32 nodes each): 36,001 targets 139 -> 114 us, a batch of
    // 64 small halos 257 -> 93, but 131,072 targets 313 -> 386.
    const bool together = 2 * groups <= wave * warps;
    int64_t grid = together ? groups : (groups + warps - 1) / warps;
    if (!together) {
        // a grid of 1.6 waves would leave 40 % of the SMs' block slots empty in its second wave
        grid = std::min(grid, wave);
        if (GF_BH_DYN) {
            GF_TRY(ctx->work.reserve(256));
            work = ctx->work.as<unsigned long long>();  // slot 0: this walk
            GF_CUDA_TRY(cudaMemsetAsync(work, 0, sizeof(unsigned long long), ctx->stream));
        }
    }
    kern<<<(int)grid, block, shmem, ctx->stream>>>(ntarget, tpos, thalo, tout, t.pos, t.root, t.rend, t.bh, t.walk,
                                                   direct, bg, pp, out, raw, counters, work, together);
    GF_LAUNCH_CHECK();
    return GF_OK;
}

// Per-halo total mass (FP64 sum of the float masses, as Self_Halo_Potent's
// Mvir += mass[i]) and background term.  Each halo's particles are summed in
// kMassSplit slices by separate blocks (a large halo no longer holds one
// block for its whole length), then the slices in order.
constexpr int kMassSplit = 16;

__global__ void halo_mass_kernel(int32_t nhalo, const int64_t *__restrict__ pstart,
                                 const float4 *__restrict__ pos, double *__restrict__ part) {
    const int h = blockIdx.x / kMassSplit, sl = blockIdx.x % kMassSplit;
    if (h >= nhalo) return;
    const int64_t a0 = pstart[h], len = pstart[h + 1] - a0;
    const int64_t a = a0 + len * sl / kMassSplit, b = a0 + len * (sl + 1) / kMassSplit;
    double s = 0.0;
    for (int64_t p = a + threadIdx.x; p < b; p += blockDim.x) s += (double)pos[p].w;
    __shared__ double red[256];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void halo_bg_kernel(int32_t nhalo, const int64_t *__restrict__ pstart,
                               const double *__restrict__ part, PotentialParams pp,
                               const int32_t *__restrict__ ntarget_halo,
                               int32_t ndirect, double *__restrict__ bg,
                               int32_t *__restrict__ direct) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= nhalo) return;
    double m = 0.0;
    for (int sl = 0; sl < kMassSplit; sl++) m += part[(int64_t)h * kMassSplit + sl];
    bg[h] = pp.add_bg ? bg_potent_dev(m, pp) : 0.0;
    const int64_t nt = ntarget_halo ? ntarget_halo[h] : pstart[h + 1] - pstart[h];
    direct[h] = nt < ndirect ? 1 : 0;
}

__global__ void bg_eval_kernel(int32_t n, const double *__restrict__ mvir, PotentialParams pp,
                               double *__restrict__ bg) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) bg[i] = bg_potent_dev(mvir[i], pp);
}

}  // namespace

// bg and direct flags of every halo of t (scratch in ctx->tmp[5]).
int launch_halo_bg(gf_ctx *ctx, const TreeView &t, const int64_t *pstart, const PotentialParams &pp,
                   const int32_t *ntarget_halo, double **bg, int32_t **direct) {
    const size_t nb = (size_t)t.nhalo * sizeof(double);
    const size_t np_ = (size_t)t.nhalo * kMassSplit * sizeof(double);
    GF_TRY(ctx->tmp[5].reserve(nb + np_ + (size_t)t.nhalo * sizeof(int32_t) + 512));
    *bg = ctx->tmp[5].as<double>();
    double *part = *bg + t.nhalo;
    *direct = reinterpret_cast<int32_t *>(part + (size_t)t.nhalo * kMassSplit);
    halo_mass_kernel<<<t.nhalo * kMassSplit, 256, 0, ctx->stream>>>(t.nhalo, pstart, t.pos, part);
    GF_LAUNCH_CHECK();
    halo_bg_kernel<<<(t.nhalo + 127) / 128, 128, 0, ctx->stream>>>(t.nhalo, pstart, part, pp, ntarget_halo,
                                                                   pp.ndirect, *bg, *direct);
    GF_LAUNCH_CHECK();
    return GF_OK;
}

// The background term of n halo masses as the potential kernels evaluate it.
int launch_bg_eval(gf_ctx *ctx, int32_t n, const double *mvir, const PotentialParams &pp, double *bg) {
    if (n <= 0) return GF_OK;
    bg_eval_kernel<<<(n + 127) / 128, 128, 0, ctx->stream>>>(n, mvir, pp, bg);
    GF_LAUNCH_CHECK();
    return GF_OK;
}

// Potential at every particle of every halo from the halo's own tree
// (self potential); outputs in batch order.
int launch_self_potential(gf_ctx *ctx, const TreeView &t, const int64_t *pstart,
                          const PotentialParams &pp, float *penergy, float *raw,
                          unsigned long long *counters, double *bg, int32_t *direct) {
    if (t.n <= 0) return GF_OK;
    // tree-ordered positions carry the masses; halo h is still [pstart[h], pstart[h+1])
    if (!bg) GF_TRY(launch_halo_bg(ctx, t, pstart, pp, nullptr, &bg, &direct));
    GF_TRY(launch_bh(ctx, t.n, t.pos, t.phalo, t.perm, t, direct, bg, pp, penergy, raw, counters));
    return GF_OK;
}

// Potential of one source tree (halo 0 of t) at arbitrary targets.
int launch_external_potential(gf_ctx *ctx, const TreeView &t, const int64_t *pstart_src,
                              int64_t ntarget, const float4 *tpos, const int32_t *thalo,
                              const int32_t *ntarget_halo, const PotentialParams &pp,
                              float *penergy, float *raw) {
    if (ntarget <= 0) return GF_OK;
    double *bg;
    int32_t *direct;
    GF_TRY(launch_halo_bg(ctx, t, pstart_src, pp, ntarget_halo, &bg, &direct));
    GF_TRY(launch_bh(ctx, ntarget, tpos, thalo, nullptr, t, direct, bg, pp, penergy, raw, nullptr));
    return GF_OK;
}

}  // namespace gf
