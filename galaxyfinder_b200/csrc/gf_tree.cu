// Level-synchronous GPU build of the centre-of-mass octree of every halo in a
// batch, following the node rules of the reference's tree builders
// (NewGalFinder/ost.c:532-640 divide_node, nnost.c:105-197 new_divide_node_Near):
//   * a node's centre of mass splits its particles into octants by
//     (x > com_x) + 2 (y > com_y) + 4 (z > com_z);
//   * an octant becomes a child node iff it holds >= 10 particles
//     (MIN_CELL_PARTICLE_NUM) and the node's size sqrt(max |x - com|^2)
//     exceeds 0.5e-6 (MINCELLWIDTH/2); smaller octants stay as loose
//     particles of the node;
//   * monopole, second moments and dist2 = max |x - com|^2 are per node.
// Nodes of more than kSmall particles are built level by level, every active
// particle of all halos at once: accumulate mass and first moments, accumulate
// extents/second moments/octant counts about the centre of mass, allocate
// children, and scatter the particles into [loose | child 0 | child 1 | ...]
// order.  A node of at most kSmall particles is left to one warp, which builds its whole
// subtree in shared memory (small_subtrees).  The nodes are then numbered in
// depth-first preorder so the walks are stackless: opening node i continues at
// i + 1, skipping it continues at skip[i].  A node's preorder number is the
// number of nodes that start before its first particle (a scan over the
// particles of the nodes starting at each), plus the ancestors starting with it.
#include <math.h>

#include <algorithm>
#include <vector>

#include "gf_tree.cuh"

namespace gf {

namespace {

constexpr int kMinCell = 10;          // MIN_CELL_PARTICLE_NUM, tree.h:20
constexpr double kMinWidth = 1.E-6;   // MINCELLWIDTH, tree.h:18
constexpr int kBlock = GF_TREE_BLOCK;

// |x - com|^2 with its roundings spelled out: a node's extent decides what a walk
// opens, so it may not depend on how a kernel's compilation pairs the products
// (one unit in the last place flips an opening in some 1e8 and moves that
// target's potential by 1e-5).
__device__ __forceinline__ float offset2(float x, float y, float z) {
    return __fmaf_rn(z, z, __fmaf_rn(x, x, __fmul_rn(y, y)));
}

// Order-preserving float <-> uint32 map for atomic min/max on any sign.
__device__ __forceinline__ unsigned fkey(float v) {
    unsigned u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fkey_inv(unsigned k) {
    unsigned u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(u);
}

// BFS-numbered node arrays used while building.
struct Build {
    int32_t *start, *count, *halo;
    // accumulators, zeroed when their node is allocated (a memset of the node
    // capacity touched ten times the nodes that a tree has)
    double *m, *mx, *my, *mz;       // mass and first moments, then COM in mx..mz
    unsigned *r2;                   // float bits of max |x - com|^2
    float *q;                       // 6 second moments
    unsigned *box;                  // 6 fkeys as maxima: ~min xyz, max xyz
    int32_t *oct;                   // 8 octant counts
    int32_t *cur;                   // 8 octant cursors
    int32_t *ochild;                // 8 child ids or -1
    int32_t *first, *nchild, *lstart, *lcount;
    int32_t *par;                   // id of the parent, -1 for roots
    int32_t *small;                 // nodes left to small_subtrees (their level stands in first until then)
    int32_t *counter;               // [0] nodes allocated, [1] overflow flags, [2] blocks done, [3] small nodes,
                                    // [4] depth of the trees, in levels
    int32_t *lev;                   // level L holds the nodes [lev[L], lev[L+1]) (while the levels run)
    int32_t *nact;                  // nodes of level L that the level passes process
};

// A node of at most kSmall particles is built with its subtree by one warp.  The
// level passes cost four launches a level (and, eagerly, a host wait) however
// few particles are left, and read every one of those from memory, so the
// lower levels, most of a small batch's, go to shared memory: the stage on a
// halo of 120 took 0.32 ms, now 0.24; on one of 131,072 1.59, now 1.40; a
// replayed graph of 64 halos 0.75, now 0.66; four gradients of one million
// particles, whose tree was their largest part, 1.35, now 1.16.  256 particles
// (two buffers, 10 KB) leave 20 warps per SM; the pass is bound by the chain
// of shuffles of a node (log2 32 steps for 17 values), 0.42 ms for 6 M
// particles.
constexpr int kSmall = 256;

__device__ __forceinline__ void zero_node(const Build &b, int node) {
    b.m[node] = b.mx[node] = b.my[node] = b.mz[node] = 0.0;
    b.r2[node] = 0u;
    float2 *q = reinterpret_cast<float2 *>(b.q + 6 * (int64_t)node);
    uint2 *box = reinterpret_cast<uint2 *>(b.box + 6 * (int64_t)node);
#pragma unroll
    for (int i = 0; i < 3; i++) {
        q[i] = make_float2(0.f, 0.f);
        box[i] = make_uint2(0u, 0u);
    }
    int4 *oct = reinterpret_cast<int4 *>(b.oct + 8 * (int64_t)node);
    oct[0] = oct[1] = make_int4(0, 0, 0, 0);
}

constexpr int kMaxLevels = 4096;

// Grid-stride range of the nodes of level L (bounds in device memory).
#define FOR_LEVEL_NODES(node, L, b)                                                          \
    for (int node = (b).lev[L] + blockIdx.x * blockDim.x + threadIdx.x; node < (b).lev[(L) + 1]; \
         node += gridDim.x * blockDim.x)

// The roots, nodes 0 .. nhalo-1 (counter and nact start zeroed), and the
// particles; those of small halos go straight to the final arrays, where
// small_subtrees orders them.
__global__ void init_build(int64_t n, const int64_t *__restrict__ pstart, int32_t nhalo,
                           const float4 *__restrict__ pos_in, float4 *__restrict__ pos, int32_t *__restrict__ perm,
                           int32_t *__restrict__ pnode, float4 *__restrict__ fpos, int32_t *__restrict__ fperm,
                           int32_t *__restrict__ phalo, Build b) {
    for (int64_t h = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; h < max(nhalo, 1);
         h += (int64_t)gridDim.x * blockDim.x) {
        if (h == 0) {
            b.counter[0] = nhalo;
            b.lev[0] = 0;
            b.lev[1] = nhalo;
        }
        if (h >= nhalo) break;
        const int c = (int32_t)(pstart[h + 1] - pstart[h]);
        b.start[h] = (int32_t)pstart[h];
        b.count[h] = c;
        b.halo[h] = (int32_t)h;
        b.par[h] = -1;
        if (c > kSmall) {
            zero_node(b, (int)h);
            atomicAdd(b.nact, 1);
        } else {
            b.first[h] = 0;
            b.small[atomicAdd(b.counter + 3, 1)] = (int32_t)h;
        }
    }
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n;
         p += (int64_t)gridDim.x * blockDim.x) {
        int lo = 0, hi = nhalo;
        while (hi - lo > 1) {
            int mid = (lo + hi) >> 1;
            if (pstart[mid] <= p) lo = mid; else hi = mid;
        }
        phalo[p] = lo;
        const bool active = pstart[lo + 1] - pstart[lo] > kSmall;
        (active ? pos : fpos)[p] = pos_in[p];
        (active ? perm : fperm)[p] = (int32_t)p;
        pnode[p] = active ? lo : -1;  // the root of halo h is node h
    }
}

// Runs of a warp: lanes with equal node ids are consecutive (a node's active
// particles are contiguous at every level), so a node's lanes form one run.
// Inclusive segmented scans over the runs (five shuffle steps whatever the
// run lengths); each run's last lane holds its reduction.
struct WarpRuns {
    int start;  // first lane of this lane's run
    bool tail;  // last lane of its run
};
__device__ __forceinline__ WarpRuns warp_runs(int node) {
    const int lane = threadIdx.x & 31;
    const int prev = __shfl_up_sync(0xffffffffu, node, 1);
    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || prev != node);
    WarpRuns r;
    r.start = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
    r.tail = lane == 31 || ((heads >> (lane + 1)) & 1u);
    return r;
}
template <class T, class Op>
__device__ __forceinline__ T run_scan(T v, const WarpRuns &r, Op op) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const T u = __shfl_up_sync(0xffffffffu, v, off);
        if (lane - off >= r.start) v = op(v, u);
    }
    return v;
}
struct AddOp {
    template <class T> __device__ __forceinline__ T operator()(T a, T b) const { return a + b; }
};
struct MaxOp {
    template <class T> __device__ __forceinline__ T operator()(T a, T b) const { return max(a, b); }
};
struct FMaxOp {
    __device__ __forceinline__ float operator()(float a, float b) const { return fmaxf(a, b); }
};

// Pass 1: mass and mass-weighted position per node (FP64 accumulation).
__global__ void __launch_bounds__(kBlock)
accum_mass(int L, int64_t n, const float4 *__restrict__ pos, const int32_t *__restrict__ pnode, Build b) {
    if (b.nact[L] == 0) return;  // a level past the last one (fixed shapes, levels run ahead of the host)
    __shared__ double s[4][kBlock / 32];
    __shared__ int s_node;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t base = blockIdx.x * (int64_t)kBlock; base < n; base += (int64_t)gridDim.x * kBlock) {
        const int64_t p = base + threadIdx.x;
        const int node = p < n ? pnode[p] : -1;
        double w = 0, wx = 0, wy = 0, wz = 0;
        if (node >= 0) {
            const float4 v = pos[p];
            // ost.c:546-552: mass += ptlmass; mono += ptlmass * x (float mass, FP64 positions)
            w = v.w;
            wx = (double)v.w * (double)v.x;
            wy = (double)v.w * (double)v.y;
            wz = (double)v.w * (double)v.z;
        }
        if (threadIdx.x == 0) s_node = node;
        __syncthreads();
        const bool uniform = __syncthreads_and(node == s_node) && s_node >= 0;
        if (uniform) {
            for (int off = 16; off; off >>= 1) {
                w += __shfl_xor_sync(0xffffffffu, w, off);
                wx += __shfl_xor_sync(0xffffffffu, wx, off);
                wy += __shfl_xor_sync(0xffffffffu, wy, off);
                wz += __shfl_xor_sync(0xffffffffu, wz, off);
            }
            if (lane == 0) { s[0][warp] = w; s[1][warp] = wx; s[2][warp] = wy; s[3][warp] = wz; }
            __syncthreads();
            if (threadIdx.x < 4) {
                double a = 0;
                for (int i = 0; i < kBlock / 32; i++) a += s[threadIdx.x][i];
                double *dst = threadIdx.x == 0 ? b.m : threadIdx.x == 1 ? b.mx : threadIdx.x == 2 ? b.my : b.mz;
                atomicAdd(dst + s_node, a);
            }
        } else if (__all_sync(0xffffffffu, node == __shfl_sync(0xffffffffu, node, 0))) {
            // one node for the whole warp (settled warps add nothing)
            if (node >= 0) {
                for (int off = 16; off; off >>= 1) {
                    w += __shfl_xor_sync(0xffffffffu, w, off);
                    wx += __shfl_xor_sync(0xffffffffu, wx, off);
                    wy += __shfl_xor_sync(0xffffffffu, wy, off);
                    wz += __shfl_xor_sync(0xffffffffu, wz, off);
                }
                if (lane == 0) {
                    atomicAdd(b.m + node, w);
                    atomicAdd(b.mx + node, wx);
                    atomicAdd(b.my + node, wy);
                    atomicAdd(b.mz + node, wz);
                }
            }
        } else {
            // several nodes: segmented sums over the warp's runs, added by
            // each run's last lane (settled runs, node < 0, add nothing)
            const WarpRuns r = warp_runs(node);
            w = run_scan(w, r, AddOp());
            wx = run_scan(wx, r, AddOp());
            wy = run_scan(wy, r, AddOp());
            wz = run_scan(wz, r, AddOp());
            if (r.tail && node >= 0) {
                atomicAdd(b.m + node, w);
                atomicAdd(b.mx + node, wx);
                atomicAdd(b.my + node, wy);
                atomicAdd(b.mz + node, wz);
            }
        }
        __syncthreads();
    }
}

// ost.c:553-555: the centre of mass of a node whose sums are complete.
__device__ __forceinline__ void centre_of(const Build &b, int node, double &x, double &y, double &z) {
    const double m = b.m[node];
    x = b.mx[node];
    y = b.my[node];
    z = b.mz[node];
    if (m > 0) {
        x /= m;
        y /= m;
        z /= m;
    }
}

// Pass 2: extents, max |x - com|^2, second moments and octant counts.
// The 13 reductions (max r2, six moment sums, min and max of the three
// coordinate keys) run over the block when all its particles share a node
// (one atomic per value and block: the top levels of large halos), over the
// warp when it does, else over the warp's runs.
__global__ void __launch_bounds__(kBlock)
accum_moments(int L, int64_t n, const float4 *__restrict__ pos, const int32_t *__restrict__ pnode,
              uint8_t *__restrict__ pkey, int q5_asbuilt, Build b) {
    if (b.nact[L] == 0) return;
    constexpr int kWarps = kBlock / 32;
    __shared__ float s_f[7][kWarps];
    __shared__ unsigned s_k[6][kWarps];
    __shared__ int s_oct[8];
    __shared__ int s_node;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 8) s_oct[threadIdx.x] = 0;
    for (int64_t base = blockIdx.x * (int64_t)kBlock; base < n; base += (int64_t)gridDim.x * kBlock) {
        const int64_t p = base + threadIdx.x;
        const int node = p < n ? pnode[p] : -1;
        float v[7] = {0, 0, 0, 0, 0, 0, 0};  // max |x - com|^2, then q0..q5
        unsigned bx[6] = {0u, 0u, 0u, 0u, 0u, 0u};  // ~min xyz, max xyz: all maxima
        int key = 0;
        if (node >= 0) {
            const float4 P = pos[p];
            double cx, cy, cz;  // (divided by every particle: cheaper than a launch per level for it)
            centre_of(b, node, cx, cy, cz);
            // ost.c:561-571: float offsets, float moments
            const float tx = (float)((double)P.x - cx);
            const float ty = (float)((double)P.y - cy);
            const float tz = (float)((double)P.z - cz);
            const float m = P.w;
            v[0] = offset2(tx, ty, tz);
            v[1] = m * tx * tx;
            v[2] = m * ty * ty;
            v[3] = m * tz * tz;
            v[4] = m * tx * ty;
            v[5] = m * tx * tz;
            v[6] = q5_asbuilt ? m * ty * tx : m * ty * tz;
            bx[3] = fkey(P.x);
            bx[4] = fkey(P.y);
            bx[5] = fkey(P.z);
            bx[0] = ~bx[3];
            bx[1] = ~bx[4];
            bx[2] = ~bx[5];
            // ost.c:589-592: SubCellDicision(x, monox) = x > monox
            key = ((double)P.x > cx ? 1 : 0) | ((double)P.y > cy ? 2 : 0) | ((double)P.z > cz ? 4 : 0);
            pkey[p] = (uint8_t)key;
        }
        if (threadIdx.x == 0) s_node = node;
        __syncthreads();
        const bool block_uniform = __syncthreads_and(node == s_node) && s_node >= 0;
        const bool warp_uniform = __all_sync(0xffffffffu, node == __shfl_sync(0xffffffffu, node, 0));
        if (block_uniform || warp_uniform) {  // butterfly over the warp (none for a settled warp)
            for (int off = 16; node >= 0 && off; off >>= 1) {
                v[0] = fmaxf(v[0], __shfl_xor_sync(0xffffffffu, v[0], off));
                for (int i = 1; i < 7; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i], off);
            }
            if (node >= 0)
                for (int i = 0; i < 6; i++) bx[i] = __reduce_max_sync(0xffffffffu, bx[i]);
        } else {  // several nodes: segmented over the warp's runs
            const WarpRuns r = warp_runs(node);
            v[0] = run_scan(v[0], r, FMaxOp());
            for (int i = 1; i < 7; i++) v[i] = run_scan(v[i], r, AddOp());
            for (int i = 0; i < 6; i++) bx[i] = run_scan(bx[i], r, MaxOp());
            if (r.tail && node >= 0) {
                atomicMax(b.r2 + node, __float_as_uint(v[0]));  // non-negative floats
                for (int i = 0; i < 6; i++) atomicAdd(b.q + 6 * (int64_t)node + i, v[1 + i]);
                for (int i = 0; i < 6; i++) atomicMax(b.box + 6 * (int64_t)node + i, bx[i]);
            }
        }
        if (block_uniform) {  // then over the block: one atomic per value
            if (lane == 0) {
                for (int i = 0; i < 7; i++) s_f[i][warp] = v[i];
                for (int i = 0; i < 6; i++) s_k[i][warp] = bx[i];
            }
            const unsigned g2 = __match_any_sync(0xffffffffu, key);
            if (lane == __ffs(g2) - 1) atomicAdd(s_oct + key, __popc(g2));
            __syncthreads();
            if (threadIdx.x < 7) {
                const int i = threadIdx.x;
                float a = s_f[i][0];
                for (int w2 = 1; w2 < kWarps; w2++) a = i == 0 ? fmaxf(a, s_f[i][w2]) : a + s_f[i][w2];
                if (i == 0) atomicMax(b.r2 + s_node, __float_as_uint(a));
                else atomicAdd(b.q + 6 * (int64_t)s_node + (i - 1), a);
            } else if (threadIdx.x < 13) {
                const int i = threadIdx.x - 7;
                unsigned a = s_k[i][0];
                for (int w2 = 1; w2 < kWarps; w2++) a = max(a, s_k[i][w2]);
                atomicMax(b.box + 6 * (int64_t)s_node + i, a);
            } else if (threadIdx.x >= 32 && threadIdx.x < 40) {
                const int c = threadIdx.x - 32;
                if (s_oct[c]) atomicAdd(b.oct + 8 * (int64_t)s_node + c, s_oct[c]);
                s_oct[c] = 0;
            }
        } else {
            if (warp_uniform && node >= 0 && lane == 0) {
                atomicMax(b.r2 + node, __float_as_uint(v[0]));
                for (int i = 0; i < 6; i++) atomicAdd(b.q + 6 * (int64_t)node + i, v[1 + i]);
                for (int i = 0; i < 6; i++) atomicMax(b.box + 6 * (int64_t)node + i, bx[i]);
            }
            // octant counts: lanes sharing (node, key)
            const unsigned g2 = __match_any_sync(0xffffffffu, node * 8 + key);
            if (node >= 0 && lane == __ffs(g2) - 1) atomicAdd(b.oct + 8 * (int64_t)node + key, __popc(g2));
        }
        __syncthreads();  // s_node, s_f, s_k and s_oct are reused by the next iteration
    }
}

// Takes nch node ids, or -1 when they do not fit (the build is flagged, and
// the ids up to the capacity become nodes that nothing refers to).
__device__ __forceinline__ int take_nodes(const Build &b, int nch, int32_t ncap) {
    const int first = atomicAdd(b.counter, nch);
    if (first + nch <= ncap) return first;
    atomicOr(b.counter + 1, 1);
    for (int id = first; id < ncap && id < first + nch; id++) {
        b.start[id] = b.count[id] = 0;
        b.halo[id] = -1;
    }
    return -1;
}

// Decides children, allocates them, and lays out [loose | children] ranges.
// last: the final level of a fixed-depth build: a node with a child that a
// further level would have to process keeps all its particles loose and flags
// the build (counter[1]).
__global__ void split_nodes(int L, int32_t ncap, int last, Build b) {
    if (b.nact[L] == 0) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicMax(b.counter + 4, L + 1);
    FOR_LEVEL_NODES(node, L, b) {
    if (b.count[node] <= kSmall) continue;
    {
        double x, y, z;
        centre_of(b, node, x, y, z);
        b.mx[node] = x;
        b.my[node] = y;
        b.mz[node] = z;
    }
    const float r2 = __uint_as_float(b.r2[node]);
    const double nodesize = sqrt((double)r2);           // ost.c:574
    const bool divide = nodesize > 0.5 * kMinWidth;     // divideThisNode, tree.h:36
    int cnt[8], cur[8], child_of[8], nch = 0;
    {
        const int4 *o = reinterpret_cast<const int4 *>(b.oct + 8 * (int64_t)node);
        const int4 o0 = o[0], o1 = o[1];
        cnt[0] = o0.x; cnt[1] = o0.y; cnt[2] = o0.z; cnt[3] = o0.w;
        cnt[4] = o1.x; cnt[5] = o1.y; cnt[6] = o1.z; cnt[7] = o1.w;
    }
#pragma unroll
    for (int c = 0; c < 8; c++)
        if (divide && cnt[c] >= kMinCell) nch++;
    int nbig = 0;
#pragma unroll
    for (int c = 0; c < 8; c++)
        if (divide && cnt[c] > kSmall) nbig++;
    if (last && nbig > 0) {
        atomicOr(b.counter + 1, 2);
        nch = nbig = 0;
    }
    int first = -1;
    if (nch > 0) {
        first = take_nodes(b, nch, ncap);
        if (first < 0) nch = nbig = 0;  // out of node capacity: keep all particles loose
    }
    if (nbig > 0) atomicAdd(b.nact + L + 1, nbig);
    int small_at = nch > nbig ? atomicAdd(b.counter + 3, nch - nbig) : 0;
    const int start = b.start[node], halo = b.halo[node];
    int off = start;
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const bool child = nch > 0 && divide && cnt[c] >= kMinCell;
        child_of[c] = -1;
        if (!child) {
            cur[c] = off;
            off += cnt[c];
        }
    }
    b.lstart[node] = start;
    b.lcount[node] = off - start;
    int k = 0;
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const bool child = nch > 0 && divide && cnt[c] >= kMinCell;
        if (child) {
            const int id = first + k++;
            cur[c] = off;
            b.start[id] = off;
            b.count[id] = cnt[c];
            b.halo[id] = halo;
            b.par[id] = node;
            if (cnt[c] > kSmall) {
                child_of[c] = id;
                zero_node(b, id);
            } else {  // its particles go to the final arrays, as loose ones
                b.first[id] = L + 1;
                b.small[small_at++] = id;
            }
            off += cnt[c];
        }
    }
    {
        int4 *u = reinterpret_cast<int4 *>(b.cur + 8 * (int64_t)node);
        int4 *v = reinterpret_cast<int4 *>(b.ochild + 8 * (int64_t)node);
        u[0] = make_int4(cur[0], cur[1], cur[2], cur[3]);
        u[1] = make_int4(cur[4], cur[5], cur[6], cur[7]);
        v[0] = make_int4(child_of[0], child_of[1], child_of[2], child_of[3]);
        v[1] = make_int4(child_of[4], child_of[5], child_of[6], child_of[7]);
    }
    b.first[node] = first;
    b.nchild[node] = nch;
    }
    // the last block to finish writes the next level's end: the nodes this
    // level allocated (its children are numbered [lev[L+1], lev[L+2]))
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(b.counter + 2, 1) == (int)gridDim.x - 1) {
            b.lev[L + 2] = min(atomicAdd(b.counter, 0), ncap);
            b.counter[2] = 0;  // for the next level's launch
        }
    }
}

// Moves the active particles into [loose | child 0 | child 1 | ...] order.
// A particle that stays loose here has its final tree-order slot: it is
// written once into the final arrays (fpos, fperm) and never copied again;
// its slot, like every earlier-settled one, carries node -1 into the next
// level.  So do the particles of small children.
__global__ void scatter_particles(int L, int64_t n, const float4 *__restrict__ pos_in,
                                  const int32_t *__restrict__ perm_in,
                                  const int32_t *__restrict__ pnode_in,
                                  const uint8_t *__restrict__ pkey, float4 *__restrict__ pos_out,
                                  int32_t *__restrict__ perm_out, int32_t *__restrict__ pnode_out,
                                  float4 *__restrict__ fpos, int32_t *__restrict__ fperm, Build b) {
    if (b.nact[L] == 0) return;
    const int lane = threadIdx.x & 31;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p - lane < n;
         p += (int64_t)gridDim.x * blockDim.x) {
        const int node = p < n ? pnode_in[p] : -2;
        const int key = node >= 0 ? pkey[p] : 0;
        const unsigned g = __match_any_sync(0xffffffffu, node * 8 + key);
        if (p >= n) continue;
        if (node < 0) {  // settled at an earlier level: already in the final arrays
            pnode_out[p] = -1;
            continue;
        }
        const int leader = __ffs(g) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(b.cur + 8 * (int64_t)node + key, __popc(g));
        base = __shfl_sync(g, base, leader);
        const int dest = base + __popc(g & ((1u << lane) - 1));
        const int child = b.ochild[8 * (int64_t)node + key];
        if (child >= 0) {
            pos_out[dest] = pos_in[p];
            perm_out[dest] = perm_in[p];
        } else {
            fpos[dest] = pos_in[p];
            fperm[dest] = perm_in[p];
        }
        pnode_out[dest] = child;
    }
}

// ---- subtrees of small nodes
struct SmallWarp {
    float4 pos[2][kSmall];
    int32_t perm[2][kSmall];
    int4 stack[kSmall / kMinCell + 1];  // (node, first place, particles, levels below the root); pending nodes are disjoint
};
constexpr int kSmallWarps = 4;

// Field key of eight 16-bit fields in four words.
__device__ __forceinline__ unsigned field16(const unsigned (&w)[4], int key) {
    const unsigned a = key & 2 ? w[1] : w[0], c = key & 2 ? w[3] : w[2];
    return ((key & 4 ? c : a) >> (16 * (key & 1))) & 0xffffu;
}

// One warp per node of at most kSmall particles: the node and all its
// descendants, with the rules and formulas of the level passes (accum_mass,
// accum_moments, split_nodes).  The particles sit in one of two shared
// buffers; a node's lanes reduce its moments, and place every particle behind
// its octant's lower lanes: loose ones into the final arrays, those of
// children into the other buffer.
__global__ void __launch_bounds__(32 * kSmallWarps)
small_subtrees(int32_t ncap, int q5_asbuilt, float4 *__restrict__ fpos, int32_t *__restrict__ fperm, Build b) {
    __shared__ SmallWarp warps[kSmallWarps];
    SmallWarp &W = warps[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int nsmall = b.counter[3];
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nsmall; i += (gridDim.x * blockDim.x) >> 5) {
        const int root = b.small[i];
        const int start = b.start[root], halo = b.halo[root], level = b.first[root];
        int depth = 0;
        for (int k = lane; k < b.count[root]; k += 32) {
            W.pos[0][k] = fpos[start + k];
            W.perm[0][k] = fperm[start + k];
        }
        if (lane == 0) W.stack[0] = make_int4(root, 0, b.count[root], 0);
        __syncwarp();
        int top = 1;
        while (top > 0) {
            const int4 e = W.stack[--top];
            const int node = e.x, off = e.y, cnt = e.z, buf = e.w & 1;
            depth = max(depth, e.w);
            const float4 *X = W.pos[buf] + off;
            const int32_t *id = W.perm[buf] + off;
            // ost.c:546-555: mass, mass-weighted position, centre of mass
            double w = 0, cx = 0, cy = 0, cz = 0;
            for (int k = lane; k < cnt; k += 32) {
                const float4 v = X[k];
                w += v.w;
                cx += (double)v.w * (double)v.x;
                cy += (double)v.w * (double)v.y;
                cz += (double)v.w * (double)v.z;
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                w += __shfl_xor_sync(0xffffffffu, w, o);
                cx += __shfl_xor_sync(0xffffffffu, cx, o);
                cy += __shfl_xor_sync(0xffffffffu, cy, o);
                cz += __shfl_xor_sync(0xffffffffu, cz, o);
            }
            if (w > 0) {
                cx /= w;
                cy /= w;
                cz /= w;
            }
            // ost.c:561-571, 589-592: float offsets and moments, octants
            float r2 = 0.f, q[6] = {0, 0, 0, 0, 0, 0};
            unsigned bx[6] = {0u, 0u, 0u, 0u, 0u, 0u};  // ~min xyz, max xyz: all maxima
            unsigned keys = 0, oct = 0;  // octant of each own particle (3 bits), own particles per octant (4 bits)
            for (int k = lane, u = 0; k < cnt; k += 32, u += 3) {
                const float4 P = X[k];
                const float tx = (float)((double)P.x - cx);
                const float ty = (float)((double)P.y - cy);
                const float tz = (float)((double)P.z - cz);
                const float m = P.w;
                r2 = fmaxf(r2, offset2(tx, ty, tz));
                q[0] += m * tx * tx;
                q[1] += m * ty * ty;
                q[2] += m * tz * tz;
                q[3] += m * tx * ty;
                q[4] += m * tx * tz;
                q[5] += q5_asbuilt ? m * ty * tx : m * ty * tz;
                const unsigned fx = fkey(P.x), fy = fkey(P.y), fz = fkey(P.z);
                bx[0] = max(bx[0], ~fx);
                bx[1] = max(bx[1], ~fy);
                bx[2] = max(bx[2], ~fz);
                bx[3] = max(bx[3], fx);
                bx[4] = max(bx[4], fy);
                bx[5] = max(bx[5], fz);
                const unsigned key = ((double)P.x > cx ? 1 : 0) | ((double)P.y > cy ? 2 : 0) | ((double)P.z > cz ? 4 : 0);
                keys |= key << u;
                oct += 1u << (4 * key);
            }
            const unsigned r2b = __reduce_max_sync(0xffffffffu, __float_as_uint(r2));  // non-negative floats
#pragma unroll
            for (int a = 0; a < 6; a++) {
                bx[a] = __reduce_max_sync(0xffffffffu, bx[a]);
#pragma unroll
                for (int o = 16; o; o >>= 1) q[a] += __shfl_xor_sync(0xffffffffu, q[a], o);
            }
            // particles of every octant in the lanes up to this one: two
            // 16-bit counts per word
            unsigned at[4], sum[4];
#pragma unroll
            for (int a = 0; a < 4; a++) {
                const unsigned own = ((oct >> (8 * a)) & 15u) | (((oct >> (8 * a + 4)) & 15u) << 16);
                unsigned v = own;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned t = __shfl_up_sync(0xffffffffu, v, o);
                    if (lane >= o) v += t;
                }
                sum[a] = __shfl_sync(0xffffffffu, v, 31);
                at[a] = v - own;  // in the lanes before
            }
            // ost.c:574, tree.h:36: children are octants of at least kMinCell
            // particles of a node that is large enough
            const bool divide = sqrt((double)__uint_as_float(r2b)) > 0.5 * kMinWidth;
            unsigned child = 0;  // octants that become children
#pragma unroll
            for (int c = 0; c < 8; c++)
                if (divide && ((sum[c >> 1] >> (16 * (c & 1))) & 0xffffu) >= (unsigned)kMinCell) child |= 1u << c;
            int first = -1;
            if (child && level + e.w + 2 > kMaxLevels) {  // only non-finite or degenerate particles nest like this
                if (lane == 0) atomicOr(b.counter + 1, 4);
                child = 0;
            }
            if (child) {
                if (lane == 0) first = take_nodes(b, __popc(child), ncap);
                first = __shfl_sync(0xffffffffu, first, 0);
                if (first < 0) child = 0;  // out of node capacity: keep all particles loose
            }
            // [loose | child 0 | child 1 | ...]: places of the octants, added
            // to the counts of the lanes before
            int place = 0, nloose = 0;
            __syncwarp();  // every lane has read this node's stack entry
#pragma unroll
            for (int pass = 0; pass < 2; pass++) {
                int k = 0;
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const int n = (sum[c >> 1] >> (16 * (c & 1))) & 0xffffu;
                    const bool is_child = (child >> c) & 1u;
                    if (is_child != (pass == 1)) continue;
                    at[c >> 1] += (unsigned)place << (16 * (c & 1));
                    if (is_child) {
                        if (lane == 0) {
                            const int kid = first + k;
                            W.stack[top + k] = make_int4(kid, off + place, n, e.w + 1);
                            b.start[kid] = start + off + place;
                            b.count[kid] = n;
                            b.halo[kid] = halo;
                            b.par[kid] = node;
                        }
                        k++;
                    }
                    place += n;
                }
                if (pass == 0) nloose = place;
            }
            top += __popc(child);
            unsigned seen = 0;  // own particles placed, per octant
            for (int k = lane; k < cnt; k += 32, keys >>= 3) {
                const int key = keys & 7;
                const int dst = (int)field16(at, key) + (int)((seen >> (4 * key)) & 15u);
                seen += 1u << (4 * key);
                const float4 v = X[k];
                const int32_t pi = id[k];
                if ((child >> key) & 1u) {
                    W.pos[buf ^ 1][off + dst] = v;
                    W.perm[buf ^ 1][off + dst] = pi;
                } else {
                    fpos[start + off + dst] = v;
                    fperm[start + off + dst] = pi;
                }
            }
            if (lane == 0) {
                b.m[node] = w;
                b.mx[node] = cx;
                b.my[node] = cy;
                b.mz[node] = cz;
                b.r2[node] = r2b;
#pragma unroll
                for (int a = 0; a < 6; a++) {
                    b.q[6 * (int64_t)node + a] = q[a];
                    b.box[6 * (int64_t)node + a] = bx[a];
                }
                b.first[node] = first;
                b.nchild[node] = __popc(child);
                b.lstart[node] = start + off;
                b.lcount[node] = nloose;
            }
            __syncwarp();  // the stack and the other buffer are written
        }
        if (lane == 0) atomicMax(b.counter + 4, level + depth + 1);
    }
}

// ---- numbering
// hist[p]: nodes whose first particle is p (nodes without particles apart).
__global__ void count_starts(int32_t ncap, Build b, int32_t *__restrict__ hist) {
    const int nn = min(b.counter[0], ncap);
    for (int node = blockIdx.x * blockDim.x + threadIdx.x; node < nn; node += gridDim.x * blockDim.x)
        if (b.count[node] > 0) atomicAdd(hist + b.start[node], 1);
}

constexpr int kScanThreads = 256, kScanItems = 16, kScanChunk = kScanThreads * kScanItems;

// Exclusive scan of `v` over the block's threads; `total` receives the sum.
template <int THREADS>
__device__ __forceinline__ int block_scan(int v, int &total, int *scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) scratch[warp] = inc;
    __syncthreads();
    int before = 0;
    total = 0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; w++) {
        if (w < warp) before += scratch[w];
        total += scratch[w];
    }
    __syncthreads();  // scratch is reused
    return before + inc - v;
}

__global__ void __launch_bounds__(kScanThreads)
scan_sums(int64_t n, const int32_t *__restrict__ hist, int32_t *__restrict__ sums) {
    __shared__ int scratch[kScanThreads / 32];
    const int64_t base = blockIdx.x * (int64_t)kScanChunk;
    int v = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        const int64_t p = base + threadIdx.x + i * kScanThreads;
        if (p < n) v += hist[p];
    }
    int total;
    block_scan<kScanThreads>(v, total, scratch);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// Per halo, the halos before it without particles (their roots are nodes too).
__device__ __forceinline__ void scan_empty(int32_t nhalo, const int64_t *__restrict__ pstart,
                                           int32_t *__restrict__ empty, int *scratch) {
    int run = 0, total;
    for (int32_t c = 0; c < nhalo; c += 1024) {
        const int h = c + threadIdx.x;
        const int v = h < nhalo && pstart[h] == pstart[h + 1];
        const int at = run + block_scan<1024>(v, total, scratch);
        if (h < nhalo) empty[h] = at;
        run += total;
    }
}

// Small batches: all of the numbering's counts and scans in one block, in place
// of a memset and four launches (the stage on 120 particles 185 us, now 172).
constexpr int kNumberMax = 8192;
__global__ void __launch_bounds__(1024)
number_small(int32_t ncap, int32_t n, Build b, int32_t nhalo, const int64_t *__restrict__ pstart,
             int32_t *__restrict__ before, int32_t *__restrict__ empty) {
    constexpr int kItems = kNumberMax / 1024 + 1;  // of the n + 1 entries
    __shared__ int hist[kItems * 1024];
    __shared__ int scratch[32];
    for (int p = threadIdx.x; p < kItems * 1024; p += 1024) hist[p] = 0;
    __syncthreads();
    const int nn = min(b.counter[0], ncap);
    for (int node = threadIdx.x; node < nn; node += 1024)
        if (b.count[node] > 0) atomicAdd(hist + b.start[node], 1);
    __syncthreads();
    int v[kItems], sum = 0, total;
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        v[i] = hist[threadIdx.x * kItems + i];
        sum += v[i];
    }
    int at = block_scan<1024>(sum, total, scratch);
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        const int p = threadIdx.x * kItems + i;
        if (p <= n) before[p] = at;
        at += v[i];
    }
    scan_empty(nhalo, pstart, empty, scratch);
}

// The chunk sums (in place) and, per halo, the halos before it without
// particles (their roots are nodes too), as exclusive prefixes: one block.
__global__ void __launch_bounds__(1024)
scan_mid(int64_t nchunk, int32_t *__restrict__ sums, int32_t nhalo, const int64_t *__restrict__ pstart,
         int32_t *__restrict__ empty) {
    __shared__ int scratch[32];
    int run = 0, total;
    for (int64_t c = 0; c < nchunk; c += 1024) {
        const int v = c + threadIdx.x < nchunk ? sums[c + threadIdx.x] : 0;
        const int at = run + block_scan<1024>(v, total, scratch);
        if (c + threadIdx.x < nchunk) sums[c + threadIdx.x] = at;
        run += total;
    }
    scan_empty(nhalo, pstart, empty, scratch);
}

__global__ void __launch_bounds__(kScanThreads)
scan_chunks(int64_t n, int32_t *__restrict__ hist, const int32_t *__restrict__ sums) {
    __shared__ int scratch[kScanThreads / 32];
    const int64_t base = blockIdx.x * (int64_t)kScanChunk + threadIdx.x * (int64_t)kScanItems;
    int v[kScanItems], s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        v[i] = base + i < n ? hist[base + i] : 0;
        s += v[i];
    }
    int total;
    int at = sums[blockIdx.x] + block_scan<kScanThreads>(s, total, scratch);
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        if (base + i < n) hist[base + i] = at;
        at += v[i];
    }
}

// Preorder number of a node and its subtree's size.  before[p]: nodes with
// particles that start before particle p.
__device__ __forceinline__ int2 number_of(const Build &b, const int32_t *__restrict__ before,
                                          const int32_t *__restrict__ empty, int node) {
    const int s = b.start[node], c = b.count[node], h = b.halo[node];
    if (c == 0) return make_int2(before[s] + empty[h], 1);
    int above = 0;  // ancestors that start with the same particle
    for (int p = b.par[node]; p >= 0 && b.start[p] == s; p = b.par[p]) above++;
    return make_int2(before[s] + above + empty[h], before[s + c] - before[s] - above);
}

// fixed: flag a build that the batch outgrew (a node of the last level that
// would have split into large ones, or the node capacity exceeded); the tree
// is consistent either way (those particles stay loose).
__global__ void emit_nodes(int32_t ncap, float theta2, Build b, const int32_t *__restrict__ before,
                           const int32_t *__restrict__ empty, int32_t nhalo, KnnNode *__restrict__ knn,
                           BhNode *__restrict__ bh, WalkNode *__restrict__ walk, int32_t *__restrict__ owner,
                           int32_t *__restrict__ root, int32_t *__restrict__ rend, int fixed, int *err) {
    if (fixed && blockIdx.x == 0 && threadIdx.x == 0 && b.counter[1]) atomicOr(err, GF_ERRBIT_PLAN);
    const int nn = min(b.counter[0], ncap);
    for (int node = blockIdx.x * blockDim.x + threadIdx.x; node < nn; node += gridDim.x * blockDim.x) {
    if (b.halo[node] < 0) continue;  // an id that the capacity cut off
    const int2 num = number_of(b, before, empty, node);
    const int i = num.x;
    if (node < nhalo) {
        root[node] = i;
        rend[node] = i + num.y;
    }
    KnnNode k;
    for (int a = 0; a < 3; a++) {
        k.lo[a] = fkey_inv(~b.box[6 * (int64_t)node + a]);
        k.hi[a] = fkey_inv(b.box[6 * (int64_t)node + 3 + a]);
    }
    k.skip = i + num.y;
    k.lstart = b.lstart[node];
    k.lcount = b.lcount[node];
    k.count = b.count[node];
    k.parent = b.par[node] >= 0 ? number_of(b, before, empty, b.par[node]).x : -1;
    k.pad = 0;
    for (int j = 0; j < k.lcount; j++) owner[k.lstart + j] = i;
    knn[i] = k;
    BhNode h;
    h.com[0] = b.mx[node];
    h.com[1] = b.my[node];
    h.com[2] = b.mz[node];
    // ost.c:573,80: dist2 = (double)distmax (a float); ratio = dist2/theta2
    // Where that is 0 the node's particles all lie at its centre, to within
    // offsets whose squares underflow a float: opened by a target there, which
    // gets the particles' terms (none) instead of a cell's at distance zero.
    // Whether such a centre rounds to the particles' very position depends on
    // the order of its sums, so their potential was finite or not by chance.
    const float far2 = __uint_as_float(b.r2[node]);
    h.open_r2 = far2 > 0.f ? (double)far2 / (double)theta2 : 4e-45;  // 3 * 2^-150 < 4e-45
    h.mass = (float)b.m[node];
    float q[6];
    for (int a = 0; a < 6; a++) q[a] = b.q[6 * (int64_t)node + a];
    for (int a = 0; a < 6; a++) h.q[a] = q[a];
    h.trq = q[0] + q[1] + q[2];
    h.skip = k.skip;
    h.lstart = k.lstart;
    h.lcount = k.lcount;
    h.count = k.count;
    bh[i] = h;
    WalkNode w;
    w.hx = (float)h.com[0];
    w.hy = (float)h.com[1];
    w.hz = (float)h.com[2];
    w.open_lo = __double2float_rd(h.open_r2 * (1.0 - 2e-6));
    if (w.open_lo < kWalkMinR2) w.open_lo = 0.f;
    w.first = b.first[node];
    w.nchild = b.nchild[node];
    w.lstart = h.lstart;
    w.lcount = h.lcount;
    w.lx = (float)(h.com[0] - (double)w.hx);
    w.ly = (float)(h.com[1] - (double)w.hy);
    w.lz = (float)(h.com[2] - (double)w.hz);
    w.mass = h.mass;
    w.pre = i;
    const double half_tr = 0.5 * ((double)q[0] + (double)q[1] + (double)q[2]);
    w.txx = (float)(1.5 * (double)q[0] - half_tr);
    w.tyy = (float)(1.5 * (double)q[1] - half_tr);
    w.tzz = (float)(1.5 * (double)q[2] - half_tr);
    w.txy = 3.f * q[3];
    w.txz = 3.f * q[4];
    w.tyz = 3.f * q[5];
    w.pad = 0;
    walk[node] = w;
    }
}

int grid_n(int64_t n) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + kBlock - 1) / kBlock, sm_count() * 8));
}
int grid_exact(int64_t n, int block) { return (int)std::max<int64_t>(1, (n + block - 1) / block); }

template <class T>
T *carve(char *&p, size_t count) {
    T *r = reinterpret_cast<T *>(p);
    p += (count * sizeof(T) + 255) & ~size_t(255);
    return r;
}

}  // namespace

int build_tree(gf_ctx *ctx, int32_t nhalo, int64_t n, const int64_t *pstart_dev,
               const float4 *pos_in, float theta2, int q5_asbuilt, TreeView *out,
               const TreeShape *fixed, TreeShape *shape, const std::function<int()> &before_wait) {
    bool waited = !before_wait;  // else the caller queues its own work before the host first waits
    if (n > 0x7fffffffLL) {
        set_status(GF_ENOTIMPL, "tree build over more than 2^31 particles in one batch");
        return GF_ENOTIMPL;
    }
    if (fixed && (fixed->levels < 1 || fixed->levels > kMaxLevels || fixed->ncap < nhalo)) {
        set_status(GF_EINVAL, "fixed tree shape: %d levels, %lld nodes", fixed ? fixed->levels : 0,
                   fixed ? (long long)fixed->ncap : 0LL);
        return GF_EINVAL;
    }
    int64_t ncap = fixed ? fixed->ncap : n / 2 + 2LL * nhalo + 1024;
    for (int attempt = 0; attempt < (fixed ? 1 : 4); attempt++, ncap *= 2) {
        // ---- particle buffers: pos x2, perm x2, pnode x2, key
        auto al = [](size_t v) { return (v + 255) & ~size_t(255); };
        const int64_t nscan = n + 1, nchunk = (nscan + kScanChunk - 1) / kScanChunk;
        const size_t pbytes = 3 * al(n * sizeof(float4)) + 6 * al(n * sizeof(int32_t)) + al(n) +
                              al(nscan * sizeof(int32_t)) + al(nchunk * sizeof(int32_t)) +
                              al(std::max(nhalo, 1) * sizeof(int32_t));
        GF_TRY(ctx->tree[0].reserve(pbytes + 256));
        char *pp = ctx->tree[0].as<char>();
        float4 *pos[2] = {carve<float4>(pp, n), carve<float4>(pp, n)};
        int32_t *perm[2] = {carve<int32_t>(pp, n), carve<int32_t>(pp, n)};
        int32_t *pnode[2] = {carve<int32_t>(pp, n), carve<int32_t>(pp, n)};
        uint8_t *pkey = carve<uint8_t>(pp, n);
        float4 *fpos = carve<float4>(pp, n);    // final tree order, written as particles settle
        int32_t *fperm = carve<int32_t>(pp, n);
        int32_t *phalo = carve<int32_t>(pp, n);
        int32_t *before = carve<int32_t>(pp, nscan);  // nodes starting at, then before, each particle
        int32_t *sums = carve<int32_t>(pp, nchunk);
        int32_t *empty = carve<int32_t>(pp, std::max(nhalo, 1));
        // ---- node buffers (BFS numbering): exactly the carves below
        const size_t nc = (size_t)ncap;
        const size_t nbytes = 3 * al(nc * 4) + 4 * al(nc * 8) + al(nc * 4) + al(nc * 24) +
                              al(nc * 24) + 3 * al(nc * 32) + 6 * al(nc * 4) + al(64) +
                              2 * al((kMaxLevels + 2) * sizeof(int32_t));
        GF_TRY(ctx->tree[1].reserve(nbytes + 256));
        char *np_ = ctx->tree[1].as<char>();
        Build b;
        b.start = carve<int32_t>(np_, nc);
        b.count = carve<int32_t>(np_, nc);
        b.halo = carve<int32_t>(np_, nc);
        b.m = carve<double>(np_, nc);
        b.mx = carve<double>(np_, nc);
        b.my = carve<double>(np_, nc);
        b.mz = carve<double>(np_, nc);
        b.r2 = carve<unsigned>(np_, nc);
        b.q = carve<float>(np_, nc * 6);
        b.box = carve<unsigned>(np_, nc * 6);
        b.oct = carve<int32_t>(np_, nc * 8);
        b.cur = carve<int32_t>(np_, nc * 8);
        b.ochild = carve<int32_t>(np_, nc * 8);
        b.first = carve<int32_t>(np_, nc);
        b.nchild = carve<int32_t>(np_, nc);
        b.lstart = carve<int32_t>(np_, nc);
        b.lcount = carve<int32_t>(np_, nc);
        b.par = carve<int32_t>(np_, nc);
        b.small = carve<int32_t>(np_, nc);
        b.counter = carve<int32_t>(np_, 16);
        b.nact = carve<int32_t>(np_, kMaxLevels + 2);
        char *const zero_end = np_;
        b.lev = carve<int32_t>(np_, kMaxLevels + 2);
        cudaStream_t s = ctx->stream;
        GF_CUDA_TRY(cudaMemsetAsync(b.counter, 0, zero_end - (char *)b.counter, s));
        if (n > kNumberMax) GF_CUDA_TRY(cudaMemsetAsync(before, 0, nscan * sizeof(int32_t), s));
        init_build<<<grid_n(std::max<int64_t>(n, nhalo)), kBlock, 0, s>>>(n, pstart_dev, nhalo, pos_in, pos[0], perm[0],
                                                                          pnode[0], fpos, fperm, phalo, b);
        GF_LAUNCH_CHECK();
        // Level by level.  Eagerly, the host looks after every third level
        // whether a level is left (levels past the last one return at once);
        // with a fixed shape fixed->levels levels run without a host round
        // trip and emit_nodes flags a tree that needed more levels or nodes.
        // A batch of at most kSmall particles has no node for these passes.
        const int fixed_grid = sm_count() * 4;
        const int level_grid = (int)std::min<int64_t>(fixed_grid, std::max<int64_t>(n / 4096, nhalo / 256) + 1);
        int cur = 0;
        int32_t hc[16] = {0}, act = 0;
        bool more = fixed || n > kSmall;
        for (int L = 0; more; L++) {
            if (fixed ? L == fixed->levels : L >= kMaxLevels) {
                if (fixed) break;
                set_status(GF_EINVAL, "octree deeper than %d levels", kMaxLevels);
                return GF_EINVAL;
            }
            accum_mass<<<grid_n(n), kBlock, 0, s>>>(L, n, pos[cur], pnode[cur], b);
            GF_LAUNCH_CHECK();
            accum_moments<<<grid_n(n), kBlock, 0, s>>>(L, n, pos[cur], pnode[cur], pkey, q5_asbuilt, b);
            GF_LAUNCH_CHECK();
            split_nodes<<<level_grid, 256, 0, s>>>(L, (int32_t)ncap, fixed && L == fixed->levels - 1, b);
            GF_LAUNCH_CHECK();
            scatter_particles<<<grid_n(n), kBlock, 0, s>>>(L, n, pos[cur], perm[cur], pnode[cur], pkey,
                                                           pos[cur ^ 1], perm[cur ^ 1],
                                                           pnode[cur ^ 1], fpos, fperm, b);
            GF_LAUNCH_CHECK();
            cur ^= 1;
            if (fixed || L % 3 != 2) continue;
            if (!waited) GF_TRY(before_wait());
            waited = true;
            GF_CUDA_TRY(cudaMemcpyAsync(&act, b.nact + L + 1, sizeof(act), cudaMemcpyDeviceToHost, s));
            GF_CUDA_TRY(cudaStreamSynchronize(s));
            more = act > 0;
        }
        small_subtrees<<<fixed ? sm_count() * 5 : (int)std::max<int64_t>(1, std::min<int64_t>(n / 64 + nhalo / 4 + 1, sm_count() * 5)),
                         32 * kSmallWarps, 0, s>>>((int32_t)ncap, q5_asbuilt, fpos, fperm, b);
        GF_LAUNCH_CHECK();
        int32_t nnode = -1;
        if (!fixed) {
            if (!waited) GF_TRY(before_wait());
            waited = true;
            GF_CUDA_TRY(cudaMemcpyAsync(hc, b.counter, sizeof(hc), cudaMemcpyDeviceToHost, s));
            GF_CUDA_TRY(cudaStreamSynchronize(s));
            if (hc[1] & 4) {
                set_status(GF_EINVAL, "octree deeper than %d levels", kMaxLevels);
                return GF_EINVAL;
            }
            if (hc[1]) continue;  // node capacity exceeded: retry with more nodes
            nnode = hc[0];
        }
        const int node_grid = fixed ? fixed_grid : grid_exact(nnode, 256);
        if (n <= kNumberMax) {
            number_small<<<1, 1024, 0, s>>>((int32_t)ncap, (int32_t)n, b, nhalo, pstart_dev, before, empty);
            GF_LAUNCH_CHECK();
        } else {
            count_starts<<<node_grid, 256, 0, s>>>((int32_t)ncap, b, before);
            GF_LAUNCH_CHECK();
            scan_sums<<<(unsigned)nchunk, kScanThreads, 0, s>>>(nscan, before, sums);
            GF_LAUNCH_CHECK();
            scan_mid<<<1, 1024, 0, s>>>(nchunk, sums, nhalo, pstart_dev, empty);
            GF_LAUNCH_CHECK();
            scan_chunks<<<(unsigned)nchunk, kScanThreads, 0, s>>>(nscan, before, sums);
            GF_LAUNCH_CHECK();
        }
        if (shape) {
            shape->levels = std::max(hc[4], 1);
            shape->ncap = ncap;
            shape->nnode = nnode;
        }
        // ---- output buffers
        const int64_t nout = fixed ? ncap : std::max(nnode, 1);  // node slots written
        const size_t obytes = al((size_t)nout * sizeof(KnnNode)) + al((size_t)nout * sizeof(BhNode)) +
                              al((size_t)nout * sizeof(WalkNode)) +
                              2 * al((size_t)std::max(nhalo, 1) * 4) + al((size_t)std::max<int64_t>(n, 1) * 4);
        GF_TRY(ctx->tree[2].reserve(obytes + 256));
        char *op = ctx->tree[2].as<char>();
        KnnNode *knn = carve<KnnNode>(op, (size_t)nout);
        BhNode *bh = carve<BhNode>(op, (size_t)nout);
        WalkNode *walk = carve<WalkNode>(op, (size_t)nout);
        int32_t *root = carve<int32_t>(op, std::max(nhalo, 1));
        int32_t *rend = carve<int32_t>(op, std::max(nhalo, 1));
        int32_t *owner = carve<int32_t>(op, std::max<int64_t>(n, 1));
        if (fixed || nnode > 0) {
            emit_nodes<<<node_grid, 256, 0, s>>>((int32_t)ncap, theta2, b, before, empty, nhalo, knn, bh, walk, owner,
                                                 root, rend, fixed ? 1 : 0, ctx->d_err);
            GF_LAUNCH_CHECK();
        }
        out->nhalo = nhalo;
        out->nnode = nnode;
        out->n = n;
        out->pos = fpos;
        out->perm = fperm;
        out->root = root;
        out->rend = rend;
        out->knn = knn;
        out->bh = bh;
        out->walk = walk;
        out->phalo = phalo;
        out->owner = owner;
        return GF_OK;
    }
    set_status(GF_ENOMEM, "octree node capacity exhausted");
    return GF_ENOMEM;
}

int export_tree(gf_ctx *ctx, const TreeView &t, void *knn_host, void *bh_host, float4 *pos_host,
                int32_t *perm_host, int32_t *root_host, int32_t *rend_host) {
    cudaStream_t s = ctx->stream;
    if (knn_host)
        GF_CUDA_TRY(cudaMemcpyAsync(knn_host, t.knn, sizeof(KnnNode) * t.nnode, cudaMemcpyDeviceToHost, s));
    if (bh_host)
        GF_CUDA_TRY(cudaMemcpyAsync(bh_host, t.bh, sizeof(BhNode) * t.nnode, cudaMemcpyDeviceToHost, s));
    if (pos_host)
        GF_CUDA_TRY(cudaMemcpyAsync(pos_host, t.pos, sizeof(float4) * t.n, cudaMemcpyDeviceToHost, s));
    if (perm_host)
        GF_CUDA_TRY(cudaMemcpyAsync(perm_host, t.perm, sizeof(int32_t) * t.n, cudaMemcpyDeviceToHost, s));
    if (root_host)
        GF_CUDA_TRY(cudaMemcpyAsync(root_host, t.root, sizeof(int32_t) * t.nhalo, cudaMemcpyDeviceToHost, s));
    if (rend_host)
        GF_CUDA_TRY(cudaMemcpyAsync(rend_host, t.rend, sizeof(int32_t) * t.nhalo, cudaMemcpyDeviceToHost, s));
    GF_CUDA_TRY(cudaStreamSynchronize(s));
    return GF_OK;
}

}  // namespace gf
