// tree.cu -- bounding box, keys, key sort, key-built octree and FP64 moments.
//
// Replaces the reference's insertion build (3D/CUDA/CUDA_NBody/src/Kernels.cu:157-377),
// its bounding box (:67-154), centre of mass (:381-399) and sort (:403-456) with a
// sort-based construction that produces the same tree:
//
//  keys     each body replays the reference's float subdivision (:200-258) for 21
//           levels; the child codes c = [x<mid] + 2[y<mid] + 4[z<mid] packed most
//           significant first give a 63-bit key whose ascending order is the
//           reference's in-order body order.  Bodies sharing all 21 levels are
//           refined to 42 levels (k_refine).
//  delta    delta(i) = number of leading levels sorted neighbours i, i+1 share.
//           A cell (a region holding >= 2 bodies) at level L starts at sorted
//           position a iff delta(a-1) < L <= delta(a); the body at position i sits
//           at level max(delta(i-1), delta(i)) + 1.  Position i therefore owns the
//           node levels lo..hi = delta(i-1)+1 .. max(delta(i-1),delta(i))+1.
//  nodes    in breadth-first order a node's index is the start of its level plus
//           the number of that level's nodes at earlier positions, so per-block
//           counts of the nodes of every level (k_delta) give every index without
//           materialising and sorting the entries.
//  links    a cell (level l, position p) has its first child at (l + 1, p); the
//           topmost node of a position that shares levels with its predecessor
//           is a later child of the last level-(lo-1) node before it.  Both are
//           ranks in their levels, so the thread of p links its nodes by itself
//           (k_nodes) -- no search, no locks, no sort.
//  moments  bottom-up FP64 sums in child order, deterministic: one BFS level
//           per launch, deepest first, or for small systems one launch in
//           which the last child to finish sums its parent.
#include <cooperative_groups.h>

#include "nbx_internal.cuh"
#include "quotient.cuh"

namespace nbx {

namespace cg = cooperative_groups;

namespace {

constexpr int kBlock = 256;
#ifndef NBX_MOMENTS_UP_MAX
#define NBX_MOMENTS_UP_MAX (1 << 21)
#endif
constexpr int kMomentsUpMaxBodies = NBX_MOMENTS_UP_MAX;  // one-launch moments up to this many bodies
constexpr int kUpRounds = 4;    // largest number of 32-node rounds a warp of k_moments_up lists at once
constexpr int kLvlRow = 64;     // per-block counts of levels 0 .. kMaxLevel, padded to a row
static_assert(kLvlRow > kMaxLevel, "a row holds every level");
// k_nodes sums the earlier blocks' counts itself up to this many blocks: every
// block reads all rows, which beyond costs more than the scan's launch
constexpr int kDirectBlocks = 256;

__device__ __forceinline__ int grid_stride_start() { return blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ int grid_stride() { return gridDim.x * blockDim.x; }

// What a build starts from: the per-build counters of the status and of the
// systems, and the nodes' meta words, which k_nodes adds up.  Only the words of
// the array's previous tree are not zero (the array is cleared when it is made):
// clearing the whole pool took 0.5 ms of a 1000-body step in a context of 2^24.
__device__ __forceinline__ void reset_build(int nsys, DevStatus *st, int *sys_lvl, int *root_nch, int4 *meta4,
                                            int *meta, const unsigned *lvl_start) {
    const int i = grid_stride_start();
    const int used = (int)lvl_start[kLvlRow - 1];  // nodes of the previous tree
    for (int j = i; j < used / 4; j += grid_stride()) meta4[j] = make_int4(0, 0, 0, 0);
    if (i < (used & 3)) meta[(used & ~3) + i] = 0;
    for (int j = i; j < nsys; j += grid_stride()) {
        sys_lvl[j] = 0;
        root_nch[j] = 0;  // k_nodes counts the root children up
    }
    if (i == 0) {
        st->refined_runs = 0;
        st->max_level = 0;
        st->interactions = 0ull;
        st->opened = 0ull;
        st->rounds = 0ull;
        st->candidates = 0ull;
    }
}

__global__ void k_step_reset(int nsys, DevStatus *st, int *sys_lvl, int *root_nch, int4 *__restrict__ meta4,
                             int *__restrict__ meta, const unsigned *__restrict__ lvl_start) {
    grid_dependency();
    reset_build(nsys, st, sys_lvl, root_nch, meta4, meta, lvl_start);
}

__device__ __forceinline__ float depth0_of(float mnx, float mxx, float theta_ref) {
    float r = __fmul_rn(__fsub_rn(mxx, mnx), 0.5f);  // Kernels.cu:477
    return __fdiv_rn(__fmul_rn(r, r), theta_ref);    // Kernels.cu:513
}

// The boxes of all systems, and the build's reset, in one launch: per-tile
// min/max of the bodies of one system.  A system of one tile has its box at once;
// of several, they are merged with ordered-int atomics, and the system's last block
// to finish writes its box and walk threshold and leaves the scratch box empty
// (boxes contain the origin: Kernels.cu:56-62) and the system's block counter at
// zero for the next build.  (One last block for the boxes of all systems took as
// long as the rest of the build for 10^5 systems.)
__global__ void __launch_bounds__(kBlock) k_bbox(const float *__restrict__ x, const float *__restrict__ y,
                                                  const float *__restrict__ z, const int4 *__restrict__ tiles,
                                                  const int2 *__restrict__ sys_tiles, unsigned *bbox_u, int nsys,
                                                  float theta_ref, float *bbox, double *bbox64, float *depth0,
                                                  unsigned *done, DevStatus *st, int *sys_lvl, int *root_nch,
                                                  int4 *__restrict__ meta4, int *__restrict__ meta,
                                                  const unsigned *__restrict__ lvl_start) {
    grid_dependency();
    reset_build(nsys, st, sys_lvl, root_nch, meta4, meta, lvl_start);
    const int4 tl = tiles[blockIdx.x];
    const int s = tl.z, ntiles = sys_tiles[s].y;
    float v[6] = {INFINITY, -INFINITY, INFINITY, -INFINITY, INFINITY, -INFINITY};
    for (int i = threadIdx.x; i < tl.y; i += kBlock) {
        float a = x[tl.x + i], b = y[tl.x + i], c = z[tl.x + i];
        v[0] = fminf(v[0], a); v[1] = fmaxf(v[1], a);
        v[2] = fminf(v[2], b); v[3] = fmaxf(v[3], b);
        v[4] = fminf(v[4], c); v[5] = fmaxf(v[5], c);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < 6; k += 2) {
            v[k] = fminf(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
            v[k + 1] = fmaxf(v[k + 1], __shfl_xor_sync(0xffffffffu, v[k + 1], o));
        }
    }
    __shared__ float part[kBlock / 32][6], box[6];
    __shared__ bool last;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, k = threadIdx.x;
    if (lane == 0)
        for (int q = 0; q < 6; q++) part[w][q] = v[q];
    __syncthreads();
    if (k < 6) {
        float r = part[0][k];
        for (int q = 1; q < kBlock / 32; q++) r = (k & 1) ? fmaxf(r, part[q][k]) : fminf(r, part[q][k]);
        const bool finite = !isnan(r) && !isinf(r);
        if (ntiles == 1) {
            box[k] = !finite ? 0.0f : ((k & 1) ? fmaxf(r, 0.0f) : fminf(r, 0.0f));
        } else {
            if (finite) {
                unsigned *dst = &bbox_u[6 * s + k];
                if (k & 1) atomicMax(dst, f2ord(r));
                else atomicMin(dst, f2ord(r));
            }
            __threadfence();
        }
    }
    if (ntiles > 1) {  // uniform over the block
        __syncthreads();
        if (k == 0) {
            last = atomicAdd(&done[s], 1u) == (unsigned)ntiles - 1u;
            __threadfence();
        }
        __syncthreads();
        if (!last) return;
        if (k == 0) done[s] = 0u;
        if (k < 6) {
            box[k] = ord2f(__ldcg(&bbox_u[6 * s + k]));
            bbox_u[6 * s + k] = f2ord(0.0f);
        }
    }
    __syncthreads();
    if (k < 6) {
        const float b = __fadd_rn(box[k], 0.0f);  // -0 -> +0
        bbox[6 * s + k] = b;
        bbox64[6 * s + k] = (double)b;
        if (k == 0) depth0[s] = depth0_of(b, __fadd_rn(box[1], 0.0f), theta_ref);
    }
}

// Single-system box supplied by the caller (reference-compatible entry points).
__global__ void k_bbox_from_ptrs(const float *mnx, const float *mxx, const float *mny,
                                 const float *mxy, const float *mnz, const float *mxz,
                                 float theta_ref, float *bbox, double *bbox64, float *depth0,
                                 DevStatus *st) {
    grid_dependency();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    float b[6] = {*mnx, *mxx, *mny, *mxy, *mnz, *mxz};
    for (int k = 0; k < 6; k++) { bbox[k] = b[k]; bbox64[k] = (double)b[k]; }
    depth0[0] = depth0_of(b[0], b[1], theta_ref);
    st->refined_runs = 0;
    st->max_level = 0;
}

// Optional Hilbert order (key_order = 1).  The 12-state Lebesgue-to-Hilbert
// tables of the reference's domain-decomposition code
// (MolecularDynamics/BarnesHutParallel/SpaceFillingCurves/src/Tree.cpp:70-104),
// indexed by the Lebesgue child number b = [x>=mid] + 2[y>=mid] + 4[z>=mid]
// = 7 - c.  Digits map one-to-one per level, so two keys share a Hilbert prefix
// exactly when they share the Lebesgue one: the same cells, siblings reordered.
__constant__ unsigned char kHilbertDigit[12][8] = {
    {0, 7, 3, 4, 1, 6, 2, 5}, {4, 3, 7, 0, 5, 2, 6, 1}, {6, 1, 5, 2, 7, 0, 4, 3}, {2, 5, 1, 6, 3, 4, 0, 7},
    {0, 1, 7, 6, 3, 2, 4, 5}, {6, 7, 1, 0, 5, 4, 2, 3}, {2, 3, 5, 4, 1, 0, 6, 7}, {4, 5, 3, 2, 7, 6, 0, 1},
    {0, 3, 1, 2, 7, 4, 6, 5}, {2, 1, 3, 0, 5, 6, 4, 7}, {4, 7, 5, 6, 3, 0, 2, 1}, {6, 5, 7, 4, 1, 2, 0, 3}};
__constant__ unsigned char kHilbertState[12][8] = {
    {8, 10, 3, 3, 4, 5, 4, 5}, {2, 2, 11, 9, 4, 5, 4, 5}, {7, 6, 7, 6, 8, 10, 1, 1}, {7, 6, 7, 6, 0, 0, 11, 9},
    {0, 8, 1, 11, 6, 8, 6, 11}, {10, 0, 9, 1, 10, 7, 9, 7}, {10, 4, 9, 4, 10, 2, 9, 3}, {5, 8, 5, 11, 2, 8, 3, 11},
    {4, 9, 0, 0, 7, 9, 2, 2}, {1, 1, 8, 5, 3, 3, 8, 6}, {11, 5, 0, 0, 11, 6, 2, 2}, {1, 1, 4, 10, 3, 3, 7, 10}};

// The lanes of a warp index the tables by their own states, which the constant
// cache would serialise: each block copies them to shared memory, one byte per
// (state, child) holding digit | next state << 3.
__device__ __forceinline__ void load_hilbert(unsigned char *t, int order) {
    if (order == 0) return;  // uniform over the launch
    for (int i = threadIdx.x; i < 96; i += blockDim.x)
        t[i] = (unsigned char)(kHilbertDigit[i >> 3][i & 7] | (kHilbertState[i >> 3][i & 7] << 3));
    __syncthreads();
}

__device__ __forceinline__ int to_digit(int c, int &state, int order, const unsigned char *t) {
    if (order == 0) return c;
    const int e = t[(state << 3) + 7 - c];
    state = e >> 3;
    return e & 7;
}

__device__ __forceinline__ unsigned long long make_key(float px, float py, float pz, const float *bb, int order,
                                                       const unsigned char *t) {
    float mnx = bb[0], mxx = bb[1], mny = bb[2], mxy = bb[3], mnz = bb[4], mxz = bb[5];
    unsigned long long key = 0ull;
    int state = 0;
#pragma unroll 3
    for (int l = 1; l <= 21; l++) {
        int c = split_axis(px, mnx, mxx) + 2 * split_axis(py, mny, mxy) + 4 * split_axis(pz, mnz, mxz);
        key = (key << 3) | (unsigned long long)to_digit(c, state, order, t);
    }
    return key;
}

// Also packs the bodies as float4 (x, y, z, m) in their original order, so that
// the gather into sorted order reads one 16-byte record per body.
__global__ void __launch_bounds__(kBlock) k_keys(const float *__restrict__ x, const float *__restrict__ y,
                                                  const float *__restrict__ z, const float *__restrict__ m,
                                                  const int *__restrict__ body_sys,
                                                  const float *__restrict__ bbox, int n,
                                                  unsigned long long *__restrict__ key, int *__restrict__ val,
                                                  float4 *__restrict__ pos4, DevStatus *st, int order) {
    grid_dependency();
    __shared__ unsigned char ht[96];
    load_hilbert(ht, order);
    for (int i = grid_stride_start(); i < n; i += grid_stride()) {
        const float px = x[i], py = y[i], pz = z[i];
        pos4[i] = make_float4(px, py, pz, m[i]);
        if (!isfinite(px) || !isfinite(py) || !isfinite(pz)) set_status(st, NBX_ERR_NONFINITE, i);
        const int s = body_sys[i];
        float bb[6];
#pragma unroll
        for (int k = 0; k < 6; k++) bb[k] = bbox[6 * s + k];
        key[i] = make_key(px, py, pz, bb, order, ht);
        val[i] = i;
    }
}

// The first runs of the merging sort (merge.cu): k_keys and a stable sort.
//
// A block's 256 keys: parts of 64 by counting, for every key, the part's keys
// before it (broadcast comparisons, no chain of passes), then the four parts by
// searching the other three.  Leaves the sorted keys and their bodies in sk, sv.
// `first` is this block's first key of the run t.  (Counting over all 256 keys
// took 220 us for a batch of 3.2 x 10^6 bodies, this 171.)
__device__ __forceinline__ void sort_block(const float *__restrict__ x, const float *__restrict__ y,
                                           const float *__restrict__ z, const float *__restrict__ m, int4 t, int first,
                                           const float *__restrict__ bbox, float4 *__restrict__ pos4, DevStatus *st,
                                           int order, const unsigned char *ht, unsigned long long *sk, int *sv,
                                           unsigned long long (*so)[kMergeTile]) {
    const int tid = (int)threadIdx.x;
    int i = t.x + first + tid;
    unsigned long long k = 1ull << 63;  // padding: above every 63-bit key
    if (first + tid < t.y) {
        const float px = x[i], py = y[i], pz = z[i];
        pos4[i] = make_float4(px, py, pz, m[i]);
        if (!isfinite(px) || !isfinite(py) || !isfinite(pz)) set_status(st, NBX_ERR_NONFINITE, i);
        float bb[6];
#pragma unroll
        for (int q = 0; q < 6; q++) bb[q] = bbox[6 * t.z + q];
        k = make_key(px, py, pz, bb, order, ht);
    }
    // 64 keys at a time by counting; the two warps of a part order their equal keys
    // by position
    const int part = tid & ~63, w0 = tid & ~31;
    int place = part;
    so[0][tid] = k;
    __syncthreads();
    const ulonglong2 *mine = reinterpret_cast<const ulonglong2 *>(&so[0][w0]);
    const ulonglong2 *other = reinterpret_cast<const ulonglong2 *>(&so[0][w0 ^ 32]);
#pragma unroll
    for (int j = 0; j < 16; j++) {
        const ulonglong2 a = mine[j];
        place += (int)(a.x < k) + ((int)(a.x == k) & (int)(w0 + 2 * j < tid)) + (int)(a.y < k) +
                 ((int)(a.y == k) & (int)(w0 + 2 * j + 1 < tid));
    }
    const unsigned long long kq = k + (w0 & 32 ? 1ull : 0ull);  // an earlier warp's equal key comes first
#pragma unroll
    for (int j = 0; j < 16; j++) {
        const ulonglong2 a = other[j];
        place += (int)(a.x < kq) + (int)(a.y < kq);
    }
    so[1][place] = k;
    __syncthreads();
    // and the four parts of 64 by search
    k = so[1][tid];
    int pos[3] = {0, 0, 0};
#pragma unroll
    for (int step = 64; step > 0; step >>= 1) {
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const int q = a + (64 * a >= part);
            const int p = min(pos[a] + step, 64);
            const bool before = so[1][64 * q + p - 1] < k + (64 * q < part ? 1ull : 0ull);
            pos[a] = (int)(pos[a] + step <= 64) & (int)before ? p : pos[a];
        }
    }
    // the body that stands at `place` of its part moves along
    reinterpret_cast<int *>(so[2])[place] = i;
    __syncthreads();
    i = reinterpret_cast<const int *>(so[2])[tid];
    place = tid - part + pos[0] + pos[1] + pos[2];
    sk[place] = k;
    sv[place] = i;
}

// Every run of 1024 keys, one cluster of four blocks per run: each sorts a
// quarter, reads the other three sorted quarters through distributed shared
// memory and searches those.  (One block of 1024 threads per run took 13.5 us at
// 16384 bodies on 16 SMs.)
__global__ void __cluster_dims__(4, 1, 1) __launch_bounds__(kMergeTile)
    k_sort_tiles(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
                 const float *__restrict__ m, const int4 *__restrict__ runs, const float *__restrict__ bbox,
                 unsigned long long *__restrict__ key, int *__restrict__ val, float4 *__restrict__ pos4, DevStatus *st,
                 int order) {
    grid_dependency();
    constexpr int kQ = kMergeTile;  // a quarter
    static_assert(kMergeRun == 4 * kQ, "four quarters");
    __shared__ unsigned char ht[96];
    __shared__ __align__(16) unsigned long long sk[kQ];     // the quarter's keys, sorted
    __shared__ __align__(16) unsigned long long so[3][kQ];  // the other quarters
    __shared__ int sv[kQ];
    load_hilbert(ht, order);
    const cg::cluster_group cluster = cg::this_cluster();
    const int quarter = (int)cluster.block_rank();
    const int4 t = runs[blockIdx.x >> 2];  // start, len, system, run of the system
    const int tid = (int)threadIdx.x;
    sort_block(x, y, z, m, t, quarter * kQ, bbox, pos4, st, order, ht, sk, sv, so);
    cluster.sync();
#pragma unroll
    for (int a = 0; a < 3; a++) so[a][tid] = cluster.map_shared_rank(sk, a + (a >= quarter))[tid];
    __syncthreads();
    // this thread's key is now the sorted quarter's tid-th; the keys of earlier
    // quarters precede an equal one
    const unsigned long long k = sk[tid];
    const int v = sv[tid];
    int pos[3] = {0, 0, 0};
#pragma unroll
    for (int step = kQ; step > 0; step >>= 1) {
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const int p = min(pos[a] + step, kQ);
            const bool before = so[a][p - 1] < k + (a < quarter ? 1ull : 0ull);
            pos[a] = (int)(pos[a] + step <= kQ) & (int)before ? p : pos[a];
        }
    }
    const int place = tid + pos[0] + pos[1] + pos[2];
    // (padding keys stay behind the valid ones: place < len marks a valid key)
    if (place < t.y) {
        key[t.x + place] = k;
        val[t.x + place] = v;
    }
    cluster.sync();  // the other blocks have read this block's quarter
}

// Runs of at most 256 keys (systems of at most so many bodies), one block each.
// (With clusters, whose other three blocks have nothing to sort, the build of 500000
// systems of four bodies took 23 ms, so 4.1; of 100000 systems of ten 4.8, so 0.94.)
__global__ void __launch_bounds__(kMergeTile)
    k_sort_small(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
                 const float *__restrict__ m, const int4 *__restrict__ runs, const float *__restrict__ bbox,
                 unsigned long long *__restrict__ key, int *__restrict__ val, float4 *__restrict__ pos4, DevStatus *st,
                 int order) {
    grid_dependency();
    __shared__ unsigned char ht[96];
    __shared__ __align__(16) unsigned long long sk[kMergeTile];
    __shared__ __align__(16) unsigned long long so[3][kMergeTile];
    __shared__ int sv[kMergeTile];
    load_hilbert(ht, order);
    const int4 t = runs[blockIdx.x];
    sort_block(x, y, z, m, t, 0, bbox, pos4, st, order, ht, sk, sv, so);
    __syncthreads();
    if ((int)threadIdx.x < t.y) {
        key[t.x + threadIdx.x] = sk[threadIdx.x];
        val[t.x + threadIdx.x] = sv[threadIdx.x];
    }
}

// Runs of equal 21-level keys: compute levels 22..42 and order the run by them.
__global__ void k_refine(const float *__restrict__ x, const float *__restrict__ y,
                         const float *__restrict__ z, const int *__restrict__ body_sys,
                         const int *__restrict__ sys_off, const float *__restrict__ bbox, int n,
                         const unsigned long long *__restrict__ key,
                         unsigned long long *__restrict__ key_lo, int *__restrict__ val,
                         DevStatus *st, int order) {
    grid_dependency();
    __shared__ unsigned char ht[96];
    load_hilbert(ht, order);
    for (int p = grid_stride_start(); p < n; p += grid_stride()) {
        const int s = body_sys[p];
        const int beg = sys_off[s], end = sys_off[s + 1];
        const unsigned long long k = key[p];
        if (p + 1 >= end || key[p + 1] != k) continue;
        if (p > beg && key[p - 1] == k) continue;
        int e = p + 1;
        while (e + 1 < end && key[e + 1] == k) e++;
        if (e - p + 1 > kMaxRun) {
            set_status(st, NBX_ERR_CLUSTER, p);
            continue;
        }
        atomicAdd(&st->refined_runs, 1);
        float bb[6];
        for (int q = 0; q < 6; q++) bb[q] = bbox[6 * s + q];
        for (int q = p; q <= e; q++) {
            const int b = val[q];
            float mnx = bb[0], mxx = bb[1], mny = bb[2], mxy = bb[3], mnz = bb[4], mxz = bb[5];
            unsigned long long lo = 0ull;
            const float px = x[b], py = y[b], pz = z[b];
            int state = 0;
            for (int l = 1; l <= 42; l++) {
                int c = split_axis(px, mnx, mxx) + 2 * split_axis(py, mny, mxy) + 4 * split_axis(pz, mnz, mxz);
                const int d = to_digit(c, state, order, ht);
                if (l > 21) lo = (lo << 3) | (unsigned long long)d;
            }
            key_lo[q] = lo;
        }
        // stable insertion sort of the run by key_lo (runs are short)
        for (int q = p + 1; q <= e; q++) {
            unsigned long long kl = key_lo[q];
            int v = val[q];
            int r = q - 1;
            while (r >= p && key_lo[r] > kl) {
                key_lo[r + 1] = key_lo[r];
                val[r + 1] = val[r];
                r--;
            }
            key_lo[r + 1] = kl;
            val[r + 1] = v;
        }
        for (int q = p; q < e; q++)
            if (key_lo[q] == key_lo[q + 1]) set_status(st, NBX_ERR_DEPTH, val[q]);
    }
}

__device__ __forceinline__ int delta_of(const unsigned long long *key, const unsigned long long *key_lo,
                                        int a) {
    const unsigned long long ka = key[a], kb = key[a + 1];
    if (ka != kb) return common_digits(ka, kb);
    int d = 21 + common_digits(key_lo[a], key_lo[a + 1]);
    return d > 41 ? 41 : d;  // equal 42-level keys were reported as NBX_ERR_DEPTH
}

// Node levels owned by sorted position p: the cells starting at p (levels
// lo..hi-1) and the body (level hi).  With leaf buckets (bucket != nullptr) the
// body hangs directly below its bucket cell (level bucket[p]): deeper cells
// are dropped and the body's level is at most bucket[p] + 1.
__device__ __forceinline__ void levels_of(const unsigned char *delta, const unsigned char *bucket, int p, int beg,
                                          int &lo, int &hi, int &dp) {
    dp = p > beg ? (int)delta[p - 1] : 0;
    const int di = delta[p];
    lo = dp + 1;
    hi = max(dp, di) + 1;
    if (bucket) {
        hi = min(hi, (int)bucket[p] + 1);
        lo = min(lo, hi);
    }
}

// The nodes of every level among a block's kPosBlock positions, stored
// [block][level] in rows of kLvlRow.  Lanes without a position pass lo > hi.
__device__ __forceinline__ void count_levels(int lo, int hi, unsigned *cnt, unsigned *__restrict__ counts) {
    for (int l = threadIdx.x; l < kLvlRow; l += blockDim.x) cnt[l] = 0u;
    __syncthreads();
    const int a = __reduce_min_sync(0xffffffffu, lo <= hi ? lo : kLvlRow);
    const int b = __reduce_max_sync(0xffffffffu, lo <= hi ? hi : 0);
    for (int l = a; l <= b; l++) {
        const unsigned m = __ballot_sync(0xffffffffu, lo <= l && l <= hi);
        if ((threadIdx.x & 31) == 0 && m) atomicAdd(&cnt[l], (unsigned)__popc(m));
    }
    __syncthreads();
    for (int l = threadIdx.x; l < kLvlRow; l += blockDim.x) counts[(size_t)blockIdx.x * kLvlRow + l] = cnt[l];
}

// Sorted bodies as float4 plus delta and (without leaf buckets) the block's
// nodes per level.  One position per thread.
__global__ void __launch_bounds__(kPosBlock) k_delta(const float4 *__restrict__ pos4,
                                                      const int *__restrict__ body_sys,
                                                      const int *__restrict__ sys_off, int n,
                                                      const unsigned long long *__restrict__ key,
                                                      const unsigned long long *__restrict__ key_lo,
                                                      const int *__restrict__ val, float4 *__restrict__ body4,
                                                      unsigned char *__restrict__ delta,
                                                      unsigned *__restrict__ counts, DevStatus *st,
                                                      int *__restrict__ sys_lvl) {
    grid_dependency();
    __shared__ unsigned cnt[kLvlRow];
    const int p = blockIdx.x * kPosBlock + threadIdx.x;
    int lo = 1, hi = 0, s = -1;
    if (p < n) {
        s = body_sys[p];
        const int beg = sys_off[s], end = sys_off[s + 1];
        body4[p] = pos4[val[p]];
        const int di = p + 1 < end ? delta_of(key, key_lo, p) : 0;
        const int dp = p > beg ? delta_of(key, key_lo, p - 1) : 0;
        delta[p] = (unsigned char)di;
        lo = dp + 1;
        hi = max(di, dp) + 1;
    }
    // each system's deepest level (the walk's depth-first reserve of its groups): one
    // check per block where the block lies in one system, else one per body, and an
    // atomic only above the L2 copy.  (An atomic per body took 13 us of a
    // 16384-body k_delta; a check per warp serialised on the one word: 122 us for a
    // batch of 3.2 x 10^6 bodies.)
    __shared__ int s_lvl;
    if (threadIdx.x == 0) s_lvl = 0;
    __syncthreads();
    const int lvl_max = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_lvl, lvl_max);
    const int last = min(n, (int)(blockIdx.x + 1) * kPosBlock) - 1;
    const bool one = body_sys[blockIdx.x * kPosBlock] == body_sys[last];
    __syncthreads();
    const int lv = one ? s_lvl : hi;
    if (s >= 0 && (!one || threadIdx.x == 0) && lv > __ldcg(&sys_lvl[s])) atomicMax(&sys_lvl[s], lv);
    if (threadIdx.x == 0 && s_lvl > __ldcg(&st->max_level)) atomicMax(&st->max_level, s_lvl);
    if (counts) count_levels(lo, hi, cnt, counts);
}

// Leaf buckets (nbx_params.leaf_size k > 1; not the reference's tree, which has
// one body per leaf): the bucket of a body is the shallowest cell around it
// holding at most k bodies.  The cell at level L around p holds more than k
// bodies exactly when some window of k+1 consecutive positions of the system
// containing p shares at least L levels, i.e. all k deltas inside the window
// are >= L; so the bucket level is 1 + the largest inner-delta minimum over
// those windows.  Counts the nodes per level accordingly.
__global__ void __launch_bounds__(kPosBlock) k_bucket(const int *__restrict__ body_sys,
                                                       const int *__restrict__ sys_off, int n, int k,
                                                       const unsigned char *__restrict__ delta,
                                                       unsigned char *__restrict__ bucket,
                                                       unsigned *__restrict__ counts) {
    grid_dependency();
    __shared__ unsigned cnt[kLvlRow];
    const int p = blockIdx.x * kPosBlock + threadIdx.x;
    int lo = 1, hi = 0;
    if (p < n) {
        const int s = body_sys[p];
        const int beg = sys_off[s], end = sys_off[s + 1];
        int best = 0;
        for (int a = max(p - k, beg); a <= p && a + k <= end - 1; a++) {
            int mn = 255;
            for (int j = a; j < a + k; j++) mn = min(mn, (int)delta[j]);
            best = max(best, mn);
        }
        bucket[p] = (unsigned char)(best + 1);
        int dp;
        levels_of(delta, bucket, p, beg, lo, hi, dp);
    }
    count_levels(lo, hi, cnt, counts);
}

// Exclusive scan of every level's counts over the blocks (one block per level),
// in place; the level's total goes to totals[level].
__global__ void __launch_bounds__(1024) k_level_scan(unsigned *__restrict__ counts, int nblk,
                                                      unsigned *__restrict__ totals) {
    grid_dependency();
    constexpr int kPer = 8;
    __shared__ unsigned wt[32];
    const int l = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned carry = 0;
    for (int b0 = 0; b0 < nblk; b0 += 1024 * kPer) {
        const int base = b0 + kPer * (int)threadIdx.x;
        unsigned v[kPer], s = 0;
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            v[k] = base + k < nblk ? counts[(size_t)(base + k) * kLvlRow + l] : 0u;
            s += v[k];
        }
        unsigned incl = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        if (lane == 31) wt[w] = incl;
        __syncthreads();
        if (w == 0) {
            unsigned t = wt[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned u = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += u;
            }
            wt[lane] = t;
        }
        __syncthreads();
        unsigned run = carry + (w ? wt[w - 1] : 0u) + incl - s;
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            if (base + k < nblk) counts[(size_t)(base + k) * kLvlRow + l] = run;
            run += v[k];
        }
        carry += wt[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) totals[l] = carry;
}

// Writes every node of the tree in breadth-first order, one position per
// thread.  The block's base in every level comes from the scanned counts, or
// (Direct, up to kDirectBlocks blocks) from a sum over the earlier blocks' raw
// counts, which saves the scan's launch; ranks inside the block are ballots.
// A cell's meta (first child, children - 1) is gathered by atomic adds on a
// zeroed word: its own thread adds the first child, every later child's thread
// adds one to the count.  Bound by its scattered writes; DRAM at large sizes.
template <bool Direct>
__global__ void __launch_bounds__(kPosBlock) k_nodes(const int *__restrict__ body_sys,
                                                      const int *__restrict__ sys_off, int n,
                                                      const unsigned char *__restrict__ delta,
                                                      const unsigned char *__restrict__ bucket,
                                                      const unsigned *__restrict__ counts, int nblk,
                                                      const unsigned *__restrict__ lvl_tot, int cap_nodes,
                                                      const float4 *__restrict__ body4, unsigned *__restrict__ totals,
                                                      unsigned long long *__restrict__ totals64,
                                                      unsigned *__restrict__ lvl_start, unsigned *__restrict__ eoff,
                                                      unsigned *__restrict__ ent, float4 *__restrict__ node4,
                                                      int *__restrict__ meta, int *__restrict__ parent,
                                                      int *__restrict__ body_node, int *__restrict__ count,
                                                      int *__restrict__ arrive, unsigned char *__restrict__ lvl8,
                                                      int *__restrict__ root_first, int *__restrict__ root_nch,
                                                      DevStatus *st) {
    grid_dependency();
    constexpr int kWarps = kPosBlock / 32, kRows = kPosBlock / kLvlRow;
    __shared__ unsigned part[2][kRows][kLvlRow];  // Direct: partial sums (all blocks, earlier blocks)
    __shared__ unsigned base[kLvlRow];            // index of the block's first node of each level
    __shared__ unsigned wcnt[kWarps][kLvlRow];    // nodes per warp and level, then the warps' bases
    __shared__ unsigned went[kWarps];             // entries per warp
    __shared__ unsigned s_T, s_ebase;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int p = blockIdx.x * kPosBlock + threadIdx.x;
    int lo = 1, hi = 0, dp = 0, s = 0, beg = 0;
    if (p < n) {
        s = body_sys[p];
        beg = sys_off[s];
        levels_of(delta, bucket, p, beg, lo, hi, dp);
    }
    // nodes and entries per warp
    const int wlo = __reduce_min_sync(0xffffffffu, lo <= hi ? lo : kLvlRow);
    const int whi = __reduce_max_sync(0xffffffffu, hi);
    wcnt[w][lane] = 0u;
    wcnt[w][lane + 32] = 0u;
    __syncwarp();
    for (int l = wlo; l <= whi; l++) {
        const unsigned m = __ballot_sync(0xffffffffu, lo <= l && l <= hi);
        if (lane == 0) wcnt[w][l] = __popc(m);
    }
    const unsigned ne = (unsigned)(hi - lo + 1);
    unsigned einc = ne;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, einc, o);
        if (lane >= o) einc += u;
    }
    if (lane == 31) went[w] = einc;
    // the level totals and the counts of the blocks before
    if (Direct) {
        const int l = threadIdx.x & (kLvlRow - 1), r = threadIdx.x / kLvlRow;
        unsigned all = 0, before = 0;
#pragma unroll 4
        for (int b = r; b < nblk; b += kRows) {
            const unsigned c = counts[(size_t)b * kLvlRow + l];
            all += c;
            if (b < (int)blockIdx.x) before += c;
        }
        part[0][r][l] = all;
        part[1][r][l] = before;
    }
    __syncthreads();
    if (w == 0) {
        unsigned tot[2], bef[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int l = 2 * lane + h;
            if (Direct) {
                tot[h] = bef[h] = 0u;
#pragma unroll
                for (int r = 0; r < kRows; r++) {
                    tot[h] += part[0][r][l];
                    bef[h] += part[1][r][l];
                }
            } else {
                tot[h] = lvl_tot[l];
                bef[h] = counts[(size_t)blockIdx.x * kLvlRow + l];
            }
        }
        unsigned incl = tot[0] + tot[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        const unsigned excl = incl - tot[0] - tot[1];
        base[2 * lane] = excl + bef[0];
        base[2 * lane + 1] = excl + tot[0] + bef[1];
        const unsigned eb = __reduce_add_sync(0xffffffffu, bef[0] + bef[1]);
        const unsigned T = __shfl_sync(0xffffffffu, incl, 31);
        if (lane == 0) {
            s_T = T;
            s_ebase = eb;
        }
        if (blockIdx.x == 0) {
            const bool fits = T <= (unsigned)cap_nodes;
            lvl_start[2 * lane] = fits ? excl : 0u;
            lvl_start[2 * lane + 1] = fits ? excl + tot[0] : 0u;
            if (lane == 0) {
                if (!fits) set_status(st, NBX_ERR_CAPACITY, (int)min(T, 0x7fffffffu));
                totals[0] = T;
                totals[1] = fits ? T : 0u;  // nothing downstream reads a partial tree
                totals64[0] = fits ? (unsigned long long)(T - (unsigned)n) << 32 : 0ull;
            }
        }
    }
    __syncthreads();
    // the warps' bases in every level, and this warp's first entry
    if (threadIdx.x < kLvlRow) {
        unsigned run = base[threadIdx.x];
#pragma unroll
        for (int v = 0; v < kWarps; v++) {
            const unsigned c = wcnt[v][threadIdx.x];
            wcnt[v][threadIdx.x] = run;
            run += c;
        }
    }
    unsigned e = s_ebase + einc - ne;
    for (int v = 0; v < w; v++) e += went[v];
    __syncthreads();
    const bool fits = s_T <= (unsigned)cap_nodes;
    const bool ok = fits && st->code == 0;  // a failed build leaves empty roots
    if (p < n) eoff[p] = e;
    if (!fits) {
        if (p < n && p == beg) root_first[s] = 0;
        return;
    }
    int b = 0;  // this position's node at the level before l
    for (int l = wlo - 1; l <= whi; l++) {
        const unsigned m = __ballot_sync(0xffffffffu, lo <= l && l <= hi);
        if (l < lo - 1 || l > hi) continue;
        const int i = (int)(wcnt[w][l] + __popc(m & lt));
        if (l == lo - 1) {
            b = i - 1;  // the last level-l node before p: the parent of p's top node
            continue;
        }
        lvl8[i] = (unsigned char)l;
        ent[i] = ((unsigned)l << kLevelShift) | (unsigned)p;
        arrive[i] = 0;
        if (l == 1) {
            parent[i] = -1 - s;
            if (p == beg) root_first[s] = ok ? i : 0;
            if (ok) atomicAdd(&root_nch[s], 1);
        } else {
            parent[i] = b;
            // the first child of the cell at this position, or a later child
            atomicAdd(&meta[b], l > lo ? i : 1 << 28);
        }
        if (l == hi) {
            node4[i] = body4[p];
            meta[i] = kBodyFlag | p;
            body_node[p] = i;
            count[i] = 1;
        }
        b = i;
    }
}

// Moments of a cell by a group of lanes (4, or 8 with quadrupoles), lane k of
// the group holding component k & 3 of (m, m x, m y, m z): the children are
// summed in child order, one FP64 instruction per child for all components
// (a body's m x is exact in FP64, so the fused product adds it with one
// rounding), and one division gives the three coordinates of the centre.
// Lanes of inactive groups pass nch = 0 and store nothing.  The loads of all
// children are issued together; a child's kind picks the value.
struct CellSum {
    double acc;
    int cnt;
};

__device__ __forceinline__ CellSum sum_cell(int k, int first, int nch, const int *__restrict__ meta,
                                            const float4 *node4, const double4 *sums, const int *count) {
    int mk[8], ck[8];
    float mb[8], fb[8];
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        if (j < nch) {
            const int c = first + j;
            mk[j] = meta[c];
            const float *q = reinterpret_cast<const float *>(&node4[c]);
            mb[j] = q[3];
            fb[j] = k == 0 ? 1.f : q[k - 1];
            v[j] = __ldcg(reinterpret_cast<const double *>(&sums[c]) + k);
            ck[j] = __ldcg(&count[c]);
        }
    }
    CellSum r{0.0, 0};
#pragma unroll
    for (int j = 0; j < 8; j++) {
        if (j < nch) {
            const bool body = mk[j] < 0;
            r.acc = __fma_rn(body ? widen(mb[j]) : v[j], body ? widen(fb[j]) : 1.0, r.acc);
            r.cnt += body ? 1 : ck[j];
        }
    }
    return r;
}

// Quadrupole mode: the FP64 second moments of a cell about its centre of mass c,
// composed from its children in child order -- M2 = sum over children of
// [M2_child + m_child d d^T], d = c_child - c (a body child: M2 = 0, c_child =
// its position) -- and the cell's traceless quadrupole Q = 3 M2 - tr(M2) I,
// stored negated in FP32 as P = -Q = tr(M2) I - 3 M2 (the walk's form of the
// term; the FP64 differences are negated before rounding, so P is exactly -Q).
// Every FP64 operation is rounded explicitly (no contraction), in the order of
// the oracle's restatement, so both give the same bits.  Lane k < 6 of the
// group holds component k of (xx, yy, zz, xy, xz, yz); com is the centres' FP64
// array, (x, y, z) per cell.
__device__ __forceinline__ void quad_cell(int k, int b, int first, int nch, double q0, const int *__restrict__ meta,
                                          const float4 *node4, const double4 *sums, double *com, double2 *m2,
                                          float4 *quad4, float2 *quad2) {
    const int ka = k < 3 ? k : (k == 5 ? 1 : 0);   // first axis of the component
    const int kb = k < 3 ? k : (k == 3 ? 1 : 2);   // second axis
    const int g = threadIdx.x & 24;                // first lane of the group
    // q0: lane 1..3 hold the cell's own centre (x, y, z)
    const double ca = __shfl_sync(0xffffffffu, q0, g + 1 + min(ka, 2));
    const double cb = __shfl_sync(0xffffffffu, q0, g + 1 + min(kb, 2));
    if (k < 3 && nch > 0) com[3 * (size_t)b + k] = ca;
    double a = 0.0;
    if (k < 6) {
#pragma unroll 4
        for (int j = 0; j < nch; j++) {
            const int c = first + j;
            double mc, xa, xb;
            if (meta[c] < 0) {
                const float *q = reinterpret_cast<const float *>(&node4[c]);
                mc = widen(q[3]);
                xa = widen(q[ka]);
                xb = widen(q[kb]);
            } else {
                mc = __ldcg(reinterpret_cast<const double *>(&sums[c]));
                xa = __ldcg(&com[3 * (size_t)c + ka]);
                xb = __ldcg(&com[3 * (size_t)c + kb]);
                a = __dadd_rn(a, __ldcg(reinterpret_cast<const double *>(&m2[3 * (size_t)c]) + k));
            }
            a = __dadd_rn(a, __dmul_rn(__dmul_rn(mc, __dsub_rn(xa, ca)), __dsub_rn(xb, cb)));
        }
    }
    const double axx = __shfl_sync(0xffffffffu, a, g), ayy = __shfl_sync(0xffffffffu, a, g + 1);
    const double azz = __shfl_sync(0xffffffffu, a, g + 2);
    const double tr = __dadd_rn(__dadd_rn(axx, ayy), azz);
    if (k < 6 && nch > 0) {
        reinterpret_cast<double *>(&m2[3 * (size_t)b])[k] = a;
        const double t3 = __dmul_rn(k < 3 ? 3.0 : -3.0, a);
        const float P = (float)(k < 3 ? __dsub_rn(tr, t3) : t3);
        if (k < 4) reinterpret_cast<float *>(&quad4[b])[k] = P;
        else reinterpret_cast<float *>(&quad2[b])[k - 4] = P;
    }
}

// A cell's sums, and (finish) its centre of mass, node record and quadrupole.
template <bool Quad>
__device__ __forceinline__ void finish_cell(int k, int b, int first, int nch, double acc, const int *__restrict__ meta,
                                              float4 *node4, const double4 *sums, double *com, double2 *m2,
                                              float4 *quad4, float2 *quad2) {
    constexpr int kLanes = Quad ? 8 : 4;
    const int kc = k & 3;
    const double m = __shfl_sync(0xffffffffu, acc, (threadIdx.x & 31) & ~(kLanes - 1));
    if (!Quad) {
        if (nch > 0) {
            const float f = kc == 0 ? (float)acc : quotient32(acc, m);
            reinterpret_cast<float *>(&node4[b])[kc == 0 ? 3 : kc - 1] = f;
        }
        return;
    }
    const double q = kc == 0 ? acc : acc / (nch > 0 ? m : 1.0);
    if (k < 4 && nch > 0) reinterpret_cast<float *>(&node4[b])[kc == 0 ? 3 : kc - 1] = (float)q;
    quad_cell(k, b, first, nch, q, meta, node4, sums, com, m2, quad4, quad2);
}

// Bottom-up FP64 moments, one BFS level per launch (deepest first): a cell sums
// its children -- contiguous, one level below, already final -- in child order,
// so the result is deterministic.  Level L occupies BFS indices
// [lvl_start[L], lvl_start[L+1]); each warp lists the cells among 32 nodes and
// gives each a group of lanes.
template <bool Quad>
__global__ void __launch_bounds__(kBlock) k_moments_level(int level, const unsigned *__restrict__ lvl_start,
                                                           const int *__restrict__ meta, float4 *node4,
                                                           double4 *sums, int *count, double *com, double2 *m2,
                                                           float4 *quad4, float2 *quad2, const DevStatus *st) {
    grid_dependency();
    constexpr int kLanes = Quad ? 8 : 4, kGroups = 32 / kLanes;
    if (st->code != 0) return;  // an inconsistent tree is never summed
    __shared__ int list[kBlock / 32][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, k = lane & (kLanes - 1);
    const unsigned lt = (1u << lane) - 1u;
    const unsigned beg = lvl_start[level], end = lvl_start[level + 1];
    for (unsigned c0 = beg + 32u * (blockIdx.x * (kBlock / 32) + w); c0 < end; c0 += 32u * gridDim.x * (kBlock / 32)) {
        const bool cell = c0 + lane < end && meta[c0 + lane] >= 0;
        const unsigned m = __ballot_sync(0xffffffffu, cell);
        __syncwarp();
        if (cell) list[w][__popc(m & lt)] = (int)c0 + lane;
        __syncwarp();
        const int nc = __popc(m);
        for (int i = lane / kLanes; i - lane / kLanes < nc; i += kGroups) {
            int b = 0, first = 0, nch = 0;
            if (i < nc) {
                b = list[w][i];
                const int pm = meta[b];
                first = pm & 0x0fffffff;
                nch = ((pm >> 28) & 7) + 1;
            }
            const CellSum r = sum_cell(k & 3, first, nch, meta, node4, sums, count);
            if (i < nc && k < 4) {
                reinterpret_cast<double *>(&sums[b])[k] = r.acc;
                if (k == 0) count[b] = r.cnt;
            }
            finish_cell<Quad>(k, b, first, nch, r.acc, meta, node4, sums, com, m2, quad4, quad2);
        }
    }
}

__device__ __forceinline__ int arrive_acq_rel(int *p) {
    int old;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(p) : "memory");
    return old;
}

// Bottom-up FP64 moments in one launch.  A warp takes kUpNodes nodes in BFS
// order and lists the cells whose children are all bodies; every group of lanes
// sums a listed cell and climbs: every child arrives once at its cell's counter
// (the body children in one step, by the warp that meets the cell; a child cell
// when it is complete), and the arrival that brings the count to the cell's
// number of children sums the cell (children in child order: the same additions
// as k_moments_level) and climbs on to the parent.  A group whose arrival is
// not the last takes the warp's next listed cell.  Nothing waits.  A cell's
// arrival is acquire-release: it publishes the group's sums (ordered before it
// by the warp barrier) and, when last, orders the reads of the siblings' sums
// (through L2) after their arrivals.  Counters are zeroed by k_nodes.
// Bound by the chain of levels, and in a level by the FP64 pipe: one thread per
// cell issued about 15 FP64 instructions per child and three divisions per
// level (4.5 us a level); the lanes share them.  The mode without quadrupoles
// arrives before its division, which then runs while the arrival returns.
template <bool Quad>
__global__ void __launch_bounds__(kBlock) k_moments_up(const unsigned *__restrict__ totals, int rounds,
                                                       const int *__restrict__ parent,
                                                       const int *__restrict__ meta, float4 *node4,
                                                       double4 *sums, int *count, int *counter, double *com,
                                                       double2 *m2, float4 *quad4, float2 *quad2,
                                                       const DevStatus *st) {
    grid_dependency();
    constexpr int kLanes = Quad ? 8 : 4;
    if (st->code != 0) return;  // an inconsistent tree is never summed
    __shared__ int list[kBlock / 32][32 * kUpRounds];
    const int T = (int)totals[1];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, k = lane & (kLanes - 1);
    const int lead = lane & ~(kLanes - 1);
    const unsigned lt = (1u << lane) - 1u;
    const int nwarps = gridDim.x * (kBlock / 32);
    for (int c0 = 32 * rounds * (blockIdx.x * (kBlock / 32) + w); c0 < T; c0 += 32 * rounds * nwarps) {
        int nlist = 0;
        __syncwarp();
        for (int r = 0; r < rounds; r++) {
            const int b = c0 + 32 * r + lane;
            const int pm = b < T ? meta[b] : -1;
            bool ready = false;
            if (pm >= 0) {
                const int first = pm & 0x0fffffff, nch = ((pm >> 28) & 7) + 1;
                int nbody = 0;
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (j < nch) nbody += meta[first + j] < 0;
                // no body child: completed by the arrival of its last child cell;
                // both kinds: the bodies arrive together (relaxed: nothing to publish)
                ready = nbody == nch;
                if (nbody > 0 && !ready) {
                    ready = atomicAdd(&counter[b], nbody) + nbody == nch;
                    if (ready) asm volatile("fence.acq_rel.gpu;" ::: "memory");
                }
            }
            const unsigned m = __ballot_sync(0xffffffffu, ready);
            if (ready) list[w][nlist + __popc(m & lt)] = b;
            nlist += __popc(m);
        }
        __syncwarp();
        int next = 0, b = -1, pm = 0, up = -1;
        for (;;) {
            // groups without a cell take the next listed ones
            const unsigned want = __ballot_sync(0xffffffffu, b < 0 && k == 0);
            if (b < 0) {
                const int i = next + __popc(want & ((1u << lead) - 1u));
                if (i < nlist) {
                    b = list[w][i];
                    pm = meta[b];
                    up = parent[b];
                }
            }
            next += __popc(want);
            const bool on = b >= 0;
            if (!__any_sync(0xffffffffu, on)) break;
            const int first = on ? pm & 0x0fffffff : 0, nch = on ? ((pm >> 28) & 7) + 1 : 0;
            // the parent's record loads with the children; in a small tree (one round
            // per warp) its parent too, which shortens the chain of a climb but is
            // one more load for every group that stops
            int upm = 0, up2 = -1;
            if (on && up >= 0) {
                upm = meta[up];
                if (rounds == 1) up2 = parent[up];
            }
            const CellSum r = sum_cell(k & 3, first, nch, meta, node4, sums, count);
            if (on && k < 4) {
                reinterpret_cast<double *>(&sums[b])[k] = r.acc;
                if (k == 0) count[b] = r.cnt;
            }
            if (Quad) finish_cell<true>(k, b, first, nch, r.acc, meta, node4, sums, com, m2, quad4, quad2);
            __syncwarp();  // the group's stores come before its arrival
            int old = -1;
            if (on && up >= 0 && k == 0) old = arrive_acq_rel(&counter[up]);
            if (!Quad) finish_cell<false>(k, b, first, nch, r.acc, meta, node4, sums, com, m2, quad4, quad2);
            old = __shfl_sync(0xffffffffu, old, lead);
            __syncwarp();  // the reads of the siblings' sums come after it
            const bool last = on && up >= 0 && old == ((upm >> 28) & 7);  // of the parent's children
            b = last ? up : -1;
            pm = upm;
            up = last && rounds > 1 ? parent[up] : up2;
        }
    }
}

}  // namespace

// ---------------------------------------------------------------------------
int build_tree(Ctx *ctx, const nbx_state *s, cudaStream_t st, bool external_bbox,
               const float *const *bbox_ptrs) {
    const int n = (int)ctx->nbodies;
    const int S = ctx->nsys;
    if (n <= 0 || S <= 0) return NBX_ERR_STATE;
    ctx->chain = false;
    const int gb = ceil_div(n, kBlock) < ctx->nsm * 8 ? ceil_div(n, kBlock) : ctx->nsm * 8;
    int4 *meta4 = reinterpret_cast<int4 *>(ctx->d_meta);
    if (!external_bbox) {
        launch_chained(ctx, st, ctx->ntiles_body, kBlock, 0, k_bbox, s->x, s->y, s->z, ctx->d_tiles, ctx->d_sys_tiles,
                       ctx->d_bbox_u, S, ctx->theta_ref, ctx->d_bbox, ctx->d_bbox64, ctx->d_depth0, ctx->d_bbox_done,
                       ctx->d_status, ctx->d_sys_lvl, ctx->d_root_nch, meta4, ctx->d_meta, ctx->d_lvl_start);
    } else {
        launch_chained(ctx, st, gb, kBlock, 0, k_step_reset, S, ctx->d_status, ctx->d_sys_lvl, ctx->d_root_nch, meta4,
                       ctx->d_meta, ctx->d_lvl_start);
        launch_chained(ctx, st, 1, 32, 0, k_bbox_from_ptrs, bbox_ptrs[0], bbox_ptrs[1], bbox_ptrs[2], bbox_ptrs[3],
                       bbox_ptrs[4], bbox_ptrs[5], ctx->theta_ref, ctx->d_bbox, ctx->d_bbox64, ctx->d_depth0,
                       ctx->d_status);
    }
    // the node array is free until the nodes are written: it holds the packed bodies
    float4 *pos4 = ctx->d_node4;
    // keys sort by merging or by radix (sorts_by_merging);
    // the last pass writes d_key / d_val: an odd pass count starts from the alternates
    const bool merge = ctx->merge;
    const bool alt = (merge ? merge_passes(ctx->max_sys) : radix_passes(ctx->radix_bits)) & 1;
    unsigned long long *key0 = alt ? ctx->d_key_alt : ctx->d_key;
    int *val0 = alt ? ctx->d_val_alt : ctx->d_val;
    if (merge) {
        if (ctx->nruns_mg)
            launch_chained(ctx, st, 4 * ctx->nruns_mg, kMergeTile, 0, k_sort_tiles, s->x, s->y, s->z, s->m,
                           ctx->d_runs_mg, ctx->d_bbox, key0, val0, pos4, ctx->d_status, ctx->key_order);
        if (ctx->nsmall_mg)
            launch_chained(ctx, st, ctx->nsmall_mg, kMergeTile, 0, k_sort_small, s->x, s->y, s->z, s->m,
                           ctx->d_runs_mg + ctx->nruns_mg, ctx->d_bbox, key0, val0, pos4, ctx->d_status, ctx->key_order);
    } else
        launch_chained(ctx, st, gb, kBlock, 0, k_keys, s->x, s->y, s->z, s->m, ctx->d_body_sys, ctx->d_bbox, n, key0,
                       val0, pos4, ctx->d_status, ctx->key_order);
    int rc = merge ? merge_runs(ctx, st) : radix_sort_bodies(ctx, st);
    if (rc) return rc;
    launch_chained(ctx, st, gb, kBlock, 0, k_refine, s->x, s->y, s->z, ctx->d_body_sys, ctx->d_sys_off, ctx->d_bbox, n,
                   ctx->d_key, ctx->d_key_lo, ctx->d_val, ctx->d_status, ctx->key_order);
    const unsigned char *bucket = ctx->leaf_size > 1 ? ctx->d_bucket : nullptr;
    const int nblk = ceil_div(n, kPosBlock);
    launch_chained(ctx, st, nblk, kPosBlock, 0, k_delta, pos4, ctx->d_body_sys, ctx->d_sys_off, n, ctx->d_key,
                   ctx->d_key_lo, ctx->d_val, ctx->d_body4, ctx->d_delta, bucket ? nullptr : ctx->d_lvl_counts,
                   ctx->d_status, ctx->d_sys_lvl);
    if (bucket)
        launch_chained(ctx, st, nblk, kPosBlock, 0, k_bucket, ctx->d_body_sys, ctx->d_sys_off, n, ctx->leaf_size,
                       ctx->d_delta, ctx->d_bucket, ctx->d_lvl_counts);
    const bool direct = nblk <= kDirectBlocks;
    if (!direct)
        launch_chained(ctx, st, kLvlRow, 1024, 0, k_level_scan, ctx->d_lvl_counts, nblk, ctx->d_lvl_tot);
    auto nodes = direct ? k_nodes<true> : k_nodes<false>;
    launch_chained(ctx, st, nblk, kPosBlock, 0, nodes, ctx->d_body_sys, ctx->d_sys_off, n, ctx->d_delta, bucket,
                   ctx->d_lvl_counts, nblk, ctx->d_lvl_tot, ctx->cap_nodes, ctx->d_body4, ctx->d_totals,
                   ctx->d_totals64, ctx->d_lvl_start, ctx->d_ecount, ctx->d_ent, ctx->d_node4, ctx->d_meta,
                   ctx->d_parent, ctx->d_body_node, ctx->d_count, ctx->d_arrive, ctx->d_lvl8, ctx->d_root_first,
                   ctx->d_root_nch, ctx->d_status);
    const int gn = ceil_div(ctx->cap_nodes, kBlock) < ctx->nsm * 8 ? ceil_div(ctx->cap_nodes, kBlock) : ctx->nsm * 8;
    // up to 2^21 bodies the 41 per-level launches cost more than the sums: one
    // bottom-up launch (2^16: 0.37 against 0.55 ms per build); above, the
    // per-level launches stream the levels.  Batches of systems, whose chains are
    // shorter and side by side, keep the one launch up to 2^22 bodies, and to 2^23
    // where no system has more than 2^16: 4 systems of 10^6 1.40 against 1.42 ms,
    // 800 of 4096 0.99 / 1.03, 250 of 32768 2.52 / 2.56, but 2 of 4 x 10^6 2.54 /
    // 2.51 and 60 of 131072 2.53 / 2.48.  With quadrupoles it loses there (8 of 2^19
    // 4.05 against 3.97 ms)
    const int mode = ctx->p.moments_mode;
    const bool quad = ctx->multipole != 0;
    if (quad && !ctx->d_m2) return NBX_ERR_STATE;
    const int up_max = S == 1 || quad ? kMomentsUpMaxBodies : (ctx->max_sys <= 1 << 16 ? 4 : 2) * kMomentsUpMaxBodies;
    if (mode == 2 || (mode == 0 && n <= up_max)) {
        // one round of 32 nodes per warp until that fills the GPU's warps (a small
        // tree wants its chains started at once), then up to four (fuller groups)
        int rounds = (int)(3ll * n / 2 / (32ll * 32 * ctx->nsm));
        rounds = rounds < 1 ? 1 : (rounds > kUpRounds ? kUpRounds : rounds);
        auto kern = quad ? k_moments_up<true> : k_moments_up<false>;
        launch_chained(ctx, st, gn, kBlock, 0, kern, ctx->d_totals, rounds, ctx->d_parent, ctx->d_meta, ctx->d_node4,
                       ctx->d_sums, ctx->d_count, ctx->d_arrive, ctx->d_com, ctx->d_m2, ctx->d_quad4, ctx->d_quad2,
                       ctx->d_status);
    } else {
        // cells exist at levels 1..41 (two bodies share at most 41 levels without error)
        auto kern = quad ? k_moments_level<true> : k_moments_level<false>;
        for (int level = kMaxLevel - 2; level >= 1; level--)
            launch_chained(ctx, st, ctx->nsm * 4, kBlock, 0, kern, level, ctx->d_lvl_start, ctx->d_meta, ctx->d_node4,
                           ctx->d_sums, ctx->d_count, ctx->d_com, ctx->d_m2, ctx->d_quad4, ctx->d_quad2,
                           ctx->d_status);
    }
    NBX_CUDA(cudaGetLastError());
    ctx->built = true;
    return NBX_OK;
}

// ---------------------------------------------------------------------------
// Export of one system's tree in the reference's array format.
namespace {

__global__ void __launch_bounds__(kBlock) k_export(const unsigned *__restrict__ ent_bfs,
                                                    const unsigned *__restrict__ totals,
                                                    const int *__restrict__ body_sys,
                                                    const int *__restrict__ sys_off,
                                                    const unsigned char *__restrict__ delta,
                                                    const unsigned *__restrict__ eoff,
                                                    const unsigned long long *__restrict__ key,
                                                    const unsigned long long *__restrict__ key_lo,
                                                    const int *__restrict__ val, const int *__restrict__ parent,
                                                    const float4 *__restrict__ node4,
                                                    const double4 *__restrict__ sums,
                                                    const int *__restrict__ count, int sys, int cells_before,
                                                    int cap_cells, int *root_child, int *cell_child,
                                                    int *cell_start, int *cell_count, int *cell_level,
                                                    float *cx, float *cy, float *cz, float *cm, int sum_mode) {
    const int T = (int)totals[1];
    const int beg = sys_off[sys];
    const int nsys_bodies = sys_off[sys + 1] - beg;
    for (int b = grid_stride_start(); b < T; b += grid_stride()) {
        const unsigned u = ent_bfs[b];
        const int l = (int)(u >> kLevelShift);
        const int p = (int)(u & ((1u << kLevelShift) - 1u));
        if (body_sys[p] != sys) continue;
        int lo, hi, dp;
        levels_of(delta, nullptr, p, beg, lo, hi, dp);
        const bool is_cell = l < hi;
        const int pre = (int)(eoff[p] - (unsigned)p) - cells_before + (l - lo);
        int value;
        if (is_cell) {
            value = nsys_bodies + pre;
            if (pre < cap_cells) {
                if (cell_start) cell_start[pre] = p - beg;
                if (cell_count) cell_count[pre] = count[b];
                if (cell_level) cell_level[pre] = l;
                if (sum_mode) {
                    const double4 q = sums[b];
                    if (cx) cx[pre] = (float)q.y;
                    if (cy) cy[pre] = (float)q.z;
                    if (cz) cz[pre] = (float)q.w;
                    if (cm) cm[pre] = (float)q.x;
                } else {
                    const float4 q = node4[b];
                    if (cx) cx[pre] = q.x;
                    if (cy) cy[pre] = q.y;
                    if (cz) cz[pre] = q.z;
                    if (cm) cm[pre] = q.w;
                }
            }
        } else {
            value = val[p] - beg;
        }
        const int slot = digit_of(key[p], key_lo[p], l);
        const int par = parent[b];
        if (par < 0) {
            if (root_child) root_child[slot] = value;
        } else if (cell_child) {
            const unsigned pu = ent_bfs[par];
            const int pl = (int)(pu >> kLevelShift);
            const int pp = (int)(pu & ((1u << kLevelShift) - 1u));
            int plo, phi, pdp;
            levels_of(delta, nullptr, pp, beg, plo, phi, pdp);
            const int ppre = (int)(eoff[pp] - (unsigned)pp) - cells_before + (pl - plo);
            if (ppre < cap_cells) cell_child[8 * ppre + slot] = value;
        }
    }
}

__global__ void k_perm_export(const int *val, int beg, int n, int *perm) {
    for (int i = grid_stride_start(); i < n; i += grid_stride()) perm[i] = val[beg + i] - beg;
}

}  // namespace

int export_tree_impl(Ctx *ctx, int sys, int *perm, int *root_child, int *cell_child, int *cell_start,
                     int *cell_count, int *cell_level, float *cx, float *cy, float *cz, float *cm,
                     int cap_cells, int64_t *ncells, cudaStream_t st, int sum_mode) {
    // the reference's array format holds the reference's tree: Lebesgue order, one body per leaf
    if (!ctx->built || ctx->key_order != 0 || ctx->leaf_size != 1) return NBX_ERR_STATE;
    if (sys < 0 || sys >= ctx->nsys) return NBX_ERR_ARG;
    // a single system's range is the whole context: only the node count is read back
    int off[2] = {0, (int)ctx->nbodies};
    unsigned e_beg = 0, e_end = 0, T = 0;
    if (ctx->nsys > 1) {
        NBX_CUDA(cudaMemcpyAsync(off, ctx->d_sys_off + sys, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
        NBX_CUDA(cudaStreamSynchronize(st));
        NBX_CUDA(cudaMemcpyAsync(&e_beg, ctx->d_ecount + off[0], sizeof(unsigned), cudaMemcpyDeviceToHost, st));
        if (off[1] < ctx->nbodies)
            NBX_CUDA(cudaMemcpyAsync(&e_end, ctx->d_ecount + off[1], sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    }
    NBX_CUDA(cudaMemcpyAsync(&T, ctx->d_totals + 0, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    NBX_CUDA(cudaStreamSynchronize(st));
    if (off[1] >= ctx->nbodies) e_end = T;
    const int cells_before = (int)e_beg - off[0];
    const int nc = (int)e_end - off[1] - cells_before;
    if (ncells) *ncells = nc;
    if (nc > cap_cells) {
        ctx->last_error = "export: cell capacity too small";
        return NBX_ERR_CAPACITY;
    }
    const int nb = off[1] - off[0];
    if (perm) {
        k_perm_export<<<ceil_div(nb, kBlock), kBlock, 0, st>>>(ctx->d_val, off[0], nb, perm);
        ++ctx->launches;
    }
    if (root_child) NBX_CUDA(cudaMemsetAsync(root_child, 0xff, 8 * sizeof(int), st));
    if (cell_child && nc > 0) NBX_CUDA(cudaMemsetAsync(cell_child, 0xff, 8 * sizeof(int) * (size_t)nc, st));
    const int gn = ceil_div(ctx->cap_nodes, kBlock) < ctx->nsm * 8 ? ceil_div(ctx->cap_nodes, kBlock) : ctx->nsm * 8;
    k_export<<<gn, kBlock, 0, st>>>(ctx->d_ent, ctx->d_totals, ctx->d_body_sys, ctx->d_sys_off,
                                    ctx->d_delta, ctx->d_ecount, ctx->d_key, ctx->d_key_lo, ctx->d_val,
                                    ctx->d_parent, ctx->d_node4, ctx->d_sums, ctx->d_count, sys, cells_before,
                                    cap_cells, root_child, cell_child, cell_start, cell_count, cell_level, cx,
                                    cy, cz, cm, sum_mode);
    ++ctx->launches;
    NBX_CUDA(cudaGetLastError());
    return NBX_OK;
}

}  // namespace nbx
