// merge.cu -- body-key sort of small and mid-size systems by ranks.
//
// The radix passes of radix.cu cost a launch and a chain of shared-memory and
// look-back round trips per 8 bits of key, whatever the size: 8 x 6 us for a
// thousand bodies, 8 x 13 us for 131072.  Here a system's keys are sorted in
// runs of kMergeRun (k_sort_tiles in tree.cu, with the keys' computation) and
// up to kMergeFan runs are merged per launch: every key's place in the merged
// run is its place in its own run plus, for each other run, the number of that
// run's keys that precede it (equal keys keep the order of the runs: the sort is
// stable).  All keys do this at once, so a launch is two dependent phases.
// Bound by the latency of its phases below about 10^5 keys, by shared-memory
// searches above (about 15 runs x 6 steps per key and launch).  Keys + sort, eight
// one-sweep passes against this: 1000 bodies 58 -> 6.5 us, 16384 80 -> 17 us,
// 131071 116 -> 43 us; at 2^20 the merges take 309 us, the passes 275 us, so
// systems above kMergeMaxBodies sort by radix (sorts_by_merging, with the rule for
// batches).
#include <utility>

#include "nbx_internal.cuh"

namespace nbx {

namespace {

constexpr int kThreads = kMergeTile;  // one key per thread
constexpr int kAhead = 4;             // runs searched together (their loads overlap)
constexpr int kProbes = 8;            // threads of a bound's search
static_assert(kThreads == 2 * kProbes * kMergeFan && kMergeFan == 16, "threads of every run's bounds, lanes of its windows");
static_assert(kMergeFan % kAhead == 0, "whole batches of runs");

// Runs [rbeg, rbeg + R), ... of one group: the key at local run position i of
// run `own` precedes or follows keys of other runs by value, then by run.
__device__ __forceinline__ bool precedes(unsigned long long x, unsigned long long k, bool earlier) {
    return earlier ? x <= k : x < k;
}

// One block per 256 keys of a run; a group is F runs of R keys (the last
// shorter).  Of every other run the stretch between the block's first and last
// key is staged in shared memory (its bounds by a nine-way search, eight threads
// each); a stretch that no longer fits is searched in global memory.
__global__ void __launch_bounds__(kThreads) k_merge(const int4 *__restrict__ tiles, const int *__restrict__ sys_off,
                                                    int R, int F, int cap,
                                                    const unsigned long long *__restrict__ key_in,
                                                    const int *__restrict__ val_in,
                                                    unsigned long long *__restrict__ key_out,
                                                    int *__restrict__ val_out) {
    grid_dependency();
    extern __shared__ __align__(16) unsigned long long stage[];  // [cap]
    __shared__ int s_lo[kMergeFan], s_len[kMergeFan], s_off[kMergeFan];
    const int4 t = tiles[blockIdx.x];  // start, len, system, tile of the system
    const int sbeg = sys_off[t.z], send = sys_off[t.z + 1];
    const int span = R * F, q0 = t.w * kMergeTile;
    const int gbeg = sbeg + q0 / span * span;
    const int gend = min(send, gbeg + span);
    const int nrun = (gend - gbeg + R - 1) / R;
    const int own = (t.x - gbeg) / R;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool valid = (int)threadIdx.x < t.y;
    const unsigned long long kk = valid ? key_in[t.x + threadIdx.x] : 0ull;
    const int vv = valid ? val_in[t.x + threadIdx.x] : 0;
    if (nrun == 1) {  // nothing to merge with (uniform over the block)
        if (valid) {
            key_out[t.x + threadIdx.x] = kk;
            val_out[t.x + threadIdx.x] = vv;
        }
        return;
    }
    {
        const unsigned long long kmin = key_in[t.x], kmax = key_in[t.x + t.y - 1];
        const int id = threadIdx.x / kProbes, j = threadIdx.x % kProbes, r = id >> 1;
        const unsigned long long k = id & 1 ? kmax : kmin;
        const unsigned long long *run = key_in + gbeg + r * R;
        int lo = 0, hi = r < nrun && r != own ? min(R, gend - gbeg - r * R) : 0;
        while (__any_sync(0xffffffffu, hi > lo)) {
            const int len = hi - lo;
            const bool c = len > 0 && precedes(run[lo + (j + 1) * len / (kProbes + 1)], k, r < own);
            const int n = __popc((__ballot_sync(0xffffffffu, c) >> (lane & ~(kProbes - 1))) & ((1u << kProbes) - 1u));
            if (len > 0) {  // probes 0 .. n-1 precede k, probe n does not
                const int a = n > 0 ? lo + n * len / (kProbes + 1) + 1 : lo;
                if (n < kProbes) hi = lo + (n + 1) * len / (kProbes + 1);
                lo = a;
            }
        }
        const int other = __shfl_xor_sync(0xffffffffu, lo, kProbes);  // the run's other bound
        if (threadIdx.x % (2 * kProbes) == 0) {
            s_lo[r] = lo;
            s_len[r] = other - lo;
        }
        __syncthreads();
        if (w == 0) {
            const int len = lane < kMergeFan ? s_len[lane] : 0;
            int incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += u;
            }
            if (lane < kMergeFan) s_off[lane] = incl <= cap ? incl - len : -1;
        }
        __syncthreads();
        for (int q = w; q < nrun; q += kThreads / 32) {
            const int off = s_off[q], len = s_len[q];
            const unsigned long long *src = key_in + gbeg + q * R + s_lo[q];
            if (off >= 0)
                for (int i = lane; i < len; i += 32) stage[off + i] = src[i];
        }
    }
    __syncthreads();
    // this warp's window of every staged stretch: lane r bounds run r from below by
    // the warp's first key, lane 16 + r from above by its last
    int win = 0;
    {
        const int nv = __popc(__ballot_sync(0xffffffffu, valid));
        const unsigned long long kfirst = __shfl_sync(0xffffffffu, kk, 0);
        const unsigned long long klast = __shfl_sync(0xffffffffu, kk, nv > 0 ? nv - 1 : 0);
        const int r = lane & 15, len = s_len[r], off = s_off[r];
        const unsigned long long k = (lane < 16 ? kfirst : klast) + (r < own ? 1ull : 0ull);
        if (off >= 0) {
            int hi = len;
            while (win < hi) {
                const int m = (win + hi) >> 1;
                if (stage[off + m] < k) win = m + 1;
                else hi = m;
            }
        }
    }
    __syncwarp();
    int place = t.x - (gbeg + own * R) + (int)threadIdx.x;  // in its own run
    for (int r0 = 0; r0 < nrun; r0 += kAhead) {
        // the keys of an earlier run precede an equal one: compare with k + 1
        int pos[kAhead], len[kAhead];
        const unsigned long long *src[kAhead];
        unsigned long long kq[kAhead];
        int longest = 0;
#pragma unroll
        for (int a = 0; a < kAhead; a++) {
            pos[a] = 0;
            const int r = r0 + a;
            const int wlo = __shfl_sync(0xffffffffu, win, r & 15), whi = __shfl_sync(0xffffffffu, win, 16 + (r & 15));
            len[a] = r < nrun ? whi - wlo : 0;
            const int off = s_off[r];
            src[a] = stage + (len[a] > 0 ? off + wlo : 0);
            kq[a] = kk + (r < own ? 1ull : 0ull);
            if (r < nrun) place += s_lo[r] + wlo;
            if (off < 0) {  // a stretch left in global memory
                const unsigned long long *run = key_in + gbeg + r * R + s_lo[r];
                int lo = 0, hi = s_len[r];
                while (lo < hi) {
                    const int m = (lo + hi) >> 1;
                    if (run[m] < kq[a]) lo = m + 1;
                    else hi = m;
                }
                place += lo;
                len[a] = 0;
                src[a] = stage;
            }
            longest = max(longest, len[a]);
        }
        // branch-free steps: the runs' loads overlap
        for (int step = longest > 0 ? 1 << (31 - __clz(longest)) : 0; step > 0; step >>= 1) {
            unsigned long long v[kAhead];
#pragma unroll
            for (int a = 0; a < kAhead; a++) v[a] = src[a][max(min(pos[a] + step, len[a]) - 1, 0)];
#pragma unroll
            for (int a = 0; a < kAhead; a++)
                pos[a] += (int)(pos[a] + step <= len[a]) & (int)(v[a] < kq[a]) ? step : 0;
        }
#pragma unroll
        for (int a = 0; a < kAhead; a++) place += pos[a];
    }
    if (valid) {
        key_out[gbeg + place] = kk;
        val_out[gbeg + place] = vv;
    }
}

// staged keys of a block: the expected stretches (its own width per run) and a
// quarter more
constexpr int stage_cap(int fan) { return fan * (kMergeTile + kMergeTile / 4); }
static_assert(stage_cap(kMergeFan) * sizeof(unsigned long long) <= 46 * 1024, "within every kernel's shared memory");

}  // namespace

int merge_passes(int max_bodies_of_a_system) {
    int passes = 0;
    for (int64_t R = kMergeRun; R < max_bodies_of_a_system; R *= kMergeFan) passes++;
    return passes;
}

// Merges the sorted runs of every system, in the fewest launches and with the
// smallest fan that they allow; the last launch writes d_key / d_val.
int merge_runs(Ctx *ctx, cudaStream_t st) {
    const int passes = merge_passes(ctx->max_sys);
    const int runs = ceil_div(ctx->max_sys, kMergeRun);
    unsigned long long *k0 = ctx->d_key, *k1 = ctx->d_key_alt;
    int *v0 = ctx->d_val, *v1 = ctx->d_val_alt;
    if (passes & 1) {
        std::swap(k0, k1);
        std::swap(v0, v1);
    }
    int fan = 1;
    for (;; fan++) {
        int64_t all = 1;
        for (int p = 0; p < passes; p++) all *= fan;
        if (all >= runs) break;
    }
    int R = kMergeRun;
    for (int pass = 0; pass < passes; pass++) {
        const int cap = stage_cap(fan);
        launch_chained(ctx, st, ctx->ntiles_mg, kThreads, sizeof(unsigned long long) * cap, k_merge, ctx->d_tiles_mg,
                       ctx->d_sys_off, R, fan, cap, k0, v0, k1, v1);
        std::swap(k0, k1);
        std::swap(v0, v1);
        R *= fan;
    }
    NBX_CUDA(cudaGetLastError());
    return NBX_OK;
}

}  // namespace nbx
