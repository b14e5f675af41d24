// walk_team.cu -- the force walk of small and mid-size systems: the interaction
// lists and evaluation of walk2.cu, with a team of warps (one block) per group
// of 32 bodies.
//
// One warp per group leaves most of the GPU idle below about 10^5 bodies, and
// the longest group's chain of rounds (load a cell, load its children, classify,
// evaluate up to 96 candidates: about 2.4 us) is the walk's time.  Here every
// warp holds the same 32 bodies and takes its own share of a round's children:
//   expand   warp 0 pops the top-of-stack cells (the shared stack holds each cell's
//            meta word, so a pop loads nothing from memory) and lists their
//            children in shared memory; the warps classify the list's 32-child
//            chunks in turn, warp w the chunks w, w + W, ...;
//   evaluate each warp evaluates and votes on its own candidates;
//   push     after a barrier the warps append their rejected cells to the stack
//            in warp order.
// The tests, and so the lists, are those of walk2.cu; the sums are the W warps'
// partial sums added in warp order, so a group's force bits depend on its own
// system only.  Which systems are walked by teams depends on the system's size
// alone (by_team): a batch gives every system the bits of its single run.
//
// Bound by latency where the GPU is not full (16384 bodies: 2.9 warps and 0.35
// instructions per scheduler and cycle).  Walk at 1000 / 16384 bodies: 38 / 212 us by
// single warps, 19 / 67 us by teams.  Four warps, three chunks: two chunks of rounds
// with 32 pops took 106 us at 16384, 64 pops 81 us, a child list with 128 pops and
// three chunks 70.
//
// Where a batch fills the GPU, teams are bound by issue and by their barriers: every
// warp pays a round's fixed instructions, and a group takes four warps' slots.  There
// one warp walks a group and takes the four shares in turn (one_warp): no barriers, no
// rejected cells to copy, empty shares skipped, and as the totals are in shared memory
// it needs no more registers.  Walks of 16384 systems of 512 bodies 3.71 ms by four
// warps, 2.59 by one; 8388 of 1000 4.54 / 3.70, 2097 of 4000 7.03 / 6.52, 512 of 16384
// 10.9 / 10.1 (rounds of walk2.cu's shape, whose sums are others: 2.2, 3.1, 5.4 and
// 9.1).  The kernel is near what the instruction cache holds: votes unrolled by eight
// cost 10 % in full batches.
#include <type_traits>

#include "nbx_internal.cuh"
#include "walk_eval.cuh"

namespace nbx {

namespace {

constexpr int kW = 4;                      // warps of a team
constexpr int kChunks = 3;                 // 32-child chunks per warp and round
constexpr int kPops = 4;                   // cells popped per lane and round, at most
constexpr int kRound = 32 * kW * kChunks;  // most children of a round
constexpr int kSlots = 32 * kChunks + 8;   // candidate slots per warp (its children, pads of the pair loops)
// Stack entries of a group.  (Of a stack_depth alone, 16384 bodies at an opening angle
// of 0.2 took 190 us instead of 140; of two, the one-warp form's warps per SM fall
// and 8388 systems of 1000 bodies take 3.80 instead of 3.70 ms.)
constexpr int team_stack(int stack_depth) { return stack_depth + stack_depth / 2; }

// Node ids of a round's candidates (recording only).
template <bool Rec>
struct TeamIds {
    int cid[kSlots];  // cells to vote on
    int bid[kSlots];  // the round's interactions
};
template <>
struct TeamIds<false> {};

// Per-warp candidate buffers.  The bodies (and, without quadrupoles, the surely
// accepted cells) fill the slots upwards, the cells to vote on downwards in
// pairs; with quadrupoles the cells are in the second arrays, those to vote on
// upwards, the surely accepted ones downwards.
template <int kN, bool Rec, bool Quad>
struct alignas(16) TeamBuf {
    Slots<kSlots> b;
    Slots<Quad ? kSlots : 4> c;  // quadrupole mode: cells
    float cd[kSlots];            // cells to vote on: opening thresholds
    int crec[kSlots];            // their stack entries
    int rej[kN > 1 ? 32 * kChunks : 4];  // rejected cells' stack entries (one warp pushes at once)
    TeamIds<Rec> ids;
    // slot of the i-th cell to vote on
    __device__ static int vote_slot(int i) { return Quad ? i : slot_down<kSlots>(i); }
    __device__ Slots<kSlots> &cells() {
        if constexpr (Quad) return c;
        else return b;
    }
};

// A share's totals over the rounds: in the plain mode the halves' sums, else the
// compensated totals and their compensations.
template <int Mode, bool Pot>
struct TeamPart {
    float a[Mode == 0 ? 3 : 6][32];
    float pot[Pot ? 32 : 4];
};

struct alignas(16) TeamShared {
    float4 cls[3];      // group box lo, hi, centre
    ulonglong2 rxy[8];  // representative bodies, in pairs: (x0,x1) (y0,y1)
    u64 rz[8];          //                                  (z0,z1)
    int4 nrej, nrec;    // per share
    int sum[kW][2];     // list length, opened cells
    int P, T;           // the round's popped cells and children
    int pad[2];
    int child[kRound];  // the round's children
};

static_assert(sizeof(TeamShared) % 16 == 0 && sizeof(TeamBuf<1, false, false>) % 16 == 0 &&
                  sizeof(TeamBuf<kW, true, false>) % 16 == 0 && sizeof(TeamBuf<kW, false, true>) % 16 == 0 &&
                  sizeof(TeamPart<0, false>) % 16 == 0 && sizeof(TeamPart<1, false>) % 16 == 0,
              "16-byte slots");

// Minimum and maximum over a warp of finite values (one instruction each).
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Ends a share's round (fold_round's rule): the plain mode's halves go to its totals
// as one sum.
template <int Mode, bool Pot>
__device__ __forceinline__ void fold_share(Sums &a, TeamPart<Mode, Pot> &t, int lane) {
    if constexpr (Mode == 0) {
        float a0, a1;
        upk(a.x, a0, a1);
        t.a[0][lane] += a0 + a1;
        upk(a.y, a0, a1);
        t.a[1][lane] += a0 + a1;
        upk(a.z, a0, a1);
        t.a[2][lane] += a0 + a1;
        a.x = a.y = a.z = 0ull;
        if constexpr (Pot) {
            upk(a.p, a0, a1);
            t.pot[lane] += a0 + a1;
            a.p = 0ull;
        }
    } else {
        Totals<Mode, Pot> none;
        fold_round(a, none, lane);
    }
}

// Barrier of a group's warps, which are a block's (kN warps).
template <int kN>
__device__ __forceinline__ void team_sync() {
    if constexpr (kN == 1) __syncwarp();
    else __syncthreads();
}

// kN warps walk a group: kW, one for each share of a round, or one that takes the
// shares in turn (the same sums: the same bits).
// With quadrupoles four warps' slots leave seven blocks an SM: 72 registers, hardly a spill
// (walk of 6000 / 12000 / 16384 bodies 54.3 / 83.2 / 91.1 us with 64, 51.4 / 78.0 / 85.7).
template <int kN, int Mode, bool Pot, bool Rec, bool Quad>
__global__ void __launch_bounds__(kN * 32, (Quad && kN > 1 ? 28 : 32) / kN)
    k_walk_team(const float4 *__restrict__ node4, const int *__restrict__ meta, const unsigned char *__restrict__ lvl8,
                const float4 *__restrict__ quad4, const float2 *__restrict__ quad2, const float4 *__restrict__ body4,
                const int *__restrict__ val, const int *__restrict__ groups, const int *__restrict__ list, int g_first,
                const int *__restrict__ body_sys, const int *__restrict__ sys_off, const float *__restrict__ depth0,
                const int *__restrict__ root_first, const int *__restrict__ root_nch, const int *__restrict__ sys_lvl,
                float eps2, int stack_cap, float *__restrict__ ax, float *__restrict__ ay, float *__restrict__ az,
                float *__restrict__ pot, int2 *__restrict__ gstat, DevStatus *st, int *__restrict__ rec_list,
                int *__restrict__ rec_len, int rec_cap) {
    grid_dependency();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // decided by the whole block: another block of this launch may report an error
    // (a full recording list) while these warps read the status, and a team that
    // lost some of its warps would run on with shared words nobody wrote
    if (kN == 1 ? __any_sync(0xffffffffu, st->code != 0) : __syncthreads_or(st->code != 0)) return;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    TeamShared &sh = *reinterpret_cast<TeamShared *>(smem_raw);
    using Buf = TeamBuf<kN, Rec, Quad>;
    using Part = TeamPart<Mode, Pot>;
    unsigned char *mem = smem_raw + sizeof(TeamShared);
    Buf &buf = reinterpret_cast<Buf *>(mem)[w];
    mem += kN * sizeof(Buf);
    QuadBuf<kSlots> &qbuf = reinterpret_cast<QuadBuf<kSlots> *>(mem)[w];
    if (Quad) mem += kN * sizeof(QuadBuf<kSlots>);
    Part *const parts = reinterpret_cast<Part *>(mem);  // of every share
    // the cells' meta words (first child, children - 1): a pop loads nothing from memory
    int *stack = reinterpret_cast<int *>(mem + kW * sizeof(Part));
    const unsigned lt = (1u << lane) - 1u;
    const u64 eps2x2 = pk(eps2, eps2);
    const int g = list ? list[g_first + blockIdx.x] : g_first + (int)blockIdx.x;
    const int p0 = groups[g];
    const int s = body_sys[p0];
    const int end = min(sys_off[s + 1], p0 + 32);
    const int reserve = 7 * min(max(sys_lvl[s], 1), 42) + 8;
    const int p = p0 + lane;
    const bool valid = p < end;
    // lanes past the end of the system take lane 0's body (their votes repeat its)
    const float4 me = body4[valid ? p : p0];
    const u64 px = pk(me.x, me.x), py = pk(me.y, me.y), pz = pk(me.z, me.z);
    const float d0 = depth0[s];
    {
        // the group's box and, per octant, its representative pair (walk2.cu): warp w
        // finds the octants w, w + kN, ...
        const float b[6] = {warp_min(me.x), warp_max(me.x), warp_min(me.y),
                            warp_max(me.y), warp_min(me.z), warp_max(me.z)};
        const float ex = me.x - 0.5f * (b[0] + b[1]), ey = me.y - 0.5f * (b[2] + b[3]);
        const float ez = me.z - 0.5f * (b[4] + b[5]);
        const unsigned key = __float_as_uint(ex * ex + ey * ey + ez * ez);
        const unsigned kmin = __reduce_min_sync(0xffffffffu, key);
        const int lc = __ffs(__ballot_sync(0xffffffffu, key == kmin)) - 1;
        if (threadIdx.x == 0) {
            sh.cls[0] = make_float4(b[0], b[2], b[4], 0.f);
            sh.cls[1] = make_float4(b[1], b[3], b[5], 0.f);
            sh.cls[2] = make_float4(0.5f * (b[0] + b[1]), 0.5f * (b[2] + b[3]), 0.5f * (b[4] + b[5]), 0.f);
        }
        const float nx = __shfl_sync(0xffffffffu, me.x, lc), ny = __shfl_sync(0xffffffffu, me.y, lc);
        const float nz = __shfl_sync(0xffffffffu, me.z, lc);
        for (int k = w; k < 8; k += kN) {
            const float pj = (k & 1 ? ex : -ex) + (k & 2 ? ey : -ey) + (k & 4 ? ez : -ez);
            const unsigned key_k = valid ? f2ord(pj) : 0u;
            const unsigned kmax = __reduce_max_sync(0xffffffffu, key_k);
            const int lf = __ffs(__ballot_sync(0xffffffffu, key_k == kmax)) - 1;
            const float xk = __shfl_sync(0xffffffffu, me.x, lf), yk = __shfl_sync(0xffffffffu, me.y, lf);
            const float zk = __shfl_sync(0xffffffffu, me.z, lf);
            if (lane == k) {
                sh.rxy[k] = make_ulonglong2(pk(xk, nx), pk(yk, ny));
                sh.rz[k] = pk(zk, nz);
            }
        }
    }
    Sums acc;
    for (int v = w; v < kW; v += kN) {
#pragma unroll
        for (int k = 0; k < (Mode == 0 ? 3 : 6); k++) parts[v].a[k][lane] = 0.f;
        if (Pot) parts[v].pot[lane] = 0.f;
    }
    int top = 0, nb = 0, len = 0, opened = 0, nrec = 0;
    unsigned rounds = 0;
    bool overflow = false;
    int *rec = Rec ? rec_list + (size_t)g * rec_cap : nullptr;

    // root children: cells are opened unconditionally, bodies interact (warp 0)
    {
        const int rf = root_first[s], rn = min(root_nch[s], 8);
        int cm = 0;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (lane < rn) {
            cm = meta[rf + lane];
            q = node4[rf + lane];
        }
        const unsigned bodies = __ballot_sync(0xffffffffu, lane < rn && cm < 0);
        const unsigned cells = __ballot_sync(0xffffffffu, lane < rn && cm >= 0);
        if (w == 0) {
            if (lane < rn && cm < 0) {
                buf.b.put(__popc(bodies & lt), q);
                if constexpr (Rec) buf.ids.bid[__popc(bodies & lt)] = rf + lane;
            }
            if (lane < rn && cm >= 0) stack[__popc(cells & lt)] = cm;
            nb = __popc(bodies);
            opened += __popc(cells);
        }
        top = __popc(cells);
    }
    const int root_cells = top;
    team_sync<kN>();

    for (bool first_round = true; top > 0 || first_round; first_round = false) {
        // ---- expand: warp 0 pops and lists the children; P = the most top-of-stack
        // cells that fit.  Lane j takes the K entries from stack[top-1-K*j] down: one
        // where that is all of the stack, else four (the list is the same; four always
        // are three times the instructions: 16384 systems of 512 bodies 3.78 -> 3.62
        // ms, 8388 of 1000 4.63 -> 4.46; a third form for two gained nothing and cost
        // 512 systems of 16384 5 %: 10.76 -> 11.34 ms)
        if (w == 0) {
            const int avail = min(top, 32 * kPops);
            const auto pop = [&](auto entries) {
                constexpr int K = decltype(entries)::value;
                int e[K];
                int n[K], x[K + 1];
                x[0] = 0;
#pragma unroll
                for (int i = 0; i < K; i++) {
                    const int at = K * lane + i;
                    e[i] = at < avail ? stack[top - 1 - at] : 0;
                    n[i] = at < avail ? ((e[i] >> 28) & 7) + 1 : 0;
                    x[i + 1] = x[i] + n[i];
                }
                int incl = x[K];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += u;
                }
                const int excl = incl - x[K];  // children before this lane's cells
                int np = 0, nt = 0;
#pragma unroll
                for (int i = 0; i < K; i++)
                    if (n[i] > 0 && excl + x[i + 1] <= kRound) {
                        np = i + 1;
                        nt = excl + x[i + 1];
                    }
                int P = __reduce_add_sync(0xffffffffu, np);
                int T = __reduce_max_sync(0xffffffffu, nt);
                // only cells that leave the depth-first reserve free, else one (walk2.cu)
                if (P > 1 && top - P + T > stack_cap - reserve) {
                    np = nt = 0;
#pragma unroll
                    for (int i = 0; i < K; i++) {
                        const int t = excl + x[i + 1], popped = K * lane + i + 1;
                        if (popped <= P && top - popped + t <= stack_cap - reserve) {
                            np = i + 1;
                            nt = t;
                        }
                    }
                    P = max(__reduce_add_sync(0xffffffffu, np), 1);
                    T = max(__reduce_max_sync(0xffffffffu, nt), __shfl_sync(0xffffffffu, n[0], 0));
                }
                if (P > 0 && top - P + T > stack_cap) P = 0;
                if (P == 0) T = 0;
                if (lane == 0) {
                    sh.P = P;
                    sh.T = T;
                }
#pragma unroll
                for (int i = 0; i < K; i++)
                    if (K * lane + i < P) {
                        const int first = e[i] & 0x0fffffff, at = excl + x[i];
#pragma unroll
                        for (int k = 0; k < 8; k++)
                            if (k < n[i]) sh.child[at + k] = first + k;
                    }
            };
            if (avail <= 32) pop(std::integral_constant<int, 1>());
            else pop(std::integral_constant<int, kPops>());
        }
        team_sync<kN>();
        const int P = sh.P, T = sh.T;
        if (P == 0 && top > 0) {
            overflow = true;
            break;
        }
        top -= P;
        rounds++;
        int pushed = 0, recorded = 0;  // by this warp's shares
#pragma unroll 1
        for (int v = w; v < kW; v += kN) {
            if (kN == 1 && 32 * v >= T && nb == 0) break;
            // one warp pushes at once: the popped cells are in the child list
            int *const rej = kN == 1 ? stack + top + pushed : buf.rej;
            Part &mine = parts[v];
            if (kN == 1 && Mode != 0) {
                acc.kx = mine.a[0][lane];
                acc.ky = mine.a[1][lane];
                acc.kz = mine.a[2][lane];
                acc.cx = mine.a[3][lane];
                acc.cy = mine.a[4][lane];
                acc.cz = mine.a[5][lane];
            }
            int nbody = nb, ncell = 0, nacc = 0, nrej = 0;
            nb = 0;
#pragma unroll
            for (int h = 0; h < kChunks; h++) {
                const int c0 = h * kW + v;  // the share's chunk: children [32 c0, 32 c0 + 32)
                if (32 * c0 >= T) break;
                const int t = 32 * c0 + lane;
                const bool ok = t < T;
                const int c = sh.child[ok ? t : 0];
                const float dpc = scale4(d0, (int)lvl8[c] - 1);  // its opening threshold, depth0 * 4^-level(popped cell)
                const int cm = ok ? meta[c] : 0;
                const float4 q = ok ? node4[c] : make_float4(0.f, 0.f, 0.f, 0.f);
                const bool isc = ok && cm >= 0;
                float4 qq4 = make_float4(0.f, 0.f, 0.f, 0.f);
                float2 qq2 = make_float2(0.f, 0.f);
                if (Quad && isc) {
                    qq4 = quad4[c];
                    qq2 = quad2[c];
                }
                // sure accepts and sure rejects, exactly as walk2.cu classifies
                bool sacc, srej;
                {
                    const float4 lo = sh.cls[0], hi = sh.cls[1], cen = sh.cls[2];
                    const float gx = fmaxf(0.f, fmaxf(__fsub_rn(lo.x, q.x), __fsub_rn(q.x, hi.x)));
                    const float gy = fmaxf(0.f, fmaxf(__fsub_rn(lo.y, q.y), __fsub_rn(q.y, hi.y)));
                    const float gz = fmaxf(0.f, fmaxf(__fsub_rn(lo.z, q.z), __fsub_rn(q.z, hi.z)));
                    sacc = dpc <= __fmaf_rn(gz, gz, __fmaf_rn(gy, gy, __fmaf_rn(gx, gx, eps2)));
                    const int oct = (q.x > cen.x ? 1 : 0) | (q.y > cen.y ? 2 : 0) | (q.z > cen.z ? 4 : 0);
                    const ulonglong2 R = sh.rxy[oct];
                    const u64 dx = sub2(pk(q.x, q.x), R.x), dy = sub2(pk(q.y, q.y), R.y);
                    const u64 dz = sub2(pk(q.z, q.z), sh.rz[oct]);
                    float ra, rb;
                    upk(fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, eps2x2))), ra, rb);
                    srej = ra < dpc || rb < dpc;
                }
                const bool tob = ok && (cm < 0 || (!Quad && isc && sacc));
                const bool toc = isc && !sacc && !srej;
                const bool tos = isc && !sacc && srej;
                const bool toa = Quad && isc && sacc;
                const unsigned bm = __ballot_sync(0xffffffffu, tob);
                const unsigned cmk = __ballot_sync(0xffffffffu, toc);
                const unsigned smk = __ballot_sync(0xffffffffu, tos);
                const unsigned amk = Quad ? __ballot_sync(0xffffffffu, toa) : 0u;
                if (toa) {  // surely accepted cells fill the cell buffer downwards
                    const int slot = kSlots - 1 - (nacc + __popc(amk & lt));
                    buf.cells().put(slot, q);
                    putq(qbuf.qa, qbuf.qb, qbuf.qc, slot, qq4, qq2);
                }
                const int vslot = ncell + __popc(cmk & lt);
                const int bslot = nbody + __popc(bm & lt);
                if (!Quad) {
                    if (tob || toc) buf.b.put(toc ? buf.vote_slot(vslot) : bslot, q);
                } else if (tob) {
                    buf.b.put(bslot, q);
                }
                if constexpr (Rec)
                    if (tob) buf.ids.bid[bslot] = c;
                if (toc) {
                    if (Quad) {
                        buf.cells().put(vslot, q);
                        putq(qbuf.qa, qbuf.qb, qbuf.qc, vslot, qq4, qq2);
                    }
                    buf.cd[vslot] = dpc;
                    buf.crec[vslot] = cm;
                    if constexpr (Rec) buf.ids.cid[vslot] = c;
                }
                if (tos) rej[nrej + __popc(smk & lt)] = cm;
                nbody += __popc(bm);
                ncell += __popc(cmk);
                nrej += __popc(smk);
                nacc += __popc(amk);
            }
            // pads: massless far-away candidates fill odd last pairs
            const int nbp = (nbody + 1) >> 1;
            if (lane == 0 && (nbody & 1)) buf.b.put(nbody, make_float4(1e18f, 1e18f, 1e18f, 0.f));
            if (lane == 8 && (ncell & 1)) {
                buf.cells().put(buf.vote_slot(ncell), make_float4(1e18f, 1e18f, 1e18f, 0.f));
                buf.cd[ncell] = -INFINITY;
                if (Quad) putq(qbuf.qa, qbuf.qb, qbuf.qc, ncell, make_float4(0.f, 0.f, 0.f, 0.f), make_float2(0.f, 0.f));
            }
            const int abeg = (kSlots - nacc) & ~1;
            if (Quad && lane == 9 && ((kSlots - nacc) & 1)) {
                buf.cells().put(abeg, make_float4(1e18f, 1e18f, 1e18f, 0.f));
                putq(qbuf.qa, qbuf.qb, qbuf.qc, abeg, make_float4(0.f, 0.f, 0.f, 0.f), make_float2(0.f, 0.f));
            }
            __syncwarp();

            // ---- evaluate bodies: no MAC
            const auto body_pair = [&](u64 x, u64 y, u64 z, u64 m) {
                const u64 dx = sub2(x, px);
                const u64 dy = sub2(y, py);
                const u64 dz = sub2(z, pz);
                u64 r = fma2(dx, dx, eps2x2);
                r = fma2(dy, dy, r);
                r = fma2(dz, dz, r);
                float ra, rb;
                upk(r, ra, rb);
                const u64 ri = pk(rsq(ra), rsq(rb));
                const u64 f = mul2(mul2(m, ri), mul2(ri, ri));
                accumulate<Mode, Pot>(acc, f, m, ri, dx, dy, dz);
            };
            const auto body_pairs = [&](int q, auto count) {  // whole double pairs from q
                constexpr int kN = decltype(count)::value;
#pragma unroll
                for (int u = 0; u < kN; u += 2) {
                    const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(&buf.b.x[2 * (q + u)]);
                    const ulonglong2 Y = *reinterpret_cast<const ulonglong2 *>(&buf.b.y[2 * (q + u)]);
                    const ulonglong2 Z = *reinterpret_cast<const ulonglong2 *>(&buf.b.z[2 * (q + u)]);
                    const ulonglong2 M = *reinterpret_cast<const ulonglong2 *>(&buf.b.m[2 * (q + u)]);
                    body_pair(X.x, Y.x, Z.x, M.x);
                    body_pair(X.y, Y.y, Z.y, M.y);
                }
            };
            int q0 = 0;
            for (; q0 + 8 <= nbp; q0 += 8) body_pairs(q0, std::integral_constant<int, 8>());
            if (nbp & 4) {
                body_pairs(q0, std::integral_constant<int, 4>());
                q0 += 4;
            }
            if (nbp & 2) {
                body_pairs(q0, std::integral_constant<int, 2>());
                q0 += 2;
            }
            if (nbp & 1)
                body_pair(reinterpret_cast<const u64 *>(buf.b.x)[q0], reinterpret_cast<const u64 *>(buf.b.y)[q0],
                          reinterpret_cast<const u64 *>(buf.b.z)[q0], reinterpret_cast<const u64 *>(buf.b.m)[q0]);
            if (Quad) {  // surely accepted cells, no vote
#pragma unroll 2
                for (int q = abeg >> 1; q < kSlots / 2; q++) {
                    const u64 dx = sub2(reinterpret_cast<const u64 *>(buf.cells().x)[q], px);
                    const u64 dy = sub2(reinterpret_cast<const u64 *>(buf.cells().y)[q], py);
                    const u64 dz = sub2(reinterpret_cast<const u64 *>(buf.cells().z)[q], pz);
                    u64 r = fma2(dx, dx, eps2x2);
                    r = fma2(dy, dy, r);
                    r = fma2(dz, dz, r);
                    float ra, rb;
                    upk(r, ra, rb);
                    const u64 ri = pk(rsq(ra), rsq(rb));
                    quad_term<Mode>(acc, qbuf, q, reinterpret_cast<const u64 *>(buf.cells().m)[q], ri, dx, dy, dz);
                }
            }
            // ---- evaluate cells: one vote per cell, accept or push
            const int ncp = (ncell + 1) >> 1;
            const int nsrej = nrej;
            int nlist = nbody;
            const auto vote_pair = [&](int q, u64 x, u64 y, u64 z, u64 m) {
                const float2 dp = reinterpret_cast<const float2 *>(buf.cd)[q];
                const float dpa = dp.x, dpb = dp.y;
                const u64 dx = sub2(x, px);
                const u64 dy = sub2(y, py);
                const u64 dz = sub2(z, pz);
                u64 r = fma2(dx, dx, eps2x2);
                r = fma2(dy, dy, r);
                r = fma2(dz, dz, r);
                float ra, rb;
                upk(r, ra, rb);
                const bool oka = __all_sync(0xffffffffu, dpa <= ra);
                const bool okb = __all_sync(0xffffffffu, dpb <= rb);
                if (oka || okb) {  // warp-uniform: a pair of rejected cells adds nothing
                    if (!Quad) {
                        float ma, mb;
                        upk(m, ma, mb);
                        const u64 ri = pk(rsq(ra), rsq(rb));
                        const u64 mm = pk(oka ? ma : 0.f, okb ? mb : 0.f);
                        const u64 f = mul2(mul2(mul2(mm, ri), ri), ri);
                        accumulate<Mode, Pot>(acc, f, mm, ri, dx, dy, dz);
                    } else {
                        const u64 ri = pk(oka ? rsq(ra) : 0.f, okb ? rsq(rb) : 0.f);
                        quad_term<Mode>(acc, qbuf, q, m, ri, dx, dy, dz);
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int slot = 2 * q + h;
                    if (!(h ? okb : oka)) {  // (a pad is accepted)
                        if (lane == 0) rej[nrej] = buf.crec[slot];
                        nrej++;
                    } else if constexpr (Rec) {
                        if (slot < ncell) {
                            if (lane == 0) buf.ids.bid[nlist] = buf.ids.cid[slot];
                            nlist++;
                        }
                    }
                }
            };
            if constexpr (Quad) for_pairs<4>(buf.cells(), 0, ncp, vote_pair);
            else for_pairs_down<4>(buf.b, ncp, vote_pair);
            len += nbody + ncell - (nrej - nsrej) + nacc;
            opened += nrej;
            if (nbody + ncell + nacc > 0) fold_share<Mode, Pot>(acc, mine, lane);
            if (kN == 1 && Mode != 0) {
                mine.a[0][lane] = acc.kx;
                mine.a[1][lane] = acc.ky;
                mine.a[2][lane] = acc.kz;
                mine.a[3][lane] = acc.cx;
                mine.a[4][lane] = acc.cy;
                mine.a[5][lane] = acc.cz;
            }
            pushed += nrej;
            if (kN > 1 && lane == 0) {
                reinterpret_cast<int *>(&sh.nrej)[w] = nrej;
                if (Rec) reinterpret_cast<int *>(&sh.nrec)[w] = nlist;
            }
            if (Rec) recorded = nlist;
            if (kN == 1) __syncwarp();  // the next share takes over the buffers
        }
        // ---- push: the shares' rejected cells, in their order
        if constexpr (kN == 1) {
            top += pushed;
        } else {
            __syncthreads();
            static_assert(kW == 4, "one int4 holds a count per share");
            const int4 nr = sh.nrej;
            const int before = (w > 0 ? nr.x : 0) + (w > 1 ? nr.y : 0) + (w > 2 ? nr.z : 0);
            for (int i = lane; i < pushed; i += 32) stack[top + before + i] = buf.rej[i];
            top += nr.x + nr.y + nr.z + nr.w;
            if constexpr (Rec) {
                const int4 nl = sh.nrec;
                const int rbefore = (w > 0 ? nl.x : 0) + (w > 1 ? nl.y : 0) + (w > 2 ? nl.z : 0);
                for (int i = lane; i < recorded; i += 32) {
                    const int at = nrec + rbefore + i;
                    if (at < rec_cap) rec[at] = buf.ids.bid[i];
                }
                nrec += nl.x + nl.y + nl.z + nl.w;
            }
            __syncthreads();
        }
    }
    if (overflow) {  // uniform over the block
        if (threadIdx.x == 0) set_status(st, NBX_ERR_STACK, g);
        return;
    }
    // ---- the shares' totals, added in their order
    if (kN > 1 && Mode != 0) {
        parts[w].a[0][lane] = acc.kx;
        parts[w].a[1][lane] = acc.ky;
        parts[w].a[2][lane] = acc.kz;
        parts[w].a[3][lane] = acc.cx;
        parts[w].a[4][lane] = acc.cy;
        parts[w].a[5][lane] = acc.cz;
    }
    if (lane == 0) {
        sh.sum[w][0] = len;
        sh.sum[w][1] = opened;
    }
    team_sync<kN>();
    for (int k = w; k < 3 && valid; k += kN) {  // component k
        float f = 0.f;
        if (Mode == 0) {
            f = parts[0].a[k][lane];
#pragma unroll
            for (int v = 1; v < kW; v++) f += parts[v].a[k][lane];
        } else {
            float c = 0.f;
#pragma unroll
            for (int v = 0; v < kW; v++) {
                kahan(f, c, parts[v].a[k][lane]);
                kahan(f, c, -parts[v].a[3 + k][lane]);
            }
            f -= c;
        }
        float *out = k == 0 ? ax : (k == 1 ? ay : az);
        out[val[p]] = f;
    }
    if (Pot && w == kN - 1 && valid) {
        float a = parts[0].pot[lane];
#pragma unroll
        for (int v = 1; v < kW; v++) a += parts[v].pot[lane];
        // remove the body's own term m * rsqrt(eps2), then phi = -sum
        pot[val[p]] = -(a - me.w * rsq(eps2));
    }
    if (threadIdx.x == 0) {
        int l = 0, o = 0;
#pragma unroll
        for (int v = 0; v < kN; v++) {
            l += sh.sum[v][0];
            o += sh.sum[v][1];
        }
        gstat[g] = make_int2(l, o);
        if (Rec) {
            rec_len[g] = nrec < rec_cap ? nrec : rec_cap;
            if (nrec > rec_cap) set_status(st, NBX_ERR_CAPACITY, g);
        }
        atomicAdd(&st->interactions, (unsigned long long)l * (unsigned long long)(end - p0));
        atomicAdd(&st->opened, (unsigned long long)o);
        atomicAdd(&st->rounds, (unsigned long long)rounds);
        // every child is a list entry or was opened (the root's cells are no one's children)
        atomicAdd(&st->candidates, (unsigned long long)(l + o - root_cells));
    }
}

template <int kN, int Mode, bool Pot, bool Rec, bool Quad>
size_t team_smem(int stack_depth) {
    return sizeof(TeamShared) + kN * (sizeof(TeamBuf<kN, Rec, Quad>) + (Quad ? sizeof(QuadBuf<kSlots>) : 0)) +
           kW * sizeof(TeamPart<Mode, Pot>) + (size_t)team_stack(stack_depth) * sizeof(int);
}

template <int kN, int Mode, bool Pot, bool Rec, bool Quad>
int launch_warps(Ctx *ctx, const nbx_state *s, float *pot, cudaStream_t st, const int *list, int first, int count,
                 int *rec_list, int *rec_len, int rec_cap) {
    const size_t smem = team_smem<kN, Mode, Pot, Rec, Quad>(ctx->p.stack_depth);
    if (smem > (size_t)ctx->smem_optin) {
        ctx->last_error = "walk: stack_depth too large for the launch shape's shared memory";
        return NBX_ERR_ARG;
    }
    // (only deep stacks and the quadrupoles' slots need more than the default limit)
    if (smem > 48 * 1024)
        NBX_CUDA(cudaFuncSetAttribute(k_walk_team<kN, Mode, Pot, Rec, Quad>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->smem_optin));
    // in plain stream order, as the walk by single warps: blocks placed while the build's
    // last kernel holds some of the SMs fill the others (eager steps of 1000 / 6000 /
    // 16000 bodies 66 / 110 / 149 us chained, 61 / 100 / 129 not; with quadrupoles 99 /
    // 168 / 215 and 94 / 154 / 192)
    ctx->chain = false;
    launch_chained(ctx, st, count, kN * 32, smem, k_walk_team<kN, Mode, Pot, Rec, Quad>, ctx->d_node4, ctx->d_meta,
                   ctx->d_lvl8, ctx->d_quad4, ctx->d_quad2, ctx->d_body4, ctx->d_val, ctx->d_groups, list, first,
                   ctx->d_body_sys, ctx->d_sys_off, ctx->d_depth0, ctx->d_root_first, ctx->d_root_nch, ctx->d_sys_lvl,
                   ctx->eps2, team_stack(ctx->p.stack_depth), s->ax, s->ay, s->az, pot, ctx->d_gstat, ctx->d_status,
                   rec_list, rec_len, rec_cap);
    NBX_CUDA(cudaGetLastError());
    return NBX_OK;
}

// One warp per group where that is faster: where the groups are enough to fill the
// GPU so many times over that a group's latency no longer counts, which is the
// sooner the smaller the systems (their rounds leave warps of a team idle).  Walks
// by one warp against four: 2180 groups of systems of 300 bodies 37 / 43 us, 34950
// 265 / 406; of 1000 bodies 2080 groups 57 / 57, 33536 467 / 570; of 4000 8125 groups
// 255 / 247, 32750 831 / 894; of 16384 16384 groups 762 / 743, 32768 1.33 / 1.40 ms.
// With quadrupoles, whose slots leave fewer warps per SM, only for small systems
// (33536 groups of 1000 bodies 926 / 1005 us, but 32750 of 4000 1.73 / 1.60 ms).
// Both forms give the same bits.
bool one_warp(const Ctx *ctx, int count, bool quad) {
    const int mean = 32 * (ctx->nteam / ctx->nteam_sys);  // bodies of a system, about
    const int per_sm = mean / 40 < 12 ? 12 : (mean / 40 > 160 ? 160 : mean / 40);
    return count > (int64_t)per_sm * ctx->nsm && !(quad && mean > 1536);
}

template <int Mode, bool Pot, bool Rec, bool Quad>
int launch_team(Ctx *ctx, const nbx_state *s, float *pot, cudaStream_t st, const int *list, int first, int count,
                int *rec_list, int *rec_len, int rec_cap) {
    if constexpr (!Rec)  // (recording walks keep their ids by warp)
        if (one_warp(ctx, count, Quad))
            return launch_warps<1, Mode, Pot, Rec, Quad>(ctx, s, pot, st, list, first, count, rec_list, rec_len, rec_cap);
    return launch_warps<kW, Mode, Pot, Rec, Quad>(ctx, s, pot, st, list, first, count, rec_list, rec_len, rec_cap);
}

}  // namespace

// The walk of `count` groups by teams: groups first, first + 1, ..., or the
// entries first, ... of `list` (device array) where it is given.  mode: -1
// potential too, 0..2 the accumulation modes; rec_list: recording (mode 0).
int walk_team(Ctx *ctx, const nbx_state *s, float *pot, int mode, bool quad, cudaStream_t st, const int *list,
              int first, int count, int *rec_list, int *rec_len, int rec_cap) {
    if (count <= 0) return NBX_OK;
    if (rec_list)
        return launch_team<0, false, true, false>(ctx, s, nullptr, st, list, first, count, rec_list, rec_len, rec_cap);
    if (pot) return launch_team<0, true, false, false>(ctx, s, pot, st, list, first, count, nullptr, nullptr, 0);
    if (quad) switch (mode) {
            case 1: return launch_team<1, false, false, true>(ctx, s, pot, st, list, first, count, nullptr, nullptr, 0);
            case 2: return launch_team<2, false, false, true>(ctx, s, pot, st, list, first, count, nullptr, nullptr, 0);
            default: return launch_team<0, false, false, true>(ctx, s, pot, st, list, first, count, nullptr, nullptr, 0);
        }
    switch (mode) {
        case 1: return launch_team<1, false, false, false>(ctx, s, pot, st, list, first, count, nullptr, nullptr, 0);
        case 2: return launch_team<2, false, false, false>(ctx, s, pot, st, list, first, count, nullptr, nullptr, 0);
        default: return launch_team<0, false, false, false>(ctx, s, pot, st, list, first, count, nullptr, nullptr, 0);
    }
}

}  // namespace nbx
