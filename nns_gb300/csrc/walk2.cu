// walk2.cu -- the production force walk: same interaction lists as walk.cu
// (the reference's warp-coherent MAC, 3D/CUDA/CUDA_NBody/src/Kernels.cu:460-577),
// organised for throughput on sm_103a.
//
// Per warp (one aligned group of 32 sorted bodies), rounds of
//   expand   the P top-of-stack cells whose children fit the buffers are popped
//            at once, one per lane; their child blocks (contiguous in the BFS
//            node array) are spread over the lanes, one child per lane.  Each
//            lane classifies its child cell against the group's box and the
//            representative pair of the child's octant (exactly, see below): surely accepted cells
//            join the bodies in the body buffer, surely rejected cells are
//            pushed at once, the rest go to the cell buffer with their
//            threshold dp = depth0 * 0.25^(L-1) and id;
//   evaluate every lane streams the buffers with broadcast shared-memory loads,
//            two candidates per instruction with the packed FP32 pair
//            instructions (add/fma/mul .rn.f32x2: each lane an IEEE FP32 op, so r
//            and the MAC decisions are bit-identical to the scalar form).  Body
//            buffer pairs go straight to the accumulation; each cell of the cell
//            buffer takes one warp vote (dp <= r on every lane) and is
//            accumulated or pushed.
// A round pops as many cells as leave a depth-first reserve free on the stack (7
// entries per level of the group's system's deepest level), and one where none do:
// that can never outgrow the reserve, so a stack of at least kDfsReserve + 7*8
// entries cannot overflow (NBX_ERR_STACK otherwise).  (Rounds near the reserve
// popped one cell each before, whatever room was left, which opening angles below
// 0.25 ran into all the time: 2^20 bodies at 0.1375 37.8 -> 33.3 ms, 131071 with a
// stack of 384 9.6 -> 4.3.)
//
// Accumulation modes: 0 plain FP32 (two packed partial sums per round, added to two
// packed totals), 1 split compensation (plain FP32 within a round, Kahan across
// rounds), 2 Kahan on every term.  Optional per-body potential for the energy
// diagnostics.
#include <algorithm>

#include "nbx_internal.cuh"
#include "walk_eval.cuh"

namespace nbx {

namespace {

// Stack entries kept free for depth-first descent: from any stack content a
// depth-first walk (one cell per round) grows the stack by at most 7 entries per
// level below the popped cell, i.e. by less than 7 * (deepest level) <= 7 * 42.
// The walk uses the bound of the tree at hand (its deepest level, recorded by
// the build); kDfsReserve is the bound for any tree.
constexpr int kDfsReserve = 7 * 42 + 8;

// Build-time tuning knobs of the evaluation loops (defaults are the measured best).
#ifndef NBX_BODY_UNROLL
#define NBX_BODY_UNROLL 16
#endif
#ifndef NBX_CELL_UNROLL
#define NBX_CELL_UNROLL 4
#endif
#ifndef NBX_WALK64_THREADS
#define NBX_WALK64_THREADS 512
#endif
#ifndef NBX_WALK64_MINB
#define NBX_WALK64_MINB 2
#endif
#ifndef NBX_WALK128_THREADS
#define NBX_WALK128_THREADS 256
#endif
#ifndef NBX_WALK128_MINB
#define NBX_WALK128_MINB 3
#endif
// (#pragma arguments are not macro-expanded: the unroll factors go through constants)
constexpr int kBodyUnroll = NBX_BODY_UNROLL;
constexpr int kCellUnroll = NBX_CELL_UNROLL;

// Per-warp candidate buffers for CB children.  The bodies (and, without
// quadrupoles, the surely accepted cells) fill the slots upwards and the cells to
// vote on downwards, so one masked store serves both; with quadrupoles the cells
// have slots of their own.  (Four slots more: each side pads to a whole pair.)
template <int CB, int Mode, bool Pot, bool Rec, bool Quad>
struct WarpBuf {
    Slots<CB + 4> b;
    Slots<Quad ? CB : 4> c; // quadrupole mode: cells
    float cd[CB];           // cells to vote on: opening thresholds
    int cid[CB];            //                   node index
    int bid[Rec ? CB : 4];  // body node ids (interaction-list recording only)
    float4 cls[3];          // group box lo, hi, centre
    ulonglong2 rxy[8];      // representative bodies, in pairs: (x0,x1) (y0,y1)
    u64 rz[8];              //                                  (z0,z1)
    Totals<Mode, Pot> tot;
};

// The buffer variants: children per round and register budget.  0: 64 children;
// 3: 128 (96 with quadrupoles and with split compensation), both at 64 registers
// (two 16-warp or four 8-warp blocks per SM); 1: 128 at up to 85 registers, for
// more loads in flight (three 8-warp blocks).  Rounds of 128 pay their fixed
// instructions less often than rounds of 96: 131071 bodies 1.69 -> 1.63 ms for
// four steps, 2^24 155.4 -> 153.7 ms.  With quadrupoles, whose slots take more
// shared memory, they cost an eighth of the warps (700001 bodies 8.21 against 7.19
// ms); split compensation (mode 1) sums plainly within a round, so a longer round
// is a longer uncompensated sum.
template <int V, int Mode, bool Quad>
struct WalkShape {
    static constexpr int kSlots = V == 0 ? 64 : (V == 3 && (Quad || Mode == 1) ? 96 : 128);
    static constexpr int kThreads = V != 1 ? NBX_WALK64_THREADS : NBX_WALK128_THREADS;
    static constexpr int kMinBlocks = V != 1 ? NBX_WALK64_MINB : NBX_WALK128_MINB;
};

template <int V, int Mode, bool Pot, bool Rec, bool Quad = false>
__global__ void __launch_bounds__(WalkShape<V, Mode, Quad>::kThreads, WalkShape<V, Mode, Quad>::kMinBlocks)
    k_walk2(const float4 *__restrict__ node4, const int *__restrict__ meta, const unsigned char *__restrict__ lvl8,
            const float4 *__restrict__ quad4, const float2 *__restrict__ quad2, const float4 *__restrict__ body4,
            const int *__restrict__ val, const int *__restrict__ groups, const int *__restrict__ list, int ngroups,
            const int *__restrict__ body_sys, const int *__restrict__ sys_off, const float *__restrict__ depth0,
            const int *__restrict__ root_first, const int *__restrict__ root_nch, const int *__restrict__ sys_lvl,
            float eps2, int stack_cap,
            float *__restrict__ ax, float *__restrict__ ay, float *__restrict__ az, float *__restrict__ pot,
            int2 *__restrict__ gstat, DevStatus *st, int *__restrict__ rec_list,
            int *__restrict__ rec_len, int rec_cap) {
    grid_dependency();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (st->code != 0) return;
    const int warps = blockDim.x >> 5;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int CB = WalkShape<V, Mode, Quad>::kSlots, kCB = CB;
    using Buf = WarpBuf<CB, Mode, Pot, Rec, Quad>;
    Buf &buf = reinterpret_cast<Buf *>(smem_raw)[w];
    constexpr size_t kQuadBytes = Quad ? sizeof(QuadBuf<CB>) : 0;
    QuadBuf<CB> &qbuf = reinterpret_cast<QuadBuf<CB> *>(smem_raw + sizeof(Buf) * warps)[w];
    int *stack = reinterpret_cast<int *>(smem_raw + (sizeof(Buf) + kQuadBytes) * warps) + w * stack_cap;
    const unsigned lt = (1u << lane) - 1u;
    const u64 eps2x2 = pk(eps2, eps2);
    unsigned long long tot_len = 0ull, tot_open = 0ull, tot_rounds = 0ull, tot_cand = 0ull;

    // groups are handed out dynamically (costs vary widely between groups); the last
    // warp to find none left leaves the counter at zero for the next launch
    for (;;) {
        int g = 0;
        if (lane == 0) g = (int)atomicAdd(&st->walk_next, 1u);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= ngroups) {
            if (lane == 0 && g - ngroups == (int)gridDim.x * warps - 1) st->walk_next = 0u;
            break;
        }
        if (list) g = list[g];
        const int p0 = groups[g];
        const int s = body_sys[p0];
        const int end = min(sys_off[s + 1], p0 + 32);
        // the depth-first reserve from this system's own tree, so that a system's
        // rounds (and force sums) do not depend on the other systems of a batch
        const int reserve = 7 * min(max(sys_lvl[s], 1), 42) + 8;
        const int p = p0 + lane;
        const bool valid = p < end;
        // lanes past the end of the system take lane 0's body: their MAC votes
        // repeat lane 0's and their results are discarded
        const float4 me = body4[valid ? p : p0];
        const u64 px = pk(me.x, me.x), py = pk(me.y, me.y), pz = pk(me.z, me.z);
        const float d0 = depth0[s];
        {
            // the group's box and representative bodies, for classifying children
            float b[6] = {me.x, me.x, me.y, me.y, me.z, me.z};
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                for (int k = 0; k < 6; k += 2) {
                    b[k] = fminf(b[k], __shfl_xor_sync(0xffffffffu, b[k], o));
                    b[k + 1] = fmaxf(b[k + 1], __shfl_xor_sync(0xffffffffu, b[k + 1], o));
                }
            }
            // the body nearest the box centre (lane lc)
            const float ex = me.x - 0.5f * (b[0] + b[1]), ey = me.y - 0.5f * (b[2] + b[3]);
            const float ez = me.z - 0.5f * (b[4] + b[5]);
            const unsigned key = __float_as_uint(ex * ex + ey * ey + ez * ez);
            const unsigned kmin = __reduce_min_sync(0xffffffffu, key);
            const int lc = __ffs(__ballot_sync(0xffffffffu, key == kmin)) - 1;
            if (lane == 0) {
                buf.cls[0] = make_float4(b[0], b[2], b[4], 0.f);
                buf.cls[1] = make_float4(b[1], b[3], b[5], 0.f);
                buf.cls[2] = make_float4(0.5f * (b[0] + b[1]), 0.5f * (b[2] + b[3]), 0.5f * (b[4] + b[5]), 0.f);
            }
            // representative pairs for the sure-reject test, one per octant k (bit
            // a set: the cell lies on the + side of axis a, seen from the box
            // centre): the body furthest along that diagonal and the body nearest
            // the centre.  Any valid body is a correct representative; these two
            // catch 86 % of the rejected cells before the vote (the first and last
            // body of the group caught 58 %).
            {
                const float nx = __shfl_sync(0xffffffffu, me.x, lc), ny = __shfl_sync(0xffffffffu, me.y, lc);
                const float nz = __shfl_sync(0xffffffffu, me.z, lc);
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const float pj = (k & 1 ? ex : -ex) + (k & 2 ? ey : -ey) + (k & 4 ? ez : -ez);
                    const unsigned key_k = valid ? f2ord(pj) : 0u;
                    const unsigned kmax = __reduce_max_sync(0xffffffffu, key_k);
                    const int le = __ffs(__ballot_sync(0xffffffffu, key_k == kmax)) - 1;
                    const float xk = __shfl_sync(0xffffffffu, me.x, le), yk = __shfl_sync(0xffffffffu, me.y, le);
                    const float zk = __shfl_sync(0xffffffffu, me.z, le);
                    if (lane == k) {
                        buf.rxy[k] = make_ulonglong2(pk(xk, nx), pk(yk, ny));
                        buf.rz[k] = pk(zk, nz);
                    }
                }
            }
            __syncwarp();
        }
        Sums acc;
        clear_totals(buf.tot, lane);
        int top = 0, nb = 0, len = 0, opened = 0, nrec = 0;
        bool overflow = false;
        int *rec = Rec ? rec_list + (size_t)g * rec_cap : nullptr;

        // root children: cells are opened unconditionally, bodies interact
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
            if (lane < rn && cm < 0) {
                buf.b.put(__popc(bodies & lt), q);
                if (Rec) buf.bid[__popc(bodies & lt)] = rf + lane;
            }
            if (lane < rn && cm >= 0) stack[__popc(cells & lt)] = rf + lane;
            nb = __popc(bodies);
            top = __popc(cells);
            opened += top;
            __syncwarp();
        }

        while (top > 0 || nb > 0) {
            // ---- expand: lane j pops stack[top-1-j] and copies its children
            // P = the most top-of-stack cells whose children fit the buffers and, if
            // all were pushed, would leave the depth-first reserve free (P cells grow
            // the stack by at most T - P, which grows with P); where not even one
            // does, one cell per round (depth-first), which cannot outgrow the reserve
            const int avail = min(top, 32);
            int first = 0, nch = 0;
            float dpp = 0.f;  // the children's opening threshold, depth0 * 4^-level(popped cell)
            if (lane < avail) {
                const int b = stack[top - 1 - lane];  // stack entries are node indices
                const int mb = meta[b];
                first = mb & 0x0fffffff;
                nch = ((mb >> 28) & 7) + 1;
                dpp = scale4(d0, lvl8[b]);
            }
            int incl = nch;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += u;
            }
            const int excl = incl - nch;
            const int cbase = first - excl;  // child t of this lane's cell is node cbase + t
            // (the quadrupole mode keeps one slot free: its two cell regions are
            // padded to whole pairs independently)
            int P = __popc(__ballot_sync(0xffffffffu, lane < avail && incl <= kCB - nb - (Quad ? 1 : 0) &&
                                                          top + incl - lane - 1 <= stack_cap - reserve));
            if (P == 0 && avail > 0) P = 1;
            int T = __shfl_sync(0xffffffffu, incl, (P + 31) & 31);
            if (P > 0 && top - P + T > stack_cap) P = 0;
            if (P == 0) T = 0;
            if (P == 0 && nb == 0) {
                overflow = true;
                break;
            }
            __syncwarp();
            top -= P;
            // the T children are spread over the lanes, 32 at a time: lane t
            // finds its popped cell j (largest j < P with excl_j <= t) by counting
            // the segment starts at or below t in a bit mask of the starts
            unsigned seg[kCB / 32];
#pragma unroll
            for (int k = 0; k < kCB / 32; k++)
                seg[k] = __reduce_or_sync(0xffffffffu, (lane < P && (excl >> 5) == k) ? 1u << (excl & 31) : 0u);
            // Each child cell is classified by its lane before any warp-wide work:
            //   sure accept: a lower bound of every lane's r (the gaps between the
            //     cell and the group box, in the walk's own FP32 operation order;
            //     rounding is monotone) is >= dp, so the vote would pass: the cell
            //     goes to the body buffer (no vote);
            //   sure reject: a representative body's r (computed exactly as its
            //     lane does) is < dp, so the vote would fail: pushed at once;
            //   otherwise it is voted on in the cell buffer.
            // The interaction lists are unchanged; only their order differs.
            int nbody = nb, ncell = 0, nsrej = 0, nacc = 0;
            int jbase = -1;
#pragma unroll
            for (int k = 0; k < kCB / 32; k++) {
                const int t0 = 32 * k;
                if (t0 >= T) break;
                const int t = t0 + lane;
                const unsigned le = lane == 31 ? 0xffffffffu : (2u << lane) - 1u;
                const int j = jbase + __popc(seg[k] & le);
                jbase += __popc(seg[k]);
                const int bj = __shfl_sync(0xffffffffu, cbase, j);
                const float dpc = __shfl_sync(0xffffffffu, dpp, j);
                const bool ok = t < T;
                const int c = bj + t;
                const int cm = ok ? meta[c] : 0;
                const float4 q = ok ? node4[c] : make_float4(0.f, 0.f, 0.f, 0.f);
                const bool isc = ok && cm >= 0;
                float4 qq4 = make_float4(0.f, 0.f, 0.f, 0.f);
                float2 qq2 = make_float2(0.f, 0.f);
                if (Quad && isc) {
                    qq4 = quad4[c];
                    qq2 = quad2[c];
                }
                bool sacc = false, srej = false;
                {  // on every lane, without a branch; the results are masked by isc below
                    const float4 lo = buf.cls[0], hi = buf.cls[1];
                    const float gx = fmaxf(0.f, fmaxf(__fsub_rn(lo.x, q.x), __fsub_rn(q.x, hi.x)));
                    const float gy = fmaxf(0.f, fmaxf(__fsub_rn(lo.y, q.y), __fsub_rn(q.y, hi.y)));
                    const float gz = fmaxf(0.f, fmaxf(__fsub_rn(lo.z, q.z), __fsub_rn(q.z, hi.z)));
                    sacc = dpc <= __fmaf_rn(gz, gz, __fmaf_rn(gy, gy, __fmaf_rn(gx, gx, eps2)));
                    // the representative pair of the cell's octant, in one packed
                    // instruction with the operations and order of the evaluation
                    // (so r is their lanes' r exactly)
                    const u64 qx = pk(q.x, q.x), qy = pk(q.y, q.y), qz = pk(q.z, q.z);
                    {
                        const float4 cen = buf.cls[2];
                        const int oct = (q.x > cen.x ? 1 : 0) | (q.y > cen.y ? 2 : 0) | (q.z > cen.z ? 4 : 0);
                        const ulonglong2 R = buf.rxy[oct];
                        const u64 dx = sub2(qx, R.x), dy = sub2(qy, R.y), dz = sub2(qz, buf.rz[oct]);
                        float ra, rb;
                        upk(fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, eps2x2))), ra, rb);
                        srej = ra < dpc || rb < dpc;
                    }
                }
                // quadrupole mode: accepted cells need their quadrupoles, so a surely
                // accepted cell goes to the top of the cell buffer (filled downwards),
                // evaluated without a vote; the cells to vote on fill it upwards
                const bool tob = ok && (cm < 0 || (!Quad && isc && sacc));
                const bool toc = isc && !sacc && !srej;
                const bool tos = isc && !sacc && srej;
                const bool toa = Quad && isc && sacc;
                const unsigned bm = __ballot_sync(0xffffffffu, tob);
                const unsigned cmk = __ballot_sync(0xffffffffu, toc);
                const unsigned smk = __ballot_sync(0xffffffffu, tos);
                if (Quad) {
                    const unsigned amk = __ballot_sync(0xffffffffu, toa);
                    if (toa) {
                        const int slot = kCB - 1 - (nacc + __popc(amk & lt));
                        buf.c.put(slot, q);
                        putq(qbuf.qa, qbuf.qb, qbuf.qc, slot, qq4, qq2);
                    }
                    nacc += __popc(amk);
                }
                const int bslot = nbody + __popc(bm & lt), vslot = ncell + __popc(cmk & lt);
                if (!Quad) {
                    if (tob || toc) buf.b.put(toc ? slot_down<CB + 4>(vslot) : bslot, q);
                } else if (tob) {
                    buf.b.put(bslot, q);
                }
                if (Rec && tob) buf.bid[bslot] = c;
                if (toc) {
                    if (Quad) {
                        buf.c.put(vslot, q);
                        putq(qbuf.qa, qbuf.qb, qbuf.qc, vslot, qq4, qq2);
                    }
                    buf.cd[vslot] = dpc;
                    buf.cid[vslot] = c;
                }
                if (tos) stack[top + nsrej + __popc(smk & lt)] = c;
                nbody += __popc(bm);
                ncell += __popc(cmk);
                nsrej += __popc(smk);
            }
            top += nsrej;
            // pad odd buffers with a massless far-away candidate that is accepted
            if (lane == 0 && (nbody & 1)) buf.b.put(nbody, make_float4(1e18f, 1e18f, 1e18f, 0.f));
            if (lane == 1 && (ncell & 1)) {
                if (Quad) buf.c.put(ncell, make_float4(1e18f, 1e18f, 1e18f, 0.f));
                else buf.b.put(slot_down<CB + 4>(ncell), make_float4(1e18f, 1e18f, 1e18f, 0.f));
                buf.cd[ncell] = -INFINITY;
                if (Quad)
                    putq(qbuf.qa, qbuf.qb, qbuf.qc, ncell, make_float4(0.f, 0.f, 0.f, 0.f), make_float2(0.f, 0.f));
            }
            // the accepted region [kCB - nacc, kCB) starts on a whole pair: a
            // massless, quadrupole-free far candidate fills its odd first slot
            // (ncell + nacc < kCB keeps it clear of the voted region's pad)
            const int abeg = (kCB - nacc) & ~1;
            if (Quad && lane == 2 && ((kCB - nacc) & 1)) {
                buf.c.put(abeg, make_float4(1e18f, 1e18f, 1e18f, 0.f));
                putq(qbuf.qa, qbuf.qb, qbuf.qc, abeg, make_float4(0.f, 0.f, 0.f, 0.f), make_float2(0.f, 0.f));
            }
            __syncwarp();

            // ---- evaluate bodies: no MAC
            for_pairs<kBodyUnroll>(buf.b, 0, (nbody + 1) >> 1, [&](int, u64 x, u64 y, u64 z, u64 m) {
                const u64 dx = sub2(x, px);
                const u64 dy = sub2(y, py);
                const u64 dz = sub2(z, pz);
                u64 r = fma2(dx, dx, eps2x2);
                r = fma2(dy, dy, r);
                r = fma2(dz, dz, r);
                float ra, rb;
                upk(r, ra, rb);
                const u64 ri = pk(rsq(ra), rsq(rb));
                // no MAC depends on this product: (m ri)(ri ri) shortens its dependency chain
                const u64 f = mul2(mul2(m, ri), mul2(ri, ri));
                accumulate<Mode, Pot>(acc, f, m, ri, dx, dy, dz);
            });
            if (Rec) {  // every body candidate is an interaction
                for (int t = lane; t < nbody; t += 32)
                    if (nrec + t < rec_cap) rec[nrec + t] = buf.bid[t];
                nrec += nbody;
            }
            // ---- quadrupole mode: surely accepted cells, no vote
            if (Quad) {
#pragma unroll (kCellUnroll)
                for (int q = abeg >> 1; q < kCB / 2; q++) {
                    const u64 dx = sub2(reinterpret_cast<const u64 *>(buf.c.x)[q], px);
                    const u64 dy = sub2(reinterpret_cast<const u64 *>(buf.c.y)[q], py);
                    const u64 dz = sub2(reinterpret_cast<const u64 *>(buf.c.z)[q], pz);
                    u64 r = fma2(dx, dx, eps2x2);
                    r = fma2(dy, dy, r);
                    r = fma2(dz, dz, r);
                    float ra, rb;
                    upk(r, ra, rb);
                    const u64 ri = pk(rsq(ra), rsq(rb));
                    quad_term<Mode>(acc, qbuf, q, reinterpret_cast<const u64 *>(buf.c.m)[q], ri, dx, dy, dz);
                }
            }
            // ---- evaluate cells: one vote per cell, accept or push
            int nrej = 0;
            const auto vote_pair = [&](int q, u64 x, u64 y, u64 z, u64 m) {
                const float2 dp = reinterpret_cast<const float2 *>(buf.cd)[q];
                const u64 dx = sub2(x, px);
                const u64 dy = sub2(y, py);
                const u64 dz = sub2(z, pz);
                u64 r = fma2(dx, dx, eps2x2);
                r = fma2(dy, dy, r);
                r = fma2(dz, dz, r);
                float ra, rb;
                upk(r, ra, rb);
                const bool oka = __all_sync(0xffffffffu, dp.x <= ra);
                const bool okb = __all_sync(0xffffffffu, dp.y <= rb);
                if (oka || okb) {  // warp-uniform: a pair of rejected cells adds nothing
                    if (!Quad) {
                        float ma, mb;
                        upk(m, ma, mb);
                        const u64 ri = pk(rsq(ra), rsq(rb));
                        const u64 mm = pk(oka ? ma : 0.f, okb ? mb : 0.f);
                        const u64 f = mul2(mul2(mul2(mm, ri), ri), ri);
                        accumulate<Mode, Pot>(acc, f, mm, ri, dx, dy, dz);
                    } else {
                        // the rejected half of the pair masked through r^-1 (its term is 0)
                        const u64 ri = pk(oka ? rsq(ra) : 0.f, okb ? rsq(rb) : 0.f);
                        quad_term<Mode>(acc, qbuf, q, m, ri, dx, dy, dz);
                    }
                }
                if (!oka) {
                    if (lane == 0) stack[top + nrej] = buf.cid[2 * q];
                    nrej++;
                } else if (Rec && 2 * q < ncell) {
                    if (lane == 0 && nrec < rec_cap) rec[nrec] = buf.cid[2 * q];
                    nrec++;
                }
                if (!okb) {
                    if (lane == 0) stack[top + nrej] = buf.cid[2 * q + 1];
                    nrej++;
                } else if (Rec && 2 * q + 1 < ncell) {
                    if (lane == 0 && nrec < rec_cap) rec[nrec] = buf.cid[2 * q + 1];
                    nrec++;
                }
            };
            if constexpr (Quad) for_pairs<kCellUnroll>(buf.c, 0, (ncell + 1) >> 1, vote_pair);
            else for_pairs_down<kCellUnroll>(buf.b, (ncell + 1) >> 1, vote_pair);
            top += nrej;
            tot_rounds += 1ull;
            tot_cand += (unsigned long long)(nbody + ncell + nsrej + nacc);
            len += nbody + ncell - nrej + nacc;
            opened += nrej + nsrej;
            nb = 0;
            fold_round(acc, buf.tot, lane);
            __syncwarp();
        }
        if (overflow) {
            if (lane == 0) set_status(st, NBX_ERR_STACK, g);
            continue;
        }
        if (Rec && lane == 0) {
            rec_len[g] = nrec < rec_cap ? nrec : rec_cap;
            if (nrec > rec_cap) set_status(st, NBX_ERR_CAPACITY, g);
        }
        if (valid) {
            float fx, fy, fz;
            if constexpr (Mode == 0) {
                float a0, a1;
                upk(buf.tot.x[lane], a0, a1);
                fx = a0 + a1;
                upk(buf.tot.y[lane], a0, a1);
                fy = a0 + a1;
                upk(buf.tot.z[lane], a0, a1);
                fz = a0 + a1;
            } else {
                fx = acc.kx - acc.cx;
                fy = acc.ky - acc.cy;
                fz = acc.kz - acc.cz;
            }
            const int ob = val[p];
            ax[ob] = fx;
            ay[ob] = fy;
            az[ob] = fz;
            if constexpr (Pot) {
                float a0, a1;
                upk(buf.tot.p[lane], a0, a1);
                // remove the body's own term m * rsqrt(eps2), then phi = -sum
                pot[ob] = -((a0 + a1) - me.w * rsq(eps2));
            }
        }
        if (lane == 0) gstat[g] = make_int2(len, opened);
        tot_len += (unsigned long long)len * (unsigned long long)(end - p0);
        tot_open += (unsigned long long)opened;
    }
    if (lane == 0 && (tot_len | tot_open)) {
        atomicAdd(&st->interactions, tot_len);
        atomicAdd(&st->opened, tot_open);
        atomicAdd(&st->rounds, tot_rounds);
        atomicAdd(&st->candidates, tot_cand);
    }
}

#ifndef NBX_SPREAD_BLOCK
#define NBX_SPREAD_BLOCK 2
#endif
constexpr int kSpreadBlock = NBX_SPREAD_BLOCK;  // warps of a block of a launch that fits the GPU at once
constexpr int kSpreadWarps = 32;                // such a launch has at most this many groups per SM

// Which groups one launch walks: `count` from the first, or the entries of a list
// (device array) from there on.
struct Share {
    const int *list;
    int first, count;
};

template <int V, int Mode, bool Pot, bool Rec = false, bool Quad = false>
int launch(Ctx *ctx, const nbx_state *s, float *pot, int warps, cudaStream_t st, Share share,
           int *rec_list = nullptr, int *rec_len = nullptr, int rec_cap = 0) {
    constexpr int kCB = WalkShape<V, Mode, Quad>::kSlots;
    const int cap = ctx->p.stack_depth;
    const size_t per_warp = sizeof(WarpBuf<kCB, Mode, Pot, Rec, Quad>) + (Quad ? sizeof(QuadBuf<kCB>) : 0) +
                            (size_t)cap * sizeof(int);
    // (the rounds' totals came later: a shape that fits without them goes out in
    // blocks that do, below)
    if ((size_t)warps * (per_warp - sizeof(Totals<Mode, Pot>)) > (size_t)ctx->smem_optin) {
        ctx->last_error = "walk: stack_depth too large for the launch shape's shared memory";
        return NBX_ERR_ARG;
    }
    if (share.count <= 0) return NBX_OK;
    // groups that all fit the GPU at once go out in small blocks, which spread
    // evenly over the SMs (the sums do not depend on the shape)
    if (share.count <= kSpreadWarps * ctx->nsm && warps > kSpreadBlock) warps = kSpreadBlock;
    while (warps > 1 && warps * per_warp > (size_t)ctx->smem_optin) warps >>= 1;
    const size_t block_smem = warps * per_warp;
    const int blocks_needed = ceil_div(share.count, warps);
    int per_sm = 1;
    NBX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_walk2<V, Mode, Pot, Rec, Quad>, warps * 32,
                                                           block_smem));
    if (per_sm < 1) per_sm = 1;
    const int grid = blocks_needed < ctx->nsm * per_sm ? blocks_needed : ctx->nsm * per_sm;
    // without a list the group arrays start at the first group
    const int off = share.list ? 0 : share.first;
    // in plain stream order: blocks that are placed while the build's last kernel still
    // holds some of the SMs fill the others, and the walk lasts as long as the fullest
    // (an eager step of 65536 bodies 396 against 287 us)
    ctx->chain = false;
    launch_chained(
        ctx, st, grid, warps * 32, block_smem, k_walk2<V, Mode, Pot, Rec, Quad>,
        ctx->d_node4, ctx->d_meta, ctx->d_lvl8, ctx->d_quad4, ctx->d_quad2, ctx->d_body4, ctx->d_val,
        ctx->d_groups + off, share.list ? share.list + share.first : nullptr, share.count, ctx->d_body_sys,
        ctx->d_sys_off, ctx->d_depth0, ctx->d_root_first, ctx->d_root_nch, ctx->d_sys_lvl, ctx->eps2, cap, s->ax,
        s->ay, s->az, pot, ctx->d_gstat + off, ctx->d_status, rec_list, rec_len, rec_cap);
    NBX_CUDA(cudaGetLastError());
    return NBX_OK;
}

template <int V, int Mode, bool Pot, bool Rec = false, bool Quad = false>
int set_attr(Ctx *ctx, int smem_max) {
    NBX_CUDA(cudaFuncSetAttribute(k_walk2<V, Mode, Pot, Rec, Quad>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  smem_max));
    return NBX_OK;
}

template <int V>
int forces_cb(Ctx *ctx, const nbx_state *s, float *pot, int warps, cudaStream_t st, Share share) {
    if (pot) return launch<V, 0, true>(ctx, s, pot, warps, st, share);
    if (ctx->multipole) {
        switch (ctx->compensated) {
            case 1: return launch<V, 1, false, false, true>(ctx, s, nullptr, warps, st, share);
            case 2: return launch<V, 2, false, false, true>(ctx, s, nullptr, warps, st, share);
            default: return launch<V, 0, false, false, true>(ctx, s, nullptr, warps, st, share);
        }
    }
    switch (ctx->compensated) {
        case 1: return launch<V, 1, false>(ctx, s, nullptr, warps, st, share);
        case 2: return launch<V, 2, false>(ctx, s, nullptr, warps, st, share);
        default: return launch<V, 0, false>(ctx, s, nullptr, warps, st, share);
    }
}

// The groups [g0, g0 + gn) of one kind (walked by teams, or by single warps), as
// a share: of a context whose groups are all of one kind, the range itself;
// of a batch of both kinds, a stretch of that kind's ascending list.
Share share_of(const Ctx *ctx, bool team, int g0, int gn) {
    const int all = team ? ctx->nteam : ctx->ngroups - ctx->nteam;
    if (all == 0) return {nullptr, 0, 0};
    if (all == ctx->ngroups) return {nullptr, g0, gn};
    const std::vector<int> &mine = team ? ctx->h_team : ctx->h_solo;
    const int a = (int)(std::lower_bound(mine.begin(), mine.end(), g0) - mine.begin());
    const int b = (int)(std::lower_bound(mine.begin(), mine.end(), g0 + gn) - mine.begin());
    return {team ? ctx->d_team : ctx->d_solo, a, b - a};
}

}  // namespace

int walk2_init(Ctx *ctx) {
    const int smem_optin = ctx->smem_optin;
    int rc = 0;
    rc |= set_attr<0, 0, false>(ctx, smem_optin);
    rc |= set_attr<0, 1, false>(ctx, smem_optin);
    rc |= set_attr<0, 2, false>(ctx, smem_optin);
    rc |= set_attr<0, 0, true>(ctx, smem_optin);
    rc |= set_attr<1, 0, false>(ctx, smem_optin);
    rc |= set_attr<1, 1, false>(ctx, smem_optin);
    rc |= set_attr<1, 2, false>(ctx, smem_optin);
    rc |= set_attr<1, 0, true>(ctx, smem_optin);
    rc |= set_attr<3, 0, false>(ctx, smem_optin);
    rc |= set_attr<3, 1, false>(ctx, smem_optin);
    rc |= set_attr<3, 2, false>(ctx, smem_optin);
    rc |= set_attr<3, 0, true>(ctx, smem_optin);
    rc |= set_attr<3, 0, false, true>(ctx, smem_optin);
    rc |= set_attr<0, 0, false, false, true>(ctx, smem_optin);
    rc |= set_attr<0, 1, false, false, true>(ctx, smem_optin);
    rc |= set_attr<0, 2, false, false, true>(ctx, smem_optin);
    rc |= set_attr<1, 0, false, false, true>(ctx, smem_optin);
    rc |= set_attr<1, 1, false, false, true>(ctx, smem_optin);
    rc |= set_attr<1, 2, false, false, true>(ctx, smem_optin);
    rc |= set_attr<3, 0, false, false, true>(ctx, smem_optin);
    rc |= set_attr<3, 1, false, false, true>(ctx, smem_optin);
    rc |= set_attr<3, 2, false, false, true>(ctx, smem_optin);
    return rc;
}

// Plain walk that also records every group's interaction list (node ids, in
// evaluation order) into rec_list[g * rec_cap ...], its length into rec_len[g].
int walk2_record(Ctx *ctx, const nbx_state *s, int *rec_list, int *rec_len, int rec_cap, cudaStream_t st) {
    const int rc = launch<3, 0, false, true>(ctx, s, nullptr, ctx->walk_warps, st,
                                              share_of(ctx, false, 0, ctx->ngroups), rec_list, rec_len, rec_cap);
    if (rc) return rc;
    const Share t = share_of(ctx, true, 0, ctx->ngroups);
    return walk_team(ctx, s, nullptr, 0, false, st, t.list, t.first, t.count, rec_list, rec_len, rec_cap);
}

// The same walk without recording: the recording adds stores only, so both
// give the same forces bit for bit (the adjoint's forward and recompute).
int walk2_unrecorded(Ctx *ctx, const nbx_state *s, cudaStream_t st) {
    const int rc = launch<3, 0, false, false>(ctx, s, nullptr, ctx->walk_warps, st,
                                               share_of(ctx, false, 0, ctx->ngroups));
    if (rc) return rc;
    const Share t = share_of(ctx, true, 0, ctx->ngroups);
    return walk_team(ctx, s, nullptr, 0, false, st, t.list, t.first, t.count, nullptr, nullptr, 0);
}

// variants 0, 1 (<= 8 warps) and 3: WalkShape
// (of the single-warp walk; small systems' groups are walked by teams, whose shape is fixed).
// Walk groups [g0, g0 + gn) of the last build (gn < 0: all groups from g0).
int walk2_forces(Ctx *ctx, const nbx_state *s, float *pot, int warps, cudaStream_t st, int g0, int gn) {
    if (gn < 0) gn = ctx->ngroups - g0;
    if (!pot && ctx->multipole && !ctx->d_quad4) return NBX_ERR_STATE;
    const Share r = share_of(ctx, false, g0, gn), t = share_of(ctx, true, g0, gn);
    // (a launch shape that does not fit is refused whatever the groups' kind)
    int rc;
    if (ctx->walk_variant == 1) rc = forces_cb<1>(ctx, s, pot, warps > 8 ? 8 : warps, st, r);
    else if (ctx->walk_variant == 3) rc = forces_cb<3>(ctx, s, pot, warps, st, r);
    else rc = forces_cb<0>(ctx, s, pot, warps, st, r);
    if (rc) return rc;
    return walk_team(ctx, s, pot, ctx->compensated, ctx->multipole != 0, st, t.list, t.first, t.count, nullptr,
                     nullptr, 0);
}

}  // namespace nbx
