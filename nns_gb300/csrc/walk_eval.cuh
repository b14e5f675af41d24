// walk_eval.cuh -- evaluation pieces shared by the force walks (walk2.cu,
// walk_team.cu): candidate slots, packed force terms, accumulation modes.
#pragma once

#include "f32x2.cuh"
#include "nbx_internal.cuh"

namespace nbx {

// depth0 * 4^-k exactly (a power-of-two product is exact unless it underflows)
__device__ __forceinline__ float scale4(float d0, int k) {
    return d0 * __int_as_float((127 - 2 * k) << 23);
}

// Kahan step s += v with compensation c (scalar, explicit rounding).
__device__ __forceinline__ void kahan(float &s, float &c, float v) {
    const float y = __fsub_rn(v, c);
    const float t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
}

// Candidate slots, one array per component: a candidate is stored with four
// 4-byte stores at one offset (consecutive slots, no bank conflicts), and two
// pairs are read with four 16-byte loads.
template <int N>
struct alignas(16) Slots {
    float x[N], y[N], z[N], m[N];
    __device__ __forceinline__ void put(int slot, float4 q) {
        x[slot] = q.x;
        y[slot] = q.y;
        z[slot] = q.z;
        m[slot] = q.w;
    }
};

// Calls f(pair index, x, y, z, m) for the packed pairs [0, n) of the slots from
// `first` (a multiple of four), two pairs per load.
template <int Unroll, int N, typename F>
__device__ __forceinline__ void for_pairs(const Slots<N> &s, int first, int n, F &&f) {
    const ulonglong2 *x = reinterpret_cast<const ulonglong2 *>(s.x + first);
    const ulonglong2 *y = reinterpret_cast<const ulonglong2 *>(s.y + first);
    const ulonglong2 *z = reinterpret_cast<const ulonglong2 *>(s.z + first);
    const ulonglong2 *m = reinterpret_cast<const ulonglong2 *>(s.m + first);
#pragma unroll (Unroll / 2)
    for (int q = 0; q < n >> 1; q++) {
        const ulonglong2 X = x[q], Y = y[q], Z = z[q], M = m[q];
        f(2 * q, X.x, Y.x, Z.x, M.x);
        f(2 * q + 1, X.y, Y.y, Z.y, M.y);
    }
    if (n & 1) {
        const int q = n >> 1;
        f(n - 1, x[q].x, y[q].x, z[q].x, m[q].x);
    }
}

// The same for pairs that fill the slots downwards: pair q in the two slots below
// N - 2 q, its first candidate in the lower one.
template <int Unroll, int N, typename F>
__device__ __forceinline__ void for_pairs_down(const Slots<N> &s, int n, F &&f) {
    static_assert(N % 4 == 0, "whole double pairs");
    const ulonglong2 *x = reinterpret_cast<const ulonglong2 *>(s.x), *y = reinterpret_cast<const ulonglong2 *>(s.y);
    const ulonglong2 *z = reinterpret_cast<const ulonglong2 *>(s.z), *m = reinterpret_cast<const ulonglong2 *>(s.m);
#pragma unroll (Unroll / 2)
    for (int q = 0; q < n >> 1; q++) {
        const int at = N / 4 - 1 - q;
        const ulonglong2 X = x[at], Y = y[at], Z = z[at], M = m[at];
        f(2 * q, X.y, Y.y, Z.y, M.y);
        f(2 * q + 1, X.x, Y.x, Z.x, M.x);
    }
    if (n & 1) {
        const int at = N / 4 - 1 - (n >> 1);
        f(n - 1, x[at].y, y[at].y, z[at].y, m[at].y);
    }
}
template <int N>
__device__ __forceinline__ constexpr int slot_down(int i) {
    return N - 2 - 2 * (i >> 1) + (i & 1);
}

// Quadrupole mode: the traceless quadrupoles of the cell buffer's slots, in
// pairs: (xx, yy), (zz, xy), (xz, yz).
template <int CB>
struct QuadBuf {
    static constexpr int kPairs = CB / 2;
    ulonglong2 qa[kPairs];
    ulonglong2 qb[kPairs];
    ulonglong2 qc[kPairs];
};

__device__ __forceinline__ void putq(ulonglong2 *qa, ulonglong2 *qb, ulonglong2 *qc, int slot, float4 q4, float2 q2) {
    float *pa = reinterpret_cast<float *>(&qa[slot >> 1]);
    float *pb = reinterpret_cast<float *>(&qb[slot >> 1]);
    float *pc = reinterpret_cast<float *>(&qc[slot >> 1]);
    const int h = slot & 1;
    pa[h] = q4.x;
    pa[2 + h] = q4.y;
    pb[h] = q4.z;
    pb[2 + h] = q4.w;
    pc[h] = q2.x;
    pc[2 + h] = q2.y;
}

struct Sums {
    u64 x = 0ull, y = 0ull, z = 0ull, p = 0ull;  // packed partial sums of the round (+0.0f, +0.0f)
    float kx = 0.f, ky = 0.f, kz = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;  // Kahan totals
};

// Plain mode: a warp's packed totals of the rounds before, in shared memory (in
// registers they cost the loops theirs: 2^20 bodies 1.85 against 1.82 ms).
template <int Mode, bool Pot>
struct Totals {};
template <>
struct Totals<0, false> {
    u64 x[32], y[32], z[32];
};
template <>
struct Totals<0, true> {
    u64 x[32], y[32], z[32], p[32];
};
template <int Mode, bool Pot>
__device__ __forceinline__ void clear_totals(Totals<Mode, Pot> &t, int lane) {
    if constexpr (Mode == 0) t.x[lane] = t.y[lane] = t.z[lane] = 0ull;
    if constexpr (Mode == 0 && Pot) t.p[lane] = 0ull;
}

// Ends a round: its sums go to the totals, plainly or compensated (mode 2 adds
// every term to the compensated totals by itself).  A term that outweighs the
// rest (a star) then rounds only what its own round still adds and one sum per
// later round, whenever it comes.  In one running sum it rounded every later term,
// and the wider a round the earlier it came: medians against FP64 sums of the same
// lists, binary disk of 2^24 bodies, rounds of 96 children 9.8e-7, of 128 10.5e-7,
// of 128 with their own sums 1.8e-7 (Plummer, 2^20: 3.5e-7, 3.5e-7, 0.7e-7), for 1 %
// of the walk's time (2^20 bodies 1.80 -> 1.82 ms).
template <int Mode, bool Pot>
__device__ __forceinline__ void fold_round(Sums &a, Totals<Mode, Pot> &t, int lane) {
    if constexpr (Mode == 0) {
        t.x[lane] = add2(t.x[lane], a.x);
        t.y[lane] = add2(t.y[lane], a.y);
        t.z[lane] = add2(t.z[lane], a.z);
        a.x = a.y = a.z = 0ull;
        if constexpr (Pot) {
            t.p[lane] = add2(t.p[lane], a.p);
            a.p = 0ull;
        }
    }
    if (Mode == 1) {
        float a0, a1;
        upk(a.x, a0, a1);
        kahan(a.kx, a.cx, a0);
        kahan(a.kx, a.cx, a1);
        upk(a.y, a0, a1);
        kahan(a.ky, a.cy, a0);
        kahan(a.ky, a.cy, a1);
        upk(a.z, a0, a1);
        kahan(a.kz, a.cz, a0);
        kahan(a.kz, a.cz, a1);
        a.x = a.y = a.z = 0ull;
    }
}

// Accumulate the packed force factor f = m*rsqrt(r)^3 of two candidates.
template <int Mode, bool Pot>
__device__ __forceinline__ void accumulate(Sums &a, u64 f, u64 mm, u64 ri, u64 dx, u64 dy, u64 dz) {
    if (Mode == 2) {
        float xa, xb, ya, yb, za, zb;
        upk(mul2(f, dx), xa, xb);
        upk(mul2(f, dy), ya, yb);
        upk(mul2(f, dz), za, zb);
        kahan(a.kx, a.cx, xa);
        kahan(a.kx, a.cx, xb);
        kahan(a.ky, a.cy, ya);
        kahan(a.ky, a.cy, yb);
        kahan(a.kz, a.cz, za);
        kahan(a.kz, a.cz, zb);
    } else {
        a.x = fma2(f, dx, a.x);
        a.y = fma2(f, dy, a.y);
        a.z = fma2(f, dz, a.z);
    }
    if (Pot) a.p = fma2(mm, ri, a.p);
}

// Accumulate r^-2 v for two candidates: the quadrupole mode's contribution.
template <int Mode>
__device__ __forceinline__ void accumulate_quad(Sums &a, u64 ri2, u64 vx, u64 vy, u64 vz) {
    if (Mode == 2) {
        float xa, xb, ya, yb, za, zb;
        upk(mul2(ri2, vx), xa, xb);
        upk(mul2(ri2, vy), ya, yb);
        upk(mul2(ri2, vz), za, zb);
        kahan(a.kx, a.cx, xa);
        kahan(a.kx, a.cx, xb);
        kahan(a.ky, a.cy, ya);
        kahan(a.ky, a.cy, yb);
        kahan(a.kz, a.cz, za);
        kahan(a.kz, a.cz, zb);
    } else {
        a.x = fma2(ri2, vx, a.x);
        a.y = fma2(ri2, vy, a.y);
        a.z = fma2(ri2, vz, a.z);
    }
}

// One pair of cells of the quadrupole mode, with the cells' negated traceless
// quadrupoles P = -Q from slot pair q of the buffer (d = cell - body,
// r^2 = |d|^2 + eps^2, e = d / r):
//   a += m d r^-3 - Q d r^-5 + 5/2 (d.Q.d) d r^-7
//      = r^-2 [ (m - 5/2 (e.P.e) r^-2) e + (P e) r^-2 ].
// In the unit-vector form every intermediate is bounded by |Q| or by the
// mass and force scales, and the only power of r^-1 is r^-2 <= 1 / eps^2.
// With d itself, r^-5 and r^-7 overflow FP32 once r is below about 1e-8, and
// d.Q.d (~ |Q| d^2) underflows for cells of about 1e-12 and less, dropping a
// term that is 1e-2 of such a pair's force.  A rejected half of a voted pair
// comes with ri = 0, so its e and r^-2, and its whole term, are 0.
template <int Mode, int CB>
__device__ __forceinline__ void quad_term(Sums &acc, const QuadBuf<CB> &qbuf, int q, u64 mm, u64 ri, u64 dx, u64 dy,
                                          u64 dz) {
    const ulonglong2 QA = qbuf.qa[q], QB = qbuf.qb[q], QC = qbuf.qc[q];
    const u64 ri2 = mul2(ri, ri);
    const u64 ex = mul2(dx, ri), ey = mul2(dy, ri), ez = mul2(dz, ri);
    // P e: P = (xx, yy, zz, xy | xz, yz) in QA = (xx, yy), QB = (zz, xy), QC = (xz, yz)
    const u64 px = fma2(QC.x, ez, fma2(QB.y, ey, mul2(QA.x, ex)));
    const u64 py = fma2(QC.y, ez, fma2(QA.y, ey, mul2(QB.y, ex)));
    const u64 pz = fma2(QB.x, ez, fma2(QC.y, ey, mul2(QC.x, ex)));
    const u64 epe = fma2(ez, pz, fma2(ey, py, mul2(ex, px)));
    const u64 mq = fma2(mul2(epe, ri2), pk(-2.5f, -2.5f), mm);
    accumulate_quad<Mode>(acc, ri2, fma2(mq, ex, mul2(px, ri2)), fma2(mq, ey, mul2(py, ri2)),
                          fma2(mq, ez, mul2(pz, ri2)));
}

}  // namespace nbx
