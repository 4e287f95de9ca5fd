// One loop-frequency node of the vertex flow, for all the triples that read the same slabs.
//
// With x the transfer frequency of a channel and a >= b the two other frequencies of a triple
// (mesh indices), the access buffers of
//     the s channel of (x, a, b) and of (x, b, a), the u channel of (b, a, x) and of (a, b, x), and
//     the t channel of (a, x, b) with its site-local vertices
// all interpolate the four magnitudes of
//     A = (x - (a - b))/2 + w,  B = (x + (a - b))/2 + w,  P = (x + (a + b))/2 + w,  Q = (x - (a + b))/2 + w
// at the loop frequency w, with the same node list (that of x).  The s and u channels read four
// planes at a stored pair with x,
//     G0: (t, u) = (|A|, |B|), G1: (|P|, |Q|), G2: (|B|, |A|), G3: (|Q|, |P|)   [slab (x, t, u)],
// and differ in the site exchange (the signs of A, B, P, Q) and in the sign of the density where
// the stored sector swaps s and u.  The t channel reads two planes at t = x,
//     T0: (s, u) = (|Q|, |P|), T1: (|A|, |B|);
// its third and fourth buffer swap s and u, the same stored slabs with the density's sign
// flipped, and its site-local vertices are the G planes at site pair 0.  So a node of (x, {a, b})
// takes 24 slab segments for two s/u-channel nodes and one t-channel node; evaluated triple by
// triple the same three nodes take 48 segments and 16 site-local reads.  For three indices
// p >= q >= r the items (p, {q, r}), (q, {p, r}), (r, {p, q}) close on the three triples
// (p, q, r), (p, r, q), (q, p, r), so one warp (or CTA) evaluates them with nothing to exchange.
//
// Density signs.  The s channel of (x, ., .) reads slab (x, t, u) with a minus where x < u
// (indices).  The u channel of (., ., x) reads the same slab as (u, t, x), with a minus where
// u < x, and enters with the opposite coefficient; written with h = -(its density) its integrand
// is the s channel's with the density output's sign reversed, and h has the s channel's signs
// except on the diagonal u = x, where it is -1 (kU) instead of +1 (kS).  The diagonal
// density vanishes for the states of a flow, but not for an arbitrary state, so it is kept.
//
// All arithmetic is spelled out in single rounded operations, so the kernels that share this
// code give the same bits.
#pragma once
#include "su2_common.cuh"
#include "su2_device.cuh"

namespace spn {
namespace dev {

// Packed single-precision pairs (f32x2): per element the IEEE round-to-nearest result.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, z, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
        "fma.rn.f32x2 w, x, y, z;\n\tmov.b64 {%0, %1}, w;\n}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
        "mul.rn.f32x2 w, x, y;\n\tmov.b64 {%0, %1}, w;\n}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
        "add.rn.f32x2 w, x, y;\n\tmov.b64 {%0, %1}, w;\n}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
        "sub.rn.f32x2 w, x, y;\n\tmov.b64 {%0, %1}, w;\n}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// (spin, density) sum of one triple at one site, Kahan-compensated: `lost` is what the last
// addition to `sum` rounded away.
struct Acc {
    float2 sum, lost;
    __device__ __forceinline__ void clear() { sum = lost = make_float2(0.0f, 0.0f); }
    __device__ __forceinline__ void add(float2 c, float2 v) {
        const float2 y = fma2(c, v, lost);
        const float2 t = add2(sum, y);
        lost = sub2(y, sub2(t, sum));
        sum = t;
    }
    __device__ __forceinline__ float2 value() const { return add2(sum, lost); }
};
__device__ __forceinline__ void swap_acc(Acc &a, Acc &b) {
    const Acc t = a;
    a = b;
    b = t;
}

// Items of an n-frequency mesh: index triples p >= q >= r.
__host__ __device__ inline int vertex_items(int n) { return int((long long)n * (n + 1) * (n + 2) / 6); }

__device__ __forceinline__ void decode_item(int item, int &p, int &q, int &r) {
    p = int(cbrtf(6.0f * float(item)));
    while (p > 0 && p * (p + 1) * (p + 2) / 6 > item) --p;
    while ((p + 1) * (p + 2) * (p + 3) / 6 <= item) ++p;
    const int rest = item - p * (p + 1) * (p + 2) / 6;
    q = int((sqrtf(8.0f * float(rest) + 1.0f) - 1.0f) * 0.5f);
    while (q * (q + 1) / 2 > rest) --q;
    while ((q + 1) * (q + 2) / 2 <= rest) ++q;
    r = rest - q * (q + 1) / 2;
}

// One transfer frequency of an item: x and the pair a >= b.  h + l is (x - m)/2, (x + m)/2,
// (x + q)/2, (x - q)/2 with m = a - b, q = a + b to twice the working precision (two-sum error
// terms), so that A, B, P, Q lose nothing where the frequencies cancel.
struct ItemFreq {
    int xi;
    bool u_signs;  // density signs of the u channel (both targets are u-channel nodes)
    float h[4], l[4];
};
// a + b = s + e exactly
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
    s = __fadd_rn(a, b);
    const float t = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t));
}
__device__ __forceinline__ ItemFreq item_freq(const float *pos, int xi, int ai, int bi, bool u_signs) {
    ItemFreq f;
    f.xi = xi;
    f.u_signs = u_signs;
    const float x = pos[xi];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float s, e, h, l;
        two_sum(pos[ai], k < 2 ? -pos[bi] : pos[bi], s, e);
        const bool minus = k == 0 || k == 3;
        two_sum(x, minus ? -s : s, h, l);
        f.h[k] = 0.5f * h;
        f.l[k] = 0.5f * __fadd_rn(l, minus ? -e : e);
    }
    return f;
}

// Node descriptor: 272 bytes, so 8 lanes' 16-byte stores to consecutive descriptors hit distinct banks.
struct __align__(16) ItemDesc {
    int4 g[4];    // element offsets of the G planes' supports: (t, u) at (lower, lower), (upper, lower), (lower,
                  // upper), (upper, upper)
    int4 t[2];    // the same of T0, (s, u) = (|Q|, |P|), and T1, (|A|, |B|)
    float4 w[4];  // A, B, P, Q: weight of the lower point, the same with the density's sign as the u coordinate of a G
                  // plane, weight of the upper point, the same with its sign
    float4 tw[2][2];  // T0, T1: per support the weight and the density's weight in the first buffer (0 on the diagonal)
    float4 td[2];     // T0, T1: per support the density's weight if it is on the diagonal, else 0
    float c;          // node coefficient (s-channel sign)
    int flags, pad[2];
};
static_assert(sizeof(ItemDesc) == 272, "ItemDesc layout");

// flags: site exchange of G0..G3 for the first target, of G0 and G2 for the second; of T0 and T2,
// T1, T3; a t plane with diagonal supports; diagonal supports of G0..G3 (u lower, upper).
enum : int {
    kFlE0 = 1 << 0, kFlE1 = 1 << 1, kFlE2 = 1 << 2, kFlE3 = 1 << 3, kFlF0 = 1 << 4, kFlF2 = 1 << 5,
    kFlT0 = 1 << 6, kFlT1 = 1 << 7, kFlT3 = 1 << 8,
    kFlDiagT = 1 << 9,
    kFlDiagShift = 10,
    kFlDiag = 0xff << kFlDiagShift,
    kFlExT = 1 << 18  // T3's site exchange is not T1's
};

__device__ __forceinline__ int su_index(int i, int j) {
    const int hi = max(i, j), lo = min(i, j);
    return hi * (hi + 1) / 2 + lo;
}

// Builds the descriptor of node (w, c) of an item; mi looks up the mesh, nl elements make a slab.
template <class Mesh>
__device__ __forceinline__ void make_item(const Mesh &mi, int nl, const ItemFreq &f, float w, float c, ItemDesc &d) {
    const float A = __fadd_rn(__fadd_rn(f.h[0], w), f.l[0]), B = __fadd_rn(__fadd_rn(f.h[1], w), f.l[1]);
    const float P = __fadd_rn(__fadd_rn(f.h[2], w), f.l[2]), Q = __fadd_rn(__fadd_rn(f.h[3], w), f.l[3]);
    const int stepT = mi.n * nl, x = f.xi;
    int flags = 0;
    const Interp<float> iA = interp_abs(mi, A), iB = interp_abs(mi, B), iP = interp_abs(mi, P), iQ = interp_abs(mi, Q);
    // outer-point weights with the density's sign; a diagonal point has sign +1 (s) or -1 (u)
    auto weights = [&](const Interp<float> &i) {
        const float n = rn_sub(1.0f, i.b);
        const bool nl_ = f.u_signs ? i.lo >= x : i.lo > x, nh = f.u_signs ? i.hi >= x : i.hi > x;
        return make_float4(n, nl_ ? -n : n, i.b, nh ? -i.b : i.b);
    };
    auto diag = [&](const Interp<float> &i, int plane) {
        flags |= (int(i.lo == x) | (int(i.hi == x) << 1)) << (kFlDiagShift + 2 * plane);
    };
    auto plane = [&](const Interp<float> &in, const Interp<float> &out) {  // slab (x, t = in, u = out)
        const int lo = su_index(x, out.lo) * stepT, hi = su_index(x, out.hi) * stepT;
        return make_int4(lo + in.lo * nl, lo + in.hi * nl, hi + in.lo * nl, hi + in.hi * nl);
    };
    // slab (s = in, t = x, u = out); the density takes a minus where in < out
    auto tplane = [&](const Interp<float> &in, const Interp<float> &out, int i) {
        const int o = x * nl;
        d.t[i] = make_int4(su_index(in.lo, out.lo) * stepT + o, su_index(in.hi, out.lo) * stepT + o,
                           su_index(in.lo, out.hi) * stepT + o, su_index(in.hi, out.hi) * stepT + o);
        const float ni = rn_sub(1.0f, in.b), no = rn_sub(1.0f, out.b);
        auto sign = [](int a, int b, float w) { return a < b ? -w : (a > b ? w : 0.0f); };
        auto on = [](int a, int b, float w) { return a == b ? w : 0.0f; };
        const float w0 = rn_mul(no, ni), w1 = rn_mul(no, in.b), w2 = rn_mul(out.b, ni), w3 = rn_mul(out.b, in.b);
        d.tw[i][0] = make_float4(w0, sign(in.lo, out.lo, w0), w1, sign(in.hi, out.lo, w1));
        d.tw[i][1] = make_float4(w2, sign(in.lo, out.hi, w2), w3, sign(in.hi, out.hi, w3));
        d.td[i] = make_float4(on(in.lo, out.lo, w0), on(in.hi, out.lo, w1), on(in.lo, out.hi, w2), on(in.hi, out.hi, w3));
        if (in.lo == out.lo || in.hi == out.lo || in.lo == out.hi || in.hi == out.hi) flags |= kFlDiagT;
    };
    d.g[0] = plane(iA, iB);
    d.g[1] = plane(iP, iQ);
    d.g[2] = plane(iB, iA);
    d.g[3] = plane(iQ, iP);
    tplane(iQ, iP, 0);
    tplane(iA, iB, 1);
    diag(iB, 0);
    diag(iQ, 1);
    diag(iA, 2);
    diag(iP, 3);
    d.w[0] = weights(iA);
    d.w[1] = weights(iB);
    d.w[2] = weights(iP);
    d.w[3] = weights(iQ);
    if (B > 0) flags |= kFlE0;
    if (Q > 0) flags |= kFlE1;
    if (A < 0) flags |= kFlE2;
    if (P < 0) flags |= kFlE3;
    if (B < 0) flags |= kFlF0;
    if (A > 0) flags |= kFlF2;
    if ((Q > 0) != (P < 0)) flags |= kFlT0;
    const bool e1 = (A > 0) != (B > 0), e3 = (A < 0) != (B < 0);
    if (e1) flags |= kFlT1;
    if (e3) flags |= kFlT3;
    if (e1 != e3) flags |= kFlExT;
    d.c = c;
    d.flags = flags;
}

// (spin, density) of G plane i at one site (v: the site's element of slab 0): four loads,
// interpolated along u (wo), then along t (wi).
__device__ __forceinline__ float2 g_value(const ItemDesc &d, const float2 *v, int i, const float4 &wi, const float4 &wo) {
    const int4 o = d.g[i];
    const float2 lo = make_float2(wo.x, wo.y), hi = make_float2(wo.z, wo.w);
    const float2 x = fma2(hi, __ldg(v + o.z), mul2(lo, __ldg(v + o.x)));
    const float2 y = fma2(hi, __ldg(v + o.w), mul2(lo, __ldg(v + o.y)));
    return make_float2(__fmaf_rn(wi.z, y.x, __fmul_rn(wi.x, x.x)), __fmaf_rn(wi.z, y.y, __fmul_rn(wi.x, x.y)));
}
// T plane i: the spin, and the density of the plane's off-diagonal supports in the first buffer
// (the second buffer's is the opposite).
__device__ __forceinline__ float2 t_value(const ItemDesc &d, const float2 *v, int i) {
    const int4 o = d.t[i];
    const float4 a = d.tw[i][0], b = d.tw[i][1];
    const float2 x = fma2(make_float2(a.z, a.w), __ldg(v + o.y), mul2(make_float2(a.x, a.y), __ldg(v + o.x)));
    return fma2(make_float2(b.z, b.w), __ldg(v + o.w), fma2(make_float2(b.x, b.y), __ldg(v + o.z), x));
}
// The density of a t plane's diagonal supports (the same in both buffers).
__device__ __forceinline__ float t_diag(const ItemDesc &d, const float2 *v, int i) {
    const int4 o = d.t[i];
    const float4 w = d.td[i];
    return __fmaf_rn(w.w, __ldg(v + o.w).y,
                     __fmaf_rn(w.z, __ldg(v + o.z).y, __fmaf_rn(w.y, __ldg(v + o.y).y, __fmul_rn(w.x, __ldg(v + o.x).y))));
}

// The density of G plane i with the u channel's sign on the diagonal, from the one with the s channel's.
__device__ __forceinline__ float diag_u(const ItemDesc &d, const float2 *v, int i, int flags, const float4 &wi,
                                        const float4 &wo, float h) {
    const int4 o = d.g[i];
    const int bits = flags >> (kFlDiagShift + 2 * i);
    if (bits & 1) h = __fmaf_rn(-2.0f * wo.x, __fmaf_rn(wi.z, __ldg(v + o.y).y, __fmul_rn(wi.x, __ldg(v + o.x).y)), h);
    if (bits & 2) h = __fmaf_rn(-2.0f * wo.z, __fmaf_rn(wi.z, __ldg(v + o.w).y, __fmul_rn(wi.x, __ldg(v + o.z).y)), h);
    return h;
}

// The s/u integrand of one target from its planes' (spin, density) (SU2FrgCore.cpp:216-226,
// 323-328; see the density note above).
__device__ __forceinline__ float2 su_term(float2 g0, float2 g1, float2 g2, float2 g3) {
    const float p = __fmaf_rn(g2.x, g3.x, __fmul_rn(g0.x, g1.x));
    float2 r;
    r.x = __fmaf_rn(-0.5f, p, __fmul_rn(g0.y, g1.x));
    r.x = __fmaf_rn(g0.x, g1.y, r.x);
    r.x = __fmaf_rn(g2.y, g3.x, r.x);
    r.x = __fmaf_rn(g2.x, g3.y, r.x);
    r.y = __fmaf_rn(3.0f / 16.0f, p, __fmul_rn(g0.y, g1.y));
    r.y = __fmaf_rn(g2.y, g3.y, r.y);
    return r;
}

// One node at the SPT sites of a lane, every pair its own exchange: adds the two s/u targets to acc1, acc2 and the t target's
// local terms to acct, and returns the t channel's panel entries pa = c * (third buffer),
// pb = fourth buffer per site.  `step` 0: both targets are s-channel nodes; 1: the first is, the
// second is a u-channel node; 2: both are u-channel nodes.  Every lane of the warp calls it, W
// lanes per node; lanes whose node is not `active` add nothing.
template <int SPT, int W>
__device__ __forceinline__ void node_eval(const float2 *sd, const ItemDesc &d, float c, int step, bool active,
                                          const int (&site)[SPT], Acc (&acc1)[SPT], Acc (&acc2)[SPT], Acc (&acct)[SPT],
                                          float2 (&pa)[SPT], float2 (&pb)[SPT]) {
    constexpr unsigned kAll = 0xffffffffu;
    const float4 wA = d.w[0], wB = d.w[1], wP = d.w[2], wQ = d.w[3];
    const int fl = d.flags;
    // density output: opposite sign in the u channel
    const float2 c1 = make_float2(c, step == 2 ? -c : c), c2 = make_float2(c, step == 0 ? c : -c);
    const bool diag = step != 2 && __any_sync(kAll, (fl & kFlDiag) != 0);
    const bool diag_t = __any_sync(kAll, (fl & kFlDiagT) != 0);
    // the t integrand's site-local coefficients: of T0 and T1, and of their diagonal densities
    float2 ka, kb;
    float kd = 0.0f, ke = 0.0f;
    float2 q0[SPT], q1[SPT], q2[SPT], q3[SPT];  // the second target's planes
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        const float2 *v = sd + site[k];
        const float2 G0 = g_value(d, v, 0, wA, wB), G1 = g_value(d, v, 1, wP, wQ);
        const float2 G2 = g_value(d, v, 2, wB, wA), G3 = g_value(d, v, 3, wQ, wP);
        const float2 T0 = t_value(d, v, 0), T1 = t_value(d, v, 1);
        const float2 r1 = su_term(G0, G1, G2, G3);
        if (active) acc1[k].add(c1, r1);
        q0[k] = G0;
        q1[k] = G1;
        q2[k] = G2;
        q3[k] = G3;
        float u0 = G0.y, u1 = G1.y, u2 = G2.y, u3 = G3.y;  // densities with the u channel's signs
        if (diag) {
            u0 = diag_u(d, v, 0, fl, wA, wB, u0);
            u1 = diag_u(d, v, 1, fl, wP, wQ, u1);
            u2 = diag_u(d, v, 2, fl, wB, wA, u2);
            u3 = diag_u(d, v, 3, fl, wQ, wP, u3);
            if (step == 1) q0[k].y = u0, q1[k].y = u1, q2[k].y = u2, q3[k].y = u3;
        }
        // t channel, SU2FrgCore.cpp:286-302: buffer 0 takes plane G2 at pair 0, 1 G1, 2 G0, 3 G3
        if (k == 0) {
            float2 L0 = make_float2(G0.x, u0), L1 = make_float2(G1.x, u1), L2 = make_float2(G2.x, u2), L3 = make_float2(G3.x, u3);
            // spin: buffers 0 and 2 (1 and 3) have equal slabs; density: opposite ones
            ka.x = __fmaf_rn(0.25f, __fadd_rn(L0.x, L2.x), __fadd_rn(L0.y, L2.y));
            kb.x = __fmaf_rn(0.25f, __fadd_rn(L1.x, L3.x), __fadd_rn(L1.y, L3.y));
            ka.y = __fmaf_rn(-0.75f, __fsub_rn(L2.x, L0.x), __fsub_rn(L2.y, L0.y));
            kb.y = __fmaf_rn(-0.75f, __fsub_rn(L1.x, L3.x), __fsub_rn(L1.y, L3.y));
            ka.x = __shfl_sync(kAll, ka.x, 0, W);
            kb.x = __shfl_sync(kAll, kb.x, 0, W);
            ka.y = __shfl_sync(kAll, ka.y, 0, W);
            kb.y = __shfl_sync(kAll, kb.y, 0, W);
            if (diag_t) {
                kd = __shfl_sync(kAll, __fmaf_rn(-0.75f, __fadd_rn(L0.x, L2.x), __fadd_rn(L0.y, L2.y)), 0, W);
                ke = __shfl_sync(kAll, __fmaf_rn(-0.75f, __fadd_rn(L1.x, L3.x), __fadd_rn(L1.y, L3.y)), 0, W);
            }
        }
        float2 r = fma2(kb, T1, mul2(ka, T0));
        pa[k] = mul2(make_float2(c, -c), T0);  // third buffer
        pb[k] = make_float2(T1.x, -T1.y);      // fourth buffer
        if (diag_t && (fl & kFlDiagT)) {
            const float e0 = t_diag(d, v, 0), e1 = t_diag(d, v, 1);
            r.y = __fmaf_rn(ke, e1, __fmaf_rn(kd, e0, r.y));
            pa[k].y = __fmaf_rn(c, e0, pa[k].y);
            pb[k].y = __fadd_rn(e1, pb[k].y);
        }
        if (active) acct[k].add(make_float2(c, c), r);
    }
    // the second target exchanges a and b: G0 and G2 trade places
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        const float2 r = su_term(q2[k], q1[k], q0[k], q3[k]);
        if (active) acc2[k].add(c2, r);
    }
}

// Site-local coefficients of a node's t integrand, of T0 and T1 (ka, kb) and of their diagonal densities (kd, ke),
// from the planes at pair 0 (as in node_eval).
struct __align__(16) LocalCoef {
    float2 ka, kb;
    float kd, ke, pad[2];
};
__device__ __forceinline__ void item_local(const float2 *sd, const ItemDesc &d, int step, LocalCoef &k) {
    const float4 wA = d.w[0], wB = d.w[1], wP = d.w[2], wQ = d.w[3];
    const int fl = d.flags;
    float2 L0 = g_value(d, sd, 0, wA, wB), L1 = g_value(d, sd, 1, wP, wQ);
    float2 L2 = g_value(d, sd, 2, wB, wA), L3 = g_value(d, sd, 3, wQ, wP);
    if (step != 2 && (fl & kFlDiag)) {
        L0.y = diag_u(d, sd, 0, fl, wA, wB, L0.y);
        L1.y = diag_u(d, sd, 1, fl, wP, wQ, L1.y);
        L2.y = diag_u(d, sd, 2, fl, wB, wA, L2.y);
        L3.y = diag_u(d, sd, 3, fl, wQ, wP, L3.y);
    }
    k.ka.x = __fmaf_rn(0.25f, __fadd_rn(L0.x, L2.x), __fadd_rn(L0.y, L2.y));
    k.kb.x = __fmaf_rn(0.25f, __fadd_rn(L1.x, L3.x), __fadd_rn(L1.y, L3.y));
    k.ka.y = __fmaf_rn(-0.75f, __fsub_rn(L2.x, L0.x), __fsub_rn(L2.y, L0.y));
    k.kb.y = __fmaf_rn(-0.75f, __fsub_rn(L1.x, L3.x), __fsub_rn(L1.y, L3.y));
    k.kd = __fmaf_rn(-0.75f, __fadd_rn(L0.x, L2.x), __fadd_rn(L0.y, L2.y));
    k.ke = __fmaf_rn(-0.75f, __fadd_rn(L1.x, L3.x), __fadd_rn(L1.y, L3.y));
}

// node_eval at one site per lane (its element v in a slab, its own exchange) with the local coefficients given: the lanes of
// a warp need not hold pair 0.
__device__ __forceinline__ void site_node(const ItemDesc &d, const LocalCoef &lc, int step, const float2 *v, Acc &acc1,
                                          Acc &acc2, Acc &acct, float2 &pa, float2 &pb) {
    constexpr unsigned kAll = 0xffffffffu;
    const float4 wA = d.w[0], wB = d.w[1], wP = d.w[2], wQ = d.w[3];
    const int fl = d.flags;
    const float c = d.c;
    // density output: opposite sign in the u channel
    const float2 c1 = make_float2(c, step == 2 ? -c : c), c2 = make_float2(c, step == 0 ? c : -c);
    const bool diag = step == 1 && __any_sync(kAll, (fl & kFlDiag) != 0);
    const bool diag_t = __any_sync(kAll, (fl & kFlDiagT) != 0);
    float2 G0 = g_value(d, v, 0, wA, wB), G1 = g_value(d, v, 1, wP, wQ);
    float2 G2 = g_value(d, v, 2, wB, wA), G3 = g_value(d, v, 3, wQ, wP);
    const float2 T0 = t_value(d, v, 0), T1 = t_value(d, v, 1);
    const float2 r1 = su_term(G0, G1, G2, G3);
    acc1.add(c1, r1);
    float2 r = fma2(lc.kb, T1, mul2(lc.ka, T0));
    pa = mul2(make_float2(c, -c), T0);  // third buffer
    pb = make_float2(T1.x, -T1.y);      // fourth buffer
    if (diag_t && (fl & kFlDiagT)) {
        const float e0 = t_diag(d, v, 0), e1 = t_diag(d, v, 1);
        r.y = __fmaf_rn(lc.ke, e1, __fmaf_rn(lc.kd, e0, r.y));
        pa.y = __fmaf_rn(c, e0, pa.y);
        pb.y = __fadd_rn(e1, pb.y);
    }
    acct.add(make_float2(c, c), r);
    // the second target exchanges a and b: G0 and G2 trade places
    if (diag) {
        G0.y = diag_u(d, v, 0, fl, wA, wB, G0.y);
        G1.y = diag_u(d, v, 1, fl, wP, wQ, G1.y);
        G2.y = diag_u(d, v, 2, fl, wB, wA, G2.y);
        G3.y = diag_u(d, v, 3, fl, wQ, wP, G3.y);
    }
    const float2 r2 = su_term(G2, G1, G0, G3);
    acc2.add(c2, r2);
}


}  // namespace dev
}  // namespace spn
