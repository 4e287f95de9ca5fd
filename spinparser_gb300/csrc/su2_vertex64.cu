// Two-particle vertex flow in double precision (flows created with SPN_SU2_FP64): the
// reference's right-hand side (SU2FrgCore::_calculateVertexTwoParticle,
// src/SU2/SU2FrgCore.cpp:171-431) evaluated entirely in FP64 on the GPU, the precision
// reference for the FP32 flows of the same task.
//
// Lattices of at most 32 sites take three triples at a time (su2_item_f64_kernel, the items of
// su2_item.cuh in double).  Larger ones run triple by triple: a persistent grid whose warps take one
// (s,t,u) triple at a time from a device counter; the lanes hold the sites (up to four each); the
// loop-frequency nodes of each channel are visited in order; every lane builds the node's
// access buffers itself; the t channel's RPA sum runs over each rid's own overlap pair list
// in the reference's order (SU2FrgCore.cpp:249-266).  The node tables (conventional and
// Katanin terms with their quadrature weights) come from the same node-table body as the
// FP32 flow, instantiated in double.
#include "su2_common.cuh"
#include "su2_device.cuh"
#include "su2_item.cuh"

namespace spn {
namespace {

using namespace spn::dev;

constexpr int kThreads64 = 128;
constexpr int kWarps64 = kThreads64 / 32;
constexpr int kSitesPerLane64 = 4;  // Nl <= 128
constexpr double kPi64 = 3.14159265358979323846;

struct Freqs {
    double s, t, u, w1p, w1, w2p, w2;
};

// Interpolated slab of one access buffer for the lane's sites (getValueSuperbundle).
__device__ __forceinline__ void gather64(const FlowArgsT<double> &a, const AB4T<double> &ab, const int *site,
                                         const int *isite, const bool *valid, double *vs, double *vd) {
#pragma unroll
    for (int k = 0; k < kSitesPerLane64; ++k) {
        double gs = 0.0, gd = 0.0;
        if (valid[k]) {
            const int st = ab.exch ? isite[k] : site[k];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double2 p = a.sd[ab.off[q] + st];
                gs += ab.w[q] * p.x;
                gd += ab.sw[q] * p.y;
            }
        }
        vs[k] = gs;
        vd[k] = gd;
    }
}

// Site-local (rid 0) value pair of an access buffer.
__device__ __forceinline__ void local64(const FlowArgsT<double> &a, const AB4T<double> &ab, double &vs, double &vd) {
    double gs = 0.0, gd = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double2 p = a.sd[ab.off[q]];
        gs += ab.w[q] * p.x;
        gd += ab.sw[q] * p.y;
    }
    vs = gs;
    vd = gd;
}

__global__ void __launch_bounds__(kThreads64) su2_vertex_flow_f64_kernel(FlowArgsT<double> a) {
    __shared__ double pos[kMaxFreq];
    extern __shared__ double xs[];  // per warp: As, Ad, Bs, Bd [nl each]
    for (int i = threadIdx.x; i < a.n; i += blockDim.x) pos[i] = a.freq[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = a.n, nl = a.nl;
    double *As = xs + size_t(warp) * 4 * nl, *Ad = As + nl, *Bs = Ad + nl, *Bd = Bs + nl;
    int site[kSitesPerLane64], isite[kSitesPerLane64], jj[kSitesPerLane64];
    bool valid[kSitesPerLane64];
#pragma unroll
    for (int k = 0; k < kSitesPerLane64; ++k) {
        jj[k] = lane + 32 * k;
        valid[k] = jj[k] < nl;
        site[k] = valid[k] ? a.sites[jj[k]] : 0;
        isite[k] = valid[k] ? a.inv_sites[jj[k]] : 0;
    }
    const double s2 = 2.0 * double(a.spin), s8 = 8.0 * double(a.spin);

    for (;;) {
        int it = 0;
        if (lane == 0) it = atomicAdd(a.work_counter, 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= a.fn) break;
        const int su = it / n, ti = it - su * n;
        int si = int((sqrt(8.0 * double(su) + 1.0) - 1.0) * 0.5);
        while (si * (si + 1) / 2 > su) --si;
        while ((si + 1) * (si + 2) / 2 <= su) ++si;
        const int ui = su - si * (si + 1) / 2;
        Freqs f;
        f.s = pos[si];
        f.t = pos[ti];
        f.u = pos[ui];
        f.w1p = 0.5 * (f.s + f.t + f.u);
        f.w1 = 0.5 * (f.s - f.t + f.u);
        f.w2p = 0.5 * (f.s - f.t - f.u);
        f.w2 = 0.5 * (f.s + f.t - f.u);

        double acc_s[kSitesPerLane64] = {}, acc_d[kSitesPerLane64] = {};
        for (int ch = 0; ch < 3; ++ch) {
            const int xi = ch == 0 ? si : (ch == 1 ? ti : ui);
            const int cnt = a.node_cnt[xi];
            const double *nwp = a.node_wp + size_t(xi) * a.max_nodes;
            const double *nc = a.node_c + size_t(xi) * a.max_nodes;
            for (int b = 0; b < cnt; ++b) {
                const double wp = nwp[b];
                const double c = ch == 2 ? -nc[b] : nc[b];
                AB4T<double> ab[4];
                double S0[kSitesPerLane64], S1[kSitesPerLane64], S2[kSitesPerLane64], S3[kSitesPerLane64];
                double D0[kSitesPerLane64], D1[kSitesPerLane64], D2[kSitesPerLane64], D3[kSitesPerLane64];
                double xv[kSitesPerLane64], yv[kSitesPerLane64];
                if (ch == 0) {  // integralKernelS, SU2FrgCore.cpp:199-227
                    access4<kS>(pos, n, nl, f.s, -f.w1 - wp, -f.w2 - wp, ab[0]);
                    access4<kS>(pos, n, nl, f.s, f.w1p + wp, -f.w2p - wp, ab[1]);
                    access4<kS>(pos, n, nl, f.s, f.w2 + wp, f.w1 + wp, ab[2]);
                    access4<kS>(pos, n, nl, f.s, -f.w2p - wp, f.w1p + wp, ab[3]);
                } else if (ch == 1) {  // integralKernelT, SU2FrgCore.cpp:229-303
                    access4<kT>(pos, n, nl, f.w1 - wp, f.t, f.w1p + wp, ab[0]);
                    access4<kT>(pos, n, nl, f.w2p - wp, f.t, -f.w2 - wp, ab[1]);
                    access4<kT>(pos, n, nl, f.w1p + wp, f.t, f.w1 - wp, ab[2]);
                    access4<kT>(pos, n, nl, f.w2 + wp, f.t, wp - f.w2p, ab[3]);
                } else {  // integralKernelU, SU2FrgCore.cpp:305-334
                    access4<kU>(pos, n, nl, f.w1 + wp, wp - f.w2p, f.u, ab[0]);
                    access4<kU>(pos, n, nl, f.w1p + wp, f.w2 - wp, f.u, ab[1]);
                    access4<kU>(pos, n, nl, f.w2p - wp, -f.w1 - wp, f.u, ab[2]);
                    access4<kU>(pos, n, nl, f.w2 - wp, f.w1p + wp, f.u, ab[3]);
                }
                gather64(a, ab[0], site, isite, valid, S0, D0);
                gather64(a, ab[1], site, isite, valid, S1, D1);
                gather64(a, ab[2], site, isite, valid, S2, D2);
                gather64(a, ab[3], site, isite, valid, S3, D3);
                if (ch != 1) {
#pragma unroll
                    for (int k = 0; k < kSitesPerLane64; ++k) {
                        double x = 0.0, y = 0.0;
                        if (ch == 0) {
                            x -= 0.5 * S0[k] * S1[k];
                            x -= 0.5 * S2[k] * S3[k];
                            x += D0[k] * S1[k];
                            x += D2[k] * S3[k];
                            x += S0[k] * D1[k];
                            x += S2[k] * D3[k];
                        } else {
                            x += 0.5 * S0[k] * S1[k];
                            x += 0.5 * S2[k] * S3[k];
                            x += S0[k] * D1[k];
                            x += S2[k] * D3[k];
                            x += D0[k] * S1[k];
                            x += D2[k] * S3[k];
                        }
                        y += (3.0 / 16.0) * S0[k] * S1[k];
                        y += (3.0 / 16.0) * S2[k] * S3[k];
                        y += D0[k] * D1[k];
                        y += D2[k] * D3[k];
                        xv[k] = x;
                        yv[k] = y;
                    }
                } else {
                    // exchange the third and fourth slabs, then the RPA sum per rid
#pragma unroll
                    for (int k = 0; k < kSitesPerLane64; ++k)
                        if (valid[k]) {
                            As[jj[k]] = S2[k];
                            Ad[jj[k]] = D2[k];
                            Bs[jj[k]] = S3[k];
                            Bd[jj[k]] = D3[k];
                        }
                    __syncwarp();
                    AB4T<double> lb;
                    double cbs, cbd, icas, icad, cbs2, cbd2, icas2, icad2;
                    access4<kU>(pos, n, nl, f.w2p - wp, -f.w2 - wp, f.t, lb);
                    local64(a, lb, cbs, cbd);
                    access4<kU>(pos, n, nl, f.w1 - wp, -f.w1p - wp, -f.t, lb);
                    local64(a, lb, icas, icad);
                    access4<kU>(pos, n, nl, f.w2 + wp, wp - f.w2p, f.t, lb);
                    local64(a, lb, cbs2, cbd2);
                    access4<kU>(pos, n, nl, f.w1p + wp, wp - f.w1, -f.t, lb);
                    local64(a, lb, icas2, icad2);
#pragma unroll
                    for (int k = 0; k < kSitesPerLane64; ++k) {
                        double rpa_s = 0.0, rpa_d = 0.0;
                        if (valid[k]) {
                            const int r = jj[k];
                            for (int i = a.ov_ptr[r]; i < a.ov_ptr[r + 1]; ++i) {
                                const int r1 = a.ov_r1[i], r2 = a.ov_r2[i];
                                rpa_s += As[r1] * Bs[r2];
                                rpa_d += Ad[r1] * Bd[r2];
                            }
                        }
                        double x = 0.0 + s2 * rpa_s;  // SU2FrgCore.cpp:265, 286-293
                        x -= cbd * S0[k];
                        x += (0.25 * cbs) * S0[k];
                        x -= icad * S1[k];
                        x += (0.25 * icas) * S1[k];
                        x -= cbd2 * S2[k];
                        x += (0.25 * cbs2) * S2[k];
                        x -= icad2 * S3[k];
                        x += (0.25 * icas2) * S3[k];
                        double y = 0.0 + s8 * rpa_d;  // SU2FrgCore.cpp:266, 295-302
                        y -= cbd * D0[k];
                        y -= (0.75 * cbs) * D0[k];
                        y -= icad * D1[k];
                        y -= (0.75 * icas) * D1[k];
                        y -= cbd2 * D2[k];
                        y -= (0.75 * cbs2) * D2[k];
                        y -= icad2 * D3[k];
                        y -= (0.75 * icas2) * D3[k];
                        xv[k] = x;
                        yv[k] = y;
                    }
                    __syncwarp();
                }
#pragma unroll
                for (int k = 0; k < kSitesPerLane64; ++k) {
                    acc_s[k] += c * xv[k];
                    acc_d[k] += c * yv[k];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < kSitesPerLane64; ++k)
            if (valid[k]) {
                const double os = acc_s[k] / (2.0 * kPi64), od = acc_d[k] / (2.0 * kPi64);
                a.dsd[size_t(it) * nl + jj[k]] = make_double2(os, od);
                if (isnan(os) || isnan(od)) atomicOr(a.status, kStatusNaN);
            }
    }
}

// ------------------------------------------------------------------------------------
// Items in double (see su2_item.cuh for the planes, signs and targets).
//
// The FP64 pipe (2 FMAs per clock and SM) bounds this flow, so what counts is FP64 instructions per warp.  Triple by
// triple every lane built every node's eight access buffers (two divisions each), four site slots were evaluated for
// any lattice, and the lattice sum ran over each site's pair list per node: 46.7 ms a launch for 12 sites, N = 32,
// cutoff 0.7.  Here a lane builds one node's supports, W lanes hold a node's sites (32 / W nodes at once), a node
// serves three triples, and the lattice sum goes through the outer-product matrix as in FP32.
// ------------------------------------------------------------------------------------
struct __align__(16) ItemDesc64 {
    double w[4][4];       // A, B, P, Q: lower weight, with the density's sign as the u coordinate, upper, with its sign
    double tw[2][4];      // T0, T1: support weights
    double ts[2][4];      // the density's off-diagonal weights in the first buffer
    int g[4][4], t[2][4];
    double c;
    int flags, pad;
};

__device__ __forceinline__ void make_item64(const double *pos, int n, int nl, int x, double fx, double fa, double fb, bool u_signs,
                                            double w, double c, ItemDesc64 &d) {
    const MeshSearch<double> m{pos, n};
    const double dm = fa - fb, dq = fa + fb;
    const double A = 0.5 * (fx - dm) + w, B = 0.5 * (fx + dm) + w, P = 0.5 * (fx + dq) + w, Q = 0.5 * (fx - dq) + w;
    const Interp<double> iA = interp_abs(m, A), iB = interp_abs(m, B), iP = interp_abs(m, P), iQ = interp_abs(m, Q);
    const int stepT = n * nl;
    int flags = 0;
    auto weights = [&](int k, const Interp<double> &i) {
        const double lo = 1.0 - i.b;
        d.w[k][0] = lo;
        d.w[k][1] = (u_signs ? i.lo >= x : i.lo > x) ? -lo : lo;
        d.w[k][2] = i.b;
        d.w[k][3] = (u_signs ? i.hi >= x : i.hi > x) ? -i.b : i.b;
    };
    auto plane = [&](int k, const Interp<double> &in, const Interp<double> &out) {
        const int lo = su_index(x, out.lo) * stepT, hi = su_index(x, out.hi) * stepT;
        d.g[k][0] = lo + in.lo * nl;
        d.g[k][1] = lo + in.hi * nl;
        d.g[k][2] = hi + in.lo * nl;
        d.g[k][3] = hi + in.hi * nl;
        flags |= (int(out.lo == x) | (int(out.hi == x) << 1)) << (kFlDiagShift + 2 * k);
    };
    auto tplane = [&](int k, const Interp<double> &in, const Interp<double> &out) {
        const int ii[4] = {in.lo, in.hi, in.lo, in.hi}, oo[4] = {out.lo, out.lo, out.hi, out.hi};
        const double wi[4] = {1.0 - in.b, in.b, 1.0 - in.b, in.b}, wo[4] = {1.0 - out.b, 1.0 - out.b, out.b, out.b};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            d.t[k][q] = su_index(ii[q], oo[q]) * stepT + x * nl;
            const double v = wo[q] * wi[q];
            d.tw[k][q] = v;
            d.ts[k][q] = ii[q] < oo[q] ? -v : (ii[q] > oo[q] ? v : 0.0);
            if (ii[q] == oo[q]) flags |= kFlDiagT;
        }
    };
    plane(0, iA, iB);
    plane(1, iP, iQ);
    plane(2, iB, iA);
    plane(3, iQ, iP);
    tplane(0, iQ, iP);
    tplane(1, iA, iB);
    weights(0, iA);
    weights(1, iB);
    weights(2, iP);
    weights(3, iQ);
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

__device__ __forceinline__ double2 g64(const ItemDesc64 &d, const double2 *v, int i, int wi, int wo) {
    const double2 a = v[d.g[i][0]], b = v[d.g[i][1]], e = v[d.g[i][2]], f = v[d.g[i][3]];
    const double *o = d.w[wo], *n = d.w[wi];
    const double2 x = make_double2(o[2] * e.x + o[0] * a.x, o[3] * e.y + o[1] * a.y);
    const double2 y = make_double2(o[2] * f.x + o[0] * b.x, o[3] * f.y + o[1] * b.y);
    return make_double2(n[2] * y.x + n[0] * x.x, n[2] * y.y + n[0] * x.y);
}
// the density with the u channel's sign on the diagonal
__device__ __forceinline__ double diag64(const ItemDesc64 &d, const double2 *v, int i, int wi, int wo, double h) {
    const int bits = d.flags >> (kFlDiagShift + 2 * i);
    const double *o = d.w[wo], *n = d.w[wi];
    if (bits & 1) h -= 2.0 * o[0] * (n[2] * v[d.g[i][1]].y + n[0] * v[d.g[i][0]].y);
    if (bits & 2) h -= 2.0 * o[2] * (n[2] * v[d.g[i][3]].y + n[0] * v[d.g[i][2]].y);
    return h;
}
// spin, off-diagonal density of the first buffer, and diagonal density of a T plane
__device__ __forceinline__ double2 t64(const ItemDesc64 &d, const double2 *v, int i, double &diag) {
    double2 r = make_double2(0.0, 0.0);
    diag = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double2 e = v[d.t[i][q]];
        r.x += d.tw[i][q] * e.x;
        r.y += d.ts[i][q] * e.y;
        if ((d.flags & kFlDiagT) && d.ts[i][q] == 0.0) diag += d.tw[i][q] * e.y;
    }
    return r;
}
__device__ __forceinline__ double2 su64(double2 g0, double2 g1, double2 g2, double2 g3) {
    const double p = g0.x * g1.x + g2.x * g3.x;
    return make_double2(-0.5 * p + g0.y * g1.x + g0.x * g1.y + g2.y * g3.x + g2.x * g3.y,
                        3.0 / 16.0 * p + g0.y * g1.y + g2.y * g3.y);
}
__device__ __forceinline__ double2 shfl64(double2 v, int width) {
    return make_double2(__shfl_sync(0xffffffffu, v.x, 0, width), __shfl_sync(0xffffffffu, v.y, 0, width));
}
__device__ __forceinline__ void acc64(double2 &a, double cs, double cd, double2 v) {
    a.x += cs * v.x;
    a.y += cd * v.y;
}

__host__ __device__ constexpr int lanes64(int MB) { return MB == 1 ? 8 : (MB == 2 ? 16 : 32); }
__host__ __device__ inline size_t warp64_bytes(int MB, int n_seg) {
    const size_t w = 8 * MB, G = 32 / lanes64(MB);
    const size_t main = 32 * sizeof(ItemDesc64) + G * 2 * w * sizeof(double2), st = sizeof(double2) * (w * w + n_seg);
    return main > st ? main : st;
}

template <int MB>
__global__ void __launch_bounds__(kThreads64) su2_item_f64_kernel(FlowArgsT<double> a) {
    constexpr int w = 8 * MB, W = lanes64(MB), G = 32 / W;
    __shared__ double pos[kMaxFreq];
    extern __shared__ __align__(16) unsigned char xs64[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane / W, jl = lane - g * W;
    const int n = a.n, nl = a.nl;
    for (int i = threadIdx.x; i < n; i += blockDim.x) pos[i] = a.freq[i];
    unsigned char *area = xs64 + warp * warp64_bytes(MB, a.rpa.n_seg);
    ItemDesc64 *desc = reinterpret_cast<ItemDesc64 *>(area);
    double2 *panel = reinterpret_cast<double2 *>(area + 32 * sizeof(ItemDesc64));
    double2 *Ms = reinterpret_cast<double2 *>(area), *slots = Ms + w * w;
    const bool valid = jl < nl;
    const int sc = min(jl, nl - 1), site = a.sites[sc], isite = a.inv_sites[sc];
    const int rb = lane >> 2, cb = lane & 3;
    __syncthreads();
    const int items = vertex_items(n);
    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(a.work_counter, 1);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= items) break;
        int p, q, r;
        decode_item(item, p, q, r);
        double2 A = make_double2(0.0, 0.0), B = A, T = A;
#pragma unroll 1
        for (int step = 0; step < 3; ++step) {
            const int xi = step == 0 ? p : (step == 1 ? q : r), ai = step == 0 ? q : p, bi = step == 2 ? q : r;
            double2 M[MB][2 * MB];
#pragma unroll
            for (int i = 0; i < MB; ++i)
#pragma unroll
                for (int j = 0; j < 2 * MB; ++j) M[i][j] = make_double2(0.0, 0.0);
            const int cnt = a.node_cnt[xi];
            const double *nwp = a.node_wp + size_t(xi) * a.max_nodes, *nc = a.node_c + size_t(xi) * a.max_nodes;
            for (int b0 = 0; b0 < cnt; b0 += 32) {
                const int nb = min(32, cnt - b0);
                if (lane < nb)
                    make_item64(pos, n, nl, xi, pos[xi], pos[ai], pos[bi], step == 2, nwp[b0 + lane], nc[b0 + lane], desc[lane]);
                __syncwarp();
#pragma unroll 1
                for (int k0 = 0; k0 < nb; k0 += G) {
                    const bool active = k0 + g < nb;
                    const ItemDesc64 &d = desc[active ? k0 + g : 0];
                    const int fl = d.flags;
                    const double c = active ? d.c : 0.0, c1 = step == 2 ? -c : c, c2 = step == 0 ? c : -c;
                    auto at = [&](int bit) { return a.sd + ((fl & bit) ? isite : site); };
                    const double2 *v0 = at(kFlE0), *v1 = at(kFlE1), *v2 = at(kFlE2), *v3 = at(kFlE3);
                    double2 G0 = g64(d, v0, 0, 0, 1), G1 = g64(d, v1, 1, 2, 3), G2 = g64(d, v2, 2, 1, 0), G3 = g64(d, v3, 3, 3, 2);
                    const double2 r1 = su64(G0, G1, G2, G3);
                    if (active) acc64(A, c, c1, r1);
                    double2 L0 = G0, L1 = G1, L2 = G2, L3 = G3;
                    const bool diag = step != 2 && (fl & kFlDiag) != 0;
                    if (diag) {
                        L0.y = diag64(d, v0, 0, 0, 1, L0.y);
                        L1.y = diag64(d, v1, 1, 2, 3, L1.y);
                        L2.y = diag64(d, v2, 2, 1, 0, L2.y);
                        L3.y = diag64(d, v3, 3, 3, 2, L3.y);
                        if (step == 1) G0 = L0, G1 = L1, G2 = L2, G3 = L3;
                    }
                    if (a.inv_kind != 0) {  // the second target's own site exchange
                        const double2 *b0p = at(kFlF0), *b2p = at(kFlF2);
                        G0 = g64(d, b0p, 0, 0, 1);
                        G2 = g64(d, b2p, 2, 1, 0);
                        if (diag && step == 1) {
                            G0.y = diag64(d, b0p, 0, 0, 1, G0.y);
                            G2.y = diag64(d, b2p, 2, 1, 0, G2.y);
                        }
                    }
                    const double2 r2 = su64(G2, G1, G0, G3);
                    if (active) acc64(B, c, c2, r2);
                    if (a.inv_kind == 2) {  // pair 0 itself
                        L0 = g64(d, a.sd, 0, 0, 1);
                        L1 = g64(d, a.sd, 1, 2, 3);
                        L2 = g64(d, a.sd, 2, 1, 0);
                        L3 = g64(d, a.sd, 3, 3, 2);
                        if (diag) {
                            L0.y = diag64(d, a.sd, 0, 0, 1, L0.y);
                            L1.y = diag64(d, a.sd, 1, 2, 3, L1.y);
                            L2.y = diag64(d, a.sd, 2, 1, 0, L2.y);
                            L3.y = diag64(d, a.sd, 3, 3, 2, L3.y);
                        }
                    }
                    L0 = shfl64(L0, W);
                    L1 = shfl64(L1, W);
                    L2 = shfl64(L2, W);
                    L3 = shfl64(L3, W);
                    const double2 *vt1 = at(kFlT1);
                    double e0, e1;
                    const double2 T0 = t64(d, at(kFlT0), 0, e0), T1 = t64(d, vt1, 1, e1);
                    double S3 = T1.x, D3 = e1 - T1.y;  // fourth buffer
                    if (fl & kFlExT) {
                        double e3;
                        const double2 T3 = t64(d, at(kFlT3), 1, e3);
                        S3 = T3.x;
                        D3 = e3 - T3.y;
                    }
                    const double D0 = e0 + T0.y, D2 = e0 - T0.y, D1 = e1 + T1.y;
                    double2 rt;
                    rt.x = (0.25 * (L0.x + L2.x) + (L0.y + L2.y)) * T0.x + (0.25 * L1.x + L1.y) * T1.x + (0.25 * L3.x + L3.y) * S3;
                    rt.y = (L2.y - 0.75 * L2.x) * D0 + (L0.y - 0.75 * L0.x) * D2 + (L1.y - 0.75 * L1.x) * D1 + (L3.y - 0.75 * L3.x) * D3;
                    if (active) acc64(T, c, c, rt);
                    if (valid) {
                        panel[g * 2 * w + jl] = make_double2(c * T0.x, c * D2);
                        panel[g * 2 * w + w + jl] = make_double2(S3, D3);
                    }
                    __syncwarp();  // panels written
                    for (int k = 0; k < G && k0 + k < nb; ++k) {
                        const double2 *pa = panel + k * 2 * w + rb * MB, *pb = panel + k * 2 * w + w + cb * 2 * MB;
#pragma unroll
                        for (int i = 0; i < MB; ++i) {
                            const double2 av = pa[i];
#pragma unroll
                            for (int j = 0; j < 2 * MB; ++j) {
                                const double2 bv = pb[j];
                                M[i][j].x += av.x * bv.x;
                                M[i][j].y += av.y * bv.y;
                            }
                        }
                    }
                    __syncwarp();  // panels read
                }
                __syncwarp();
            }
            // lattice sum: M staged, the merged pair list walked once
#pragma unroll
            for (int i = 0; i < MB; ++i)
#pragma unroll
                for (int j = 0; j < 2 * MB; ++j) Ms[(rb * MB + i) * w + cb * 2 * MB + j] = M[i][j];
            __syncwarp();
            {
                const int len = a.rpa.count[lane];
                int slot = a.rpa.slot_base[lane];
                double2 sum = make_double2(0.0, 0.0);
                for (int i = 0; i < len; ++i) {
                    const int e = a.rpa.sched[i * a.rpa.lanes + lane];
                    const double m = double((e >> 16) & 0xff);
                    const double2 v = Ms[(e & 0xffff) >> 3];
                    sum.x += m * v.x;
                    sum.y += m * v.y;
                    if (e < 0) {
                        slots[slot++] = sum;
                        sum = make_double2(0.0, 0.0);
                    }
                }
            }
            __syncwarp();
            if (g == 0 && valid) {
                double2 sum = make_double2(0.0, 0.0);
                for (int k = a.rpa.seg_ptr[jl]; k < a.rpa.seg_ptr[jl + 1]; ++k) {
                    sum.x += slots[k].x;
                    sum.y += slots[k].y;
                }
                acc64(T, 2.0 * double(a.spin), 8.0 * double(a.spin), sum);
            }
            __syncwarp();
            if (step == 0) { const double2 t = A; A = T; T = t; }
            if (step == 1) { const double2 t = B; B = T; T = t; }
        }
        auto store = [&](double2 v, int s, int t, int u) {
#pragma unroll
            for (int o = W; o < 32; o <<= 1) {
                v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
                v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
            }
            if (g == 0 && valid) {
                const double os = v.x / (2.0 * kPi64), od = v.y / (2.0 * kPi64);
                a.dsd[(size_t(su_index(s, u)) * n + t) * nl + jl] = make_double2(os, od);
                if (isnan(os) || isnan(od)) atomicOr(a.status, kStatusNaN);
            }
        };
        store(B, p, q, r);
        if (q != r) store(T, p, r, q);
        if (p != q) store(A, q, p, r);
    }
}

using Kernel64 = void (*)(FlowArgsT<double>);
Kernel64 kernel64(int nl) {
    if (nl <= 8) return su2_item_f64_kernel<1>;
    if (nl <= 16) return su2_item_f64_kernel<2>;
    if (nl <= 24) return su2_item_f64_kernel<3>;
    if (nl <= 32) return su2_item_f64_kernel<4>;
    return su2_vertex_flow_f64_kernel;
}
size_t smem64(int nl, int n_seg) {
    return nl <= 32 ? kWarps64 * warp64_bytes(rpa_outer_width(nl) / 8, n_seg) : size_t(kWarps64) * 4 * nl * sizeof(double);
}

}  // namespace

int vertex_flow_f64_blocks_per_sm(int nl, const RpaSchedule &rpa) {
    const size_t smem = smem64(nl, rpa.n_seg);
    if (allow_shared(kernel64(nl), smem) != cudaSuccess) return -1;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel64(nl), kThreads64, smem) != cudaSuccess) return -1;
    return per_sm;
}

void launch_vertex_flow_f64(const FlowArgsT<double> &a, int grid, cudaStream_t stream) {
    const size_t smem = smem64(a.nl, a.rpa.n_seg);
    kernel64(a.nl)<<<grid, kThreads64, smem, stream>>>(a);
}

}  // namespace spn
