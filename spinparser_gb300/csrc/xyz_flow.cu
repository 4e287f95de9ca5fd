// GB300 kernels of the XYZ pf-FRG flow right-hand side (models with diagonal, possibly
// anisotropic couplings: Heisenberg-Kitaev, XXZ, ...) and the device half of the spn_xyz_* C
// ABI in include/spn_su2.h.  Restates XYZFrgCore (src/XYZ/XYZFrgCore.cpp:161-570), the XYZ
// vertex access (src/XYZ/XYZVertexTwoParticle.hpp:185-612) and XYZMeasurementCorrelation
// (src/XYZ/XYZMeasurementCorrelation.cpp:98-184).
//
// The vertex has four components per element, X, Y, Z and density D, stored as one float4
// per element ((s(s+1)/2+u)*N + t)*Nl + rid, so an interpolation support is one 16-byte load.
// A lattice symmetry map may permute X, Y, Z: site j of the superbundle reads component
// perm[p_j][c] of its representative, and each RPA pair carries the permutations of its two
// factors (spn_lattice_get_spin_tables).
//
// A step: the self-energy flow (one CTA per frequency), the loop-frequency node tables (the
// SU(2) core's, shared), the vertex flow and the Euler update.  The vertex-flow kernel runs a
// persistent grid whose warps take one (s,t,u) triple at a time from a device counter.  Per
// channel, nodes go in batches of 16: first a lane builds one node's access buffers (and
// the t channel's site-local values) into a shared-memory descriptor, then the lanes hold
// the sites (up to four each) and walk the batch's nodes in order.  The t channel's RPA sum
// exchanges the first two slabs of a node through shared memory in all six spin
// permutations, so a pair (rid1, rid2, perm1, perm2) is two 16-byte loads and four FMAs.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>
#include "su2_common.cuh"
#include "su2_device.cuh"
#include "su2_kernels.cuh"
#include "su2_item.cuh"
#include "cuda_host.cuh"
#include "host/capi_common.hpp"
#include "host/pair_order.hpp"
#include "../../include/spn_su2.h"

using namespace spn;
using namespace spn::dev;

namespace {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kSpt = 4;  // sites per lane at most (Nl <= 128); the vertex kernel takes 1, 2 or 4
constexpr int X = 0, Y = 1, Z = 2, D = 3;

// The six spin permutations (X,Y,Z) (X,Z,Y) (Y,X,Z) (Y,Z,X) (Z,X,Y) (Z,Y,X): 2 bits per image
// component, 6 bits per permutation.
constexpr unsigned long long kPermBits =
    36ull | (24ull << 6) | (33ull << 12) | (9ull << 18) | (18ull << 24) | (6ull << 30);
__host__ __device__ __forceinline__ int perm_c(int p, int c) { return int((kPermBits >> (6 * p + 2 * c)) & 3ull); }

SPN_HDI float comp_of(const float4 &v, int c) { return c == 0 ? v.x : (c == 1 ? v.y : (c == 2 ? v.z : v.w)); }

struct XyzArgs {
    int n, nl, fn, max_nodes, n_range, n_corr;
    float cutoff;
    const float *freq;
    const float4 *sd;  // state
    float4 *dsd;       // flow
    const float *v2;
    float *dv2;
    const int *sites, *sites_perm, *inv_sites, *inv_sites_perm;
    // the t channel's RPA pairs of all sites in one lane-balanced walk (lane_schedule): entry i
    // of lane l is sched[32 i + l], the pair's word rid1 | rid2 << 7 | perm1 << 14 | perm2 << 17
    // (order_rpa_pairs) with bit 20 set on the last entry of a site's run in the lane; count[l]
    // entries; the runs' partial sums go to slots slot_base[l], ... and site j sums slots
    // seg_ptr[j] .. seg_ptr[j + 1] - 1
    const int *rpa_sched, *rpa_count, *rpa_slot_base, *rpa_seg_ptr;
    int rpa_n_seg;
    int site_kind;  // lattices of at most 32 sites: xyz_site_kind (below); their walk is cut into kItemThreads chunks
    const int *range_rid, *range_inv;
    const float *node_wp, *node_c;
    const int *node_cnt;
    int *work_counter;
    unsigned *status;
    const int *corr_rid, *corr_perm;
    double *partial;  // [kMaxCorrNodes][4][nl]
    float *out;       // [4][n_corr] correlations, then chi [4][nl]
};

// One component of the state for value_none (su2_device.cuh): c < 3 reads X, Y or Z (its
// "spin" accessor), c == 3 the density (with the density's sign on an s <-> u swap).
struct QuadComp {
    const float4 *v;
    int c;
    SPN_HDI float spin(int i) const { return comp_of(ro_load(v + i), c); }
    SPN_HDI float density(int i) const { return ro_load(v + i).w; }
};

SPN_HDI float value4(const float *pos, const XyzArgs &a, int c, int rid12, int rid21, float s, float t, float u) {
    return value_none(pos, a.n, a.nl, QuadComp{a.sd, c}, c == D, rid12, rid21, s, t, u);
}

// ------------------------------------------------------------------------------------
// self-energy flow, one CTA per frequency (XYZFrgCore.cpp:161-194)
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) xyz_self_energy_kernel(XyzArgs a) {
    __shared__ float pos[kMaxFreq];
    __shared__ double red[4];
    for (int i = threadIdx.x; i < a.n; i += blockDim.x) pos[i] = a.freq[i];
    __syncthreads();
    const int i = blockIdx.x;
    const float w = pos[i], L = a.cutoff;
    const float wpl = w + L, wml = w - L;
    double part = 0.0;
    for (int j = threadIdx.x; j < a.n_range; j += blockDim.x) {
        const int r12 = a.range_rid[j], r21 = a.range_inv[j];
        part += double(value4(pos, a, D, r12, r21, wpl, 0.0f, wml)) - double(value4(pos, a, D, r12, r21, wml, 0.0f, wpl));
    }
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int k = 0; k < int(blockDim.x >> 5); ++k) sum += red[k];
        double val = -2.0 * sum;
        for (int c = 0; c < 4; ++c)
            val += double(value4(pos, a, c, 0, 0, wpl, wml, 0.0f)) - double(value4(pos, a, c, 0, 0, wml, wpl, 0.0f));
        val /= (2.0 * kPiD * (double(L) + odd_interp(pos, a.n, a.v2, L)));
        const float outv = float(val);
        a.dv2[i] = outv;
        if (isnan(outv)) atomicOr(a.status, kStatusNaN);
    }
}

// Loop-frequency node tables: the SU(2) core's body on an argument block of this flow.
__global__ void __launch_bounds__(kNodeThreads) xyz_node_table_kernel(FlowArgs f) { node_table_body(f, blockIdx.x); }

// ------------------------------------------------------------------------------------
// vertex flow
// ------------------------------------------------------------------------------------
template <int SPT>
struct LaneT {
    int j[SPT], rid[SPT], prm[SPT], irid[SPT], iprm[SPT];
    bool valid[SPT];
};
using Lane4 = LaneT<kSpt>;

// Interpolated slab of one access buffer for the lane's sites (getValueSuperbundle): X, Y, Z
// of site j read the permuted components of its representative, D the signed density.  The
// four supports are summed per stored component (one fused multiply-add each) and the sums
// permuted once, instead of selecting a permuted component of every support.
template <int SPT>
SPN_HDI void gather4(const XyzArgs &a, const AB4 &ab, const LaneT<SPT> &ln, float4 *out) {
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (ln.valid[k]) {
            const int r = ab.exch ? ln.irid[k] : ln.rid[k];
            const int p = ab.exch ? ln.iprm[k] : ln.prm[k];
            float4 h = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 v = ro_load(a.sd + ab.off[q] + r);
                h.x += ab.w[q] * v.x;
                h.y += ab.w[q] * v.y;
                h.z += ab.w[q] * v.z;
                h.w += ab.sw[q] * v.w;
            }
            g = make_float4(comp_of(h, perm_c(p, 0)), comp_of(h, perm_c(p, 1)), comp_of(h, perm_c(p, 2)), h.w);
        }
        out[k] = g;
    }
}

// getValueLocal of the four components at rid 0 (identity permutation).
SPN_HDI float4 local4(const XyzArgs &a, const AB4 &ab) {
    float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float4 v = ro_load(a.sd + ab.off[q]);
        g.x += ab.w[q] * v.x;
        g.y += ab.w[q] * v.y;
        g.z += ab.w[q] * v.z;
        g.w += ab.sw[q] * v.w;
    }
    return g;
}

// The products of a pair of slabs (a, b) in the s integrand: per component (D,c) and (c,D)
// added, the two others crossed and subtracted (XYZFrgCore.cpp:230-261).
__device__ __forceinline__ float4 s_terms(const float4 &a, const float4 &b) {
    float4 r;
    r.x = a.w * b.x + a.x * b.w - a.z * b.y - a.y * b.z;
    r.y = a.w * b.y + a.y * b.w - a.z * b.x - a.x * b.z;
    r.z = a.w * b.z + a.z * b.w - a.x * b.y - a.y * b.x;
    r.w = a.w * b.w + a.x * b.x + a.y * b.y + a.z * b.z;
    return r;
}

// The u integrand subtracts all four products of every component (XYZFrgCore.cpp:436-469):
// the cross terms keep the sign of the others, unlike the s integrand.
__device__ __forceinline__ float4 u_terms(const float4 &a, const float4 &b) {
    float4 r;
    r.x = -(a.w * b.x + a.x * b.w + a.z * b.y + a.y * b.z);
    r.y = -(a.w * b.y + a.y * b.w + a.z * b.x + a.x * b.z);
    r.z = -(a.w * b.z + a.z * b.w + a.x * b.y + a.y * b.x);
    r.w = -(a.w * b.w + a.x * b.x + a.y * b.y + a.z * b.z);
    return r;
}

// v with X, Y, Z replaced by components perm[p][0..2] of v (density unchanged).
template <int P>
__device__ __forceinline__ float4 permuted(const float4 &v) {
    constexpr int c0 = int((kPermBits >> (6 * P)) & 3ull), c1 = int((kPermBits >> (6 * P + 2)) & 3ull),
                  c2 = int((kPermBits >> (6 * P + 4)) & 3ull);
    return make_float4(comp_of(v, c0), comp_of(v, c1), comp_of(v, c2), v.w);
}

// Node descriptor (lane = node in phase A): the four access buffers of the node and, for the
// t channel, the four site-local values (getValueLocal of ab4..ab7, four components each).
struct __align__(16) XDesc {
    int4 off[4];
    float4 w[4], sw[4];
    float4 lv[4];
    int exch;  // bit i: buffer i reads the site-exchanged pairs
    float c;   // node coefficient
    int pad[2];
};

__device__ __forceinline__ void put_desc(XDesc &d, int i, const AB4 &ab) {
    d.off[i] = make_int4(ab.off[0], ab.off[1], ab.off[2], ab.off[3]);
    d.w[i] = make_float4(ab.w[0], ab.w[1], ab.w[2], ab.w[3]);
    d.sw[i] = make_float4(ab.sw[0], ab.sw[1], ab.sw[2], ab.sw[3]);
}

// Phase A: the descriptor of one node of channel ch (0 = s, 1 = t, 2 = u).  The channel's own
// coordinate is a mesh value, so its offset is the triple's index e.
__device__ __forceinline__ void make_xdesc(const XyzArgs &a, const float *pos, int ch, int e, float s, float t, float u,
                                           float w1p, float w1, float w2p, float w2, float wp, float c, XDesc &d) {
    const MeshSearch<float> m{pos, a.n};
    const int nl = a.nl, n = a.n;
    AB4 ab;
    int ex = 0;
    // each pair of buffers interpolates two of the node's four distinct magnitudes (a
    // coordinate and its negation fold alike; -a - b is bitwise -(a + b))
    if (ch == 0) {  // integralKernelS, XYZFrgCore.cpp:218-224
        {
            const Interp<float> iA = interp_abs(m, w1 + wp), iB = interp_abs(m, w2 + wp);
            access4i<kS>(n, nl, s, -w1 - wp, -w2 - wp, iA, iB, e, ab); put_desc(d, 0, ab); ex |= ab.exch << 0;
            access4i<kS>(n, nl, s, w2 + wp, w1 + wp, iB, iA, e, ab); put_desc(d, 2, ab); ex |= ab.exch << 2;
        }
        {
            const Interp<float> iP = interp_abs(m, w1p + wp), iQ = interp_abs(m, w2p + wp);
            access4i<kS>(n, nl, s, w1p + wp, -w2p - wp, iP, iQ, e, ab); put_desc(d, 1, ab); ex |= ab.exch << 1;
            access4i<kS>(n, nl, s, -w2p - wp, w1p + wp, iQ, iP, e, ab); put_desc(d, 3, ab); ex |= ab.exch << 3;
        }
    } else if (ch == 1) {  // integralKernelT, XYZFrgCore.cpp:268-276, 323-345
        {
            const Interp<float> iC = interp_abs(m, w1 - wp), iP = interp_abs(m, w1p + wp);
            access4i<kT>(n, nl, w1 - wp, t, w1p + wp, iC, iP, e, ab); put_desc(d, 0, ab); ex |= ab.exch << 0;
            access4i<kT>(n, nl, w1p + wp, t, w1 - wp, iP, iC, e, ab); put_desc(d, 2, ab); ex |= ab.exch << 2;
            access4i<kU>(n, nl, w1 - wp, -w1p - wp, -t, iC, iP, e, ab); d.lv[1] = local4(a, ab);
            access4i<kU>(n, nl, w1p + wp, wp - w1, -t, iP, iC, e, ab); d.lv[3] = local4(a, ab);
        }
        {
            const Interp<float> iD = interp_abs(m, w2p - wp), iB = interp_abs(m, w2 + wp);
            access4i<kT>(n, nl, w2p - wp, t, -w2 - wp, iD, iB, e, ab); put_desc(d, 1, ab); ex |= ab.exch << 1;
            access4i<kT>(n, nl, w2 + wp, t, wp - w2p, iB, iD, e, ab); put_desc(d, 3, ab); ex |= ab.exch << 3;
            access4i<kU>(n, nl, w2p - wp, -w2 - wp, t, iD, iB, e, ab); d.lv[0] = local4(a, ab);
            access4i<kU>(n, nl, w2 + wp, wp - w2p, t, iB, iD, e, ab); d.lv[2] = local4(a, ab);
        }
    } else {  // integralKernelU, XYZFrgCore.cpp:424-430
        {
            const Interp<float> iA = interp_abs(m, w1 + wp), iD = interp_abs(m, w2p - wp);
            access4i<kU>(n, nl, w1 + wp, wp - w2p, u, iA, iD, e, ab); put_desc(d, 0, ab); ex |= ab.exch << 0;
            access4i<kU>(n, nl, w2p - wp, -w1 - wp, u, iD, iA, e, ab); put_desc(d, 2, ab); ex |= ab.exch << 2;
        }
        {
            const Interp<float> iP = interp_abs(m, w1p + wp), iE = interp_abs(m, w2 - wp);
            access4i<kU>(n, nl, w1p + wp, w2 - wp, u, iP, iE, e, ab); put_desc(d, 1, ab); ex |= ab.exch << 1;
            access4i<kU>(n, nl, w2 - wp, w1p + wp, u, iE, iP, e, ab); put_desc(d, 3, ab); ex |= ab.exch << 3;
        }
    }
    d.exch = ex;
    d.c = c;
}

// Phase B gather of buffer i of a descriptor (see gather4).
template <int SPT>
__device__ __forceinline__ void gather_desc(const XyzArgs &a, const XDesc &d, int i, const LaneT<SPT> &ln, float4 *out) {
    AB4 ab;
    const int4 o = d.off[i];
    const float4 w = d.w[i], sw = d.sw[i];
    ab.off[0] = o.x; ab.off[1] = o.y; ab.off[2] = o.z; ab.off[3] = o.w;
    ab.w[0] = w.x; ab.w[1] = w.y; ab.w[2] = w.z; ab.w[3] = w.w;
    ab.sw[0] = sw.x; ab.sw[1] = sw.y; ab.sw[2] = sw.z; ab.sw[3] = sw.w;
    ab.exch = (d.exch >> i) & 1;
    gather4(a, ab, ln, out);
}

constexpr int kXBatch = 4;  // nodes whose descriptors a warp builds at once

template <int SPT>
__global__ void __launch_bounds__(kThreads) xyz_vertex_kernel(XyzArgs a) {
    __shared__ float pos[kMaxFreq];
    // per warp: kXBatch node descriptors, then the first two t slabs of every site in all six
    // spin permutations, A6[p][nl] and B6[p][nl], then the RPA walk's run partials
    extern __shared__ float4 xs[];
    for (int i = threadIdx.x; i < a.n; i += blockDim.x) pos[i] = a.freq[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = a.n, nl = a.nl;
    const int warp_f4 = kXBatch * int(sizeof(XDesc) / sizeof(float4)) + 12 * nl + a.rpa_n_seg;
    XDesc *desc = reinterpret_cast<XDesc *>(xs + size_t(warp) * warp_f4);
    float4 *A6 = xs + size_t(warp) * warp_f4 + kXBatch * (sizeof(XDesc) / sizeof(float4)), *B6 = A6 + 6 * nl;
    float4 *slots = B6 + 6 * nl;
    const int rpa_cnt = a.rpa_count[lane], rpa_base = a.rpa_slot_base[lane];
    LaneT<SPT> ln;
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        const int j = lane + 32 * k;
        ln.j[k] = j;
        ln.valid[k] = j < nl;
        ln.rid[k] = ln.valid[k] ? a.sites[j] : 0;
        ln.prm[k] = ln.valid[k] ? a.sites_perm[j] : 0;
        ln.irid[k] = ln.valid[k] ? a.inv_sites[j] : 0;
        ln.iprm[k] = ln.valid[k] ? a.inv_sites_perm[j] : 0;
    }
    const float two_pi = 2.0f * float(kPiD);

    for (;;) {
        int it = 0;
        if (lane == 0) it = atomicAdd(a.work_counter, 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= a.fn) break;
        const int su = it / n, ti = it - su * n;
        int si = int((sqrtf(8.0f * float(su) + 1.0f) - 1.0f) * 0.5f);
        while (si * (si + 1) / 2 > su) --si;
        while ((si + 1) * (si + 2) / 2 <= su) ++si;
        const int ui = su - si * (si + 1) / 2;
        const float s = pos[si], t = pos[ti], u = pos[ui];
        const float w1p = 0.5f * (s + t + u), w1 = 0.5f * (s - t + u), w2p = 0.5f * (s - t - u), w2 = 0.5f * (s + t - u);

        float4 acc[SPT];
#pragma unroll
        for (int k = 0; k < SPT; ++k) acc[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (int ch = 0; ch < 3; ++ch) {
            const int xi = ch == 0 ? si : (ch == 1 ? ti : ui);
            const int cnt = a.node_cnt[xi];
            const float *nwp = a.node_wp + size_t(xi) * a.max_nodes;
            const float *nc = a.node_c + size_t(xi) * a.max_nodes;
            for (int b0 = 0; b0 < cnt; b0 += kXBatch) {
                const int nb = min(kXBatch, cnt - b0);
                if (lane < nb)  // phase A: lane = node
                    make_xdesc(a, pos, ch, xi, s, t, u, w1p, w1, w2p, w2, nwp[b0 + lane], nc[b0 + lane], desc[lane]);
                __syncwarp();
                for (int b = 0; b < nb; ++b) {  // phase B: lane = site
                    const XDesc &d = desc[b];
                    float4 S0[SPT], S1[SPT], S2[SPT], S3[SPT], r[SPT];
                    gather_desc(a, d, 0, ln, S0);
                    gather_desc(a, d, 1, ln, S1);
                    gather_desc(a, d, 2, ln, S2);
                    gather_desc(a, d, 3, ln, S3);
                    if (ch == 0) {  // XYZFrgCore.cpp:229-261
#pragma unroll
                        for (int k = 0; k < SPT; ++k) {
                            const float4 p = s_terms(S0[k], S1[k]), q = s_terms(S2[k], S3[k]);
                            r[k] = make_float4(p.x + q.x, p.y + q.y, p.z + q.z, p.w + q.w);
                        }
                    } else if (ch == 2) {  // XYZFrgCore.cpp:436-469
#pragma unroll
                        for (int k = 0; k < SPT; ++k) {
                            const float4 p = u_terms(S0[k], S1[k]), q = u_terms(S2[k], S3[k]);
                            r[k] = make_float4(p.x + q.x, p.y + q.y, p.z + q.z, p.w + q.w);
                        }
                    } else {  // t channel: RPA over the first two slabs of all sites, then local terms
#pragma unroll
                        for (int k = 0; k < SPT; ++k)
                            if (ln.valid[k]) {
                                const int j = ln.j[k];
                                A6[0 * nl + j] = permuted<0>(S0[k]);
                                A6[1 * nl + j] = permuted<1>(S0[k]);
                                A6[2 * nl + j] = permuted<2>(S0[k]);
                                A6[3 * nl + j] = permuted<3>(S0[k]);
                                A6[4 * nl + j] = permuted<4>(S0[k]);
                                A6[5 * nl + j] = permuted<5>(S0[k]);
                                B6[0 * nl + j] = permuted<0>(S1[k]);
                                B6[1 * nl + j] = permuted<1>(S1[k]);
                                B6[2 * nl + j] = permuted<2>(S1[k]);
                                B6[3 * nl + j] = permuted<3>(S1[k]);
                                B6[4 * nl + j] = permuted<4>(S1[k]);
                                B6[5 * nl + j] = permuted<5>(S1[k]);
                            }
                        __syncwarp();
                        const float4 cb = d.lv[0], ica = d.lv[1], cb2 = d.lv[2], ica2 = d.lv[3];
                        const float cbv[4] = {cb.x, cb.y, cb.z, cb.w}, icav[4] = {ica.x, ica.y, ica.z, ica.w};
                        const float cb2v[4] = {cb2.x, cb2.y, cb2.z, cb2.w}, ica2v[4] = {ica2.x, ica2.y, ica2.z, ica2.w};
                        {  // RPA (XYZFrgCore.cpp:282-305): every site's pairs in one lane-balanced walk
                            float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                            int slot = rpa_base;
                            for (int i = 0; i < rpa_cnt; ++i) {
                                const int e = __ldg(a.rpa_sched + 32 * i + lane);
                                const float4 x1 = A6[((e >> 14) & 7) * nl + (e & 127)];
                                const float4 x2 = B6[((e >> 17) & 7) * nl + ((e >> 7) & 127)];
                                p.x += x1.x * x2.x;
                                p.y += x1.y * x2.y;
                                p.z += x1.z * x2.z;
                                p.w += x1.w * x2.w;
                                if (e & (1 << 20)) {
                                    slots[slot++] = p;
                                    p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                                }
                            }
                        }
                        __syncwarp();
#pragma unroll
                        for (int k = 0; k < SPT; ++k) {
                            float rp[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                            if (ln.valid[k]) {  // the site's run partials, in order
                                for (int q = a.rpa_seg_ptr[ln.j[k]]; q < a.rpa_seg_ptr[ln.j[k] + 1]; ++q) {
                                    const float4 v = slots[q];
                                    rp[0] += v.x;
                                    rp[1] += v.y;
                                    rp[2] += v.z;
                                    rp[3] += v.w;
                                }
                            }
                            const float a0[4] = {S0[k].x, S0[k].y, S0[k].z, S0[k].w};
                            const float a1[4] = {S1[k].x, S1[k].y, S1[k].z, S1[k].w};
                            const float a2[4] = {S2[k].x, S2[k].y, S2[k].z, S2[k].w};
                            const float a3[4] = {S3[k].x, S3[k].y, S3[k].z, S3[k].w};
                            float rv[4];
#pragma unroll
                            for (int cc = 0; cc < 3; ++cc) {  // XYZFrgCore.cpp:347-401
                                const int pA = cc == X ? Y : X, pB = cc == Z ? Y : Z;
                                const int qA = cc == Z ? X : Z, qB = cc == X ? Y : (cc == Y ? X : Y);
                                float v = 4.0f * rp[cc];
                                v -= a0[cc] * cbv[D];
                                v += a0[cc] * cbv[pA];
                                v += a0[cc] * cbv[pB];
                                v -= a0[cc] * cbv[cc];
                                v -= icav[D] * a1[cc];
                                v += icav[qA] * a1[cc];
                                v += icav[qB] * a1[cc];
                                v -= icav[cc] * a1[cc];
                                v -= a2[cc] * cb2v[D];
                                v += a2[cc] * cb2v[pA];
                                v += a2[cc] * cb2v[pB];
                                v -= a2[cc] * cb2v[cc];
                                v -= ica2v[D] * a3[cc];
                                v += ica2v[qA] * a3[cc];
                                v += ica2v[qB] * a3[cc];
                                v -= ica2v[cc] * a3[cc];
                                rv[cc] = v;
                            }
                            {  // XYZFrgCore.cpp:402-417
                                float v = 4.0f * rp[D];
                                v -= a0[D] * cbv[D];
                                v -= a0[D] * cbv[X];
                                v -= a0[D] * cbv[Y];
                                v -= a0[D] * cbv[Z];
                                v -= icav[D] * a1[D];
                                v -= icav[X] * a1[D];
                                v -= icav[Y] * a1[D];
                                v -= icav[Z] * a1[D];
                                v -= a2[D] * cb2v[D];
                                v -= a2[D] * cb2v[X];
                                v -= a2[D] * cb2v[Y];
                                v -= a2[D] * cb2v[Z];
                                v -= ica2v[D] * a3[D];
                                v -= ica2v[X] * a3[D];
                                v -= ica2v[Y] * a3[D];
                                v -= ica2v[Z] * a3[D];
                                rv[D] = v;
                            }
                            r[k] = make_float4(rv[0], rv[1], rv[2], rv[3]);
                        }
                        __syncwarp();
                    }
                    const float c = d.c;
#pragma unroll
                    for (int k = 0; k < SPT; ++k) {
                        acc[k].x += c * r[k].x;
                        acc[k].y += c * r[k].y;
                        acc[k].z += c * r[k].z;
                        acc[k].w += c * r[k].w;
                    }
                }
                __syncwarp();
            }
        }
#pragma unroll
        for (int k = 0; k < SPT; ++k)
            if (ln.valid[k]) {
                const float4 o = make_float4(acc[k].x / two_pi, acc[k].y / two_pi, acc[k].z / two_pi, acc[k].w / two_pi);
                a.dsd[size_t(it) * nl + ln.j[k]] = o;
                if (isnan(o.x) || isnan(o.y) || isnan(o.z) || isnan(o.w)) atomicOr(a.status, kStatusNaN);
            }
    }
}

// ------------------------------------------------------------------------------------
// Vertex flow of lattices of at most 32 sites: a CTA per item of three triples (su2_item.cuh).
//
// A warp takes a node, lane = site: it reads the node's six planes (24 segments of 16-byte elements)
// and adds the node's s/u terms to two triples and its t terms to the third, with the site-local
// vertices of the t channel from the lane that holds pair 0.  The t channel's lattice sum
// sum over pairs of A[perm1 c][rid1] B[perm2 c][rid2] (A, B: the first and second slab) is linear in the node, so the
// CTA accumulates, over the nodes of a transfer frequency, the matrix of products of every spin component of A
// with every spin component of B (3w x 3w) and of the densities (w x w) in registers (a 16 x 16 grid of
// threads, 6 x 6 + 2 x 2 elements each at w = 32), and walks the pairs once per transfer frequency instead of
// once per node.
//
// Honeycomb r9 (28 sites, 2308 pairs), N = 48, cutoff 1: triple by triple, with the pairs walked for every node (577
// wavefronts of 16-byte shared reads), 14.2 ms a launch, bound by the shared-memory path; by items 5.6 ms, bound by
// instruction issue and the latency of the slab reads at two CTAs an SM.
// ------------------------------------------------------------------------------------
constexpr int kItemThreads = 256, kItemWarps = kItemThreads / 32;
constexpr int kItemBatch = 64;  // node descriptors built at once

// Exchange of a flow's pairs, as site_exchange_kind: 0 every pair is its own exchange with identity
// spin maps, 1 the exchange is an involution of the sites that fixes pair 0 and the direct pairs have
// identity spin maps, 2 any tables.
int xyz_site_kind(int nl, const int *sites, const int *perm, const int *inv, const int *inv_perm) {
    int kind = site_exchange_kind(nl, sites, inv);
    for (int j = 0; j < nl; ++j) {
        if (perm[j] != 0) return 2;
        if (kind == 0 && inv_perm[j] != 0) kind = 1;
    }
    return kind;
}

// (X, Y) and (Z, density) of an element.
struct Quad {
    float2 a, b;
};
__device__ __forceinline__ Quad load_quad(const float4 *p) {
    const float4 v = __ldg(p);
    return Quad{make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ float2 dup(float x) { return make_float2(x, x); }
// w1 * x + w2 * y, the density with its own weights
__device__ __forceinline__ Quad quad_mix(float w1, float d1, const Quad &x, float w2, float d2, const Quad &y) {
    return Quad{fma2(dup(w2), y.a, mul2(dup(w1), x.a)), fma2(make_float2(w2, d2), y.b, mul2(make_float2(w1, d1), x.b))};
}
__device__ __forceinline__ Quad quad_g(const ItemDesc &d, const float4 *v, int i, const float4 &wi, const float4 &wo) {
    const int4 o = d.g[i];
    const Quad x = quad_mix(wo.x, wo.y, load_quad(v + o.x), wo.z, wo.w, load_quad(v + o.z));
    const Quad y = quad_mix(wo.x, wo.y, load_quad(v + o.y), wo.z, wo.w, load_quad(v + o.w));
    return quad_mix(wi.x, wi.x, x, wi.z, wi.z, y);
}
// T plane i: the density of its off-diagonal supports in the first buffer (the second buffer's is the opposite).
__device__ __forceinline__ Quad quad_t(const ItemDesc &d, const float4 *v, int i) {
    const int4 o = d.t[i];
    const float4 p = d.tw[i][0], q = d.tw[i][1];
    const Quad x = quad_mix(p.x, p.y, load_quad(v + o.x), p.z, p.w, load_quad(v + o.y));
    const Quad y = quad_mix(q.x, q.y, load_quad(v + o.z), q.z, q.w, load_quad(v + o.w));
    return Quad{add2(x.a, y.a), add2(x.b, y.b)};
}
__device__ __forceinline__ float quad_t_diag(const ItemDesc &d, const float4 *v, int i) {
    const int4 o = d.t[i];
    const float4 w = d.td[i];
    return __fmaf_rn(w.w, __ldg(&v[o.w].w), __fmaf_rn(w.z, __ldg(&v[o.z].w), __fmaf_rn(w.y, __ldg(&v[o.y].w), __fmul_rn(w.x, __ldg(&v[o.x].w)))));
}
// the density of G plane i with the u channel's sign on the diagonal
__device__ __forceinline__ float quad_diag_u(const ItemDesc &d, const float4 *v, int i, const float4 &wi, const float4 &wo, float h) {
    const int4 o = d.g[i];
    const int bits = d.flags >> (kFlDiagShift + 2 * i);
    if (bits & 1) h = __fmaf_rn(-2.0f * wo.x, __fmaf_rn(wi.z, __ldg(&v[o.y].w), __fmul_rn(wi.x, __ldg(&v[o.x].w))), h);
    if (bits & 2) h = __fmaf_rn(-2.0f * wo.z, __fmaf_rn(wi.z, __ldg(&v[o.w].w), __fmul_rn(wi.x, __ldg(&v[o.z].w))), h);
    return h;
}
// X, Y, Z replaced by components perm[p][0..2]
__device__ __forceinline__ Quad quad_perm(const Quad &q, int p) {
    const float4 v = make_float4(q.a.x, q.a.y, q.b.x, q.b.y);
    return Quad{make_float2(comp_of(v, perm_c(p, 0)), comp_of(v, perm_c(p, 1))), make_float2(comp_of(v, perm_c(p, 2)), v.w)};
}
// adds the s/u integrand's products of a pair of slabs (s_terms)
__device__ __forceinline__ void add_su(const Quad &p, const Quad &q, float4 &r) {
    r.x = fmaf(p.b.y, q.a.x, fmaf(p.a.x, q.b.y, fmaf(-p.b.x, q.a.y, fmaf(-p.a.y, q.b.x, r.x))));
    r.y = fmaf(p.b.y, q.a.y, fmaf(p.a.y, q.b.y, fmaf(-p.b.x, q.a.x, fmaf(-p.a.x, q.b.x, r.y))));
    r.z = fmaf(p.b.y, q.b.x, fmaf(p.b.x, q.b.y, fmaf(-p.a.x, q.a.y, fmaf(-p.a.y, q.a.x, r.z))));
    r.w = fmaf(p.b.y, q.b.y, fmaf(p.a.x, q.a.x, fmaf(p.a.y, q.a.y, fmaf(p.b.x, q.b.x, r.w))));
}
__device__ __forceinline__ void add_acc(float4 &acc, float c, float cd, const float4 &r) {
    acc.x = fmaf(c, r.x, acc.x);
    acc.y = fmaf(c, r.y, acc.y);
    acc.z = fmaf(c, r.z, acc.z);
    acc.w = fmaf(cd, r.w, acc.w);
}
// Factors of the t channel's slab components for one site-local vertex l (XYZFrgCore.cpp:347-417), its density with
// the u channel's sign reversed: component c takes the two other spin components minus its own.
__device__ __forceinline__ float4 local_factors(const Quad &l) {
    const float x = l.a.x, y = l.a.y, z = l.b.x, h = l.b.y;
    return make_float4(y + z - x + h, x + z - y + h, x + y - z + h, h - x - y - z);
}
__device__ __forceinline__ float4 shfl4(const float4 &v) {
    constexpr unsigned kAll = 0xffffffffu;
    return make_float4(__shfl_sync(kAll, v.x, 0), __shfl_sync(kAll, v.y, 0), __shfl_sync(kAll, v.z, 0), __shfl_sync(kAll, v.w, 0));
}
__device__ __forceinline__ Quad shfl_quad(const Quad &q, int src) {
    constexpr unsigned kAll = 0xffffffffu;
    return Quad{make_float2(__shfl_sync(kAll, q.a.x, src), __shfl_sync(kAll, q.a.y, src)),
                make_float2(__shfl_sync(kAll, q.b.x, src), __shfl_sync(kAll, q.b.y, src))};
}

// One node at the lane's site, by a whole warp: adds the two s/u targets to acc1, acc2 and the t target's local terms
// to acct, and returns the first two t slabs (a times c) for the lattice sum.
__device__ __forceinline__ void xyz_node(const XyzArgs &a, const ItemDesc &d, int step, int rid, int prm, int irid, int iprm,
                                         int lane, float4 &acc1, float4 &acc2, float4 &acct, Quad &pa, Quad &pb) {
    const int fl = d.flags, kind = a.site_kind;
    const float c = d.c, c1 = step == 2 ? -c : c, c2 = step == 0 ? c : -c;
    const float4 wA = d.w[0], wB = d.w[1], wP = d.w[2], wQ = d.w[3];
    auto at = [&](int bit) { return a.sd + (fl & bit ? irid : rid); };
    auto site = [&](const Quad &q, int bit) {  // the site's components: its representative's, permuted
        if (fl & bit) return kind ? quad_perm(q, iprm) : q;
        return kind == 2 ? quad_perm(q, prm) : q;
    };
    const float4 *v0 = at(kFlE0), *v1 = at(kFlE1), *v2 = at(kFlE2), *v3 = at(kFlE3);
    Quad R0 = quad_g(d, v0, 0, wA, wB), R1 = quad_g(d, v1, 1, wP, wQ), R2 = quad_g(d, v2, 2, wB, wA), R3 = quad_g(d, v3, 3, wQ, wP);
    {
        float4 r = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        add_su(site(R0, kFlE0), site(R1, kFlE1), r);
        add_su(site(R2, kFlE2), site(R3, kFlE3), r);
        add_acc(acc1, c, c1, r);
    }
    const bool diag = step != 2 && (fl & kFlDiag) != 0;
    Quad U0 = R0, U1 = R1, U2 = R2, U3 = R3;  // densities with the u channel's signs
    if (diag) {
        U0.b.y = quad_diag_u(d, v0, 0, wA, wB, U0.b.y);
        U1.b.y = quad_diag_u(d, v1, 1, wP, wQ, U1.b.y);
        U2.b.y = quad_diag_u(d, v2, 2, wB, wA, U2.b.y);
        U3.b.y = quad_diag_u(d, v3, 3, wQ, wP, U3.b.y);
        if (step == 1) R0 = U0, R1 = U1, R2 = U2, R3 = U3;
    }
    // second target: a and b exchanged, G0 and G2 trade places with their own site exchange
    {
        Quad q0 = R0, q2 = R2;
        const bool f0 = ((fl & kFlE0) != 0) != ((fl & kFlF0) != 0), f2 = ((fl & kFlE2) != 0) != ((fl & kFlF2) != 0);
        if (kind == 1) {
            if (f0) q0 = shfl_quad(q0, irid);
            if (f2) q2 = shfl_quad(q2, irid);
        } else if (kind == 2) {
            const float4 *b0 = at(kFlF0), *b2 = at(kFlF2);
            q0 = quad_g(d, b0, 0, wA, wB);
            q2 = quad_g(d, b2, 2, wB, wA);
            if (diag && step == 1) {
                q0.b.y = quad_diag_u(d, b0, 0, wA, wB, q0.b.y);
                q2.b.y = quad_diag_u(d, b2, 2, wB, wA, q2.b.y);
            }
        }
        float4 r = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        add_su(site(q2, kFlF2), site(R1, kFlE1), r);
        add_su(site(q0, kFlF0), site(R3, kFlE3), r);
        add_acc(acc2, c, c2, r);
    }
    // t channel: buffers 0, 2 (1, 3) have equal spin slabs and opposite off-diagonal densities, and the local vertices
    // of planes G2, G0 (G1, G3) at pair 0
    if (kind == 2) {
        U0 = quad_g(d, a.sd, 0, wA, wB);
        U1 = quad_g(d, a.sd, 1, wP, wQ);
        U2 = quad_g(d, a.sd, 2, wB, wA);
        U3 = quad_g(d, a.sd, 3, wQ, wP);
        if (diag) {
            U0.b.y = quad_diag_u(d, a.sd, 0, wA, wB, U0.b.y);
            U1.b.y = quad_diag_u(d, a.sd, 1, wP, wQ, U1.b.y);
            U2.b.y = quad_diag_u(d, a.sd, 2, wB, wA, U2.b.y);
            U3.b.y = quad_diag_u(d, a.sd, 3, wQ, wP, U3.b.y);
        }
    }
    const float4 m0 = local_factors(U2), m1 = local_factors(U1), m2 = local_factors(U0), m3 = local_factors(U3);
    const float4 k0 = shfl4(make_float4(m0.x + m2.x, m0.y + m2.y, m0.z + m2.z, m0.w - m2.w));
    const float4 k1 = shfl4(make_float4(m1.x + m3.x, m1.y + m3.y, m1.z + m3.z, m1.w - m3.w));
    const float4 *vt0 = at(kFlT0), *vt1 = at(kFlT1);
    Quad T0 = site(quad_t(d, vt0, 0), kFlT0), T1 = site(quad_t(d, vt1, 1), kFlT1);
    float4 r = make_float4(fmaf(k1.x, T1.a.x, k0.x * T0.a.x), fmaf(k1.y, T1.a.y, k0.y * T0.a.y),
                           fmaf(k1.z, T1.b.x, k0.z * T0.b.x), fmaf(k1.w, T1.b.y, k0.w * T0.b.y));
    if (fl & (kFlDiagT | kFlExT)) {
        const float d0 = __shfl_sync(0xffffffffu, m0.w + m2.w, 0), d1 = __shfl_sync(0xffffffffu, m1.w + m3.w, 0);
        const float e0 = quad_t_diag(d, vt0, 0), e1 = quad_t_diag(d, vt1, 1);
        r.w = fmaf(d0, e0, fmaf(d1, e1, r.w));
        if (fl & kFlExT) {  // the fourth buffer reads the other site
            const float4 f = shfl4(m3);
            const float4 *vt3 = at(kFlT3);
            const Quad T3 = site(quad_t(d, vt3, 1), kFlT3);
            const float e3 = quad_t_diag(d, vt3, 1);
            r.x = fmaf(f.x, T3.a.x - T1.a.x, r.x);
            r.y = fmaf(f.y, T3.a.y - T1.a.y, r.y);
            r.z = fmaf(f.z, T3.b.x - T1.b.x, r.z);
            r.w = fmaf(f.w, (e3 - T3.b.y) - (e1 - T1.b.y), r.w);
        }
        T0.b.y += e0;
        T1.b.y += e1;
    }
    add_acc(acct, c, c, r);
    pa = Quad{mul2(dup(c), T0.a), mul2(dup(c), T0.b)};
    pb = T1;
}

struct XyzItemSmem {
    size_t u, ms, panels, parts, rpa, total;
};
__host__ __device__ inline XyzItemSmem xyz_item_smem(int R, bool once, int n_seg) {
    const int w = 16 * R;
    XyzItemSmem L;
    size_t o = 0;
    // a batch's descriptors and (after a transfer frequency) the product matrices and the walk's partials, in a union but for `once`
    L.u = o;
    const size_t d = kItemBatch * sizeof(ItemDesc), m = sizeof(float) * size_t(10 * w * w) + sizeof(float4) * size_t(n_seg);
    L.ms = once ? o + d : o;
    o += ((once ? d + m : (d > m ? d : m)) + 15) / 16 * 16;
    L.panels = o; o += sizeof(float) * 2 * kItemWarps * 8 * size_t(w);  // 2 buffers x nodes x (A, B) x 4 components
    L.parts = o; o += sizeof(float4) * 3 * kItemWarps * size_t(w);
    L.rpa = o; o += sizeof(float4) * 3 * size_t(w);
    L.total = o;
    return L;
}

// Adds a panel to the thread's block of the product matrices.  Panel: A's components X, Y, Z, D of w sites each,
// then B's.
template <int R>
__device__ __forceinline__ void xyz_outer(const float *pan, int tr, int tc, float2 (&S)[3 * R][(3 * R + 1) / 2],
                                          float (&Dm)[R][R]) {
    constexpr int w = 16 * R, K = 3 * R, K2 = (K + 1) / 2;
    float av[K], ad[R], bd[R];
    float2 bv[K2];
    if constexpr (K % 2 == 0) {  // 8-byte reads
        const float2 *pa = reinterpret_cast<const float2 *>(pan + tr * K), *pb = reinterpret_cast<const float2 *>(pan + 4 * w + tc * K);
#pragma unroll
        for (int i = 0; i < K2; ++i) {
            const float2 v = pa[i];
            av[2 * i] = v.x;
            av[2 * i + 1] = v.y;
            bv[i] = pb[i];
        }
    } else {
#pragma unroll
        for (int i = 0; i < K; ++i) av[i] = pan[tr * K + i];
#pragma unroll
        for (int j = 0; j < K2; ++j)
            bv[j] = make_float2(pan[4 * w + tc * K + 2 * j], 2 * j + 1 < K ? pan[4 * w + tc * K + 2 * j + 1] : 0.0f);
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        ad[i] = pan[3 * w + tr * R + i];
        bd[i] = pan[7 * w + tc * R + i];
    }
#pragma unroll
    for (int i = 0; i < K; ++i)
#pragma unroll
        for (int j = 0; j < K2; ++j) S[i][j] = fma2(dup(av[i]), bv[j], S[i][j]);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) Dm[i][j] = fmaf(ad[i], bd[j], Dm[i][j]);
}

// ONCE: the nodes of any three transfer frequencies together are at most kItemBatch, so an item's descriptors are built at once.  At so few nodes,
// as early in a flow, the builds before each transfer frequency are most of an item's time: at 3 sites, N = 32, cutoff 20 a
// right-hand side took 496 us with them (429 triple by triple), 416 without; later in the flow the form costs 1 to 2 %
// (registers), so it is a kernel by itself.
template <int R, bool ONCE>
__global__ void __launch_bounds__(kItemThreads, 2) xyz_item_kernel(XyzArgs a) {
    constexpr int w = 16 * R, K = 3 * R, K2 = (K + 1) / 2;
    extern __shared__ float4 xs[];
    __shared__ float pos[kMaxFreq];
    __shared__ int s_item;
    unsigned char *smem = reinterpret_cast<unsigned char *>(xs);
    const XyzItemSmem L = xyz_item_smem(R, ONCE, a.rpa_n_seg);
    ItemDesc *desc = reinterpret_cast<ItemDesc *>(smem + L.u);
    float *Ms = reinterpret_cast<float *>(smem + L.ms);  // spin (3w x 3w), then density (w x w)
    float4 *slots = reinterpret_cast<float4 *>(Ms + 10 * w * w);
    float *panels = reinterpret_cast<float *>(smem + L.panels);
    float4 *parts = reinterpret_cast<float4 *>(smem + L.parts);
    float4 *rpa = reinterpret_cast<float4 *>(smem + L.rpa);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tr = tid >> 4, tc = tid & 15;
    const int n = a.n, nl = a.nl;
    for (int i = tid; i < n; i += blockDim.x) pos[i] = a.freq[i];
    const bool valid = lane < nl;
    const int sc = min(lane, nl - 1);  // a lane without a site reads the last one's elements
    const int rid = a.sites[sc], prm = a.sites_perm[sc], irid = a.inv_sites[sc], iprm = a.inv_sites_perm[sc];
    const int rpa_cnt = a.rpa_count[tid], rpa_base = a.rpa_slot_base[tid];
    const float two_pi = 2.0f * float(kPiD);
    const int items = vertex_items(n);
    const MeshSearch<float> mesh{pos, n};
    int round = 0;
    for (;;) {
        __syncthreads();  // the previous item is finished with shared memory
        if (tid == 0) s_item = atomicAdd(a.work_counter, 1);
        __syncthreads();
        const int item = s_item;
        if (item >= items) break;
        int p, q, r;
        decode_item(item, p, q, r);
        float4 A = make_float4(0.0f, 0.0f, 0.0f, 0.0f), B = A, T = A;
        // transfer p: targets (p,q,r), (p,r,q) and the t channel of (q,p,r); q: (q,p,r), (p,r,q), t of (p,q,r);
        // r: (q,p,r), (p,q,r), t of (p,r,q)
        [[maybe_unused]] int first = 0;  // the transfer frequency's first descriptor
        if constexpr (ONCE) {
            const int n0 = __ldg(a.node_cnt + p), n1 = __ldg(a.node_cnt + q), step = tid < n0 ? 0 : (tid < n0 + n1 ? 1 : 2);
            const ItemFreq f = item_freq(pos, step == 0 ? p : (step == 1 ? q : r), step == 0 ? q : p, step == 2 ? q : r, step == 2);
            const int node = tid - (step == 0 ? 0 : (step == 1 ? n0 : n0 + n1));
            const size_t k = size_t(f.xi) * a.max_nodes + node;
            if (tid < kItemBatch && node < __ldg(a.node_cnt + f.xi)) make_item(mesh, nl, f, __ldg(a.node_wp + k), __ldg(a.node_c + k), desc[tid]);
            __syncthreads();
        }
#pragma unroll 1
        for (int step = 0; step < 3; ++step) {
            const ItemFreq f = item_freq(pos, step == 0 ? p : (step == 1 ? q : r), step == 0 ? q : p, step == 2 ? q : r, step == 2);
            float2 S[K][K2];
            float Dm[R][R];
#pragma unroll
            for (int i = 0; i < K; ++i)
#pragma unroll
                for (int j = 0; j < K2; ++j) S[i][j] = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int i = 0; i < R; ++i)
#pragma unroll
                for (int j = 0; j < R; ++j) Dm[i][j] = 0.0f;
            const int cnt = __ldg(a.node_cnt + f.xi);
            const float *nwp = a.node_wp + size_t(f.xi) * a.max_nodes;
            const float *nc = a.node_c + size_t(f.xi) * a.max_nodes;
#pragma unroll 1
            for (int b0 = 0; b0 < cnt; b0 += kItemBatch) {
                const int nb = min(kItemBatch, cnt - b0);
                if constexpr (!ONCE) {
                    __syncthreads();  // the previous batch's descriptors (or the matrices) are no longer read
                    if (tid < nb) make_item(mesh, nl, f, __ldg(nwp + b0 + tid), __ldg(nc + b0 + tid), desc[tid]);
                    __syncthreads();
                }
#pragma unroll 1
                for (int r0 = 0; r0 < nb; r0 += kItemWarps, ++round) {
                    float *buf = panels + size_t(round & 1) * kItemWarps * 8 * w;
                    if (r0 + warp < nb) {
                        Quad pa, pb;
                        xyz_node(a, desc[ONCE ? first + r0 + warp : r0 + warp], step, rid, prm, irid, iprm, lane, A, B, T, pa, pb);
                        if (valid) {
                            float *pan = buf + warp * 8 * w + lane;
                            pan[0] = pa.a.x;
                            pan[w] = pa.a.y;
                            pan[2 * w] = pa.b.x;
                            pan[3 * w] = pa.b.y;
                            pan[4 * w] = pb.a.x;
                            pan[5 * w] = pb.a.y;
                            pan[6 * w] = pb.b.x;
                            pan[7 * w] = pb.b.y;
                        }
                    }
                    __syncthreads();  // the round's panels are written
                    const int np = min(kItemWarps, nb - r0);
#pragma unroll 1
                    for (int k = 0; k < np; ++k) xyz_outer<R>(buf + k * 8 * w, tr, tc, S, Dm);
                }
            }
            __syncthreads();  // every descriptor read is done
#pragma unroll
            for (int i = 0; i < K; ++i)
#pragma unroll
                for (int j = 0; j < K; ++j) Ms[(tr * K + i) * 3 * w + tc * K + j] = (j & 1) ? S[i][j / 2].y : S[i][j / 2].x;
#pragma unroll
            for (int i = 0; i < R; ++i)
#pragma unroll
                for (int j = 0; j < R; ++j) Ms[9 * w * w + (tr * R + i) * w + tc * R + j] = Dm[i][j];
            __syncthreads();
            {  // XYZFrgCore.cpp:282-305, every site's pairs in one walk
                float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                int slot = rpa_base;
                for (int i = 0; i < rpa_cnt; ++i) {
                    const int e = __ldg(a.rpa_sched + kItemThreads * i + tid);
                    const int r1 = e & 127, r2 = (e >> 7) & 127, p1 = (e >> 14) & 7, p2 = (e >> 17) & 7;
                    sum.x += Ms[(perm_c(p1, 0) * w + r1) * 3 * w + perm_c(p2, 0) * w + r2];
                    sum.y += Ms[(perm_c(p1, 1) * w + r1) * 3 * w + perm_c(p2, 1) * w + r2];
                    sum.z += Ms[(perm_c(p1, 2) * w + r1) * 3 * w + perm_c(p2, 2) * w + r2];
                    sum.w += Ms[9 * w * w + r1 * w + r2];
                    if (e & (1 << 20)) {
                        slots[slot++] = sum;
                        sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    }
                }
            }
            __syncthreads();
            if (tid < nl) {
                float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                for (int k = a.rpa_seg_ptr[tid]; k < a.rpa_seg_ptr[tid + 1]; ++k) {
                    const float4 v = slots[k];
                    sum.x += v.x;
                    sum.y += v.y;
                    sum.z += v.z;
                    sum.w += v.w;
                }
                rpa[step * w + tid] = sum;
            }
            if constexpr (ONCE) first += cnt;
            if (step == 0) { const float4 t = A; A = T; T = t; }
            if (step == 1) { const float4 t = B; B = T; T = t; }
        }
        if (valid) {
            parts[(0 * kItemWarps + warp) * w + lane] = B;  // (p,q,r), t channel of transfer q
            parts[(1 * kItemWarps + warp) * w + lane] = T;  // (p,r,q), r
            parts[(2 * kItemWarps + warp) * w + lane] = A;  // (q,p,r), p
        }
        __syncthreads();
        for (int e = tid; e < 3 * nl; e += kItemThreads) {
            const int k = e / nl, j = e - k * nl;
            if ((k == 1 && q == r) || (k == 2 && p == q)) continue;  // the same triple again
            float4 v[kItemWarps];
#pragma unroll
            for (int u = 0; u < kItemWarps; ++u) v[u] = parts[(k * kItemWarps + u) * w + j];
#pragma unroll
            for (int o = 1; o < kItemWarps; o <<= 1)
#pragma unroll
                for (int u = 0; u + o < kItemWarps; u += 2 * o)
                    v[u] = make_float4(v[u].x + v[u + o].x, v[u].y + v[u + o].y, v[u].z + v[u + o].z, v[u].w + v[u + o].w);
            const float4 g = rpa[((k + 1) % 3) * w + j];
            const int ts = k == 2 ? q : p, tt = k == 0 ? q : (k == 1 ? r : p), tu = k == 1 ? q : r;
            const float4 o = make_float4((v[0].x + 4.0f * g.x) / two_pi, (v[0].y + 4.0f * g.y) / two_pi,
                                         (v[0].z + 4.0f * g.z) / two_pi, (v[0].w + 4.0f * g.w) / two_pi);
            a.dsd[(size_t(su_index(ts, tu)) * n + tt) * nl + j] = o;
            if (isnan(o.x) || isnan(o.y) || isnan(o.z) || isnan(o.w)) atomicOr(a.status, kStatusNaN);
        }
    }
}

// ------------------------------------------------------------------------------------
// correlation measurement at nu = 0 (XYZMeasurementCorrelation.cpp:98-184): one CTA per
// outer node accumulates the inner integral per site in FP64, a final CTA adds the outer
// weights and the on-site term and scatters to (basis, site in range) entries.
// ------------------------------------------------------------------------------------
// getValueSuperbundle through a trilinear buffer for one site: X, Y, Z the components of the
// representative r under permutation p, D the signed density.
SPN_HDI void bundle8(const XyzArgs &a, const AB8 &ab, int r, int p, float g[4]) {
    g[0] = g[1] = g[2] = g[3] = 0.0f;
    for (int q = 0; q < 8; ++q) {
        const float4 v = ro_load(a.sd + ab.off[q] + r);
        for (int c = 0; c < 3; ++c) g[c] += ab.w[q] * comp_of(v, perm_c(p, c));
        g[3] += ab.sw[q] * v.w;
    }
}

// Linear in the vertex, as the SU(2) core's (corr_inner_body): sums of g * vertex per site and, a
// thread per node, of the on-site reads.
constexpr int kCorrXWarps = 8, kCorrXThreads = 32 * kCorrXWarps;

__global__ void __launch_bounds__(kCorrXThreads) xyz_corr_inner_kernel(XyzArgs a) {
    __shared__ float pos[kMaxFreq];
    __shared__ float nwp[kMaxCorrNodes];
    __shared__ double nw[kMaxCorrNodes], ng[kMaxCorrNodes];
    __shared__ double red[kCorrXWarps][4][32 * kSpt];
    __shared__ double egg[kCorrXWarps][4];
    for (int i = threadIdx.x; i < a.n; i += blockDim.x) pos[i] = a.freq[i];
    __syncthreads();
    const int ncnt = corr_nodes(pos, a.n, a.cutoff, nwp, nw, ng, [&](float x) { return odd_interp(pos, a.n, a.v2, x); });
    const int ia = blockIdx.x;
    if (ia >= ncnt) return;
    const float w = nwp[ia];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nl = a.nl;
    Lane4 ln;
#pragma unroll
    for (int k = 0; k < kSpt; ++k) {
        const int j = lane + 32 * k;
        ln.j[k] = j;
        ln.valid[k] = j < nl;
        ln.rid[k] = ln.valid[k] ? a.sites[j] : 0;
        ln.prm[k] = ln.valid[k] ? a.sites_perm[j] : 0;
        ln.irid[k] = ln.valid[k] ? a.inv_sites[j] : 0;
        ln.iprm[k] = ln.valid[k] ? a.inv_sites_perm[j] : 0;
    }
    double e[4] = {0.0, 0.0, 0.0, 0.0};
    for (int q = threadIdx.x; q < 4 * ncnt; q += blockDim.x) {  // a thread per node and component
        const int c = q & 3, b = q >> 2;
        const float wp = nwp[b];
        const double v = nw[b] * ng[b] * double(value4(pos, a, c, 0, 0, w + wp + 0.0f, w - wp, 0.0f));
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k == c) e[k] += v;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        for (int o = 16; o > 0; o >>= 1) e[c] += __shfl_xor_sync(0xffffffffu, e[c], o);
        if (lane == 0) egg[warp][c] = e[c];
    }
    double acc[kSpt][4];
#pragma unroll
    for (int k = 0; k < kSpt; ++k)
        for (int c = 0; c < 4; ++c) acc[k][c] = 0.0;
    for (int b = warp; b < ncnt; b += kCorrXWarps) {
        const float wp = nwp[b];
        AB8 ab;
        access8(pos, a.n, nl, w + wp + 0.0f, 0.0f, w - wp, ab);
        const double cw = nw[b] * ng[b];
#pragma unroll
        for (int k = 0; k < kSpt; ++k) {
            if (!ln.valid[k]) continue;
            float g[4];
            bundle8(a, ab, ab.exch ? ln.irid[k] : ln.rid[k], ab.exch ? ln.iprm[k] : ln.prm[k], g);
            for (int c = 0; c < 4; ++c) acc[k][c] += cw * double(g[c]);
        }
    }
#pragma unroll
    for (int k = 0; k < kSpt; ++k)
        for (int c = 0; c < 4; ++c) red[warp][c][lane + 32 * k] = acc[k][c];
    __syncthreads();
    const double norm = ng[ia] / (4.0 * kPiD * kPiD);
    for (int p = threadIdx.x; p < 4 * nl; p += blockDim.x) {
        const int c = p / nl, j = p - c * nl;
        double sum = 0.0;
        for (int q = 0; q < kCorrXWarps; ++q) sum += red[q][c][j];
        sum *= c == D ? -4.0 : -1.0;  // dumbbell
        if (j == 0) {                 // egg diagram
            double v[4] = {0.0, 0.0, 0.0, 0.0};
            for (int q = 0; q < kCorrXWarps; ++q)
                for (int k = 0; k < 4; ++k) v[k] += egg[q][k];
            if (c == D) sum += 2.0 * (v[0] + v[1] + v[2] + v[3]);
            else sum += 0.5 * (2.0 * v[c] - v[0] - v[1] - v[2] + v[3]);
        }
        a.partial[(size_t(ia) * 4 + c) * nl + j] = sum * norm;
    }
}

__global__ void __launch_bounds__(kCorrThreads) xyz_corr_final_kernel(XyzArgs a) {
    __shared__ float pos[kMaxFreq];
    __shared__ float nwp[kMaxCorrNodes];
    __shared__ double nw[kMaxCorrNodes], ng[kMaxCorrNodes];
    extern __shared__ double chi[];  // [4][nl] and the reduction's slices
    for (int i = threadIdx.x; i < a.n; i += blockDim.x) pos[i] = a.freq[i];
    __syncthreads();
    const int ncnt = corr_nodes(pos, a.n, a.cutoff, nwp, nw, ng, [&](float x) { return odd_interp(pos, a.n, a.v2, x); });
    const int nl = a.nl;
    column_sums(ncnt, 4 * nl, chi, [&](int ia, int e) { return nw[ia] * a.partial[size_t(ia) * 4 * nl + e]; });
    if (threadIdx.x < 32) {  // on-site term
        double s = 0.0;
        for (int k = threadIdx.x; k < ncnt; k += 32) s += nw[k] * ng[k];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (threadIdx.x < 4) chi[threadIdx.x * nl] += threadIdx.x == D ? s / kPiD : s / (4.0 * kPiD);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 4 * nl; e += blockDim.x) a.out[4 * size_t(a.n_corr) + e] = float(chi[e]);
    for (int q = threadIdx.x; q < a.n_corr; q += blockDim.x) {
        const int r = a.corr_rid[q], p = a.corr_perm[q];
        for (int c = 0; c < 3; ++c) a.out[size_t(c) * a.n_corr + q] = float(chi[perm_c(p, c) * nl + r]);
        a.out[3 * size_t(a.n_corr) + q] = float(chi[3 * nl + r]);
    }
}

// ------------------------------------------------------------------------------------
// Euler step, state layout changes
// ------------------------------------------------------------------------------------
__global__ void xyz_euler_kernel(float *__restrict__ x, const float *__restrict__ dx, long long n, float step) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        x[i] = __fadd_rn(x[i], __fmul_rn(step, dx[i]));
}

// stage[c * n + i] (four arrays in the reference layout) <-> v[i] (one float4 per element)
__global__ void xyz_pack_kernel(const float *__restrict__ stage, float4 *__restrict__ v, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        v[i] = make_float4(stage[i], stage[n + i], stage[2 * n + i], stage[3 * n + i]);
}
__global__ void xyz_unpack_kernel(const float4 *__restrict__ v, float *__restrict__ stage, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float4 e = v[i];
        stage[i] = e.x;
        stage[n + i] = e.y;
        stage[2 * n + i] = e.z;
        stage[3 * n + i] = e.w;
    }
}

using cuh::check_cuda;
using cuh::copy_grid;
using cuh::dalloc;
using cuh::h2d;

}  // namespace

struct spn_xyz {
    int device = 0, n = 0, nl = 0, n_range = 0, n_corr = 0, n_overlap = 0, max_nodes = 0, sms = 0, grid = 0;
    long long fn = 0;
    float cutoff = 0.0f;
    std::vector<float> mesh;
    cudaStream_t stream = nullptr;
    float *freq = nullptr, *v2 = nullptr, *dv2 = nullptr, *stage = nullptr, *node_wp = nullptr, *node_c = nullptr,
          *corr_out = nullptr;
    float4 *sd = nullptr, *dsd = nullptr;
    int *ints = nullptr;  // all integer tables in one allocation
    int *sites, *sites_perm, *inv_sites, *inv_sites_perm, *range_rid, *range_inv, *corr_rid, *corr_perm, *node_cnt,
        *work_counter, *rpa_sched, *rpa_count, *rpa_slot_base, *rpa_seg_ptr;
    int rpa_n_seg = 0, site_kind = 0;
    unsigned *status = nullptr;  // in ints, behind the work counters
    spn::cuh::HostResults results;  // measurements and the status word on the host
    double *partial = nullptr;

    XyzArgs args() const {
        XyzArgs a;
        a.n = n;
        a.nl = nl;
        a.fn = int(fn);
        a.max_nodes = max_nodes;
        a.n_range = n_range;
        a.n_corr = n_corr;
        a.cutoff = cutoff;
        a.freq = freq;
        a.sd = sd;
        a.dsd = dsd;
        a.v2 = v2;
        a.dv2 = dv2;
        a.sites = sites;
        a.sites_perm = sites_perm;
        a.inv_sites = inv_sites;
        a.inv_sites_perm = inv_sites_perm;
        a.rpa_sched = rpa_sched;
        a.rpa_count = rpa_count;
        a.rpa_slot_base = rpa_slot_base;
        a.rpa_seg_ptr = rpa_seg_ptr;
        a.rpa_n_seg = rpa_n_seg;
        a.site_kind = site_kind;
        a.range_rid = range_rid;
        a.range_inv = range_inv;
        a.node_wp = node_wp;
        a.node_c = node_c;
        a.node_cnt = node_cnt;
        a.work_counter = work_counter;
        a.status = status;
        a.corr_rid = corr_rid;
        a.corr_perm = corr_perm;
        a.partial = partial;
        a.out = corr_out;
        return a;
    }

    // argument block of the SU(2) node-table body (self-energy, mesh, node tables only)
    FlowArgs node_args() const {
        FlowArgs f;
        std::memset(&f, 0, sizeof(f));
        f.n = n;
        f.nl = nl;
        f.max_nodes = max_nodes;
        f.cutoff = cutoff;
        f.freq = freq;
        f.v2 = v2;
        f.dv2 = dv2;
        f.fp64_sigma = 0;
        f.node_wp = node_wp;
        f.node_c = node_c;
        f.node_cnt = node_cnt;
        f.status = status;
        return f;
    }

    void release() {
        cudaSetDevice(device);
        void *ptrs[] = {freq, v2, dv2, stage, node_wp, node_c, corr_out, sd, dsd, ints, partial};
        for (void *p : ptrs)
            if (p) cudaFree(p);
        if (stream) cudaStreamDestroy(stream);
    }
};

namespace {

void validate(const spn_xyz_desc *d) {
    if (!d) throw Error(ErrorType::Argument, "null descriptor");
    if (d->n_freq < 2 || d->n_freq > kMaxFreq)
        throw Error(ErrorType::Unsupported, "n_freq must be in [2, " + std::to_string(kMaxFreq) + "]");
    if (d->n_sites < 1 || d->n_sites > 32 * kSpt)
        throw Error(ErrorType::Unsupported, "n_sites must be in [1, " + std::to_string(32 * kSpt) + "]");
    if (!d->freq || !d->sites_rid || !d->sites_perm || !d->inv_sites_rid || !d->inv_sites_perm || !d->overlap_ptr ||
        (d->n_range > 0 && (!d->range_rid || !d->range_inv_rid)) || (d->n_corr > 0 && (!d->corr_rid || !d->corr_perm)))
        throw Error(ErrorType::Argument, "descriptor table pointer is NULL");
    for (int i = 0; i < d->n_freq; ++i) {
        if (!(d->freq[i] > 0.0f)) throw Error(ErrorType::Argument, "frequencies must be positive");
        if (i > 0 && !(d->freq[i] > d->freq[i - 1])) throw Error(ErrorType::Argument, "frequencies must be strictly ascending");
    }
    const long long fn = (long long)d->n_freq * d->n_freq * (d->n_freq + 1) / 2;
    if (fn * d->n_sites >= (1ll << 31)) throw Error(ErrorType::Unsupported, "vertex larger than 2^31 elements");
    const int nl = d->n_sites;
    auto in_range = [&](const int *v, int cnt, int hi, const char *what) {
        for (int i = 0; i < cnt; ++i)
            if (v[i] < 0 || v[i] >= hi) throw Error(ErrorType::Argument, std::string(what) + " entry out of range");
    };
    in_range(d->sites_rid, nl, nl, "sites_rid");
    in_range(d->inv_sites_rid, nl, nl, "inv_sites_rid");
    in_range(d->sites_perm, nl, 6, "sites_perm");
    in_range(d->inv_sites_perm, nl, 6, "inv_sites_perm");
    if (d->overlap_ptr[0] != 0) throw Error(ErrorType::Argument, "overlap_ptr[0] must be 0");
    for (int r = 0; r < nl; ++r)
        if (d->overlap_ptr[r + 1] < d->overlap_ptr[r]) throw Error(ErrorType::Argument, "overlap_ptr must be non-decreasing");
    const int nov = d->overlap_ptr[nl];
    if (nov > 0 && (!d->overlap_rid1 || !d->overlap_rid2 || !d->overlap_perm1 || !d->overlap_perm2))
        throw Error(ErrorType::Argument, "overlap pair table is NULL");
    in_range(d->overlap_rid1, nov, nl, "overlap_rid1");
    in_range(d->overlap_rid2, nov, nl, "overlap_rid2");
    in_range(d->overlap_perm1, nov, 6, "overlap_perm1");
    in_range(d->overlap_perm2, nov, 6, "overlap_perm2");
    in_range(d->range_rid, d->n_range, nl, "range_rid");
    in_range(d->range_inv_rid, d->n_range, nl, "range_inv_rid");
    in_range(d->corr_rid, d->n_corr, nl, "corr_rid");
    in_range(d->corr_perm, d->n_corr, 6, "corr_perm");
}

// The vertex kernel: by items for Nl <= 32, else by triples with SPT sites per lane (2 for Nl <= 64, else 4).
const void *vertex_kernel(int nl, bool once) {
    if (nl <= 16) return once ? reinterpret_cast<const void *>(&xyz_item_kernel<1, true>) : reinterpret_cast<const void *>(&xyz_item_kernel<1, false>);
    if (nl <= 32) return reinterpret_cast<const void *>(&xyz_item_kernel<2, false>);
    if (nl <= 64) return reinterpret_cast<const void *>(&xyz_vertex_kernel<2>);
    return reinterpret_cast<const void *>(&xyz_vertex_kernel<4>);
}
int vertex_threads(int nl) { return nl <= 32 ? kItemThreads : kThreads; }

// The RPA pairs of each site in the order of host/pair_order (against bank collisions of the
// kernel's 16-byte reads of A6 and B6), packed rid1 | rid2 << 7 | perm1 << 14 | perm2 << 17.
std::vector<int> order_rpa_pairs(const spn_xyz_desc *d) {
    const int nl = d->n_sites;
    const std::vector<int> order =
        order_pairs_by_banks(nl, d->overlap_ptr, xyz_rpa_model(),
                             xyz_rpa_words(nl, d->overlap_rid1, d->overlap_rid2, d->overlap_perm1, d->overlap_perm2));
    std::vector<int> out(order.size());
    for (size_t k = 0; k < order.size(); ++k) {
        const int i = order[k];
        out[k] = d->overlap_rid1[i] | d->overlap_rid2[i] << 7 | d->overlap_perm1[i] << 14 | d->overlap_perm2[i] << 17;
    }
    return out;
}

size_t vertex_smem(const spn_xyz *h, bool once) {
    if (h->nl <= 32) return xyz_item_smem(h->nl <= 16 ? 1 : 2, once, h->rpa_n_seg).total;
    return size_t(kWarps) * (kXBatch * sizeof(XDesc) + (12 * size_t(h->nl) + size_t(h->rpa_n_seg)) * sizeof(float4));
}

// Whether the items' descriptors are built at once (xyz_item_kernel<1, true>), at the flow's cutoff.
bool build_once(const spn_xyz *h) {
    if (h->nl > 16) return false;
    int most = 0;
    for (int i = 0; i < h->n; ++i) {
        QuadRule<float> r[3];
        int cnt[3];
        const int conv = node_rules(h->mesh.data(), h->n, i, h->cutoff, r, cnt);
        most = std::max(most, conv + cnt[0] + cnt[1] + cnt[2]);
    }
    return 3 * most <= kItemBatch;
}

void launch_correlation(spn_xyz *h) {
    const XyzArgs a = h->args();
    xyz_corr_inner_kernel<<<2 * h->n + 4, kCorrXThreads, 0, h->stream>>>(a);
    check_cuda(cudaGetLastError(), "correlation launch");
    xyz_corr_final_kernel<<<1, kCorrThreads, corr_final_smem(4 * h->nl), h->stream>>>(a);
    check_cuda(cudaGetLastError(), "correlation final launch");
}

}  // namespace

extern "C" int spn_xyz_create(const spn_xyz_desc *d, spn_xyz **out) {
    return guarded([&] {
        if (!out) throw Error(ErrorType::Argument, "null output handle");
        validate(d);
        auto *h = new spn_xyz;
        try {
            h->device = d->device;
            check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
            h->n = d->n_freq;
            h->nl = d->n_sites;
            h->fn = (long long)h->n * h->n * (h->n + 1) / 2;
            h->n_range = d->n_range;
            h->n_corr = d->n_corr;
            h->n_overlap = d->overlap_ptr[d->n_sites];
            h->max_nodes = 2 * h->n + 8;
            check_cuda(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking), "cudaStreamCreate");
            const size_t vsz = size_t(h->fn) * h->nl;
            h->freq = dalloc<float>(h->n, "alloc freq");
            h->v2 = dalloc<float>(h->n, "alloc v2");
            h->dv2 = dalloc<float>(h->n, "alloc dv2");
            h->sd = dalloc<float4>(vsz, "alloc vertex state");
            h->dsd = dalloc<float4>(vsz, "alloc vertex flow");
            h->node_wp = dalloc<float>(size_t(h->n) * h->max_nodes, "alloc node table");
            h->node_c = dalloc<float>(size_t(h->n) * h->max_nodes, "alloc node table");
            h->corr_out = dalloc<float>(4 * size_t(h->n_corr) + 4 * h->nl, "alloc correlation output");
            h->partial = dalloc<double>(size_t(kMaxCorrNodes) * 4 * h->nl, "alloc correlation scratch");
            // integer tables, one allocation
            const int nl = h->nl, nr = h->n_range, nc = h->n_corr;
            std::vector<int> img;
            std::vector<size_t> at;
            auto put = [&](const int *src, int cnt) {
                at.push_back(img.size());
                if (src) img.insert(img.end(), src, src + cnt);
                else img.insert(img.end(), size_t(cnt), 0);
            };
            put(d->sites_rid, nl);
            put(d->sites_perm, nl);
            put(d->inv_sites_rid, nl);
            put(d->inv_sites_perm, nl);
            const std::vector<int> packed = order_rpa_pairs(d);
            const int lanes = nl <= 32 ? kItemThreads : 32;
            const LaneSchedule rpa = nl <= 32 ? lane_schedule(nl, d->overlap_ptr, packed, kItemThreads, 20)
                                              : xyz_lane_schedule(nl, d->overlap_ptr, packed);
            h->rpa_n_seg = rpa.n_seg;
            put(d->range_rid, nr);
            put(d->range_inv_rid, nr);
            put(d->corr_rid, nc);
            put(d->corr_perm, nc);
            put(nullptr, h->n);  // node counts
            put(nullptr, 2);     // work counter, status
            put(rpa.sched.data(), int(rpa.sched.size()));
            put(rpa.count.data(), lanes);
            put(rpa.slot_base.data(), lanes);
            put(rpa.seg_ptr.data(), nl + 1);
            h->site_kind = xyz_site_kind(nl, d->sites_rid, d->sites_perm, d->inv_sites_rid, d->inv_sites_perm);
            h->ints = dalloc<int>(img.size(), "alloc lattice tables");
            h2d(h->ints, img.data(), img.size(), h->stream);
            int **fields[] = {&h->sites, &h->sites_perm, &h->inv_sites, &h->inv_sites_perm, &h->range_rid, &h->range_inv,
                              &h->corr_rid, &h->corr_perm, &h->node_cnt, &h->work_counter, &h->rpa_sched,
                              &h->rpa_count, &h->rpa_slot_base, &h->rpa_seg_ptr};
            for (size_t k = 0; k < at.size(); ++k) *fields[k] = h->ints + at[k];
            h->status = reinterpret_cast<unsigned *>(h->work_counter + 1);
            h2d(h->freq, d->freq, h->n, h->stream);
            check_cuda(cudaMemsetAsync(h->sd, 0, vsz * sizeof(float4), h->stream), "memset");
            check_cuda(cudaMemsetAsync(h->dsd, 0, vsz * sizeof(float4), h->stream), "memset");
            check_cuda(cudaMemsetAsync(h->v2, 0, h->n * sizeof(float), h->stream), "memset");
            check_cuda(cudaMemsetAsync(h->dv2, 0, h->n * sizeof(float), h->stream), "memset");
            check_cuda(cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, h->device), "device attribute");
            h->mesh.assign(d->freq, d->freq + h->n);
            for (const bool once : {true, false}) {
                if (once && h->nl > 16) continue;
                int per_sm = 0;
                const void *fn = vertex_kernel(h->nl, once);
                check_cuda(allow_shared(fn, vertex_smem(h, once)), "shared memory limit");
                check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, vertex_threads(h->nl), vertex_smem(h, once)), "occupancy");
                if (per_sm < 1) throw Error(ErrorType::Unsupported, "XYZ vertex-flow kernel does not fit on this device");
                h->grid = h->sms * per_sm;
            }
            check_cuda(cudaStreamSynchronize(h->stream), "create sync");
        } catch (...) {
            h->release();
            delete h;
            throw;
        }
        *out = h;
    });
}

extern "C" int spn_xyz_destroy(spn_xyz *h) {
    if (!h) return SPN_OK;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    h->release();
    delete h;
    return SPN_OK;
}

namespace {
float *stage_of(spn_xyz *h) {
    if (!h->stage) h->stage = dalloc<float>(4 * size_t(h->fn) * h->nl, "alloc state stage");
    return h->stage;
}
}  // namespace

extern "C" int spn_xyz_set_state(spn_xyz *h, float cutoff, const float *v2, const float *xx, const float *yy, const float *zz,
                                 const float *dd) {
    return guarded([&] {
        if (!h || !v2 || !xx || !yy || !zz || !dd) throw Error(ErrorType::Argument, "null argument");
        check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
        const size_t vsz = size_t(h->fn) * h->nl;
        float *st = stage_of(h);
        const float *src[4] = {xx, yy, zz, dd};
        for (int c = 0; c < 4; ++c) h2d(st + c * vsz, src[c], vsz, h->stream);
        xyz_pack_kernel<<<copy_grid((long long)vsz), 256, 0, h->stream>>>(st, h->sd, (long long)vsz);
        check_cuda(cudaGetLastError(), "pack launch");
        h2d(h->v2, v2, h->n, h->stream);
        h->cutoff = cutoff;
        check_cuda(cudaStreamSynchronize(h->stream), "set_state sync");
    });
}

namespace {
void copy_out(spn_xyz *h, const float4 *src, float *const dst[4]) {
    const size_t vsz = size_t(h->fn) * h->nl;
    float *st = stage_of(h);
    xyz_unpack_kernel<<<copy_grid((long long)vsz), 256, 0, h->stream>>>(src, st, (long long)vsz);
    check_cuda(cudaGetLastError(), "unpack launch");
    for (int c = 0; c < 4; ++c)
        if (dst[c])
            check_cuda(cudaMemcpyAsync(dst[c], st + c * vsz, vsz * sizeof(float), cudaMemcpyDeviceToHost, h->stream), "D2H");
}
}  // namespace

extern "C" int spn_xyz_get_state(spn_xyz *h, float *cutoff, float *v2, float *xx, float *yy, float *zz, float *dd) {
    return guarded([&] {
        if (!h) throw Error(ErrorType::Argument, "null handle");
        check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
        if (cutoff) *cutoff = h->cutoff;
        if (v2) check_cuda(cudaMemcpyAsync(v2, h->v2, h->n * sizeof(float), cudaMemcpyDeviceToHost, h->stream), "D2H");
        float *const dst[4] = {xx, yy, zz, dd};
        copy_out(h, h->sd, dst);
        check_cuda(cudaStreamSynchronize(h->stream), "get_state sync");
    });
}

extern "C" int spn_xyz_get_flow(spn_xyz *h, float *dv2, float *xx, float *yy, float *zz, float *dd) {
    return guarded([&] {
        if (!h) throw Error(ErrorType::Argument, "null handle");
        check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
        if (dv2) check_cuda(cudaMemcpyAsync(dv2, h->dv2, h->n * sizeof(float), cudaMemcpyDeviceToHost, h->stream), "D2H");
        float *const dst[4] = {xx, yy, zz, dd};
        copy_out(h, h->dsd, dst);
        check_cuda(cudaStreamSynchronize(h->stream), "get_flow sync");
    });
}

extern "C" int spn_xyz_compute_step(spn_xyz *h) {
    return guarded([&] {
        if (!h) throw Error(ErrorType::Argument, "null handle");
        check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
        check_cuda(cudaMemsetAsync(h->work_counter, 0, 2 * sizeof(int), h->stream), "memset counter and status");
        const XyzArgs a = h->args();
        xyz_self_energy_kernel<<<h->n, 128, 0, h->stream>>>(a);
        check_cuda(cudaGetLastError(), "self-energy launch");
        xyz_node_table_kernel<<<h->n, kNodeThreads, 0, h->stream>>>(h->node_args());
        check_cuda(cudaGetLastError(), "node table launch");
        const bool once = build_once(h);
        const void *fn = vertex_kernel(h->nl, once);
        XyzArgs arg = a;
        void *params[] = {&arg};
        check_cuda(cudaLaunchKernel(fn, dim3(h->grid), dim3(vertex_threads(h->nl)), params, vertex_smem(h, once), h->stream), "vertex flow launch");
        check_cuda(cudaGetLastError(), "vertex flow launch");
    });
}

extern "C" int spn_xyz_finalize_step(spn_xyz *h, float new_cutoff) {
    return guarded([&] {
        if (!h) throw Error(ErrorType::Argument, "null handle");
        check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
        const float step = new_cutoff - h->cutoff;
        const long long n4 = 4 * h->fn * h->nl;
        xyz_euler_kernel<<<1, 64, 0, h->stream>>>(h->v2, h->dv2, h->n, step);
        xyz_euler_kernel<<<copy_grid(n4), 256, 0, h->stream>>>(reinterpret_cast<float *>(h->sd),
                                                              reinterpret_cast<const float *>(h->dsd), n4, step);
        check_cuda(cudaGetLastError(), "euler launch");
        h->cutoff = new_cutoff;
    });
}

extern "C" int spn_xyz_measure_correlation(spn_xyz *h, float *xx, float *yy, float *zz, float *dd, float *chi) {
    return guarded([&] {
        if (!h) throw Error(ErrorType::Argument, "null handle");
        check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
        launch_correlation(h);
        const float *v = h->results.fetch(h->corr_out, 4 * size_t(h->n_corr) + 4 * h->nl, h->stream);
        float *const dst[4] = {xx, yy, zz, dd};
        for (int c = 0; c < 4; ++c)
            if (dst[c]) std::copy(v + size_t(c) * h->n_corr, v + size_t(c + 1) * h->n_corr, dst[c]);
        if (chi) std::copy(v + 4 * size_t(h->n_corr), v + 4 * size_t(h->n_corr) + 4 * h->nl, chi);
    });
}

extern "C" int spn_xyz_is_diverged(spn_xyz *h, int *diverged) {
    return guarded([&] {
        if (!h || !diverged) throw Error(ErrorType::Argument, "null argument");
        check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
        const unsigned st = *h->results.fetch(h->status, 1, h->stream);
        if (st & kStatusNodeOverflow) throw Error(ErrorType::Device, "loop-frequency node table overflow");
        *diverged = (st & kStatusNaN) ? 1 : 0;
    });
}

extern "C" int spn_xyz_vertex_probe(const float *pos, int n, int n_sites, const float *xx, const float *yy,
                                    const float *zz, const float *dd, int rid12, int rid21, int perm12, int perm21,
                                    float s, float t, float u, int channel, int local, float *value) {
    return guarded([&] {
        cuh::check_mesh(pos, n, kMaxFreq);
        if (n_sites < 1 || n_sites > 32 * kSpt || !xx || !yy || !zz || !dd || !value || rid12 < 0 ||
            rid12 >= n_sites || rid21 < 0 || rid21 >= n_sites || perm12 < 0 || perm12 > 5 || perm21 < 0 ||
            perm21 > 5 || channel < -1 || channel > 3 || (channel < 0 && (local || perm12 || perm21)))
            throw Error(ErrorType::Argument, "spn_xyz_vertex_probe: bad argument");
        // the device layout: one float4 (X, Y, Z, D) per element
        const size_t vsz = size_t(n) * n * (n + 1) / 2 * n_sites;
        std::vector<float4> sd(vsz);
        for (size_t i = 0; i < vsz; ++i) sd[i] = make_float4(xx[i], yy[i], zz[i], dd[i]);
        XyzArgs a{};
        a.n = n;
        a.nl = n_sites;
        a.sd = sd.data();
        float g[4];
        if (channel < 0) {
            for (int c = 0; c < 4; ++c) g[c] = value4(pos, a, c, rid12, rid21, s, t, u);
        } else if (channel == 3) {
            AB8 ab;
            access8(pos, n, n_sites, s, t, u, ab);
            if (local) bundle8(a, ab, 0, 0, g);
            else bundle8(a, ab, ab.exch ? rid21 : rid12, ab.exch ? perm21 : perm12, g);
        } else {
            // the channel's own frequency is a mesh value; the two others are interpolated in
            // the order access4i takes them (t, u for S; s, u for T; s, t for U)
            const MeshSearch<float> m{pos, n};
            const float own[3] = {s, t, u};
            const int e = cuh::mesh_index_of(pos, n, own[channel]);
            const Interp<float> ia = interp_abs(m, channel == 0 ? t : s), ib = interp_abs(m, channel == 2 ? t : u);
            AB4 ab;
            if (channel == 0) access4i<kS>(n, n_sites, s, t, u, ia, ib, e, ab);
            else if (channel == 1) access4i<kT>(n, n_sites, s, t, u, ia, ib, e, ab);
            else access4i<kU>(n, n_sites, s, t, u, ia, ib, e, ab);
            float4 v;
            if (local) {
                v = local4(a, ab);
            } else {
                LaneT<1> ln;
                ln.j[0] = 0;
                ln.valid[0] = true;
                ln.rid[0] = rid12;
                ln.prm[0] = perm12;
                ln.irid[0] = rid21;
                ln.iprm[0] = perm21;
                gather4(a, ab, ln, &v);
            }
            g[0] = v.x;
            g[1] = v.y;
            g[2] = v.z;
            g[3] = v.w;
        }
        for (int c = 0; c < 4; ++c) value[c] = g[c];
    });
}
