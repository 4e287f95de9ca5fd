// GB300 kernels of the TRI pf-FRG flow right-hand side (time-reversal-invariant spin models
// with general, also off-diagonal, couplings: Heisenberg-Kitaev-Gamma, ...) and the device
// half of the spn_tri_* C ABI in include/spn_su2.h.  Restates TRIFrgCore
// (src/TRI/TRIFrgCore.cpp:122-3001), the TRI vertex access (src/TRI/TRIVertexTwoParticle.hpp:
// 190-677) and TRIMeasurementCorrelation (src/TRI/TRIMeasurementCorrelation.cpp:147-285).
//
// The vertex keeps the reference's layout: 16 components (a, b) per element, a, b in X, Y, Z,
// density, as [(s(s+1)/2+u)*N + t][4a+b][site].  An access buffer carries, besides offsets and
// weights, the sign rules of TRIVertexTwoParticleAccessBuffer: a zeta(a) zeta(b) factor when
// exactly one of t, u was negated, and -zeta of the stored second component for a support
// whose s and u were exchanged.  A lattice symmetry map permutes X, Y, Z of both indices.
// The flow equations' coefficients come from tri_algebra.hpp (Pauli products) and fold to
// constants in the unrolled loops.
//
// A step: the self-energy flow (one CTA per frequency), the loop-frequency node tables (the
// SU(2) core's, shared), the vertex flow and the Euler update.  The vertex-flow kernels run persistent
// grids that take (s,t,u) triples from a device counter: a CTA per triple (tri_site_kernel and, for the t channel,
// tri_lattice_kernel) for at most 32 sites, a warp per triple above (tri_vertex_kernel).
#include <cuda_runtime.h>
#include <algorithm>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>
#include "su2_common.cuh"
#include "su2_device.cuh"
#include "su2_item.cuh"
#include "su2_kernels.cuh"
#include "umma.cuh"
#include "tri_algebra.hpp"
#include "cuda_host.cuh"
#include "host/capi_common.hpp"
#include "host/pair_order.hpp"
#include "../../include/spn_su2.h"

using namespace spn;
using namespace spn::dev;

namespace {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxSites = 128;
constexpr int kTBatch = 4;  // nodes whose descriptors a warp builds at once (a quad of lanes each): above 32 sites
constexpr int kSiteBatch = 8;  // at most 32 sites
constexpr int kCorrOut = 10;  // XX XY XZ YX YY YZ ZX ZY ZZ DD

// The six spin permutations (X,Y,Z) (X,Z,Y) (Y,X,Z) (Y,Z,X) (Z,X,Y) (Z,Y,X): 2 bits per image
// component, 6 bits per permutation; the density maps to itself.
constexpr unsigned long long kPermBits =
    36ull | (24ull << 6) | (33ull << 12) | (9ull << 18) | (18ull << 24) | (6ull << 30);
__host__ __device__ __forceinline__ int permc(int p, int c) {
    return c == 3 ? 3 : int((kPermBits >> (6 * p + 2 * c)) & 3ull);
}
SPN_HDI float zeta(int c) { return c <= 2 ? -1.0f : 1.0f; }

struct TriArgs {
    int n, nl, fn, max_nodes, n_range, n_corr;
    float cutoff;
    const float *freq;
    const float *v4;  // state [F_N][16][nl]
    float *dv4;       // flow
    const float *v2;
    float *dv2;
    const int *sites, *sites_perm, *inv_sites, *inv_sites_perm;
    // the t channel's RPA pairs of all sites in one lane-balanced walk (lane_schedule): entry i of
    // lane l is sched[32 i + l], the pair's word rid1 | rid2 << 7 | the images of X, Y, Z under
    // perm1 (2 bits each) << 14 | the same for perm2 << 20 (order_rpa_pairs), bit 26 set on the
    // last entry of a site's run in the lane; the runs' partial sums (16 components) go to slots
    // slot_base[l], ... and site j sums slots seg_ptr[j] .. seg_ptr[j + 1] - 1
    const int *rpa_sched, *rpa_count, *rpa_slot_base, *rpa_seg_ptr;
    int rpa_n_seg;
    // instead of them, the pairs for the lattice sum on the tensor cores (tri_lattice_kernel): site j's are dealt to groups
    // prod_group[j] .. prod_group[j + 1] - 1; the words of the inner components (k2, k1) and group g at
    // prod_words[2 prod_ptr[(4 k2 + k1) kLatGroups + g]] ..; the CTAs' operand scratch
    const int *prod_ptr, *prod_words, *prod_group;
    unsigned char *prod_scratch;
    const int *range_rid, *range_inv;
    const float *node_wp, *node_c;
    const int *node_cnt;
    int *work_counter;  // two: the vertex-flow kernel's and tri_lattice_kernel's
    unsigned *status;
    const int *corr_rid, *corr_perm;
    double *partial;  // [kMaxCorrNodes][16][nl]
    float *out;       // [10][n_corr] correlations, then chi [16][nl]
};

// ---- access buffers (TRIVertexTwoParticleAccessBuffer) ----
constexpr int kFlExch = 1 << 8;  // read the site-exchanged pair
constexpr int kFlTu = 1 << 9;    // zeta(a) zeta(b): exactly one of t, u negated
// bits 0..7: support i's s and u offsets were exchanged

template <int K>
struct TABT {
    int off[K];
    float w[K];
    int fl;
};
using TAB4 = TABT<4>;
using TAB8 = TABT<8>;

// sign[i][a][b] of the access buffer (TRIVertexTwoParticle.hpp:401-448, 643-671)
SPN_HDI float tab_sign(int fl, int i, int a, int b) {
    float s = 1.0f;
    if (fl & kFlTu) s *= zeta(a) * zeta(b);
    if ((fl >> i) & 1) s *= -((fl & kFlExch) ? zeta(a) : zeta(b));
    return s;
}

SPN_HDI int tri_fold(float &s, float &t, float &u) {
    int fl = 0;
    if (s < 0) {
        s = -s;
        fl ^= kFlExch;
    }
    if (t < 0) {
        t = -t;
        fl ^= kFlTu;
    }
    if (u < 0) {
        u = -u;
        fl ^= kFlExch | kFlTu;
    }
    return fl;
}

SPN_HDI void tri_slab(int si, int ti, int ui, int step_su, int step_t, int i, int &off, int &fl) {
    if (si < ui) {
        off = (ui * (ui + 1) / 2 + si) * step_su + ti * step_t;
        fl |= 1 << i;
    } else {
        off = (si * (si + 1) / 2 + ui) * step_su + ti * step_t;
    }
}

// generateAccessBuffer(s, t, u, channel) (TRIVertexTwoParticle.hpp:401-505) with e the exact mesh
// index of the channel's own coordinate, which every caller knows, and the two interpolations
// given (interp_abs of the interpolated coordinates, as for access4i): a node's buffers
// interpolate four distinct magnitudes, each looked up once.
template <int CH>
SPN_HDI void tri_access4i(int n, int nl, float s, float t, float u, int e, const Interp<float> &ia,
                          const Interp<float> &ib, TAB4 &ab) {
    int fl = tri_fold(s, t, u);
    const int step_t = 16 * nl, step_su = n * step_t;
    const int la = ia.lo, ua = ia.hi, lb = ib.lo, ub = ib.hi;
    const float ba = ia.b, bb = ib.b;
    const float na = rn_sub(1.0f, ba), nb = rn_sub(1.0f, bb);
    ab.w[0] = rn_mul(nb, na);
    ab.w[1] = rn_mul(nb, ba);
    ab.w[2] = rn_mul(bb, na);
    ab.w[3] = rn_mul(bb, ba);
    if (CH == kS) {
        tri_slab(e, la, lb, step_su, step_t, 0, ab.off[0], fl);
        tri_slab(e, ua, lb, step_su, step_t, 1, ab.off[1], fl);
        tri_slab(e, la, ub, step_su, step_t, 2, ab.off[2], fl);
        tri_slab(e, ua, ub, step_su, step_t, 3, ab.off[3], fl);
    } else if (CH == kT) {
        tri_slab(la, e, lb, step_su, step_t, 0, ab.off[0], fl);
        tri_slab(ua, e, lb, step_su, step_t, 1, ab.off[1], fl);
        tri_slab(la, e, ub, step_su, step_t, 2, ab.off[2], fl);
        tri_slab(ua, e, ub, step_su, step_t, 3, ab.off[3], fl);
    } else {
        tri_slab(la, lb, e, step_su, step_t, 0, ab.off[0], fl);
        tri_slab(ua, lb, e, step_su, step_t, 1, ab.off[1], fl);
        tri_slab(la, ub, e, step_su, step_t, 2, ab.off[2], fl);
        tri_slab(ua, ub, e, step_su, step_t, 3, ab.off[3], fl);
    }
    ab.fl = fl;
}

// generateAccessBuffer(s, t, u): trilinear (TRIVertexTwoParticle.hpp:514-584)
SPN_HDI void tri_access8(const float *pos, int n, int nl, float s, float t, float u, TAB8 &ab) {
    int fl = tri_fold(s, t, u);
    const int step_t = 16 * nl, step_su = n * step_t;
    int ls, us, lt, ut, lu, uu;
    float bs, bt, bu;
    mesh_interp(pos, n, s, ls, us, bs);
    mesh_interp(pos, n, t, lt, ut, bt);
    mesh_interp(pos, n, u, lu, uu, bu);
    const float ns = rn_sub(1.0f, bs), nt = rn_sub(1.0f, bt), nu = rn_sub(1.0f, bu);
    ab.w[0] = rn_mul(rn_mul(nt, ns), nu);
    ab.w[1] = rn_mul(rn_mul(nt, bs), nu);
    ab.w[2] = rn_mul(rn_mul(bt, ns), nu);
    ab.w[3] = rn_mul(rn_mul(bt, bs), nu);
    ab.w[4] = rn_mul(rn_mul(nt, ns), bu);
    ab.w[5] = rn_mul(rn_mul(nt, bs), bu);
    ab.w[6] = rn_mul(rn_mul(bt, ns), bu);
    ab.w[7] = rn_mul(rn_mul(bt, bs), bu);
    tri_slab(ls, lt, lu, step_su, step_t, 0, ab.off[0], fl);
    tri_slab(us, lt, lu, step_su, step_t, 1, ab.off[1], fl);
    tri_slab(ls, ut, lu, step_su, step_t, 2, ab.off[2], fl);
    tri_slab(us, ut, lu, step_su, step_t, 3, ab.off[3], fl);
    tri_slab(ls, lt, uu, step_su, step_t, 4, ab.off[4], fl);
    tri_slab(us, lt, uu, step_su, step_t, 5, ab.off[5], fl);
    tri_slab(ls, ut, uu, step_su, step_t, 6, ab.off[6], fl);
    tri_slab(us, ut, uu, step_su, step_t, 7, ab.off[7], fl);
    ab.fl = fl;
}

// getValueLocal(a, b, ab) (TRIVertexTwoParticle.hpp:347-356): the components are exchanged
// first and index the sign table in that order.  getValue and getValueSuperbundle (tri_bundle)
// index it with the original order, so for a site-exchanging buffer the two differ in the sign
// of the mixed spin/density components on supports whose stored sector swaps s and u; this is
// the reference's convention, kept.
template <int K>
SPN_HDI float tri_local(const float *v4, int nl, const TABT<K> &ab, int ca, int cb) {
    if (ab.fl & kFlExch) {
        const int x = ca;
        ca = cb;
        cb = x;
    }
    const int o = (4 * ca + cb) * nl;
    float v = 0.0f;
#pragma unroll
    for (int i = 0; i < K; ++i) v += tab_sign(ab.fl, i, ca, cb) * ab.w[i] * ro_load(v4 + ab.off[i] + o);
    return v;
}

// getValueSuperbundle component c of site j (TRIVertexTwoParticle.hpp:364-391): the
// (exchanged, then permuted) component of the site's representative.
template <int K>
SPN_HDI float tri_bundle(const float *v4, int nl, const TABT<K> &ab, int c, int r, int p) {
    const int ca = c >> 2, cb = c & 3;
    const bool ex = ab.fl & kFlExch;
    const int o = (4 * permc(p, ex ? cb : ca) + permc(p, ex ? ca : cb)) * nl + r;
    float v = 0.0f;
#pragma unroll
    for (int i = 0; i < K; ++i) v += tab_sign(ab.fl, i, ca, cb) * ab.w[i] * ro_load(v4 + ab.off[i] + o);
    return v;
}

// getValue(i1, i2, s, t, u, a, b, FrequencyChannel::None) (TRIVertexTwoParticle.hpp:190-312)
// for the pairs the self-energy reads: through rid12 / rid21 with identity spin maps, on the
// state v4 of n frequencies and nl sites.
__host__ __device__ float tri_value_none(const float *pos, int n, int nl, const float *v4, int ca, int cb, int rid12,
                                         int rid21, float s, float t, float u) {
    float sign = 1.0f;
    bool sw = false;
    if (s < 0) {
        s = -s;
        const int x = ca; ca = cb; cb = x;
        sw = !sw;
    }
    if (t < 0) {
        t = -t;
        sign *= zeta(ca) * zeta(cb);
    }
    if (u < 0) {
        u = -u;
        const int x = ca; ca = cb; cb = x;
        sw = !sw;
        sign *= zeta(ca) * zeta(cb);
    }
    const int site = sw ? rid21 : rid12;
    const int step_t = 16 * nl, step_su = n * step_t, co = (4 * ca + cb) * nl + site;
    const float zb = -zeta(cb);
    int ls, us, lt, ut, lu, uu;
    float bs, bt, bu;
    mesh_interp(pos, n, s, ls, us, bs);
    mesh_interp(pos, n, t, lt, ut, bt);
    mesh_interp(pos, n, u, lu, uu, bu);
    auto Dv = [&](int x, int y, int z) {
        if (x >= z) return ro_load(v4 + (x * (x + 1) / 2 + z) * step_su + y * step_t + co);
        return zb * ro_load(v4 + (z * (z + 1) / 2 + x) * step_su + y * step_t + co);
    };
    return sign * ((1 - bu) * ((1 - bt) * ((1 - bs) * Dv(ls, lt, lu) + bs * Dv(us, lt, lu)) +
                               bt * ((1 - bs) * Dv(ls, ut, lu) + bs * Dv(us, ut, lu))) +
                   bu * ((1 - bt) * ((1 - bs) * Dv(ls, lt, uu) + bs * Dv(us, lt, uu)) +
                         bt * ((1 - bs) * Dv(ls, ut, uu) + bs * Dv(us, ut, uu))));
}

// ------------------------------------------------------------------------------------
// self-energy flow, one CTA per frequency (TRIFrgCore.cpp:122-151)
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) tri_self_energy_kernel(TriArgs a) {
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
        part += double(tri_value_none(pos, a.n, a.nl, a.v4, 3, 3, r12, r21, wpl, 0.0f, wml)) -
                double(tri_value_none(pos, a.n, a.nl, a.v4, 3, 3, r12, r21, wml, 0.0f, wpl));
    }
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int k = 0; k < int(blockDim.x >> 5); ++k) sum += red[k];
        double val = -2.0 * sum;
        for (int c = 0; c < 4; ++c)
            val += double(tri_value_none(pos, a.n, a.nl, a.v4, c, c, 0, 0, wpl, wml, 0.0f)) -
                   double(tri_value_none(pos, a.n, a.nl, a.v4, c, c, 0, 0, wml, wpl, 0.0f));
        val /= (2.0 * kPiD * (double(L) + odd_interp(pos, a.n, a.v2, L)));
        const float outv = float(val);
        a.dv2[i] = outv;
        if (isnan(outv)) atomicOr(a.status, kStatusNaN);
    }
}

// Loop-frequency node tables: the SU(2) core's body on an argument block of this flow.
__global__ void __launch_bounds__(kNodeThreads) tri_node_table_kernel(FlowArgs f) { node_table_body(f, blockIdx.x); }

// ------------------------------------------------------------------------------------
// vertex flow
// ------------------------------------------------------------------------------------
// Node descriptor (built by a quad of lanes, make_tpart): the four access buffers of the channel's
// integrand and, for the t channel, the four of the chalice diagrams' site-local values.
struct __align__(16) TDesc {
    TAB4 ab[8];
    float c;  // node coefficient
    int pad[3];
};

// Phase A: the descriptor of one node of channel ch (0 = s, 1 = t, 2 = u), built by the four
// lanes of a quad (q = 0..3): integralKernelS (TRIFrgCore.cpp:184-188), integralKernelT
// (TRIFrgCore.cpp:718-724, 1257-1259, 1814-1816) and integralKernelU (TRIFrgCore.cpp:2375-2379)
// read four access buffers each (the t channel four more for its chalice diagrams' site-local
// values), and every buffer interpolates two of the node's four distinct magnitudes A = |w1 + wp|,
// B = |w2 + wp|, C = |w1 - wp|, D = |w2p - wp|, E = |w2 - wp|, P = |w1p + wp|, Q = |w2p + wp|
// (a coordinate and its negation fold alike; -a - b is bitwise -(a + b), -a + b is b - a).  Lane
// q builds the buffers of one pair of magnitudes, with the coordinates from selects, so the quad
// runs one instruction stream: slot q ^ 2 (s channel), slot q (u channel), slots (q & 1) << 1 |
// q >> 1 and 4 + (q ^ 2) (t channel).
__device__ __forceinline__ void make_tpart(const TriArgs &a, const float *pos, int ch, int e, float s, float t, float u,
                                           float w1p, float w1, float w2p, float w2, float wp, int q, TDesc &d) {
    const MeshSearch<float> m{pos, a.n};
    const int nl = a.nl, n = a.n;
    const bool lo2 = q < 2, odd = q & 1;
    if (ch == 0) {
        // slots (t, u): 2 (-A, -B), 3 (P, -Q), 0 (B, A), 1 (-Q, P); (y1, y2) = (A, B) or (P, Q)
        const float y1 = odd ? w1p + wp : w1 + wp, y2 = odd ? w2p + wp : w2 + wp;
        const Interp<float> i1 = interp_abs(m, y1), i2 = interp_abs(m, y2);
        tri_access4i<kS>(n, nl, s, lo2 ? (odd ? y1 : -y1) : (odd ? -y2 : y2), lo2 ? -y2 : y1, e, lo2 ? i1 : i2,
                         lo2 ? i2 : i1, d.ab[q ^ 2]);
    } else if (ch == 2) {
        // slots (s, t): 0 (A, -D), 1 (P, E), 2 (D, -A), 3 (E, P); (y1, y2) = (A, D) or (P, E)
        const float y1 = odd ? w1p + wp : w1 + wp, y2 = odd ? w2 - wp : w2p - wp;
        const Interp<float> i1 = interp_abs(m, y1), i2 = interp_abs(m, y2);
        tri_access4i<kU>(n, nl, lo2 ? y1 : y2, lo2 ? (odd ? y2 : -y2) : (odd ? y1 : -y1), u, e, lo2 ? i1 : i2,
                         lo2 ? i2 : i1, d.ab[q]);
    } else {
        // main slots (s, u): 0 (C, P), 2 (P, C), 1 (D, -B), 3 (B, -D); chalice slots (s, t, u):
        // 6 (C, -P, -t), 7 (P, -C, -t), 4 (D, -B, t), 5 (B, -D, t); (y1, y2) = (C, P), (P, C),
        // (D, B), (B, D) for q = 0..3
        const float x1 = lo2 ? w1 - wp : w2p - wp, x2 = lo2 ? w1p + wp : w2 + wp;
        const float y1 = odd ? x2 : x1, y2 = odd ? x1 : x2;
        const Interp<float> i1 = interp_abs(m, y1), i2 = interp_abs(m, y2);
        tri_access4i<kT>(n, nl, y1, t, lo2 ? y2 : -y2, e, i1, i2, d.ab[(int(odd) << 1) | (q >> 1)]);
        tri_access4i<kU>(n, nl, y1, -y2, lo2 ? -t : t, e, i1, i2, d.ab[4 + (q ^ 2)]);
    }
}

// Entry goff[e][c][j] of gather_slab's offsets: component c = 4a + b of the site whose
// representative is r under spin permutation p; e = 1 for the site-exchanged pair (components
// swapped, then permuted).
SPN_HDI int gather_offset(int e, int c, int nl, int r, int p) {
    const int ca = c >> 2, cb = c & 3;
    return (4 * permc(p, e ? cb : ca) + permc(p, e ? ca : cb)) * nl + r;
}

// One slab of a node for all sites (getValueSuperbundle): goff[e][c][j] is the offset of
// component c of site j (gather_offset of the site's representative and permutation).  The sign of support i depends on the component only through
// zeta(a) and zeta(b), so the four signed weights of each zeta class are formed once.
SPN_HDI void gather_slab(const float *__restrict__ v4, const TAB4 &ab, const int *goff, int nl, int lane, float *S) {
    const int fl = ab.fl;
    const bool ex = fl & kFlExch, tu = fl & kFlTu;
    float sw[4][4];  // [class: bit 0 a is a spin component, bit 1 b is][support]
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float za = (k & 1) ? -1.0f : 1.0f, zb = (k & 2) ? -1.0f : 1.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float sg = tu ? za * zb : 1.0f;
            if ((fl >> i) & 1) sg *= -(ex ? za : zb);
            sw[k][i] = sg * ab.w[i];
        }
    }
    const int *g = goff + (ex ? 16 * nl : 0);
    for (int j = lane; j < nl; j += 32) {
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            const int k = ((c >> 2) < 3 ? 1 : 0) | ((c & 3) < 3 ? 2 : 0);
            const int o = g[c * nl + j];
            float v = 0.0f;
#pragma unroll
            for (int i = 0; i < 4; ++i) v += sw[k][i] * ro_load(v4 + ab.off[i] + o);
            S[c * nl + j] = v;
        }
    }
}

// The two ladders for one site: per output c, a = 15..0 with the slab pairs (0,1) and (2,3)
// (TRIFrgCore.cpp:198-711 particle-particle, 2389-2902 particle-hole).
template <bool PH>
__device__ __forceinline__ void ladder(const float *S, int nl, int j, float *r) {
    float A0[16], A1[16], A2[16], A3[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        A0[c] = S[c * nl + j];
        A1[c] = S[(16 + c) * nl + j];
        A2[c] = S[(32 + c) * nl + j];
        A3[c] = S[(48 + c) * nl + j];
    }
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        float v = 0.0f;
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            const int x = 15 - n, y = x ^ c ^ 15;
            if ((PH ? tri::ph_sign(c, x) : tri::pp_sign(c, x)) > 0) {
                v += A0[x] * A1[y];
                v += A2[x] * A3[y];
            } else {
                v -= A0[x] * A1[y];
                v -= A2[x] * A3[y];
            }
        }
        r[c] = v;
    }
}

// One overlap pair (packed word e) of the t integrand's RPA lattice sum (TRIFrgCore.cpp:733-2368)
// added to v[16]: 4x4 products over the inner spin index, the factors' components permuted by the
// pair's maps.  The RPA reads component (P a, P b) of a factor at (4 P(a) + P(b)) nl + rid: a row
// base per a plus a column offset per b, from the permutation images packed into the pair word.
// The products are summed without the factor 2 of the reference's terms; t_terms doubles the sum
// (scaling by 2 commutes with every rounding).
__device__ __forceinline__ void rpa_pair(const float *S, int nl, int e, float *v) {
    const float *S0 = S, *S1 = S + 16 * nl, *S2 = S + 32 * nl, *S3 = S + 48 * nl;
    {
        const int r1 = e & 127, r2 = (e >> 7) & 127;
        int col1[4], col2[4];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            col1[q] = ((e >> (14 + 2 * q)) & 3) * nl;
            col2[q] = ((e >> (20 + 2 * q)) & 3) * nl;
        }
        col1[3] = col2[3] = 3 * nl;
        float x0[16], x2[16], y1[16], y3[16];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int ra = 4 * col1[q] + r1, rb = 4 * col2[q] + r2;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                x0[4 * q + u] = S0[ra + col1[u]];
                x2[4 * q + u] = S2[ra + col1[u]];
                y1[4 * q + u] = S1[rb + col2[u]];
                y3[4 * q + u] = S3[rb + col2[u]];
            }
        }
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            const int mu = c >> 2, nu = c & 3;
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const int k = tri::inner(n);
                if (tri::rpa_sign(c, k) > 0) {
                    v[c] += x0[4 * mu + k] * y1[4 * k + nu];
                    v[c] += x2[4 * mu + k] * y3[4 * k + nu];
                } else {
                    v[c] -= x0[4 * mu + k] * y1[4 * k + nu];
                    v[c] -= x2[4 * mu + k] * y3[4 * k + nu];
                }
            }
        }
    }
}

// The lane-balanced walk of the RPA pairs of all sites (TriArgs::rpa_*) for the t-channel node
// whose slabs are in S: each lane sums its chunk's runs into slots (16 floats per run).
__device__ __forceinline__ void rpa_walk(const TriArgs &a, const float *S, int nl, int lane, int cnt, int base,
                                         float *slots) {
    float p[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) p[c] = 0.0f;
    int slot = base;
    for (int i = 0; i < cnt; ++i) {
        const int e = __ldg(a.rpa_sched + 32 * i + lane);
        rpa_pair(S, nl, e, p);
        if (e & (1 << 26)) {
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                slots[16 * slot + c] = p[c];
                p[c] = 0.0f;
            }
            ++slot;
        }
    }
}

// The t integrand for one site j (TRIFrgCore.cpp:733-2368): the RPA lattice sum (the site's run
// partials of rpa_walk, in order, doubled), then the chalice diagrams with the site-local values L.
__device__ __forceinline__ void t_terms(const TriArgs &a, const float *S, const float *L, const float *slots, int nl,
                                        int j, float *r) {
    const float *S0 = S, *S1 = S + 16 * nl, *S2 = S + 32 * nl, *S3 = S + 48 * nl;
    float v[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) v[c] = 0.0f;
    for (int q = a.rpa_seg_ptr[j]; q < a.rpa_seg_ptr[j + 1]; ++q)  // the site's run partials, in order
#pragma unroll
        for (int c = 0; c < 16; ++c) v[c] += slots[16 * q + c];
#pragma unroll
    for (int c = 0; c < 16; ++c) v[c] *= 2.0f;
    {  // chalice: slabs 0 and 2 with the local values of ab4, ab5.  For an inner pair (kappa,
       // lambda) the outputs (c1, c2) read the row L(lambda, .) at rho = c2 ^ kappa ^ lambda, so
       // the row is loaded once; every output still adds its terms in (kappa, lambda) order.
        float X0[16], X2[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            X0[c] = S0[c * nl + j];
            X2[c] = S2[c * nl + j];
        }
        const float4 *L4 = reinterpret_cast<const float4 *>(L), *L5 = reinterpret_cast<const float4 *>(L + 16);
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            const int kap = tri::inner(n >> 2), lam = tri::inner(n & 3);
            const float4 q4 = L4[lam], q5 = L5[lam];
            const float r4[4] = {q4.x, q4.y, q4.z, q4.w}, r5[4] = {q5.x, q5.y, q5.z, q5.w};
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                const int ai = 4 * (c >> 2) + kap, rho = (c & 3) ^ kap ^ lam;
                if (tri::chal_sign(c, kap, lam) > 0) {
                    v[c] += X0[ai] * r4[rho];
                    v[c] += X2[ai] * r5[rho];
                } else {
                    v[c] -= X0[ai] * r4[rho];
                    v[c] -= X2[ai] * r5[rho];
                }
            }
        }
    }
    {  // inverse chalice: the local values of ab6, ab7 with slabs 1 and 3, each value loaded
       // once; every output adds its terms in the order l = 15 .. 0
        float X1[16], X3[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            X1[c] = S1[c * nl + j];
            X3[c] = S3[c * nl + j];
        }
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            const int l = 15 - n;
            const float l6 = L[32 + l], l7 = L[48 + l];
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                const int bi = 4 * ((c >> 2) ^ (l >> 2) ^ (l & 3)) + (c & 3);
                if (tri::ichal_sign(c, l) > 0) {
                    v[c] += l6 * X1[bi];
                    v[c] += l7 * X3[bi];
                } else {
                    v[c] -= l6 * X1[bi];
                    v[c] -= l7 * X3[bi];
                }
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 16; ++c) r[c] = v[c];
}

__host__ __device__ constexpr size_t tri_warp_floats(int nl, int n_seg) {
    return 80 * size_t(nl) + 64 + kTBatch * (sizeof(TDesc) / sizeof(float)) + 16 * size_t(n_seg);
}
// per CTA: the gather offsets goff[2][16][nl] (ints), then the warps' areas
__host__ __device__ constexpr size_t tri_cta_head_floats(int nl) { return (32 * size_t(nl) + 3) / 4 * 4; }

// Above 32 sites.  Per channel, nodes go in batches of four: a quad of lanes builds one node's access buffers into a
// shared-memory descriptor; then, node by node, the warp gathers the four 16-component slabs of all sites into shared
// memory (t: and the 64 site-local values of the chalice diagrams), and each lane evaluates the products for its sites from
// registers.
__global__ void __launch_bounds__(kThreads) tri_vertex_kernel(TriArgs a) {
    __shared__ float pos[kMaxFreq];
    // per CTA: gather offsets goff[2][16][nl]; per warp: slabs S[4][16][nl], accumulator
    // acc[16][nl], local values L[64], node descriptors
    extern __shared__ __align__(16) float tsm[];
    const int n = a.n, nl = a.nl;
    int *goff = reinterpret_cast<int *>(tsm);
    for (int i = threadIdx.x; i < n; i += blockDim.x) pos[i] = a.freq[i];
    for (int i = threadIdx.x; i < 32 * nl; i += blockDim.x) {
        const int e = i / (16 * nl), c = (i / nl) & 15, j = i % nl;
        const int r = e ? a.inv_sites[j] : a.sites[j], p = e ? a.inv_sites_perm[j] : a.sites_perm[j];
        goff[i] = gather_offset(e, c, nl, r, p);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *S = tsm + tri_cta_head_floats(nl) + size_t(warp) * tri_warp_floats(nl, a.rpa_n_seg);
    float *acc = S + 64 * nl;
    float *L = acc + 16 * nl;
    TDesc *desc = reinterpret_cast<TDesc *>(L + 64);
    float *slots = reinterpret_cast<float *>(desc + kTBatch);
    const int rpa_cnt = a.rpa_count[lane], rpa_base = a.rpa_slot_base[lane];
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
        for (int q = lane; q < 16 * nl; q += 32) acc[q] = 0.0f;
        __syncwarp();
        for (int ch = 0; ch < 3; ++ch) {
            const int xi = ch == 0 ? si : (ch == 1 ? ti : ui);
            const int cnt = a.node_cnt[xi];
            const float *nwp = a.node_wp + size_t(xi) * a.max_nodes;
            const float *nc = a.node_c + size_t(xi) * a.max_nodes;
            for (int b0 = 0; b0 < cnt; b0 += kTBatch) {
                const int nb = min(kTBatch, cnt - b0);
                if ((lane >> 2) < nb) {  // phase A: a quad of lanes per node
                    const int k = lane >> 2;
                    make_tpart(a, pos, ch, xi, s, t, u, w1p, w1, w2p, w2, nwp[b0 + k], lane & 3, desc[k]);
                    if ((lane & 3) == 0) desc[k].c = nc[b0 + k];
                }
                __syncwarp();
                for (int b = 0; b < nb; ++b) {
                    const TDesc &d = desc[b];
                    // gather the four slabs of all sites
#pragma unroll 1
                    for (int q = 0; q < 4; ++q) gather_slab(a.v4, d.ab[q], goff, nl, lane, S + q * 16 * nl);
                    if (ch == 1)
                        for (int q = lane; q < 64; q += 32) L[q] = tri_local(a.v4, nl, d.ab[4 + (q >> 4)], (q & 15) >> 2, q & 3);
                    __syncwarp();
                    if (ch == 1) {
                        rpa_walk(a, S, nl, lane, rpa_cnt, rpa_base, slots);
                        __syncwarp();
                    }
                    const float cw = d.c;
                    for (int j = lane; j < nl; j += 32) {
                        float r[16];
                        if (ch == 0) ladder<false>(S, nl, j, r);
                        else if (ch == 2) ladder<true>(S, nl, j, r);
                        else t_terms(a, S, L, slots, nl, j, r);
#pragma unroll
                        for (int c = 0; c < 16; ++c) acc[c * nl + j] += cw * r[c];
                    }
                    __syncwarp();
                }
            }
        }
        float *dst = a.dv4 + size_t(it) * 16 * nl;
        bool bad = false;
        for (int q = lane; q < 16 * nl; q += 32) {
            const float o = acc[q] / two_pi;
            dst[q] = o;
            bad |= isnan(o);
        }
        if (bad) atomicOr(a.status, kStatusNaN);
        __syncwarp();
    }
}

// ------------------------------------------------------------------------------------
// Lattices of at most 32 sites: a CTA per triple, whose warps take the nodes of all channels; lane = site
// (8 or 16 lanes a node where they hold the sites, so a warp takes several nodes at once).
//
// A lane gathers its own site's components straight into registers and keeps its sums there.  Above 32 sites the
// slabs go through shared memory with a warp per triple (tri_vertex_kernel): 64 stores and loads a node and site, and on a
// small mesh a warp's nodes one after the other.  The ladders of 28 sites, N = 32 take 3.35 ms here, about 8 there; all of
// 8 sites, N = 15 0.47 ms, 1.3 there.
// ------------------------------------------------------------------------------------
constexpr int kGoffRow = 20;  // gather offsets of a site: 16, rows 16 bytes aligned and in distinct banks
constexpr int kCoefRow = 260;  // chalice coefficients of a node: 256

__host__ __device__ inline int site_lanes(int nl) { return nl <= 8 ? 8 : (nl <= 16 ? 16 : 32); }

// The 16 components of a slab at site j (gather_slab for one site).
__device__ __forceinline__ void gather_site(const float *__restrict__ v4, const TAB4 &ab, const int *goff, int nl, int j, float (&x)[16]) {
    const int fl = ab.fl;
    const bool ex = fl & kFlExch, tu = fl & kFlTu;
    float sw[4][4];  // [class: bit 0 a is a spin component, bit 1 b is][support]
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float za = (k & 1) ? -1.0f : 1.0f, zb = (k & 2) ? -1.0f : 1.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float sg = tu ? za * zb : 1.0f;
            if ((fl >> i) & 1) sg *= -(ex ? za : zb);
            sw[k][i] = sg * ab.w[i];
        }
    }
    const int4 *g = reinterpret_cast<const int4 *>(goff + ((ex ? nl : 0) + j) * kGoffRow);
    const float *p[4] = {v4 + ab.off[0], v4 + ab.off[1], v4 + ab.off[2], v4 + ab.off[3]};
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int4 o4 = g[a];
        const int o[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int k = (a < 3 ? 1 : 0) | (b < 3 ? 2 : 0);
            float v = 0.0f;
#pragma unroll
            for (int i = 0; i < 4; ++i) v += sw[k][i] * ro_load(p[i] + o[b]);
            x[4 * a + b] = v;
        }
    }
}

// Slabs q and q + 2 of a t-channel node at site j.  Their coordinates are the same two magnitudes with s and u
// exchanged, and a slab is stored for s >= u alone, so both interpolate the same four stored slabs (supports 1
// and 2 trade places); their site exchanges differ only where a loop frequency cancels to zero.
__device__ __forceinline__ void gather_site_pair(const float *__restrict__ v4, const TAB4 &ab, const TAB4 &cd, const int *goff, int nl, int j,
                                                 float (&x)[16], float (&y)[16]) {
    if ((ab.fl ^ cd.fl) & kFlExch) {
        gather_site(v4, ab, goff, nl, j, x);
        gather_site(v4, cd, goff, nl, j, y);
        return;
    }
    const bool ex = ab.fl & kFlExch;
    float sx[4][4], sy[4][4];  // as gather_site's
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float za = (k & 1) ? -1.0f : 1.0f, zb = (k & 2) ? -1.0f : 1.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float sg = (ab.fl & kFlTu) ? za * zb : 1.0f, sh = (cd.fl & kFlTu) ? za * zb : 1.0f;
            if ((ab.fl >> i) & 1) sg *= -(ex ? za : zb);
            if ((cd.fl >> i) & 1) sh *= -(ex ? za : zb);
            sx[k][i] = sg * ab.w[i];
            sy[k][i] = sh * cd.w[i];
        }
    }
    const int4 *g = reinterpret_cast<const int4 *>(goff + ((ex ? nl : 0) + j) * kGoffRow);
    const float *p[4] = {v4 + ab.off[0], v4 + ab.off[1], v4 + ab.off[2], v4 + ab.off[3]};
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int4 o4 = g[a];
        const int o[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int k = (a < 3 ? 1 : 0) | (b < 3 ? 2 : 0);
            float r[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) r[i] = ro_load(p[i] + o[b]);
            x[4 * a + b] = sx[k][0] * r[0] + sx[k][1] * r[1] + sx[k][2] * r[2] + sx[k][3] * r[3];
            y[4 * a + b] = sy[k][0] * r[0] + sy[k][1] * r[2] + sy[k][2] * r[1] + sy[k][3] * r[3];
        }
    }
}

__device__ __forceinline__ void site_offsets(const TriArgs &a, int *goff) {
    for (int i = threadIdx.x; i < 32 * a.nl; i += blockDim.x) {
        const int e = i / (16 * a.nl), j = (i >> 4) % a.nl, c = i & 15;
        const int r = e ? a.inv_sites[j] : a.sites[j], p = e ? a.inv_sites_perm[j] : a.sites_perm[j];
        goff[(e * a.nl + j) * kGoffRow + c] = gather_offset(e, c, a.nl, r, p);
    }
}

// The two ladders for one site (as ladder): X holds slabs (0, 2), Y slabs (1, 3), so a packed product takes both
// slab pairs; terms of either sign are summed apart.  Adds cw times the result to acc.
template <bool PH>
__device__ __forceinline__ void site_ladder(const float2 (&X)[16], const float2 (&Y)[16], float cw, float (&acc)[16]) {
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        float2 vp = make_float2(0.0f, 0.0f), vn = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            const int x = 15 - n, y = x ^ c ^ 15;
            if ((PH ? tri::ph_sign(c, x) : tri::pp_sign(c, x)) > 0) vp = fma2(X[x], Y[y], vp);
            else vn = fma2(X[x], Y[y], vn);
        }
        acc[c] += cw * ((vp.x + vp.y) - (vn.x + vn.y));
    }
}

// The chalice diagrams are linear in a slab's components with coefficients that are sums of four
// site-local values each, the same for all sites: slab q's coefficient of output c and component k is word
// 64 q + 4 c + k, the indices of the four among the slab's 16 (4 bits) with their signs.
__device__ __forceinline__ void chalice_words(int *words) {
    for (int e = threadIdx.x; e < 256; e += blockDim.x) {
        const int q = e >> 6, c = (e >> 2) & 15, k = e & 3;
        int w = 0;
        for (int i = 0; i < 4; ++i) {
            const int l = (q & 1) ? 4 * i + (i ^ (c >> 2) ^ k) : 4 * i + ((c & 3) ^ k ^ i);
            const int sg = (q & 1) ? tri::ichal_sign(c, l) : tri::chal_sign(c, k, i);
            w |= (l | (sg < 0 ? 16 : 0)) << (5 * i);
        }
        words[e] = w;
    }
}
// Site-local value e of a node (tri_local): those of slab q are 16 ((q & 1) 2 + (q >> 1)) .. + 15.
__device__ __forceinline__ float local_value(const TriArgs &a, const TDesc &d, int e) {
    return tri_local(a.v4, a.nl, d.ab[4 + (e >> 4)], (e & 15) >> 2, e & 3);
}
__device__ __forceinline__ int local_first(int q) { return ((q & 1) << 5) | ((q >> 1) << 4); }
// A chalice coefficient from its slab's 16 site-local values.
__device__ __forceinline__ float chalice_coef(const float *L, int w) {
    float v = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = w >> (5 * i);
        v += __int_as_float(__float_as_int(L[t & 15]) ^ ((t & 16) << 27));
    }
    return v;
}
// Adds a slab's chalice terms of one site to v: chalice (slabs 0, 2) over the second component, inverse (1, 3) over the
// first.
template <bool INVERSE>
__device__ __forceinline__ void chalice_terms(const float (&x)[16], const float *coef, float (&v)[16]) {
    const float4 *C = reinterpret_cast<const float4 *>(coef);
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        const float4 k = C[c];
        const int m = c >> 2, n = c & 3;
        if (INVERSE) v[c] += x[n] * k.x + x[4 + n] * k.y + x[8 + n] * k.z + x[12 + n] * k.w;
        else v[c] += x[4 * m] * k.x + x[4 * m + 1] * k.y + x[4 * m + 2] * k.z + x[4 * m + 3] * k.w;
    }
}

// index triple of flow element `it`
__device__ __forceinline__ void decode_triple(int it, int n, int &si, int &ti, int &ui) {
    const int su = it / n;
    ti = it - su * n;
    si = int((sqrtf(8.0f * float(su) + 1.0f) - 1.0f) * 0.5f);
    while (si * (si + 1) / 2 > su) --si;
    while ((si + 1) * (si + 2) / 2 <= su) ++si;
    ui = su - si * (si + 1) / 2;
}

// shared memory, in floats: head (gather offsets, chalice words, the warps' sums) and a warp's area
__host__ __device__ inline size_t site_head_floats(int nl) { return 2 * size_t(nl) * kGoffRow + 256 + size_t(kWarps) * 512; }
__host__ __device__ inline size_t site_warp_floats(int nl, int n_seg, bool walk) {
    const size_t g = 32 / site_lanes(nl);
    return kSiteBatch * (sizeof(TDesc) / sizeof(float)) + (walk ? g * (64 + kCoefRow + 64 * size_t(nl) + 16 * size_t(n_seg)) : 0);
}

// WALK: the t channel too, with the RPA pairs walked for every node; otherwise tri_lattice_kernel adds the t channel.
template <bool WALK>
__global__ void __launch_bounds__(kThreads, 4) tri_site_kernel(TriArgs a) {
    __shared__ float pos[kMaxFreq];
    __shared__ int s_item;
    extern __shared__ __align__(16) float tsm[];
    const int n = a.n, nl = a.nl, W = site_lanes(nl), G = 32 / W, n_seg = WALK ? a.rpa_n_seg : 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane / W, jl = lane - sub * W, j = min(jl, nl - 1);
    int *goff = reinterpret_cast<int *>(tsm), *words = goff + 2 * nl * kGoffRow;
    float *red = reinterpret_cast<float *>(words + 256);
    float *area = red + kWarps * 512 + warp * site_warp_floats(nl, n_seg, WALK);
    TDesc *desc = reinterpret_cast<TDesc *>(area);
    float *coef = area + kSiteBatch * (sizeof(TDesc) / sizeof(float));  // [G][kCoefRow]
    float *L = coef + G * kCoefRow, *S = L + G * 64, *slots = S + G * 64 * nl;  // [G] of each
    for (int i = threadIdx.x; i < n; i += blockDim.x) pos[i] = a.freq[i];
    site_offsets(a, goff);
    if (WALK) chalice_words(words);
    const int rpa_cnt = WALK ? a.rpa_count[lane] : 0, rpa_base = WALK ? a.rpa_slot_base[lane] : 0;
    const float two_pi = 2.0f * float(kPiD);

    for (;;) {
        __syncthreads();  // the previous triple's sums are read
        if (threadIdx.x == 0) s_item = atomicAdd(a.work_counter, 1);
        __syncthreads();
        const int it = s_item;
        if (it >= a.fn) break;
        int si, ti, ui;
        decode_triple(it, n, si, ti, ui);
        const float s = pos[si], t = pos[ti], u = pos[ui];
        const float w1p = 0.5f * (s + t + u), w1 = 0.5f * (s - t + u), w2p = 0.5f * (s - t - u), w2 = 0.5f * (s + t - u);
        float acc[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) acc[c] = 0.0f;
#pragma unroll 1
        for (int ch = 0; ch < 3; ch += WALK ? 1 : 2) {
            const int xi = ch == 0 ? si : (ch == 1 ? ti : ui);
            const int mine = (a.node_cnt[xi] - warp + kWarps - 1) / kWarps;  // nodes warp, warp + kWarps, ...
            const float *nwp = a.node_wp + size_t(xi) * a.max_nodes + warp, *nc = a.node_c + size_t(xi) * a.max_nodes + warp;
#pragma unroll 1
            for (int b0 = 0; b0 < mine; b0 += kSiteBatch) {
                const int nb = min(kSiteBatch, mine - b0);
                if ((lane >> 2) < nb) {  // a quad of lanes per node
                    const int k = lane >> 2;
                    make_tpart(a, pos, ch, xi, s, t, u, w1p, w1, w2p, w2, nwp[kWarps * (b0 + k)], lane & 3, desc[k]);
                    if ((lane & 3) == 0) desc[k].c = nc[kWarps * (b0 + k)];
                }
                __syncwarp();
#pragma unroll 1
                for (int b = 0; b < nb; b += G) {
                    const bool active = b + sub < nb;
                    const TDesc &d = desc[active ? b + sub : b];
                    if (!WALK || ch != 1) {
                        float2 X[16], Y[16];
                        {
                            float x0[16], x1[16];
                            gather_site(a.v4, d.ab[0], goff, nl, j, x0);
                            gather_site(a.v4, d.ab[2], goff, nl, j, x1);
#pragma unroll
                            for (int c = 0; c < 16; ++c) X[c] = make_float2(x0[c], x1[c]);
                            gather_site(a.v4, d.ab[1], goff, nl, j, x0);
                            gather_site(a.v4, d.ab[3], goff, nl, j, x1);
#pragma unroll
                            for (int c = 0; c < 16; ++c) Y[c] = make_float2(x0[c], x1[c]);
                        }
                        if (active) {
                            if (ch == 0) site_ladder<false>(X, Y, d.c, acc);
                            else site_ladder<true>(X, Y, d.c, acc);
                        }
                    } else {
                        float *Sn = S + sub * 64 * nl, *Ln = L + sub * 64, *Cn = coef + sub * kCoefRow;
#pragma unroll 1
                        for (int q = 0; q < 4; ++q) {
                            float x[16];
                            gather_site(a.v4, d.ab[q], goff, nl, j, x);
                            if (jl < nl)
#pragma unroll
                                for (int c = 0; c < 16; ++c) Sn[(16 * q + c) * nl + jl] = x[c];
                        }
                        for (int e = jl; e < 64; e += W) Ln[e] = local_value(a, d, e);
                        __syncwarp();
                        for (int e = jl; e < 256; e += W) Cn[e] = chalice_coef(Ln + local_first(e >> 6), words[e]);
                        for (int g = 0; g < min(G, nb - b); ++g)
                            rpa_walk(a, S + g * 64 * nl, nl, lane, rpa_cnt, rpa_base, slots + g * 16 * n_seg);
                        __syncwarp();
                        if (active) {
                            float v[16], x[16];
                            const float *sl = slots + sub * 16 * n_seg;
#pragma unroll
                            for (int c = 0; c < 16; ++c) v[c] = 0.0f;
                            for (int q = a.rpa_seg_ptr[j]; q < a.rpa_seg_ptr[j + 1]; ++q)  // the site's run partials, in order
#pragma unroll
                                for (int c = 0; c < 16; ++c) v[c] += sl[16 * q + c];
#pragma unroll
                            for (int c = 0; c < 16; ++c) v[c] *= 2.0f;
#pragma unroll
                            for (int c = 0; c < 16; ++c) x[c] = Sn[c * nl + j];
                            chalice_terms<false>(x, Cn, v);
#pragma unroll
                            for (int c = 0; c < 16; ++c) x[c] = Sn[(16 + c) * nl + j];
                            chalice_terms<true>(x, Cn + 64, v);
#pragma unroll
                            for (int c = 0; c < 16; ++c) x[c] = Sn[(32 + c) * nl + j];
                            chalice_terms<false>(x, Cn + 128, v);
#pragma unroll
                            for (int c = 0; c < 16; ++c) x[c] = Sn[(48 + c) * nl + j];
                            chalice_terms<true>(x, Cn + 192, v);
#pragma unroll
                            for (int c = 0; c < 16; ++c) acc[c] += d.c * v[c];
                        }
                        __syncwarp();
                    }
                }
                __syncwarp();
            }
        }
#pragma unroll
        for (int c = 0; c < 16; ++c) red[warp * 512 + c * 32 + lane] = acc[c];
        __syncthreads();
        float *dst = a.dv4 + size_t(it) * 16 * nl;
        bool bad = false;
        for (int e = threadIdx.x; e < 16 * nl; e += kThreads) {
            const int c = e / nl, k = e - c * nl;
            float v = 0.0f;
            for (int w = 0; w < kWarps; ++w)
                for (int g = 0; g < G; ++g) v += red[w * 512 + c * 32 + g * W + k];
            const float o = v / two_pi;
            dst[e] = o;
            bad |= isnan(o);
        }
        if (bad) atomicOr(a.status, kStatusNaN);
    }
}

// ------------------------------------------------------------------------------------
// The t channel with its lattice sum on the tensor cores (use_products).
//
// For output (mu, nu) of site j the sum over its pairs and the inner index k of
//   sign(mu, nu, k) A[rid1][P1 mu, P1 k] B[rid2][P2 k, P2 nu]
// is linear in the node's slab products, so per triple the kernel forms, for the inner components k1 = P1 k and
// k2 = P2 k that pairs have (10 of 16 at most: the density maps to itself),
//   M = sum over nodes of c S0 x S1 + c S2 x S3      (4 Nl rows (rid1, P1 mu) x 4 Nl columns (rid2, P2 nu))
// as a matrix product over K = 2 x nodes, and adds each pair's elements of M once per triple, where the walk
// adds 128 products for every pair and node.
//
// A CTA takes a triple.  Its 14 worker warps gather the nodes' slabs, a slab at a time, add the chalice terms and leave
// the slabs as operands (three bf16 terms of each FP32 value, umma.cuh) in the CTA's scratch (0.4 MB at the nodes of N = 32 and
// cutoff 0.5, room for 0.9: with 152 CTAs 65 MB are in use, of which L2 writes 4.5 GB a launch back to DRAM).  Then one
// thread copies the operands of every (k2, k1) to shared memory in chunks of 32 slab pairs, another issues the products, up
// to two accumulators ahead of the workers, which stage M in shared memory and add their outputs' elements.
//
// 28 sites, N = 32, cutoff 0.5: 6.7 ms, where the walk took about 19 of the vertex flow's 31.5.  A triple takes 117,000
// cycles: 47,000 gather and split the slabs (latency of the slab reads, sectors written), 29,000 add the pairs' elements, 20,000
// are the products (62 cycles each, the reads of their operands), the rest is waiting between the stages.
// ------------------------------------------------------------------------------------
// From here on the products pay, but for the fewest nodes (honeycomb, a right-hand side at cutoffs 20 and 0.1, us, by products and with
// the pairs walked): 8 sites, N = 8 91, 128 and 62, 103; N = 32 3103, 9239 and 2139, 9719.  11 sites, N = 8 93, 140 and 64, 118; N = 16 406, 851
// and 290, 974; N = 32 3315, 10091 and 2759, 12777.  14 sites, N = 8 95, 142 and 73, 145; N = 32 3369, 10351 and 3340, 16651.  28 sites, N = 4
// 89, 103 and 150, 217; N = 32 4686, 13697 and 7124, 39820.  A product takes 16 slab pairs at least and its staging and pair sums
// do not shrink with N; most of a flow's time is at low cutoffs, where the line is between 8 and 11 sites from N = 12 on.
constexpr int kLatMinSites = 10;
constexpr int kLatWarps = 14, kLatWorkers = 32 * kLatWarps, kLatThreads = kLatWorkers + 64;
constexpr int kLatReaders = kLatWarps / 4 * 4;  // warps that stage M: every four of them, the 128 rows
constexpr int kLatGroups = kLatWorkers / 4;  // groups of four threads, one for each mu, that share the sites' pairs
constexpr int kLatAhead = 6;     // pairs of words loaded before M is complete
constexpr int kLatK = 32;        // slab pairs of a chunk
// Chunks of A in shared memory (as many as fit) and of B, which are kept for all products of a k2 where its K has no
// more.
constexpr int kLatStages = 4, kLatSlotsB = 3;
constexpr int kLatKeep = kLatSlotsB * kLatK;
// Slab pairs that one accumulator takes where there are more than kLatKeep.  The tensor cores cut what they add, by 0.4 units in the last
// place of the sum for every 16 slab pairs and always towards zero.  A right-hand side of operands of one sign is 2.6e-7 off in norm
// over 90 slab pairs, with the pairs walked in FP32 3.9e-7; over 144 (N = 32), 240 (N = 56) and 416 (N = 100) it would be 5.0e-7,
// 1.1e-6 and 2.1e-6 off, walked 3.8e-7, 3.6e-7 and 7.5e-7.  So longer sums are made of parts, added rounded: 3.0e-7, 1.2e-7 and
// 3.6e-7 (with parts of 96 6.4e-7 at N = 56; parts of 32 take 7 % longer).
constexpr int kLatPart = 2 * kLatK;
constexpr int kLatNodes = kLatWorkers / 4;  // nodes whose descriptors are built at once (a quad of threads each)
constexpr uint32_t kLatCols = 512;  // tensor memory: accumulator b's high products at column 256 b, low ones 128 on

__host__ __device__ inline int lat_rows(int nl) { return (4 * nl + 15) / 16 * 16; }
__host__ __device__ inline int lat_stride(int nl) { return lat_rows(nl) + 4; }  // of the staged M: an odd number of 16-byte units
// scratch of a CTA: [A of k1 = 0 .. 3, B of k2 = 0 .. 3][term][k / 8][two row blocks] (umma.cuh)
constexpr int kLatGroup = 2048;  // bytes of 8 slab pairs of 128 rows
__host__ __device__ inline int lat_blocks(int max_nodes) { return (2 * max_nodes + 15) / 16 * 2; }
__host__ __device__ inline size_t lat_scratch_bytes(int max_nodes) { return 24 * size_t(lat_blocks(max_nodes)) * kLatGroup; }

constexpr int kLatSmemMax = 227 * 1024 - 2048;  // dynamic; the rest is the kernel's static variables

struct LatSmem {
    size_t words, u, locals, coef, stage, total;
    int stages;
};
__host__ __device__ inline LatSmem lat_smem(int nl) {
    LatSmem L;
    L.words = sizeof(int) * 2 * size_t(nl) * kGoffRow;
    L.u = (L.words + sizeof(int) * 256 + 1023) / 1024 * 1024;
    // union: the nodes' descriptors and the warps' local values and coefficients, or the chunks of operands
    L.locals = L.u + sizeof(TDesc) * kLatNodes;
    L.coef = L.locals + sizeof(float) * 32 * kLatWarps;
    const size_t red = sizeof(float) * 512 * kLatWarps, st = sizeof(float) * (lat_rows(nl) * size_t(lat_stride(nl)) + 4);
    const size_t chunk = 3 * size_t(kLatGroup) * (kLatK / 8), tail = (red > st ? red : st) + 1024;  // aligned to 1024 in the kernel
    const size_t gather = L.coef + sizeof(float) * 128 * kLatWarps;
    for (L.stages = kLatStages;; --L.stages) {
        const size_t ring = L.u + (L.stages + kLatSlotsB) * chunk;
        L.stage = gather > ring ? (gather + 1023) / 1024 * 1024 : ring;
        L.total = L.stage + tail;  // the stage is a union: the warps' sums, or M and four zeros
        if (L.total <= kLatSmemMax || L.stages == 2) break;
    }
    return L;
}

__device__ __forceinline__ void worker_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kLatWorkers) : "memory"); }

// Stores the lane's rows 4 lane .. 4 lane + 3 of slab pair k, four operands of three terms: x[operand][row].  The lanes fill
// whole sectors.
template <class Split>
__device__ __forceinline__ void lat_store(unsigned char *dst, int blocks, int k, int lane, const float (&x)[4][4], Split &&split) {
    unsigned char *p = dst + (k >> 3) * kLatGroup + (lane >> 4) * 1024 + umma::block_offset(lane & 15, k & 7);
    const size_t term = size_t(blocks) * kLatGroup;
#pragma unroll
    for (int o = 0; o < 4; ++o) {
        uint2 h, m, l;
        split(x[o][0], x[o][1], h.x, m.x, l.x);
        split(x[o][2], x[o][3], h.y, m.y, l.y);
        *reinterpret_cast<uint2 *>(p + 3 * o * term) = h;
        *reinterpret_cast<uint2 *>(p + (3 * o + 1) * term) = m;
        *reinterpret_cast<uint2 *>(p + (3 * o + 2) * term) = l;
    }
}
__device__ __forceinline__ void lat_store(unsigned char *dst, int blocks, int k, int lane, const float (&x)[4][4]) {
    float top = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) top = fmaxf(top, fabsf(x[i >> 2][i & 3]));
    if (top <= umma::kSplitMax)
        lat_store(dst, blocks, k, lane, x, [](float u, float v, uint32_t &h, uint32_t &m, uint32_t &l) { umma::split2(u, v, h, m, l); });
    else
        lat_store(dst, blocks, k, lane, x, [](float u, float v, uint32_t &h, uint32_t &m, uint32_t &l) { umma::split2_any(u, v, h, m, l); });
}

// Copies the three terms of a chunk.
__device__ __forceinline__ void copy_terms(uint32_t dst, uint32_t dst_term, const unsigned char *src, size_t src_term, uint32_t bytes,
                                           uint64_t *bar) {
    umma::bar_expect(bar, 3 * bytes);
#pragma unroll
    for (int t = 0; t < 3; ++t) umma::bulk_load(dst + t * dst_term, src + t * src_term, bytes, bar);
}

__global__ void __launch_bounds__(kLatThreads, 1) tri_lattice_kernel(TriArgs a) {
    extern __shared__ __align__(1024) unsigned char lat_sm[];
    __shared__ float pos[kMaxFreq];
    // chunk of A there / read, chunk of B, accumulator complete / read
    __shared__ uint64_t full[kLatStages], empty[kLatStages], full_b[kLatSlotsB], empty_b[kLatSlotsB], done[2], drained[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_item, s_combos[16], s_ncombo;
    __shared__ int s_dead, s_late;  // a wait ran out: the copying or issuing thread's, a worker's
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = a.n, nl = a.nl, rows = lat_rows(nl), stride = lat_stride(nl), blocks = lat_blocks(a.max_nodes);
    const LatSmem L = lat_smem(nl);
    unsigned char *psm = lat_sm + (-umma::smem_addr(lat_sm) & 1023);
    int *goff = reinterpret_cast<int *>(psm), *words = reinterpret_cast<int *>(psm + L.words);
    TDesc *desc = reinterpret_cast<TDesc *>(psm + L.u);
    float *stage = reinterpret_cast<float *>(psm + L.stage), *red = stage;
    unsigned char *scratch = a.prod_scratch + lat_scratch_bytes(a.max_nodes) * blockIdx.x;
    const size_t operand = size_t(blocks) * kLatGroup;  // scratch bytes of an operand's term
    for (int i = tid; i < n; i += kLatThreads) pos[i] = a.freq[i];
    site_offsets(a, goff);
    chalice_words(words);
    if (warp == 0) umma::tmem_alloc(&tmem_slot, kLatCols);
    if (tid == 0) {
        for (int b = 0; b < kLatStages; ++b) {
            umma::bar_init(full + b);
            umma::bar_init(empty + b);
        }
        for (int b = 0; b < kLatSlotsB; ++b) {
            umma::bar_init(full_b + b);
            umma::bar_init(empty_b + b);
        }
        for (int b = 0; b < 2; ++b) {
            umma::bar_init(done + b);
            umma::bar_init(drained + b, kLatReaders);
        }
        s_dead = s_late = 0;
        s_ncombo = 0;
        for (int cb = 0; cb < 16; ++cb)
            if (a.prod_ptr[cb * kLatGroups] != a.prod_ptr[(cb + 1) * kLatGroups]) s_combos[s_ncombo++] = cb;
    }
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = tmem_slot;
    const float two_pi = 2.0f * float(kPiD);
    const int combos = s_ncombo;
    const int group = tid >> 2, mu = tid & 3;  // a worker's group of pairs and output row
    const uint32_t term = kLatK / 8 * kLatGroup;  // bytes of an operand's term of a chunk
    uint32_t combo_no = 0;                   // accumulators so far
    const uint32_t ring = umma::smem_addr(psm + L.u), ring_b = ring + L.stages * 3 * term;
    // the copying and the issuing thread's next chunk of A, its barrier's phase and those of B's slots (a bit each); the first
    // wait for an empty slot passes
    int stage_no = 0;
    uint32_t phase = warp == kLatWarps ? 1 : 0, phase_b = warp == kLatWarps ? ~0u : 0;

    while (!s_dead && !s_late) {
        __syncthreads();  // the previous triple is finished with shared memory
        if (tid == 0) s_item = atomicAdd(a.work_counter + 1, 1);
        __syncthreads();
        const int it = s_item;
        if (it >= a.fn) break;
        int si, ti, ui;
        decode_triple(it, n, si, ti, ui);
        const int cnt = a.node_cnt[ti], kn = (2 * cnt + 15) / 16 * 16;

        if (warp < kLatWarps) {
            const float s = pos[si], t = pos[ti], u = pos[ui];
            const float w1p = 0.5f * (s + t + u), w1 = 0.5f * (s - t + u), w2p = 0.5f * (s - t - u), w2 = 0.5f * (s + t - u);
            const float *nwp = a.node_wp + size_t(ti) * a.max_nodes, *nc = a.node_c + size_t(ti) * a.max_nodes;
            float *Ln = reinterpret_cast<float *>(psm + L.locals) + warp * 32, *coef = reinterpret_cast<float *>(psm + L.coef) + warp * 128;
            float acc[16];
#pragma unroll
            for (int c = 0; c < 16; ++c) acc[c] = 0.0f;
#pragma unroll 1
            for (int b0 = 0; b0 < cnt; b0 += kLatNodes) {
                const int nb = min(kLatNodes, cnt - b0);
                if (b0) worker_sync();  // the previous batch's descriptors are read
                if ((tid >> 2) < nb) {
                    const int k = tid >> 2;
                    make_tpart(a, pos, 1, ti, s, t, u, w1p, w1, w2p, w2, nwp[b0 + k], tid & 3, desc[k]);
                    if ((tid & 3) == 0) desc[k].c = nc[b0 + k];
                }
                worker_sync();
#pragma unroll 1
                for (int task = warp; task < 2 * nb; task += kLatWarps) {  // slabs q and q + 2 of a node
                    const int q = task & 1, k = 2 * (cnt - 1 - b0 - (task >> 1));
                    const TDesc &d = desc[task >> 1];
                    float x[16], y[16], v[16], f[4][4], g[4][4];
                    const float lv = local_value(a, d, 32 * q + lane);
                    gather_site_pair(a.v4, d.ab[q], d.ab[q + 2], goff, nl, min(lane, nl - 1), x, y);
                    Ln[lane] = lv;
                    __syncwarp();
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        coef[32 * e + lane] = chalice_coef(Ln + 16 * (e >> 1), words[64 * (q + (e & 2)) + 32 * (e & 1) + lane]);
                    __syncwarp();
                    const float c1 = d.c;
                    unsigned char *dst = scratch + q * 12 * operand;
#pragma unroll
                    for (int c = 0; c < 16; ++c) v[c] = 0.0f;
                    if (q) {  // operand k, row nu
                        chalice_terms<true>(x, coef, v);
                        chalice_terms<true>(y, coef + 64, v);
#pragma unroll
                        for (int c = 0; c < 16; ++c) f[c >> 2][c & 3] = x[c], g[c >> 2][c & 3] = y[c];
                    } else {  // operand k, row mu
                        chalice_terms<false>(x, coef, v);
                        chalice_terms<false>(y, coef + 64, v);
#pragma unroll
                        for (int c = 0; c < 16; ++c) f[c & 3][c >> 2] = c1 * x[c], g[c & 3][c >> 2] = c1 * y[c];
                    }
                    if (lane < nl) {
                        lat_store(dst, blocks, k, lane, f);
                        lat_store(dst, blocks, k + 1, lane, g);
                    }
#pragma unroll
                    for (int c = 0; c < 16; ++c) acc[c] += c1 * v[c];
                }
            }
            for (int task = warp + 4 * cnt; task < 2 * kn; task += kLatWarps) {  // zero up to a multiple of 16
                const float z[4][4] = {};
                if (lane < nl) lat_store(scratch + (task & 1) * 12 * operand, blocks, task >> 1, lane, z);
            }
#pragma unroll
            for (int c = 0; c < 16; ++c) red[warp * 512 + c * 32 + lane] = acc[c];
            umma::fence_copies();
        }
        __syncthreads();

        const bool keep = kn <= kLatKeep;  // the whole B of a k2 stays in shared memory
        const int part_len = keep ? kLatKeep : kLatPart, parts = keep ? 1 : (kn + kLatPart - 1) / kLatPart;
        if (warp == kLatWarps) {
            if (lane == 0) {  // copies
                bool ok = true;
                int slot = 0;
                for (int i = 0; i < combos && ok; ++i) {
                    const int cb = s_combos[i];
                    const bool with_b = !keep || i == 0 || s_combos[i - 1] >> 2 != cb >> 2;
                    const unsigned char *src_a = scratch + 3 * (cb & 3) * operand, *src_b = scratch + (12 + 3 * (cb >> 2)) * operand;
                    if (keep) slot = 0;
                    for (int k0 = 0; k0 < kn; k0 += kLatK) {
                        const uint32_t bytes = min(kLatK, kn - k0) / 8 * kLatGroup;
                        if (with_b) {
                            ok = umma::bar_wait(empty_b + slot, phase_b >> slot & 1);
                            if (!ok) break;
                            phase_b ^= 1u << slot;
                            copy_terms(ring_b + slot * 3 * term, term, src_b, operand, bytes, full_b + slot);
                        }
                        ok = umma::bar_wait(empty + stage_no, phase);
                        if (!ok) break;
                        copy_terms(ring + stage_no * 3 * term, term, src_a, operand, bytes, full + stage_no);
                        src_a += bytes;
                        src_b += bytes;
                        if (++slot == kLatSlotsB) slot = 0;
                        if (++stage_no == L.stages) stage_no = 0, phase ^= 1;
                    }
                }
                if (!ok) s_dead = 1;
            }
            __syncwarp();
        } else if (warp == kLatWarps + 1) {
            if (lane == 0) {  // products
                bool ok = true;
                int slot = 0;
                uint32_t ci = combo_no;
                for (int i = 0; i < combos && ok; ++i) {
                    const bool release_b = !keep || i + 1 == combos || s_combos[i + 1] >> 2 != s_combos[i] >> 2;
                    if (keep) slot = 0;
                    for (int part = 0; part < kn && ok; part += part_len, ++ci) {
                        const uint32_t d = tmem + 256 * (ci & 1);
                        if (ci >= 2) ok = umma::bar_wait(drained + (ci & 1), ((ci >> 1) - 1) & 1);
                        for (int k0 = part; k0 < min(kn, part + part_len) && ok; k0 += kLatK) {
                            ok = umma::bar_wait(full_b + slot, phase_b >> slot & 1) && umma::bar_wait(full + stage_no, phase);
                            if (!ok) break;
                            umma::fence_after();
                            umma::product(d, d + 128, ring + stage_no * 3 * term, kLatGroup, term, ring_b + slot * 3 * term, kLatGroup, term, rows,
                                          min(kLatK, kn - k0) / 16, k0 > part);
                            umma::commit(empty + stage_no);
                            if (release_b) {
                                umma::commit(empty_b + slot);
                                phase_b ^= 1u << slot;
                            }
                            if (++slot == kLatSlotsB) slot = 0;
                            if (++stage_no == L.stages) stage_no = 0, phase ^= 1;
                        }
                        umma::commit(done + (ci & 1));
                    }
                }
                if (!ok) s_dead = 1;
            }
            __syncwarp();
        } else {
            float sum[2] = {0.0f, 0.0f};  // outputs o = 16 site + component: tid, tid + kLatWorkers
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (const int o = tid + h * kLatWorkers; o < 16 * nl)
                    for (int w = 0; w < kLatWarps; ++w) sum[h] += red[w * 512 + (o & 15) * 32 + (o >> 4)];
            worker_sync();  // M takes the place of the sums
            if (tid < 4) stage[rows * stride + tid] = 0.0f;  // for the padding words
            float rpa[4] = {};
            const int2 *list = reinterpret_cast<const int2 *>(a.prod_words);
            const int *ptr = a.prod_ptr + group;
            int w0 = 0, w1 = 0;
            if (combos) {
                w0 = __ldg(ptr + s_combos[0] * kLatGroups);
                w1 = __ldg(ptr + s_combos[0] * kLatGroups + 1);
            }
            uint32_t ci = combo_no;
            for (int i = 0; i < combos && kn > 0; ++i) {
                const int cb = s_combos[i];
                int2 ahead[kLatAhead];
#pragma unroll
                for (int e = 0; e < kLatAhead; ++e) ahead[e] = w0 + e < w1 ? __ldg(list + w0 + e) : make_int2(rows * stride, rows * stride);
                // the reading warps alone wait for the products: the others are not held to their pace, and would miss a phase
                auto drain = [&](auto more) {
                    const uint32_t b = ci & 1;
                    if (!umma::bar_wait(done + b, (ci >> 1) & 1)) s_late = 1;
                    umma::fence_after();
                    const int row = (warp & 3) * 32 + lane;
                    for (int c0 = (warp >> 2) * 16; c0 < rows; c0 += 4 * kLatReaders) {
                        float hi[16], lo[16];
                        const uint32_t addr = tmem + 256 * b + (uint32_t(warp & 3) << 21) + c0;
                        umma::load16(addr, hi);
                        umma::load16(addr + 128, lo);
                        umma::load_wait();
                        if (row < rows)
#pragma unroll
                            for (int k = 0; k < 16; k += 4) {
                                float4 v = make_float4(umma::add_terms(hi[k], lo[k]), umma::add_terms(hi[k + 1], lo[k + 1]),
                                                       umma::add_terms(hi[k + 2], lo[k + 2]), umma::add_terms(hi[k + 3], lo[k + 3]));
                                float4 *m = reinterpret_cast<float4 *>(stage + row * stride + c0 + k);
                                if constexpr (decltype(more)::value) {  // this thread's own elements
                                    const float4 u = *m;
                                    v = make_float4(u.x + v.x, u.y + v.y, u.z + v.z, u.w + v.w);
                                }
                                *m = v;
                            }
                    }
                    umma::fence_before();
                    __syncwarp();
                    if (lane == 0) umma::bar_arrive(drained + b);
                    ++ci;
                };
                if (warp < kLatReaders) {
                    drain(std::false_type{});
#pragma unroll 1
                    for (int part = 1; part < parts; ++part) drain(std::true_type{});
                }
                worker_sync();
                if (s_late) break;  // the workers write it before this barrier alone, so they agree
                int n0 = 0, n1 = 0;
                if (i + 1 < combos) {
                    n0 = __ldg(ptr + s_combos[i + 1] * kLatGroups);
                    n1 = __ldg(ptr + s_combos[i + 1] * kLatGroups + 1);
                }
                float part[4] = {};
                auto pair = [&](int w) {  // row mu of the pair's element block, its columns permuted
                    const float *m = stage + (w & 0x7fff) + ((w >> (15 + 2 * mu)) & 3) * stride;
                    part[0] += m[(w >> 23) & 3];
                    part[1] += m[(w >> 25) & 3];
                    part[2] += m[(w >> 27) & 3];
                    part[3] += m[3];
                };
#pragma unroll
                for (int e = 0; e < kLatAhead; ++e) {
                    pair(ahead[e].x);
                    pair(ahead[e].y);
                }
#pragma unroll 4
                for (int e = w0 + kLatAhead; e < w1; ++e) {
                    const int2 w = __ldg(list + e);
                    pair(w.x);
                    pair(w.y);
                }
#pragma unroll
                for (int nu = 0; nu < 4; ++nu)  // tri::rpa_sign: the inner index is the density for k1 = 3 alone
                    rpa[nu] += (mu == 3) == (nu == 3) && ((cb & 3) == 3) != (mu == 3) ? -part[nu] : part[nu];
                w0 = n0;
                w1 = n1;
                worker_sync();  // M is read
            }
#pragma unroll
            for (int nu = 0; nu < 4; ++nu) stage[16 * group + 4 * mu + nu] = rpa[nu];
            worker_sync();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int o = tid + h * kLatWorkers, j = o >> 4;
                if (o >= 16 * nl) continue;
                float r = 0.0f;
                for (int g = __ldg(a.prod_group + j); g < __ldg(a.prod_group + j + 1); ++g) r += stage[16 * g + (o & 15)];
                float *p = a.dv4 + size_t(it) * 16 * nl + (o & 15) * nl + j;
                const float v = *p + (sum[h] + 2.0f * r) / two_pi;
                *p = v;
                if (isnan(v)) atomicOr(a.status, kStatusNaN);
            }
        }
        combo_no += combos * parts;
        __syncthreads();  // s_dead, s_late
    }
    // a copy or a product did not complete in time (each wait is long enough for those in flight to end)
    if ((s_dead || s_late) && tid == 0) atomicOr(a.status, kStatusProductTimeout);
    umma::fence_before();
    __syncthreads();
    if (warp == 0) {
        umma::fence_after();
        umma::tmem_free(tmem, kLatCols);
    }
}

// ------------------------------------------------------------------------------------
// correlation measurement at nu = 0 (TRIMeasurementCorrelation.cpp:147-285): one CTA per
// outer node accumulates the inner integral per site and component in FP64, a final CTA adds
// the outer weights and the on-site term and scatters to (basis, site in range) entries.
// ------------------------------------------------------------------------------------
__constant__ int kOutComp[kCorrOut] = {0, 1, 2, 4, 5, 6, 8, 9, 10, 15};

// Linear in the vertex, as the SU(2) core's (corr_inner_body): sums of g * vertex per site and
// component and, a thread per node and component, of the egg diagram's site-local reads (lane 0
// alone took 320 reads a node: 289 us at N = 32, 28 sites, now 29).
constexpr int kCorrTWarps = 8, kCorrTThreads = 32 * kCorrTWarps;

__global__ void __launch_bounds__(kCorrTThreads) tri_corr_inner_kernel(TriArgs a) {
    __shared__ float pos[kMaxFreq];
    __shared__ float nwp[kMaxCorrNodes];
    __shared__ double nw[kMaxCorrNodes], ng[kMaxCorrNodes];
    __shared__ double egg[kCorrTThreads];
    extern __shared__ double red[];  // [kCorrTWarps][kCorrOut][nl]
    for (int i = threadIdx.x; i < a.n; i += blockDim.x) pos[i] = a.freq[i];
    __syncthreads();
    const int ncnt = corr_nodes(pos, a.n, a.cutoff, nwp, nw, ng, [&](float x) { return odd_interp(pos, a.n, a.v2, x); });
    const int ia = blockIdx.x;
    if (ia >= ncnt) return;
    const float w = nwp[ia];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nl = a.nl;
    {  // site-local vertex component tid & 15 at nodes tid >> 4, ...
        const int c = threadIdx.x & 15;
        double sum = 0.0;
        for (int b = threadIdx.x >> 4; b < ncnt; b += kCorrTThreads / 16) {
            const float wp = nwp[b];
            TAB8 ab;
            tri_access8(pos, a.n, nl, w + wp + 0.0f, w - wp, 0.0f, ab);
            sum += nw[b] * ng[b] * double(tri_local(a.v4, nl, ab, c >> 2, c & 3));
        }
        egg[threadIdx.x] = sum;
        __syncthreads();
        if (threadIdx.x < 16) {
            for (int q = 16 + threadIdx.x; q < kCorrTThreads; q += 16) sum += egg[q];
            egg[threadIdx.x] = sum;
        }
    }
    for (int j0 = 0; j0 < nl; j0 += 32) {
        const int j = j0 + lane;
        const bool valid = j < nl;
        const int r0 = valid ? a.sites[j] : 0, p0 = valid ? a.sites_perm[j] : 0;
        const int r1 = valid ? a.inv_sites[j] : 0, p1 = valid ? a.inv_sites_perm[j] : 0;
        double acc[kCorrOut];
#pragma unroll
        for (int q = 0; q < kCorrOut; ++q) acc[q] = 0.0;
        for (int b = warp; b < ncnt; b += kCorrTWarps) {
            const float wp = nwp[b];
            TAB8 ab;
            tri_access8(pos, a.n, nl, w + wp + 0.0f, 0.0f, w - wp, ab);
            const double cw = nw[b] * ng[b];
            if (!valid) continue;
            const bool ex = ab.fl & kFlExch;
#pragma unroll
            for (int q = 0; q < kCorrOut; ++q)
                acc[q] += cw * double(tri_bundle(a.v4, nl, ab, kOutComp[q], ex ? r1 : r0, ex ? p1 : p0));
        }
        if (valid)
            for (int q = 0; q < kCorrOut; ++q) red[(size_t(warp) * kCorrOut + q) * nl + j] = acc[q];
    }
    __syncthreads();
    const double norm = ng[ia] / (4.0 * kPiD * kPiD);
    for (int e = threadIdx.x; e < kCorrOut * nl; e += blockDim.x) {
        const int q = e / nl, c = kOutComp[q];
        double sum = 0.0;
        for (int k = 0; k < kCorrTWarps; ++k) sum += red[size_t(k) * kCorrOut * nl + e];
        sum *= c == 15 ? -4.0 : -1.0;  // dumbbell
        if (e == q * nl) {             // egg diagram, TRIMeasurementCorrelation.cpp:211-251
            const double f = c == 15 ? 2.0 : 0.5;
            for (int k = 0; k < 4; ++k) {
                const int lam = tri::inner(k), rho = (c >> 2) ^ (c & 3) ^ lam;
                sum += f * tri::egg_sign(c, lam) * egg[4 * lam + rho];
            }
        }
        a.partial[size_t(ia) * kCorrOut * nl + e] = sum * norm;
    }
}

// Shared memory of the final kernel: chi[16][nl], then the reduction's slices.
size_t tri_final_smem(int nl) { return 16 * size_t(nl) * sizeof(double) + corr_final_smem(kCorrOut * nl); }

__global__ void __launch_bounds__(kCorrThreads) tri_corr_final_kernel(TriArgs a) {
    __shared__ float pos[kMaxFreq];
    __shared__ float nwp[kMaxCorrNodes];
    __shared__ double nw[kMaxCorrNodes], ng[kMaxCorrNodes];
    extern __shared__ double chi[];  // [16][nl]
    for (int i = threadIdx.x; i < a.n; i += blockDim.x) pos[i] = a.freq[i];
    __syncthreads();
    const int ncnt = corr_nodes(pos, a.n, a.cutoff, nwp, nw, ng, [&](float x) { return odd_interp(pos, a.n, a.v2, x); });
    const int nl = a.nl;
    double *sums = chi + 16 * nl;
    column_sums(ncnt, kCorrOut * nl, sums, [&](int ia, int e) { return nw[ia] * a.partial[size_t(ia) * kCorrOut * nl + e]; });
    for (int e = threadIdx.x; e < 16 * nl; e += blockDim.x) chi[e] = 0.0;
    __syncthreads();
    for (int e = threadIdx.x; e < kCorrOut * nl; e += blockDim.x) chi[kOutComp[e / nl] * nl + e % nl] = sums[e];
    __syncthreads();
    if (threadIdx.x < 32) {  // on-site term
        double s = 0.0;
        for (int k = threadIdx.x; k < ncnt; k += 32) s += nw[k] * ng[k];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (threadIdx.x < 4) chi[5 * threadIdx.x * nl] += threadIdx.x == 3 ? s / kPiD : s / (4.0 * kPiD);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 16 * nl; e += blockDim.x) a.out[size_t(kCorrOut) * a.n_corr + e] = float(chi[e]);
    for (int q = threadIdx.x; q < a.n_corr; q += blockDim.x) {
        const int r = a.corr_rid[q], p = a.corr_perm[q];
        int k = 0;
        for (int x = 0; x < 3; ++x)
            for (int y = 0; y < 3; ++y, ++k)
                a.out[size_t(k) * a.n_corr + q] = float(chi[(4 * permc(p, x) + permc(p, y)) * nl + r]);
        a.out[size_t(9) * a.n_corr + q] = float(chi[15 * nl + r]);
    }
}

__global__ void tri_euler_kernel(float *__restrict__ x, const float *__restrict__ dx, long long n, float step) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        x[i] = __fadd_rn(x[i], __fmul_rn(step, dx[i]));
}

using cuh::check_cuda;
using cuh::copy_grid;
using cuh::dalloc;
using cuh::h2d;

}  // namespace

struct spn_tri {
    int device = 0, n = 0, nl = 0, n_range = 0, n_corr = 0, n_overlap = 0, max_nodes = 0, sms = 0, grid = 0;
    long long fn = 0;
    float cutoff = 0.0f;
    cudaStream_t stream = nullptr;
    float *freq = nullptr, *v2 = nullptr, *dv2 = nullptr, *v4 = nullptr, *dv4 = nullptr, *node_wp = nullptr,
          *node_c = nullptr, *corr_out = nullptr;
    int *ints = nullptr;  // all integer tables in one allocation
    int *sites, *sites_perm, *inv_sites, *inv_sites_perm, *range_rid, *range_inv, *corr_rid,
        *corr_perm, *node_cnt, *work_counter, *rpa_sched, *rpa_count, *rpa_slot_base, *rpa_seg_ptr, *prod_ptr, *prod_words, *prod_group;
    int rpa_n_seg = 0;
    unsigned char *prod_scratch = nullptr;  // tri_lattice_kernel's, of prod_ctas CTAs; it runs when not NULL
    int prod_ctas = 0;
    unsigned *status = nullptr;  // in ints, behind the work counters
    spn::cuh::HostResults results;  // measurements and the status word on the host
    double *partial = nullptr;

    long long vsize() const { return 16 * fn * nl; }

    TriArgs args() const {
        TriArgs a;
        a.n = n;
        a.nl = nl;
        a.fn = int(fn);
        a.max_nodes = max_nodes;
        a.n_range = n_range;
        a.n_corr = n_corr;
        a.cutoff = cutoff;
        a.freq = freq;
        a.v4 = v4;
        a.dv4 = dv4;
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
        a.prod_ptr = prod_ptr;
        a.prod_words = prod_words;
        a.prod_group = prod_group;
        a.prod_scratch = prod_scratch;
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
        void *ptrs[] = {freq, v2, dv2, v4, dv4, node_wp, node_c, corr_out, ints, partial, prod_scratch};
        for (void *p : ptrs)
            if (p) cudaFree(p);
        if (stream) cudaStreamDestroy(stream);
    }
};

namespace {

void validate(const spn_tri_desc *d) {
    if (!d) throw Error(ErrorType::Argument, "null descriptor");
    if (d->n_freq < 2 || d->n_freq > kMaxFreq)
        throw Error(ErrorType::Unsupported, "n_freq must be in [2, " + std::to_string(kMaxFreq) + "]");
    if (d->n_sites < 1 || d->n_sites > kMaxSites)
        throw Error(ErrorType::Unsupported, "n_sites must be in [1, " + std::to_string(kMaxSites) + "]");
    if (!d->freq || !d->sites_rid || !d->sites_perm || !d->inv_sites_rid || !d->inv_sites_perm || !d->overlap_ptr ||
        (d->n_range > 0 && (!d->range_rid || !d->range_inv_rid)) || (d->n_corr > 0 && (!d->corr_rid || !d->corr_perm)))
        throw Error(ErrorType::Argument, "descriptor table pointer is NULL");
    for (int i = 0; i < d->n_freq; ++i) {
        if (!(d->freq[i] > 0.0f)) throw Error(ErrorType::Argument, "frequencies must be positive");
        if (i > 0 && !(d->freq[i] > d->freq[i - 1])) throw Error(ErrorType::Argument, "frequencies must be strictly ascending");
    }
    const long long fn = (long long)d->n_freq * d->n_freq * (d->n_freq + 1) / 2;
    if (16 * fn * d->n_sites >= (1ll << 31)) throw Error(ErrorType::Unsupported, "vertex larger than 2^31 elements");
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

size_t vertex_smem(const spn_tri *h) {
    const int nl = h->nl, n_seg = h->rpa_n_seg;
    if (nl > 32) return (tri_cta_head_floats(nl) + size_t(kWarps) * tri_warp_floats(nl, n_seg)) * sizeof(float);
    return (site_head_floats(nl) + size_t(kWarps) * site_warp_floats(nl, n_seg, !h->prod_scratch)) * sizeof(float);
}
void (*vertex_kernel(const spn_tri *h))(TriArgs) {
    return h->nl > 32 ? tri_vertex_kernel : (h->prod_scratch ? tri_site_kernel<false> : tri_site_kernel<true>);
}

// Whether the t channel runs on the tensor cores (tri_lattice_kernel).
bool use_products(int nl) { return nl >= kLatMinSites && nl <= 32; }

// CTAs of tri_lattice_kernel: `want`, or as many of them as the device has memory for, by halves; 0 if there is none for one.  The flow
// is the same with any number, as each triple is one CTA's.
template <class TryAlloc>
int scratch_ctas(int want, size_t bytes, TryAlloc &&try_alloc) {
    for (; want > 0; want /= 2)
        if (try_alloc(want * bytes)) return want;
    return 0;
}

// The RPA pairs as tri_lattice_kernel reads them, two words at a time: the element of the staged M (15 bits) and the
// images of the four components under perm1 and perm2 (2 bits each); an odd list ends with the zero behind M.  A site's pairs are
// dealt to as many groups as keep every group's share below the smallest bound that suffices.
void product_pairs(const spn_tri_desc *d, std::vector<int> &ptr, std::vector<int> &words, std::vector<int> &group) {
    const int nl = d->n_sites, stride = lat_stride(nl);
    int bound = 1;
    for (;; ++bound) {
        group.assign(1, 0);
        for (int j = 0; j < nl; ++j) group.push_back(group.back() + (d->overlap_ptr[j + 1] - d->overlap_ptr[j] + bound - 1) / bound);
        if (group.back() <= kLatGroups) break;
    }
    std::vector<int> site(kLatGroups, -1);
    for (int j = 0; j < nl; ++j) std::fill(site.begin() + group[j], site.begin() + group[j + 1], j);
    ptr.assign(1, 0);
    for (int k2 = 0; k2 < 4; ++k2)
        for (int k1 = 0; k1 < 4; ++k1)
            for (int g = 0; g < kLatGroups; ++g) {
                const int j = site[g], step = j < 0 ? 1 : group[j + 1] - group[j];
                const int first = j < 0 ? 0 : d->overlap_ptr[j] + g - group[j], last = j < 0 ? 0 : d->overlap_ptr[j + 1];
                for (int i = first; i < last; i += step) {
                    const int p1 = d->overlap_perm1[i], p2 = d->overlap_perm2[i];
                    for (int k = 0; k < 4; ++k) {
                        if (permc(p1, k) != k1 || permc(p2, k) != k2) continue;
                        unsigned w = 4 * d->overlap_rid1[i] * stride + 4 * d->overlap_rid2[i];
                        for (int q = 0; q < 4; ++q) w |= unsigned(permc(p1, q)) << (15 + 2 * q) | unsigned(permc(p2, q)) << (23 + 2 * q);
                        words.push_back(int(w));
                    }
                }
                if (words.size() % 2) words.push_back(lat_rows(nl) * stride);
                ptr.push_back(int(words.size() / 2));
            }
}

// The RPA pairs of each site in the order of host/pair_order (against bank collisions of the
// kernel's shared-memory reads), packed as the words of TriArgs::rpa_sched.
std::vector<int> order_rpa_pairs(const spn_tri_desc *d) {
    const int nl = d->n_sites;
    const std::vector<int> order =
        order_pairs_by_banks(nl, d->overlap_ptr, tri_rpa_model(),
                             tri_rpa_words(nl, d->overlap_rid1, d->overlap_rid2, d->overlap_perm1, d->overlap_perm2));
    std::vector<int> out(order.size());
    for (size_t k = 0; k < order.size(); ++k) {
        const int i = order[k];
        int word = d->overlap_rid1[i] | d->overlap_rid2[i] << 7;
        for (int q = 0; q < 3; ++q)
            word |= permc(d->overlap_perm1[i], q) << (14 + 2 * q) | permc(d->overlap_perm2[i], q) << (20 + 2 * q);
        out[k] = word;
    }
    return out;
}

void launch_correlation(spn_tri *h) {
    const TriArgs a = h->args();
    const size_t smem = size_t(kCorrTWarps) * kCorrOut * h->nl * sizeof(double);
    tri_corr_inner_kernel<<<2 * h->n + 4, kCorrTThreads, smem, h->stream>>>(a);
    check_cuda(cudaGetLastError(), "correlation launch");
    tri_corr_final_kernel<<<1, kCorrThreads, tri_final_smem(h->nl), h->stream>>>(a);
    check_cuda(cudaGetLastError(), "correlation final launch");
}

}  // namespace

extern "C" int spn_tri_create(const spn_tri_desc *d, spn_tri **out) {
    return guarded([&] {
        if (!out) throw Error(ErrorType::Argument, "null output handle");
        validate(d);
        auto *h = new spn_tri;
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
            const size_t vsz = size_t(h->vsize());
            h->freq = dalloc<float>(h->n, "alloc freq");
            h->v2 = dalloc<float>(h->n, "alloc v2");
            h->dv2 = dalloc<float>(h->n, "alloc dv2");
            h->v4 = dalloc<float>(vsz, "alloc vertex state");
            h->dv4 = dalloc<float>(vsz, "alloc vertex flow");
            h->node_wp = dalloc<float>(size_t(h->n) * h->max_nodes, "alloc node table");
            h->node_c = dalloc<float>(size_t(h->n) * h->max_nodes, "alloc node table");
            h->corr_out = dalloc<float>(size_t(kCorrOut) * h->n_corr + 16 * h->nl, "alloc correlation output");
            h->partial = dalloc<double>(size_t(kMaxCorrNodes) * kCorrOut * h->nl, "alloc correlation scratch");
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
            LaneSchedule rpa;  // of the flows whose pairs are walked
            if (!use_products(nl)) rpa = tri_lane_schedule(nl, d->overlap_ptr, order_rpa_pairs(d));
            h->rpa_n_seg = rpa.n_seg;
            put(d->range_rid, nr);
            put(d->range_inv_rid, nr);
            put(d->corr_rid, nc);
            put(d->corr_perm, nc);
            put(nullptr, h->n);  // node counts
            put(nullptr, 3);     // work counters, status
            put(rpa.sched.data(), int(rpa.sched.size()));
            put(rpa.count.data(), int(rpa.count.size()));
            put(rpa.slot_base.data(), int(rpa.slot_base.size()));
            put(rpa.seg_ptr.data(), int(rpa.seg_ptr.size()));
            std::vector<int> prod_ptr, prod_words, prod_group;
            if (use_products(nl)) product_pairs(d, prod_ptr, prod_words, prod_group);
            put(prod_ptr.data(), int(prod_ptr.size()));
            img.resize((img.size() + 1) / 2 * 2);  // read two words at a time
            put(prod_words.data(), int(prod_words.size()));
            put(prod_group.data(), int(prod_group.size()));
            h->ints = dalloc<int>(img.size(), "alloc lattice tables");
            h2d(h->ints, img.data(), img.size(), h->stream);
            int **fields[] = {&h->sites, &h->sites_perm, &h->inv_sites, &h->inv_sites_perm,
                              &h->range_rid, &h->range_inv, &h->corr_rid, &h->corr_perm, &h->node_cnt, &h->work_counter,
                              &h->rpa_sched, &h->rpa_count, &h->rpa_slot_base, &h->rpa_seg_ptr, &h->prod_ptr, &h->prod_words, &h->prod_group};
            for (size_t k = 0; k < at.size(); ++k) *fields[k] = h->ints + at[k];
            h->status = reinterpret_cast<unsigned *>(h->work_counter + 2);
            h2d(h->freq, d->freq, h->n, h->stream);
            check_cuda(cudaMemsetAsync(h->v4, 0, vsz * sizeof(float), h->stream), "memset");
            check_cuda(cudaMemsetAsync(h->dv4, 0, vsz * sizeof(float), h->stream), "memset");
            check_cuda(cudaMemsetAsync(h->v2, 0, h->n * sizeof(float), h->stream), "memset");
            check_cuda(cudaMemsetAsync(h->dv2, 0, h->n * sizeof(float), h->stream), "memset");
            check_cuda(cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, h->device), "device attribute");
            if (use_products(nl)) {
                check_cuda(allow_shared(tri_lattice_kernel, lat_smem(nl).total), "shared memory limit");
                void *p = nullptr;
                h->prod_ctas = scratch_ctas(h->sms, lat_scratch_bytes(h->max_nodes), [&](size_t bytes) {
                    const bool ok = cudaMalloc(&p, bytes) == cudaSuccess;
                    if (!ok) cudaGetLastError();
                    return ok;
                });
                if (!h->prod_ctas) throw Error(ErrorType::Cuda, "alloc operand scratch: out of memory");
                h->prod_scratch = static_cast<unsigned char *>(p);
            }
            int per_sm = 0;
            const auto fn = vertex_kernel(h);
            check_cuda(allow_shared(fn, vertex_smem(h)), "shared memory limit");
            check_cuda(allow_shared(tri_corr_inner_kernel, size_t(kCorrTWarps) * kCorrOut * nl * sizeof(double)), "shared memory limit");
            check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kThreads, vertex_smem(h)), "occupancy");
            if (per_sm < 1) throw Error(ErrorType::Unsupported, "TRI vertex-flow kernel does not fit on this device");
            h->grid = h->sms * per_sm;
            check_cuda(cudaStreamSynchronize(h->stream), "create sync");
        } catch (...) {
            h->release();
            delete h;
            throw;
        }
        *out = h;
    });
}

extern "C" int spn_tri_destroy(spn_tri *h) {
    if (!h) return SPN_OK;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    h->release();
    delete h;
    return SPN_OK;
}

extern "C" int spn_tri_set_state(spn_tri *h, float cutoff, const float *v2, const float *v4) {
    return guarded([&] {
        if (!h || !v2 || !v4) throw Error(ErrorType::Argument, "null argument");
        check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
        h2d(h->v4, v4, size_t(h->vsize()), h->stream);
        h2d(h->v2, v2, h->n, h->stream);
        h->cutoff = cutoff;
        check_cuda(cudaStreamSynchronize(h->stream), "set_state sync");
    });
}

extern "C" int spn_tri_get_state(spn_tri *h, float *cutoff, float *v2, float *v4) {
    return guarded([&] {
        if (!h) throw Error(ErrorType::Argument, "null handle");
        check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
        if (cutoff) *cutoff = h->cutoff;
        if (v2) check_cuda(cudaMemcpyAsync(v2, h->v2, h->n * sizeof(float), cudaMemcpyDeviceToHost, h->stream), "D2H");
        if (v4)
            check_cuda(cudaMemcpyAsync(v4, h->v4, size_t(h->vsize()) * sizeof(float), cudaMemcpyDeviceToHost, h->stream), "D2H");
        check_cuda(cudaStreamSynchronize(h->stream), "get_state sync");
    });
}

extern "C" int spn_tri_get_flow(spn_tri *h, float *dv2, float *dv4) {
    return guarded([&] {
        if (!h) throw Error(ErrorType::Argument, "null handle");
        check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
        if (dv2) check_cuda(cudaMemcpyAsync(dv2, h->dv2, h->n * sizeof(float), cudaMemcpyDeviceToHost, h->stream), "D2H");
        if (dv4)
            check_cuda(cudaMemcpyAsync(dv4, h->dv4, size_t(h->vsize()) * sizeof(float), cudaMemcpyDeviceToHost, h->stream),
                       "D2H");
        check_cuda(cudaStreamSynchronize(h->stream), "get_flow sync");
    });
}

extern "C" int spn_tri_compute_step(spn_tri *h) {
    return guarded([&] {
        if (!h) throw Error(ErrorType::Argument, "null handle");
        check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
        check_cuda(cudaMemsetAsync(h->work_counter, 0, 3 * sizeof(int), h->stream), "memset counters and status");
        const TriArgs a = h->args();
        tri_self_energy_kernel<<<h->n, 128, 0, h->stream>>>(a);
        check_cuda(cudaGetLastError(), "self-energy launch");
        tri_node_table_kernel<<<h->n, kNodeThreads, 0, h->stream>>>(h->node_args());
        check_cuda(cudaGetLastError(), "node table launch");
        const auto fn = vertex_kernel(h);
        fn<<<h->grid, kThreads, vertex_smem(h), h->stream>>>(a);
        if (h->prod_scratch) {
            check_cuda(cudaGetLastError(), "vertex flow launch");
            const size_t smem = lat_smem(h->nl).total;
            tri_lattice_kernel<<<h->prod_ctas, kLatThreads, smem, h->stream>>>(a);
        }
        check_cuda(cudaGetLastError(), "vertex flow launch");
    });
}

extern "C" int spn_tri_finalize_step(spn_tri *h, float new_cutoff) {
    return guarded([&] {
        if (!h) throw Error(ErrorType::Argument, "null handle");
        check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
        const float step = new_cutoff - h->cutoff;
        tri_euler_kernel<<<1, 64, 0, h->stream>>>(h->v2, h->dv2, h->n, step);
        tri_euler_kernel<<<copy_grid(h->vsize()), 256, 0, h->stream>>>(h->v4, h->dv4, h->vsize(), step);
        check_cuda(cudaGetLastError(), "euler launch");
        h->cutoff = new_cutoff;
    });
}

extern "C" int spn_tri_measure_correlation(spn_tri *h, float *corr, float *chi) {
    return guarded([&] {
        if (!h) throw Error(ErrorType::Argument, "null handle");
        check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
        launch_correlation(h);
        const size_t n = size_t(kCorrOut) * h->n_corr;
        const float *v = h->results.fetch(h->corr_out, n + 16 * h->nl, h->stream);
        if (corr) std::copy(v, v + n, corr);
        if (chi) std::copy(v + n, v + n + 16 * h->nl, chi);
    });
}

extern "C" int spn_tri_scratch(int n_freq, int n_sites, int n_ctas, long long free_bytes, int *ctas, long long *bytes) {
    return guarded([&] {
        if (n_freq < 2 || n_freq > kMaxFreq || n_sites < 1 || n_sites > kMaxSites || n_ctas < 1 || free_bytes < 0 || !ctas || !bytes)
            throw Error(ErrorType::Argument, "spn_tri_scratch: bad argument");
        *ctas = 0;
        *bytes = 0;
        if (!use_products(n_sites)) return;
        *ctas = scratch_ctas(n_ctas, lat_scratch_bytes(2 * n_freq + 8), [&](size_t want) {
            if (want > size_t(free_bytes)) return false;
            *bytes = (long long)want;
            return true;
        });
        if (!*ctas) throw Error(ErrorType::Cuda, "alloc operand scratch: out of memory");
    });
}

extern "C" int spn_tri_is_diverged(spn_tri *h, int *diverged) {
    return guarded([&] {
        if (!h || !diverged) throw Error(ErrorType::Argument, "null argument");
        check_cuda(cudaSetDevice(h->device), "cudaSetDevice");
        const unsigned st = *h->results.fetch(h->status, 1, h->stream);
        if (st & kStatusNodeOverflow) throw Error(ErrorType::Device, "loop-frequency node table overflow");
        if (st & kStatusProductTimeout) throw Error(ErrorType::Device, "a tensor-core product of the vertex flow did not complete");
        *diverged = (st & kStatusNaN) ? 1 : 0;
    });
}

extern "C" int spn_tri_vertex_probe(const float *pos, int n, int n_sites, const float *v4, int rid12, int rid21,
                                    int perm12, int perm21, float s, float t, float u, int channel, int local,
                                    float *value) {
    return guarded([&] {
        cuh::check_mesh(pos, n, kMaxFreq);
        if (n_sites < 1 || n_sites > kMaxSites || !v4 || !value || rid12 < 0 || rid12 >= n_sites || rid21 < 0 ||
            rid21 >= n_sites || perm12 < 0 || perm12 > 5 || perm21 < 0 || perm21 > 5 || channel < -1 || channel > 3 ||
            (channel < 0 && (local || perm12 || perm21)))
            throw Error(ErrorType::Argument, "spn_tri_vertex_probe: bad argument");
        const int nl = n_sites;
        if (channel < 0) {
            for (int c = 0; c < 16; ++c) value[c] = tri_value_none(pos, n, nl, v4, c >> 2, c & 3, rid12, rid21, s, t, u);
            return;
        }
        if (channel == 3) {
            TAB8 ab;
            tri_access8(pos, n, nl, s, t, u, ab);
            const bool ex = ab.fl & kFlExch;
            for (int c = 0; c < 16; ++c)
                value[c] = local ? tri_local(v4, nl, ab, c >> 2, c & 3)
                                 : tri_bundle(v4, nl, ab, c, ex ? rid21 : rid12, ex ? perm21 : perm12);
            return;
        }
        // the channel's own frequency is a mesh value; the two others are interpolated in the
        // order tri_access4i takes them (t, u for S; s, u for T; s, t for U)
        const MeshSearch<float> m{pos, n};
        const float own[3] = {s, t, u};
        const int e = cuh::mesh_index_of(pos, n, own[channel]);
        const Interp<float> ia = interp_abs(m, channel == 0 ? t : s), ib = interp_abs(m, channel == 2 ? t : u);
        TAB4 ab;
        if (channel == 0) tri_access4i<kS>(n, nl, s, t, u, e, ia, ib, ab);
        else if (channel == 1) tri_access4i<kT>(n, nl, s, t, u, e, ia, ib, ab);
        else tri_access4i<kU>(n, nl, s, t, u, e, ia, ib, ab);
        if (local) {
            for (int c = 0; c < 16; ++c) value[c] = tri_local(v4, nl, ab, c >> 2, c & 3);
            return;
        }
        // the vertex kernel's slab gather, every site of the table standing for the probed pair
        std::vector<int> goff(32 * size_t(nl));
        for (int i = 0; i < 32 * nl; ++i) {
            const int ex = i / (16 * nl), c = (i / nl) & 15;
            goff[i] = gather_offset(ex, c, nl, ex ? rid21 : rid12, ex ? perm21 : perm12);
        }
        std::vector<float> S(16 * size_t(nl));
        gather_slab(v4, ab, goff.data(), nl, 0, S.data());
        for (int c = 0; c < 16; ++c) value[c] = S[size_t(c) * nl];
    });
}
