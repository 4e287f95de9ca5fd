// Device bodies of the SU(2) flow kernels besides the vertex flow: self-energy flow, loop-
// frequency node tables, correlation measurement and the Euler update.  The single-flow
// kernels (su2_flow.cu) and the batched kernels (su2_batch.cu) call the same bodies, so a
// flow's numbers do not depend on whether it runs alone or in a batch.
#pragma once
#include "su2_common.cuh"
#include "su2_device.cuh"

namespace spn {
namespace dev {

constexpr double kPiD = 3.14159265358979323846;
constexpr int kCorrWarps = 16;  // warps of a correlation block
constexpr int kCorrThreads = 32 * kCorrWarps;
constexpr int kNodeThreads = 128;  // threads of a node-table block

// ------------------------------------------------------------------------------------
// 1. self-energy flow
// ------------------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ void self_energy_body(const FlowArgsT<T> &a, int blk) {
    __shared__ T pos[kMaxFreq];
    __shared__ double red[4];
    __shared__ T onsite[4];
    for (int i = threadIdx.x; i < a.n; i += blockDim.x) pos[i] = a.freq[i];
    __syncthreads();
    const int i = blk;
    const T w = pos[i], L = T(a.cutoff);
    const T wpl = w + L, wml = w - L;
    const PairedState<T> st{a.sd};
    if (threadIdx.x < 4) {  // spin, density at (w + L, w - L) and exchanged
        const int k = threadIdx.x;
        const T s = (k & 1) ? wml : wpl, t = (k & 1) ? wpl : wml;
        onsite[k] = value_none(pos, a.n, a.nl, st, k >= 2, 0, 0, s, t, T(0));
    }
    double part = 0.0;
    for (int j = threadIdx.x; j < a.n_range; j += blockDim.x) {
        const int r12 = a.range_rid[j], r21 = a.range_inv[j];
        T x1 = value_none(pos, a.n, a.nl, st, true, r12, r21, wpl, T(0), wml);
        T x2 = value_none(pos, a.n, a.nl, st, true, r12, r21, wml, T(0), wpl);
        part += double(x1) - double(x2);
    }
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int k = 0; k < int(blockDim.x >> 5); ++k) sum += red[k];
        double val = -4.0 * double(a.spin) * sum;
        val += 0.75 * (double(onsite[0]) - double(onsite[1]));
        val += (double(onsite[2]) - double(onsite[3]));
        const double sig = a.fp64_sigma ? odd_interp(pos, a.n, a.v2d, L) : odd_interp(pos, a.n, a.v2, L);
        val /= (2.0 * kPiD * (double(L) + sig));
        T out = T(val);
        a.dv2[i] = out;
        if (a.fp64_sigma) a.dv2d[i] = val;
        if (isnan(out)) atomicOr(a.status, kStatusNaN);
    }
}

// ------------------------------------------------------------------------------------
// 2. loop-frequency node tables
// ------------------------------------------------------------------------------------
// Of transfer frequency x = pos[xi] at cutoff L: the conventional nodes (SU2FrgCore.cpp:351-371: L, and -L if x > 2 L) and the rules of the
// Katanin contribution (SU2FrgCore.cpp:374-424), cnt[] nodes each.
template <class T>
SPN_HDI int node_rules(const T *pos, int n, int xi, T L, QuadRule<T> (&r)[3], int (&cnt)[3]) {
    const T x = pos[xi];
    cnt[0] = cnt[1] = cnt[2] = 0;
    if (-(x + L) > -pos[n - 1]) r[0] = rule_right(pos, n, -(x + L)), cnt[0] = r[0].count;
    if (x - L > L) r[1] = rule_both(pos, n, L - x, -L), cnt[1] = r[1].count;
    if (L < pos[n - 1]) r[2] = rule_left(pos, n, L), cnt[2] = r[2].count;
    return x > T(2) * L ? 2 : 1;
}

// One block per transfer frequency x, one thread per node.  A thread that walked a frequency's list
// alone (2N + 8 nodes of three FP64 reads and a division each, at 2 FP64 FMAs per clock and SM) took
// 150 us at N = 32 and 230 us at N = 64; the nodes side by side take 10 us.
template <class T>
__device__ __forceinline__ void node_table_body(const FlowArgsT<T> &a, int xi) {
    __shared__ T pos[kMaxFreq];
    for (int i = threadIdx.x; i < a.n; i += blockDim.x) pos[i] = a.freq[i];
    __syncthreads();
    if (xi >= a.n) return;
    const int n = a.n;
    const T x = pos[xi], L = T(a.cutoff);
    T *wp_out = a.node_wp + size_t(xi) * a.max_nodes;
    T *c_out = a.node_c + size_t(xi) * a.max_nodes;
    auto sig = [&](T w) { return a.fp64_sigma ? odd_interp(pos, n, a.v2d, w) : odd_interp(pos, n, a.v2, w); };
    auto dsig = [&](T w) { return a.fp64_sigma ? odd_interp(pos, n, a.dv2d, w) : odd_interp(pos, n, a.dv2, w); };
    auto p = [&](T w1, T w2) { return 1.0 / ((double(w1) + sig(w1)) * (double(w2) + sig(w2))); };
    auto pk = [&](T w1, T w2) {
        double d1 = double(w1) + sig(w1);
        return dsig(w1) / (d1 * d1 * (double(w2) + sig(w2)));
    };
    QuadRule<T> r[3];
    int cnt[3];
    const int conv = node_rules(pos, n, xi, L, r, cnt);
    const int total = conv + cnt[0] + cnt[1] + cnt[2];
    for (int k = threadIdx.x; k < min(total, a.max_nodes); k += blockDim.x) {
        T wp;
        double c;
        if (k < conv) {
            wp = k == 0 ? L : -L;
            c = p(L, k == 0 ? L + x : L - x);
        } else {
            int q = k - conv;
            double weight;
            if (q < cnt[0]) r[0].node(q, wp, weight);
            else if ((q -= cnt[0]) < cnt[1]) r[1].node(q, wp, weight);
            else r[2].node(q - cnt[1], wp, weight);
            c = weight * pk(wp, x + wp);
        }
        wp_out[k] = wp;
        c_out[k] = T(c);
    }
    if (threadIdx.x == 0) {
        a.node_cnt[xi] = min(total, a.max_nodes);
        if (total > a.max_nodes) atomicOr(a.status, kStatusNodeOverflow);
    }
}

// ------------------------------------------------------------------------------------
// Euler update of one element, x + step * dx, rounded like the reference (product, then sum;
// SU2FrgCore.cpp:111-137)
// ------------------------------------------------------------------------------------
__device__ __forceinline__ float euler_update(float x, float dx, float step) { return __fadd_rn(x, __fmul_rn(step, dx)); }
// FP64 self-energy (SPN_SU2_FP64_SELF_ENERGY) and the FP64 flow: the same update in double.
__device__ __forceinline__ double euler_update_f64(double x, double dx, double step) {
    return __dadd_rn(x, __dmul_rn(step, dx));
}

// ------------------------------------------------------------------------------------
// correlation measurement (nu = 0), SU2MeasurementCorrelation.cpp:77-177
// ------------------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ double corr_sigma(const CorrArgsT<T> &a, const T *pos, T w) {
    return a.v2d ? odd_interp(pos, a.n, a.v2d, w) : odd_interp(pos, a.n, a.v2, w);
}

constexpr int kMaxCorrNodes = 2 * kMaxFreq + 8;

// Loop-frequency nodes of the measurement's trapezoid rules at nu = 0 (outer and inner
// integrals use the same ranges): (-inf, -cutoff] and [cutoff, inf).  All threads of the block
// call it with shared arrays; returns the node count.  Also the squared propagator of each node,
// g = 1 / (w + Sigma(w))^2, from sigma(w).
template <class T, class Sigma>
__device__ __forceinline__ int corr_nodes(const T *pos, int n, T cut, T *wp, double *weight, double *g, Sigma &&sigma) {
    QuadRule<T> r[2];
    int cnt[2] = {0, 0};
    if (-(T(0) + cut) > -pos[n - 1]) r[0] = rule_right(pos, n, -cut - T(0)), cnt[0] = r[0].count;
    if (cut < pos[n - 1]) r[1] = rule_left(pos, n, cut), cnt[1] = r[1].count;
    for (int k = threadIdx.x; k < cnt[0] + cnt[1]; k += blockDim.x) {
        T w;
        double q;
        if (k < cnt[0]) r[0].node(k, w, q);
        else r[1].node(k - cnt[0], w, q);
        const double d = double(w) + sigma(w);
        wp[k] = w;
        weight[k] = q;
        g[k] = 1.0 / (d * d);
    }
    __syncthreads();
    return cnt[0] + cnt[1];
}

// Sums of `cols` columns of a matrix with `rows` rows over the rows, by the whole block: column e of
// row i is value(i, e).  red: max(cols, blockDim.x) doubles of shared memory; the sums are in
// red[0 .. cols) when it returns.  A column is cut into about as many slices as each has rows: the threads add
// rows / slices values and then one of them `slices` (with a slice for every thread that 4 sites' columns leave, 64 of them
// for 10 rows, a measurement took 9 us longer than the sums one after the other).
template <class F>
__device__ __forceinline__ void column_sums(int rows, int cols, double *red, F &&value) {
    const int slices = max(1, min(int(blockDim.x) / cols, int(ceilf(sqrtf(float(rows))))));
    __syncthreads();
    if (slices == 1) {
        for (int e = threadIdx.x; e < cols; e += blockDim.x) {
            double s = 0.0;
            for (int i = 0; i < rows; ++i) s += value(i, e);
            red[e] = s;
        }
        __syncthreads();
        return;
    }
    const int sl = threadIdx.x / cols, e = threadIdx.x - sl * cols;
    double s = 0.0;
    if (sl < slices)
        for (int i = sl; i < rows; i += slices) s += value(i, e);
    if (sl < slices) red[sl * cols + e] = s;
    __syncthreads();
    if (sl == 0) {
        for (int q = 1; q < slices; ++q) s += red[q * cols + e];
        red[e] = s;
    }
    __syncthreads();
}

// The measurement is linear in the vertex, so the inner integral of one outer node is, per site,
// sum over nodes of g * (interpolated vertex), with the outer node's propagator, the spin factors and the
// on-site (egg) diagram, a sum of its own, applied once.  Per node and lane that leaves two
// conversions and two FMAs in FP64 (GB300: 2 FP64 FMAs per clock and SM); with the propagators
// divided out per node in every lane the kernel took 69 us (cubic r6, N = 64), now 18; the final
// kernel, a thread per site walking all nodes, 60 to 120 us, now 10.
// `st`: the state (PairedState of a flow, or SplitState of an allocation-free call).
template <int SPT, class T, class View>
__device__ __forceinline__ void corr_inner_body(const CorrArgsT<T> &a, const View &st, int blk) {
    __shared__ T pos[kMaxFreq];
    __shared__ T nwp[kMaxCorrNodes];
    __shared__ double nw[kMaxCorrNodes], ng[kMaxCorrNodes];
    __shared__ double red[kCorrWarps][2][32 * SPT];
    __shared__ double egg[kCorrWarps][2];
    for (int i = threadIdx.x; i < a.n; i += blockDim.x) pos[i] = a.freq[i];
    __syncthreads();
    const int ncnt = corr_nodes(pos, a.n, T(a.cutoff), nwp, nw, ng, [&](T x) { return corr_sigma(a, pos, x); });
    const int ia = blk;
    if (ia >= ncnt) return;
    const T w = nwp[ia];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int W = (SPT == 1) ? a.wsite : 32;
    const int G = 32 / W;
    const int g = lane / W, jl = lane - g * W;
    const int nl = a.nl;
    int site[SPT], isite[SPT];
    bool valid[SPT];
    for (int k = 0; k < SPT; ++k) {
        const int j = jl + k * W;
        valid[k] = j < nl;
        site[k] = valid[k] ? a.sites[j] : 0;
        isite[k] = valid[k] ? a.inv_sites[j] : 0;
    }
    // on-site diagram, a thread per node, from the last warp on: the first ones have nodes of the loop below
    double es = 0.0, ed = 0.0;
    for (int b = blockDim.x - 1 - threadIdx.x; b < ncnt; b += blockDim.x) {
        const T wp = nwp[b];
        const double vs = value_none(pos, a.n, nl, st, false, 0, 0, w + wp + T(0), w - wp, T(0));
        const double vd = value_none(pos, a.n, nl, st, true, 0, 0, w + wp + T(0), w - wp, T(0));
        const double cw = nw[b] * ng[b];
        es += cw * (-vs / 4.0 + vd);
        ed += cw * (3.0 * vs + 4.0 * vd);
    }
    for (int o = 16; o > 0; o >>= 1) {
        es += __shfl_xor_sync(0xffffffffu, es, o);
        ed += __shfl_xor_sync(0xffffffffu, ed, o);
    }
    if (lane == 0) {
        egg[warp][0] = es;
        egg[warp][1] = ed;
    }
    double acc_s[SPT], acc_d[SPT];
    for (int k = 0; k < SPT; ++k) acc_s[k] = acc_d[k] = 0.0;
    const int groups = kCorrWarps * G;
    const int gid = warp * G + g;
    for (int b = gid; b < ncnt; b += groups) {
        const T wp = nwp[b];
        AB8T<T> ab;
        access8(pos, a.n, nl, w + wp + T(0), T(0), w - wp, ab);
        const double cw = nw[b] * ng[b];
        for (int k = 0; k < SPT; ++k) {
            const int site_k = ab.exch ? isite[k] : site[k];
            T gs = T(0), gd = T(0);
            for (int q = 0; q < 8; ++q) {
                const pair_t<T> p = st.both(ab.off[q] + site_k);
                gs += ab.w[q] * p.x;
                gd += ab.sw[q] * p.y;
            }
            if (valid[k]) {
                acc_s[k] += cw * double(gs);
                acc_d[k] += cw * double(gd);
            }
        }
    }
    for (int k = 0; k < SPT; ++k) {
        for (int o = W; o < 32; o <<= 1) {
            acc_s[k] += __shfl_xor_sync(0xffffffffu, acc_s[k], o);
            acc_d[k] += __shfl_xor_sync(0xffffffffu, acc_d[k], o);
        }
        if (g == 0) {
            red[warp][0][jl + k * W] = acc_s[k];
            red[warp][1][jl + k * W] = acc_d[k];
        }
    }
    __syncthreads();
    const double S = a.spin, norm = ng[ia] / (4.0 * kPiD * kPiD);
    for (int j = threadIdx.x; j < nl; j += blockDim.x) {
        double s = 0.0, d = 0.0;
        for (int q = 0; q < kCorrWarps; ++q) {
            s += red[q][0][j];
            d += red[q][1][j];
        }
        s *= -S * S;
        d *= -16.0 * S * S;
        if (j == 0)
            for (int q = 0; q < kCorrWarps; ++q) {
                s += S * egg[q][0];
                d += S * egg[q][1];
            }
        a.partial[(size_t(ia) * 2 + 0) * nl + j] = s * norm;
        a.partial[(size_t(ia) * 2 + 1) * nl + j] = d * norm;
    }
}

// Outer integral, on-site propagator term and scatter.  Shared memory: corr_final_smem.
constexpr size_t corr_final_smem(int cols) { return sizeof(double) * size_t(cols > kCorrThreads ? cols : kCorrThreads); }

template <class T>
__device__ __forceinline__ void corr_final_body(const CorrArgsT<T> &a) {
    __shared__ T pos[kMaxFreq];
    __shared__ T nwp[kMaxCorrNodes];
    __shared__ double nw[kMaxCorrNodes], ng[kMaxCorrNodes];
    __shared__ double bubble;
    extern __shared__ double chi[];  // [2][nl] and the reduction's slices
    for (int i = threadIdx.x; i < a.n; i += blockDim.x) pos[i] = a.freq[i];
    __syncthreads();
    const int ncnt = corr_nodes(pos, a.n, T(a.cutoff), nwp, nw, ng, [&](T x) { return corr_sigma(a, pos, x); });
    if (threadIdx.x < 32) {  // the on-site propagator term
        double s = 0.0;
        for (int k = threadIdx.x; k < ncnt; k += 32) s += nw[k] * ng[k];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) bubble = s;
    }
    const double S = a.spin;
    const int nl = a.nl;
    column_sums(ncnt, 2 * nl, chi, [&](int ia, int e) { return nw[ia] * a.partial[size_t(ia) * 2 * nl + e]; });
    if (threadIdx.x == 0) {
        chi[0] += S / (2.0 * kPiD) * bubble;
        chi[nl] += 2.0 * S / kPiD * bubble;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 2 * nl; e += blockDim.x) a.out[2 * a.n_corr + e] = T(chi[e]);
    for (int q = threadIdx.x; q < a.n_corr; q += blockDim.x) {
        const int r = a.corr_rid[q];
        // an entry outside [0, nl) (possible only with caller-owned device tables) reads
        // nothing and yields NaN
        double zz = __longlong_as_double(0x7ff8000000000000LL), dd = zz;
        if (r >= 0 && r < a.nl) {
            zz = chi[r];
            dd = chi[a.nl + r];
        }
        a.out[q] = T(zz);
        a.out[a.n_corr + q] = T(dd);
    }
}


}  // namespace dev
}  // namespace spn
