// Network-side kernels: branch admittances, Ybus assembly, the fused
// measurement evaluation (h(x), residual, weights, Jacobian values), the
// gain right-hand side, state update / convergence and the result pass.
#include "kernels.cuh"
#include "round32.h"

#include <cfloat>

namespace sle_gb300 {
namespace {

constexpr double kEps = 1e-12;   // SLE_REAL_EPSILON of the FP64 build (sle_types.cuh:62)
constexpr int kBlock = 256;

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// Deterministic block sum (fixed tree), result valid in thread 0.
__device__ double block_sum(double v, double* sh) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    v = (threadIdx.x < (blockDim.x >> 5)) ? sh[lane] : 0.0;
    if (wid == 0) v = warp_sum(v);
    __syncthreads();
    return v;
}
__device__ double block_max(double v, double* sh) {
    v = warp_max(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    v = (threadIdx.x < (blockDim.x >> 5)) ? sh[lane] : 0.0;
    if (wid == 0) v = warp_max(v);
    __syncthreads();
    return v;
}

// a1: per-branch series admittance and charging split
// (network_model.cu:595-612 / sparse_matrix.cu:321-355).
__global__ void k_admittance(DevNet net) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= net.n_branch) return;
    const double r = net.br_r[k], x = net.br_x[k], bt = net.br_bch[k], a = net.br_tap[k];
    double den = r * r + x * x;
    if (den < kEps) den = kEps;
    net.br_g[k] = r / den;
    net.br_b[k] = -x / den;
    net.br_bsf[k] = bt / (2.0 * a * a);
    net.br_bst[k] = bt / 2.0;
    const double A = fmax(a, kEps), ia = 1.0 / A;
    net.br_itap[k] = ia;
    net.br_itap2[k] = 1.0 / (A * A);
}

// a2: Ybus values on the canonical pattern, one thread per bus row; the
// diagonal accumulates the row's branch contributions in entry order
// (sparse_matrix.cu:410-492 without floating-point atomics).
__global__ void k_ybus(DevNet net) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= net.n_bus) return;
    const int e0 = net.y_ptr[i], e1 = net.y_ptr[i + 1];
    double dg = 0.0, db = 0.0;
    for (int e = e0 + 1; e < e1; ++e) {
        const int src = net.y_src[e];
        const int k = src >> 1, end = src & 1;
        // an open branch in the pattern (batch patterns keep every branch)
        // contributes nothing
        const double on = net.br_closed[k] ? 1.0 : 0.0;
        const double g = net.br_g[k] * on, b = net.br_b[k] * on;
        const double a = fmax(net.br_tap[k], kEps);
        const double phi = net.br_shift[k];
        double sph, cph;
        sincos(phi, &sph, &cph);
        const double inv_a = 1.0 / a;
        if (end == 0) {  // row = from bus: Y_ij = -(g+jb) e^{-j phi} / a
            net.y_g[e] = -(g * cph + b * sph) * inv_a;
            net.y_b[e] = -(-g * sph + b * cph) * inv_a;
            dg += g / (a * a);
            db += b / (a * a) + net.br_bsf[k] * on;
        } else {         // row = to bus: Y_ji = -(g+jb) e^{+j phi} / a
            net.y_g[e] = -(g * cph - b * sph) * inv_a;
            net.y_b[e] = -(g * sph + b * cph) * inv_a;
            dg += g;
            db += b + net.br_bst[k] * on;
        }
    }
    net.y_g[e0] = dg;
    net.y_b[e0] = db;
}

// A flow row's value and derivatives by the row's own end (o) and the other (x).
struct FlowTerms {
    double val;
    double dto, dvo, dvx;  // theta_o (theta_x has the opposite sign), V_o, V_x
};

// What the P and Q flow at one end of branch k share (a4 + a8 flow rows).
// With s the sine of the angle from that end, both rows are
//   h = V_o^2 q - V_o V_x inv A,  dh/dtheta_o = V_o V_x inv B
// with (A, B) = (g c + b s, g s - b c) for P and (g s - b c, -(g c + b s)) for
// Q, q the end's own admittance (over the tap squared at the from end).
//
// An SM finishes one FP64 warp instruction in 19 cycles whatever lanes it has,
// and the evaluation is bound by that.  One sequence serves the four kinds of
// flow row and both kinds of injection (selects on the integer pipe instead of
// branches, which a warp of mixed rows runs one after the other); sums that few
// rows need are behind calls, and the H entries are rounded to FP32 on the
// integer pipe (round32.h).  Products are rounded and fused as in the formulas
// one by one, so the bits are theirs: the mixed pipeline's estimates of stiff
// grids move by up to 3e-8 when an ulp of H does.  The evaluation of 512 grids
// (pairs) went from 311 to 243 us, of 200k buses from 153 to 122, of 20k
// (rows) from 39 to 33.
struct FlowEnd {
    double Vo, Vx, gc, gs;  // g c + b s, g s - b c
    double inv, w;          // 1 / a; 1 / a^2 at the from end, 1 at the to end
};

__device__ __forceinline__ double flip(double v, bool neg) {  // the sign bit, off the FP64 pipe
    return __hiloint2double(__double2hiint(v) ^ (neg ? static_cast<int>(0x80000000) : 0), __double2loint(v));
}
// A sum that few lanes need.  A call, so that it is behind a branch: an FP64
// instruction takes its pipe's time with every lane off as well.
__device__ __noinline__ double add_apart(double a, double b) { return a + b; }
__device__ __noinline__ double fma_apart(double a, double b, double c) { return fma(a, b, c); }
// v * 0.0: a zero of v's sign, NaN for an infinity or NaN; off the FP64 pipe
__device__ __forceinline__ double times_zero(double v) {
    const int hi = __double2hiint(v);
    return __hiloint2double((hi & 0x7ff00000) == 0x7ff00000 ? 0x7ff80000 : hi & static_cast<int>(0x80000000), 0);
}
// v == 0, off the FP64 pipe
__device__ __forceinline__ bool is_zero(double v) { return ((__double2hiint(v) & 0x7fffffff) | __double2loint(v)) == 0; }

// s, c: sin, cos of theta_i - theta_j - shift.  1 / a and 1 / a^2 of the tap a
// (clamped as the reference clamps it) are computed once per branch.
__device__ __forceinline__ FlowEnd flow_end(const DevNet& net, const double* v, int k, bool to_end, double s, double c) {
    const double Vi = v[net.br_from[k]], Vj = v[net.br_to[k]];
    const double g = net.br_g[k], b = net.br_b[k], inv = net.br_itap[k], ia2 = net.br_itap2[k];
    s = flip(s, to_end);
    FlowEnd E;
    E.Vo = to_end ? Vj : Vi;
    E.Vx = to_end ? Vi : Vj;
    E.gc = g * c + b * s;
    E.gs = g * s - b * c;
    E.inv = inv;
    E.w = to_end ? 1.0 : ia2;
    return E;
}

template <bool exact>
__device__ __forceinline__ FlowTerms flow_row(const DevNet& net, const FlowEnd& E, int k, bool is_q, bool to_end) {
    const double g = net.br_g[k], b = net.br_b[k];
    const double q0 = is_q ? -(b + (to_end ? net.br_bst[k] : net.br_bsf[k])) : g;
    const double A = is_q ? E.gs : E.gc, B = is_q ? flip(E.gc, true) : E.gs;
    const double vv = E.Vo * E.Vx * E.inv;
    FlowTerms f;
    // (which product of a difference is rounded follows the formulas' signs)
    const bool second = is_q && to_end;
    const double s2 = E.Vo * E.Vo * E.w;
    f.val = fma(second ? -vv : s2, second ? A : q0, second ? s2 * q0 : -(vv * A));
    const double qd = exact || !is_q ? q0 : -b;  // the reference leaves the charging out of dQ/dV
    const double t1 = 2.0 * E.Vo * (is_q ? qd : E.w), t2 = is_q ? E.w : qd, xi = E.Vx * E.inv;
    f.dvo = fma(second ? -xi : t1, second ? A : t2, second ? t1 * t2 : -(xi * A));
    f.dvx = flip(E.Vo * E.inv * A, true);
    f.dto = vv * B;
    // the reference flips the sign of dP/dtheta at the to end
    if (!exact && to_end && !is_q) f.dto = flip(f.dto, true);
    const bool closed = net.br_closed[k] != 0;
    f.val = closed ? f.val : times_zero(f.val);
    if (exact) {
        f.dto = closed ? f.dto : times_zero(f.dto);
        f.dvo = closed ? f.dvo : times_zero(f.dvo);
        f.dvx = closed ? f.dvx : times_zero(f.dvx);
    }
    return f;
}

// sin and cos of theta_i - theta_j from the buses' (cos, sin): four FMAs in
// place of an FP64 sincos per use (the evaluation meets each angle difference
// in up to eight rows); absolute error a few ulps of 1.
__device__ __forceinline__ void angle_diff(const double2 a, const double2 b, double* s, double* c) {
    *c = a.x * b.x + a.y * b.y;
    *s = a.y * b.x - a.x * b.y;
}

// sin and cos of theta_i - theta_j - shift of branch k.
__device__ __forceinline__ void branch_angle(const DevNet& net, const double2* cs, int k, double* s, double* c) {
    angle_diff(cs[net.br_from[k]], cs[net.br_to[k]], s, c);
    const double phi = net.br_shift[k];
    if (!is_zero(phi)) {
        double sp, cp;
        sincos(phi, &sp, &cp);
        const double c2 = *c * cp + *s * sp;
        *s = *s * cp - *c * sp;
        *c = c2;
    }
}

// cos and sin of every bus angle of the grids being evaluated.
__global__ void k_bus_trig(DevNet net, DevWork w, SolveParams sp) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= net.n_bus) return;
    if (net.bus_grid) {
        const uint32_t gf = w.grid_flags[net.bus_grid[i]];
        if ((gf & sp.skip_flags) || (gf & sp.need_flags) != sp.need_flags) return;
    }
    double s, c;
    sincos(w.th[i], &s, &c);
    w.bus_cs[i] = make_double2(c, s);
}

// Adds a flow row's derivatives to its (zeroed) H row; fpos: positions of
// theta_i, V_i, theta_j, V_j, i the from bus (0xFF: none).  The four are
// distinct columns, so they are stored, unless the branch ends where it starts.
__device__ __forceinline__ void put_flow(double* hrow, int fpos, bool to_end, const FlowTerms& f) {
    const double dtx = flip(f.dto, true);
    const double d[4] = {to_end ? dtx : f.dto, to_end ? f.dvx : f.dvo, to_end ? f.dto : dtx, to_end ? f.dvo : f.dvx};
    const bool loop = ((fpos >> 8) & 0xFF) == ((fpos >> 24) & 0xFF);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        const int p = (fpos >> (8 * x)) & 0xFF;
        if (p == 0xFF) continue;
        hrow[p] = loop ? add_apart(hrow[p], d[x]) : d[x];
    }
}

// Current magnitude |S| / V at one end of branch k.
template <bool exact>
__device__ __forceinline__ FlowTerms current_row(const DevNet& net, const DevWork& w, int k, bool to_end) {
    double s, c;
    branch_angle(net, w.bus_cs, k, &s, &c);
    const FlowEnd E = flow_end(net, w.v, k, to_end, s, c);
    const FlowTerms P = flow_row<exact>(net, E, k, false, to_end), Q = flow_row<exact>(net, E, k, true, to_end);
    const double on = net.br_closed[k] ? 1.0 : 0.0;
    const double vs = fmax(E.Vo, kEps);
    const double S = sqrt(P.val * P.val + Q.val * Q.val);
    FlowTerms f;
    f.val = S / vs * on;
    if (!exact) {  // the reference reuses the P-flow derivatives
        f.dto = P.dto;
        f.dvo = P.dvo;
        f.dvx = P.dvx;
    } else {
        auto d = [&](double p, double q) { return (S > 0.0) ? (P.val * p + Q.val * q) / (S * vs) * on : 0.0; };
        f.dto = d(P.dto, Q.dto);
        f.dvo = d(P.dvo, Q.dvo);
        f.dvx = d(P.dvx, Q.dvx);
        if (E.Vo > kEps) f.dvo -= S / (vs * vs) * on;
    }
    return f;
}

// float(v) off the FP64 pipe where the result is a normal number.
__device__ __forceinline__ float to_f32(double v) {
    const uint32_t hi = static_cast<uint32_t>(__double2hiint(v)), lo = static_cast<uint32_t>(__double2loint(v));
    if (round32_takes(hi)) return __uint_as_float(round32_bits(hi, lo));
    return static_cast<float>(v);
}

// H entries of a warp's rows (a contiguous range of the CSR values) staged
// in shared memory by k_evaluate.
constexpr int kEvalSpan = 512;

// a3/a6/a7/a8/a9 fused, one thread per evaluation unit (one row, or a P row
// and its Q twin): h(x), the H row values, the residual, the (Huber) weight,
// the FP32 and weighted copies of the H row, and per-block partials of the
// objective.  A warp's 32 units cover a contiguous range of rows whenever
// the rows come in order (the usual case); their H entries are then built in
// shared memory and the warp writes the range out coalesced, skipping rows
// it does not evaluate.  Otherwise each thread writes its rows in place.
template <bool exact>
__global__ void __launch_bounds__(kBlock) k_evaluate_pairs(DevNet net, DevWork w, SolveParams sp) {
    __shared__ double sh[32];
    __shared__ double hs[kBlock / 32][kEvalSpan];
    __shared__ uint8_t hrow_id[kBlock / 32][kEvalSpan];  // row - lo of each entry; 0xFF = not evaluated
    __shared__ double wes[kBlock / 32][64];
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gidx = u >> 5;
    const int2 grp = (u - lane) < net.n_units ? net.ev_grp[gidx] : make_int2(-1, -1);
    const int hw0 = grp.x >= 0 ? net.h_ptr[grp.x] : 0;
    const int hw1 = grp.x >= 0 ? net.h_ptr[grp.y] : 0;
    const bool staged = grp.x >= 0 && hw1 - hw0 <= kEvalSpan && grp.y - grp.x <= 64;  // warp-uniform
    if (staged) {
        for (int x = lane; x < hw1 - hw0; x += 32) {
            hs[warp][x] = 0.0;
            hrow_id[warp][x] = 0xFF;
        }
        __syncwarp();
    }
    double obj = 0.0, hub = 0.0;
    const int2 un = u < net.n_units ? net.ev_unit[u] : make_int2(-1, -1);
    bool skip = un.x < 0;
    if (!skip && net.meas_grid) {
        const uint32_t gf = w.grid_flags[net.meas_grid[un.x]];
        skip = (gf & sp.skip_flags) || (gf & sp.need_flags) != sp.need_flags;
    }
    // the H row of row q: in the warp's staged range or in place (zeroed)
    auto row_of = [&](int q) -> double* {
        const int base = net.h_ptr[q], nh = net.h_ptr[q + 1] - base;
        if (staged) {
            for (int x = 0; x < nh; ++x) hrow_id[warp][base - hw0 + x] = static_cast<uint8_t>(q - grp.x);
            return &hs[warp][base - hw0];
        }
        double* hrow = w.hval + base;
        for (int x = 0; x < nh; ++x) hrow[x] = 0.0;
        return hrow;
    };
    // residual, weight, outputs and objective of row q with value hv
    auto finish = [&](int q, int kind, double hv, const double* hrow) {
        const int base = net.h_ptr[q], nh = net.h_ptr[q + 1] - base;
        if (sp.mixed && !staged)
            for (int x = 0; x < nh; ++x) w.hval32[base + x] = static_cast<float>(hrow[x]);
        double rr = 0.0, we = 0.0;
        if (kind != 5) {
            rr = w.z[q] - hv;
            const double wb = net.m_w[q];
            we = wb;
            if (sp.robust) {  // kernels.cu:634-671
                const double sg = net.m_sigma[q];
                const double rn = fabs(rr / sg);
                if (!(rn <= sp.huber_gamma)) we = sp.huber_gamma / (sg * fabs(rr) + kEps);
            }
            obj += wb * rr * rr;
            if (sp.huber_objective) {  // rho(u) = u^2 / 2 inside gamma, gamma |u| - gamma^2 / 2 outside
                const double uu = fabs(rr) / fmax(net.m_sigma[q], kEps);
                hub += (uu <= sp.huber_gamma) ? 0.5 * uu * uu
                                              : sp.huber_gamma * uu - 0.5 * sp.huber_gamma * sp.huber_gamma;
            }
        } else {
            hv = 0.0;
        }
        w.h[q] = hv;
        w.r[q] = rr;
        w.w_eff[q] = we;
        w.wr[q] = we * rr;
        // weighted H entries for the gain sums G_ij = sum (w h_a) h_b
        if (staged) {
            wes[warp][q - grp.x] = we;
        } else if (sp.mixed && w.hw32) {
            for (int x = 0; x < nh; ++x) w.hw32[base + x] = static_cast<float>(we * hrow[x]);
        } else if (!sp.mixed && w.hw) {
            for (int x = 0; x < nh; ++x) w.hw[base + x] = we * hrow[x];
        }
    };
    if (!skip) {
        const int qa = un.x, qb = un.y;
        const int kind = net.m_kind[qa];
        const int ty = net.m_type[qa];
        const int loc = net.m_loc[qa];
        if (kind == 0) {  // V_MAG
            double* hrow = row_of(qa);
            hrow[0] = 1.0;
            finish(qa, kind, w.v[loc], hrow);
        } else if (kind == 1) {  // V_ANGLE
            double* hrow = row_of(qa);
            if (net.h_ptr[qa + 1] > net.h_ptr[qa]) hrow[0] = 1.0;
            finish(qa, kind, w.th[loc], hrow);
        } else if (kind == 2) {  // P/Q injection or pseudo; with its twin when qb >= 0
            // slot 0: the P row, slot 1: the Q row (either may be absent)
            const bool a_is_q = (ty == 3 || ty == 8);
            const int qp = a_is_q ? qb : qa, qq = a_is_q ? qa : qb;
            double* hp = qp >= 0 ? row_of(qp) : nullptr;
            double* hq = qq >= 0 ? row_of(qq) : nullptr;
            const double Vi = w.v[loc];
            const double2 cs_i = w.bus_cs[loc];
            double hvp = 0.0, dVip = 0.0, dTip = 0.0, hvq = 0.0, dViq = 0.0, dTiq = 0.0;
            const int e0 = net.y_ptr[loc], e1 = net.y_ptr[loc + 1];
            {
                const double G = net.y_g[e0], B = net.y_b[e0];  // the diagonal comes first
                hvp = __dmul_rn(Vi * Vi, G);
                dVip = __dmul_rn(2.0 * Vi, G);
                hvq = __dmul_rn(Vi * Vi, -B);
                dViq = __dmul_rn(2.0 * Vi, -B);
                if (!exact) {
                    dTip = __dmul_rn(Vi * Vi, B);
                    dTiq = hvp;
                }
            }
            for (int e = e0 + 1; e < e1; ++e) {
                const int j = net.y_col[e];
                const double G = net.y_g[e], B = net.y_b[e];
                if (j == loc) {  // a branch that ends where it starts
                    hvp = fma_apart(Vi * Vi, G, hvp);
                    dVip = fma_apart(2.0 * Vi, G, dVip);
                    hvq = fma_apart(Vi * Vi, -B, hvq);
                    dViq = fma_apart(2.0 * Vi, -B, dViq);
                    if (!exact) {
                        dTip = fma_apart(Vi * Vi, B, dTip);
                        dTiq = fma_apart(Vi * Vi, G, dTiq);
                    }
                } else {
                    const double Vj = w.v[j];
                    double sn, cn;
                    angle_diff(cs_i, w.bus_cs[j], &sn, &cn);
                    const double gcbs = G * cn + B * sn, gsbc = G * sn - B * cn;
                    const int pt = net.y_hpos_t[e], pv = net.y_hpos_v[e];
                    if (hp) {
                        hvp += Vi * Vj * gcbs;
                        dVip += Vj * gcbs;
                        dTip -= Vi * Vj * gsbc;
                        if (pt >= 0) hp[pt] += Vi * Vj * gsbc;
                        hp[pv] += Vi * gcbs;
                    }
                    if (hq) {
                        hvq += Vi * Vj * gsbc;
                        dViq += Vj * gsbc;
                        dTiq += Vi * Vj * gcbs;
                        if (pt >= 0) hq[pt] += -Vi * Vj * gcbs;
                        hq[pv] += Vi * gsbc;
                    }
                }
            }
            const int pt = net.y_hpos_t[e0], pv = net.y_hpos_v[e0];
            if (hp) {
                if (pt >= 0) hp[pt] += dTip;
                hp[pv] += dVip;
                finish(qp, kind, hvp, hp);
            }
            if (hq) {
                if (pt >= 0) hq[pt] += dTiq;
                hq[pv] += dViq;
                finish(qq, kind, hvq, hq);
            }
        } else if (kind == 3) {  // P/Q flow; with its twin at the same end when qb >= 0
            const bool to_end = net.m_end[qa] != 0;
            const bool a_is_q = ty == 5;
            double sn, cn;
            branch_angle(net, w.bus_cs, loc, &sn, &cn);
            const FlowEnd E = flow_end(net, w.v, loc, to_end, sn, cn);
            double* ha = row_of(qa);
            const FlowTerms fa = flow_row<exact>(net, E, loc, a_is_q, to_end);
            put_flow(ha, net.m_fpos[qa], to_end, fa);
            finish(qa, kind, fa.val, ha);
            if (qb >= 0) {
                double* hb = row_of(qb);
                const FlowTerms fb = flow_row<exact>(net, E, loc, !a_is_q, to_end);
                put_flow(hb, net.m_fpos[qb], to_end, fb);
                finish(qb, kind, fb.val, hb);
            }
        } else if (kind == 4) {  // current magnitude
            double* hrow = row_of(qa);
            const bool to_end = net.m_end[qa] != 0;
            const FlowTerms f = current_row<exact>(net, w, loc, to_end);
            put_flow(hrow, net.m_fpos[qa], to_end, f);
            finish(qa, kind, f.val, hrow);
        } else {
            double* hrow = row_of(qa);
            finish(qa, kind, 0.0, hrow);
        }
    }
    if (staged) {
        __syncwarp();
        for (int x = lane; x < hw1 - hw0; x += 32) {
            const int r = hrow_id[warp][x];
            if (r == 0xFF) continue;
            const double v = hs[warp][x];
            w.hval[hw0 + x] = v;
            if (sp.mixed) {
                w.hval32[hw0 + x] = to_f32(v);
                if (w.hw32) w.hw32[hw0 + x] = to_f32(wes[warp][r] * v);
            } else if (w.hw) {
                w.hw[hw0 + x] = wes[warp][r] * v;
            }
        }
    }
    const double s = block_sum(obj, sh);
    if (threadIdx.x == 0) w.part[blockIdx.x] = s;
    if (sp.huber_objective) {
        __syncthreads();  // sh is reused
        const double hs2 = block_sum(hub, sh);
        if (threadIdx.x == 0) w.hpart[blockIdx.x] = hs2;
    }
}

// a3/a6/a7/a8/a9 fused, one thread per measurement row (the form for
// evaluations with no paired rows: twice the threads of k_evaluate_pairs,
// which a small grid needs to fill the GPU).

template <bool exact>
__global__ void __launch_bounds__(kBlock) k_evaluate_rows(DevNet net, DevWork w, SolveParams sp) {
    __shared__ double sh[32];
    // A warp's rows own the contiguous H range [hw0, hw1).  When it fits,
    // each row is built in shared memory and the warp writes the range out
    // coalesced (H in FP64, FP32 and weighted), skipping rows it did not
    // evaluate; otherwise each thread writes its own row in place.
    __shared__ double hs[kBlock / 32][kEvalSpan];
    __shared__ uint16_t hlane[kBlock / 32][kEvalSpan];
    __shared__ double wes[kBlock / 32][32];
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int qw0 = q - lane;
    const int hw0 = qw0 < net.n_meas ? net.h_ptr[qw0] : 0;
    const int hw1 = qw0 < net.n_meas ? net.h_ptr[min(qw0 + 32, net.n_meas)] : 0;
    const bool staged = hw1 - hw0 <= kEvalSpan;  // warp-uniform
    if (staged) {
        for (int x = lane; x < hw1 - hw0; x += 32) {
            hs[warp][x] = 0.0;
            hlane[warp][x] = 0xFFFF;  // not evaluated: left as it is
        }
        __syncwarp();
    }
    double obj = 0.0, hub = 0.0;
    bool skip = false;
    if (q < net.n_meas && net.meas_grid) {
        const uint32_t gf = w.grid_flags[net.meas_grid[q]];
        skip = (gf & sp.skip_flags) || (gf & sp.need_flags) != sp.need_flags;
    }
    if (q < net.n_meas && !skip) {
        const int kind = net.m_kind[q];
        const int ty = net.m_type[q];
        const int loc = net.m_loc[q];
        const int base = net.h_ptr[q];
        const int nh = net.h_ptr[q + 1] - base;
        double* hrow = staged ? &hs[warp][base - hw0] : w.hval + base;
        if (staged) {
            for (int x = 0; x < nh; ++x) hlane[warp][base - hw0 + x] = static_cast<uint16_t>(lane);
        } else {
            for (int x = 0; x < nh; ++x) hrow[x] = 0.0;
        }
        double hv = 0.0;
        if (kind == 0) {  // V_MAG
            hv = w.v[loc];
            hrow[0] = 1.0;
        } else if (kind == 1) {  // V_ANGLE
            hv = w.th[loc];
            if (nh > 0) hrow[0] = 1.0;
        } else if (kind == 2) {  // P/Q injection or pseudo
            const bool isq = (ty == 3 || ty == 8);
            const double Vi = w.v[loc];
            const double2 cs_i = w.bus_cs[loc];
            // One sequence for P and Q: (A, D) = (gcbs, gsbc) or (gsbc, -gcbs)
            double dVi = 0.0, dTi = 0.0;
            const int e0 = net.y_ptr[loc], e1 = net.y_ptr[loc + 1];
            {
                const double G = __ldg(net.y_g + e0), B = __ldg(net.y_b + e0);  // the diagonal comes first
                const double c = isq ? flip(B, true) : G;
                hv = __dmul_rn(Vi * Vi, c);
                dVi = __dmul_rn(2.0 * Vi, c);
                if (!exact) dTi = __dmul_rn(Vi * Vi, isq ? G : B);
            }
            for (int e = e0 + 1; e < e1; ++e) {
                const int j = __ldg(net.y_col + e);
                const double G = __ldg(net.y_g + e), B = __ldg(net.y_b + e);
                const double Vj = __ldg(w.v + j);
                const int pt = __ldg(net.y_hpos_t + e), pv = __ldg(net.y_hpos_v + e);
                if (j == loc) {  // a branch that ends where it starts
                    const double c = isq ? flip(B, true) : G;
                    hv = fma_apart(Vi * Vi, c, hv);
                    dVi = fma_apart(2.0 * Vi, c, dVi);
                    if (!exact) dTi = fma_apart(Vi * Vi, isq ? G : B, dTi);
                    continue;
                }
                double s, c;
                angle_diff(cs_i, __ldg(w.bus_cs + j), &s, &c);
                const double gcbs = G * c + B * s, gsbc = G * s - B * c;
                const double A = isq ? gsbc : gcbs, D = isq ? flip(gcbs, true) : gsbc;
                const double vv = Vi * Vj, p = __dmul_rn(vv, D);
                hv = __dadd_rn(hv, __dmul_rn(vv, A));
                dVi = fma(Vj, A, dVi);
                dTi = fma(isq ? vv : p, isq ? flip(D, true) : -1.0, dTi);
                if (pt >= 0) hrow[pt] += p;
                hrow[pv] += __dmul_rn(Vi, A);
            }
            const int pt = net.y_hpos_t[e0];
            if (pt >= 0) hrow[pt] += dTi;
            hrow[net.y_hpos_v[e0]] += dVi;
        } else if (kind == 3) {  // P/Q flow
            const bool to_end = net.m_end[q] != 0;
            double sn, cn;
            branch_angle(net, w.bus_cs, loc, &sn, &cn);
            const FlowTerms f = flow_row<exact>(net, flow_end(net, w.v, loc, to_end, sn, cn), loc, ty == 5, to_end);
            hv = f.val;
            put_flow(hrow, net.m_fpos[q], to_end, f);
        } else if (kind == 4) {  // current magnitude
            const bool to_end = net.m_end[q] != 0;
            const FlowTerms f = current_row<exact>(net, w, loc, to_end);
            hv = f.val;
            put_flow(hrow, net.m_fpos[q], to_end, f);
        }
        if (sp.mixed && !staged)
            for (int x = 0; x < nh; ++x) w.hval32[base + x] = static_cast<float>(hrow[x]);
        double rr = 0.0, we = 0.0;
        if (kind != 5) {
            rr = w.z[q] - hv;
            const double wb = net.m_w[q];
            we = wb;
            if (sp.robust) {  // kernels.cu:634-671
                const double sg = net.m_sigma[q];
                const double rn = fabs(rr / sg);
                if (!(rn <= sp.huber_gamma)) we = sp.huber_gamma / (sg * fabs(rr) + kEps);
            }
            obj = wb * rr * rr;
            if (sp.huber_objective) {  // rho(u) = u^2 / 2 inside gamma, gamma |u| - gamma^2 / 2 outside
                const double u = fabs(rr) / fmax(net.m_sigma[q], kEps);
                hub = (u <= sp.huber_gamma) ? 0.5 * u * u : sp.huber_gamma * u - 0.5 * sp.huber_gamma * sp.huber_gamma;
            }
        } else {
            hv = 0.0;
        }
        w.h[q] = hv;
        w.r[q] = rr;
        w.w_eff[q] = we;
        w.wr[q] = we * rr;
        // weighted H entries for the gain sums G_ij = sum (w h_a) h_b
        if (staged) {
            wes[warp][lane] = we;
        } else if (sp.mixed && w.hw32) {
            for (int x = 0; x < nh; ++x) w.hw32[base + x] = static_cast<float>(we * hrow[x]);
        } else if (!sp.mixed && w.hw) {
            for (int x = 0; x < nh; ++x) w.hw[base + x] = we * hrow[x];
        }
    }
    if (staged) {
        __syncwarp();
        for (int x = lane; x < hw1 - hw0; x += 32) {
            const int r = hlane[warp][x];
            if (r == 0xFFFF) continue;
            const double v = hs[warp][x];
            w.hval[hw0 + x] = v;
            if (sp.mixed) {
                w.hval32[hw0 + x] = to_f32(v);
                if (w.hw32) w.hw32[hw0 + x] = to_f32(wes[warp][r] * v);
            } else if (w.hw) {
                w.hw[hw0 + x] = wes[warp][r] * v;
            }
        }
    }
    const double s = block_sum(obj, sh);
    if (threadIdx.x == 0) w.part[blockIdx.x] = s;
    if (sp.huber_objective) {
        __syncthreads();  // sh is reused
        const double hs = block_sum(hub, sh);
        if (threadIdx.x == 0) w.hpart[blockIdx.x] = hs;
    }
}

// Huber objective of the last evaluation (block partials in order).
__global__ void k_huber_objective(DevWork w, int nblk) {
    __shared__ double sh[32];
    double acc = 0.0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) acc += w.hpart[b];
    acc = block_sum(acc, sh);
    if (threadIdx.x == 0) w.status->huber_objective = acc;
}

// Mixed-precision refinement of one Gauss-Newton step (FP32 factor M ~ G):
//   dx0 = M^-1 b;  repeat: rho = b - H^T W (H dx) in FP64, dx += M^-1 rho.
__global__ void k_refine_begin(DevFactor f, DevWork w) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= f.n_state) return;
    w.b0[t] = w.rhs[t];
    w.dx[t] = static_cast<double>(w.sol32[t]);
}

__global__ void k_refine_spmv(DevNet net, DevWork w) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= net.n_meas) return;
    double acc = 0.0;
    for (int h = net.h_ptr[q]; h < net.h_ptr[q + 1]; ++h)
        acc += static_cast<double>(w.hval32[h]) * w.dx[net.h_pcol[h]];
    w.hdx[q] = w.w_eff[q] * acc;
}

__global__ void k_refine_rhs(DevNet net, DevFactor f, DevWork w) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= f.n_state) return;
    double acc = 0.0;
    for (int x = f.rhs_ptr[t]; x < f.rhs_ptr[t + 1]; ++x) {
        const int hidx = f.rhs_h[x];
        acc += static_cast<double>(w.hval32[hidx]) * w.hdx[net.h_row[hidx]];
    }
    w.rhs32[t] = static_cast<float>(w.b0[t] - acc);
}

__global__ void k_refine_accumulate(DevFactor f, DevWork w) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= f.n_state) return;
    w.dx[t] += static_cast<double>(w.sol32[t]);
}

// Objective, largest |r| (lowest index on ties) and the bad-data count
// (active rows with sigma > 0 and |r| / sigma > threshold,
// sle_engine.cu:959-977).  Two deterministic passes: per-block partials over
// the rows, then one block over the partials in block order.
__global__ void __launch_bounds__(kBlock) k_objective_part(DevNet net, DevWork w, double bad_threshold) {
    __shared__ double sb[kBlock];
    __shared__ int si[kBlock];
    __shared__ int sc[kBlock];
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    double best = -1.0;
    int bidx = 0x7fffffff, cnt = 0;
    if (q < net.n_meas && net.m_kind[q] != 5) {
        const double a = fabs(w.r[q]);
        best = a;
        bidx = q;
        const double sg = net.m_sigma[q];
        if (sg > 0.0 && a / sg > bad_threshold) cnt = 1;
    }
    sb[threadIdx.x] = best;
    si[threadIdx.x] = bidx;
    sc[threadIdx.x] = cnt;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            const double b2 = sb[threadIdx.x + o];
            const int i2 = si[threadIdx.x + o];
            if (b2 > sb[threadIdx.x] || (b2 == sb[threadIdx.x] && i2 < si[threadIdx.x])) {
                sb[threadIdx.x] = b2;
                si[threadIdx.x] = i2;
            }
            sc[threadIdx.x] += sc[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        w.opart[blockIdx.x] = sb[0];
        w.oidx[blockIdx.x] = si[0];
        w.ocnt[blockIdx.x] = sc[0];
    }
}

// nblk: blocks of k_objective_part (rows); nblk_eval: blocks of the last
// k_evaluate (evaluation units), whose objective partials are summed.
__global__ void k_objective(DevNet net, DevWork w, int nblk, int nblk_eval) {
    __shared__ double sh[32];
    __shared__ double sb[1024];
    __shared__ int si[1024];
    __shared__ int sc[1024];
    double acc = 0.0;
    for (int b = threadIdx.x; b < nblk_eval; b += blockDim.x) acc += w.part[b];
    const double tot = block_sum(acc, sh);
    double best = -1.0;
    int bidx = 0x7fffffff, cnt = 0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
        const double a = w.opart[b];
        const int i = w.oidx[b];
        if (a > best || (a == best && i < bidx)) { best = a; bidx = i; }
        cnt += w.ocnt[b];
    }
    sb[threadIdx.x] = best;
    si[threadIdx.x] = bidx;
    sc[threadIdx.x] = cnt;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            const double b2 = sb[threadIdx.x + o];
            const int i2 = si[threadIdx.x + o];
            if (b2 > sb[threadIdx.x] || (b2 == sb[threadIdx.x] && i2 < si[threadIdx.x])) {
                sb[threadIdx.x] = b2;
                si[threadIdx.x] = i2;
            }
            sc[threadIdx.x] += sc[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        w.status->objective = tot;
        w.status->largest_residual = sb[0] < 0.0 ? 0.0 : sb[0];
        w.status->largest_idx = si[0] == 0x7fffffff ? -1 : si[0];
        w.status->bad_count = sc[0];
    }
}

// Counts the CTA in and tells whether it is the grid's last: what the others
// wrote before is then visible to all of its threads.  The counter wraps back
// to zero.
__device__ __forceinline__ bool last_block(uint32_t* done) {
    __shared__ bool last;
    __syncthreads();  // the CTA's writes are made
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicInc(done, gridDim.x - 1) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    return last;
}

// One bus's step: x += dx (slack angle fixed), V clamped.  Returns |dx|, 0 for
// a NaN; bad is set when the step is not finite.
template <typename V>
__device__ __forceinline__ double update_bus(const DevFactor& f, const DevWork& w, const SolveParams& sp,
                                             const V* step, int i, int& bad) {
    const int pt = f.bus_ps_theta[i];
    const double dv = static_cast<double>(step[f.bus_ps_v[i]]);
    double dt = 0.0;
    if (pt >= 0) {
        dt = static_cast<double>(step[pt]);
        w.th[i] += dt;
    }
    double vn = w.v[i] + dv;
    vn = fmax(vn, sp.vmin);
    vn = fmin(vn, sp.vmax);
    w.v[i] = vn;
    if (!isfinite(dt) || !isfinite(dv)) bad = 1;
    const double m = fmax(fabs(dt), fabs(dv));
    return m != m ? 0.0 : m;
}

// a13: x += dx, block maxima of |dx|; the last CTA takes the maximum over them
// and writes the step's status, on the device and in host memory (a second
// kernel and a copy node before; figures at k_gain_values).
//
// A step with a non-finite entry (FLAG_NONFINITE) is never converged and
// reports a NaN max |dx|: the reference's max reduction turns NaN once a NaN
// step fills its blocks (kernels.cu:557-574,752-782), so "max |dx| < tol"
// fails and checkValidityKernel's flag decides: DIVERGED
// (wls_solver.cu:493-517, 343-352).
template <typename V>
__global__ void __launch_bounds__(kBlock) k_update(DevNet net, DevFactor f, DevWork w, SolveParams sp,
                                                   const V* step, DevStatus* host) {
    __shared__ double sh[32];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double mx = 0.0;
    int bad = 0;
    if (i < net.n_bus) mx = update_bus(f, w, sp, step, i, bad);
    bad = __syncthreads_or(bad);
    const double m = block_max(mx, sh);
    if (threadIdx.x == 0) {
        w.part[blockIdx.x] = m;
        if (bad) atomicOr(&w.status->flags, FLAG_NONFINITE);
    }
    if (!last_block(&w.status->blocks_done)) return;
    mx = 0.0;
    for (int b = threadIdx.x; b < gridDim.x; b += blockDim.x) mx = fmax(mx, __ldcg(w.part + b));
    mx = block_max(mx, sh);
    if (threadIdx.x == 0) {
        uint32_t fl = atomicOr(&w.status->flags, 0u);
        const bool nonfinite = (fl & FLAG_NONFINITE) != 0;
        if (!nonfinite && mx < sp.tol) fl |= FLAG_CONVERGED;
        w.status->flags = fl;
        w.status->max_mismatch = nonfinite ? __longlong_as_double(0x7ff8000000000000LL) : mx;
        if (host) *host = *w.status;
    }
}

// kernels.cu:799-817
__global__ void k_flat_start(DevNet net, DevWork w) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= net.n_bus) return;
    const int t = net.bus_type[i];
    w.v[i] = (t == 1 || t == 2) ? net.v_setpoint[i] : 1.0;
    w.th[i] = 0.0;
}

__global__ void k_injections(DevNet net, DevWork w) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= net.n_bus) return;
    const double Vi = w.v[i], ti = w.th[i];
    double P = 0.0, Q = 0.0;
    for (int e = net.y_ptr[i]; e < net.y_ptr[i + 1]; ++e) {
        const int j = net.y_col[e];
        const double G = net.y_g[e], B = net.y_b[e];
        double s = 0.0, c = 1.0;
        if (j != i) sincos(ti - w.th[j], &s, &c);
        const double vv = Vi * w.v[j];
        P += vv * (G * c + B * s);
        Q += vv * (G * s - B * c);
    }
    w.p_inj[i] = P;
    w.q_inj[i] = Q;
}

__global__ void k_flows(DevNet net, DevWork w) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= net.n_branch) return;
    double s, c;
    sincos(w.th[net.br_from[k]] - w.th[net.br_to[k]] - net.br_shift[k], &s, &c);
    const FlowEnd F = flow_end(net, w.v, k, false, s, c), T = flow_end(net, w.v, k, true, s, c);
    w.pf[k] = flow_row<true>(net, F, k, false, false).val;
    w.qf[k] = flow_row<true>(net, F, k, true, false).val;
    w.pt[k] = flow_row<true>(net, T, k, false, true).val;
    w.qt[k] = flow_row<true>(net, T, k, true, true).val;
}

// Batch: one block per grid.  Clears the grid's flags (FROZEN for grids not
// in this solve) and applies a flat start where requested.
__global__ void k_batch_begin(DevNet net, DevWork w, DevBatch b) {
    const int g = blockIdx.x;
    const bool act = b.active[g] != 0;
    if (threadIdx.x == 0) {
        b.flags[g] = act ? 0u : (FLAG_FROZEN | FLAG_INACTIVE);
        b.iters[g] = 0;
        b.mismatch[g] = 0.0;
    }
    if (!act || !b.flat[g]) return;
    for (int i = b.bus_off[g] + threadIdx.x; i < b.bus_off[g + 1]; i += blockDim.x) {
        const int t = net.bus_type[i];
        w.v[i] = (t == 1 || t == 2) ? net.v_setpoint[i] : 1.0;
        w.th[i] = 0.0;
    }
}

// f2: islands of the closed-branch graph (the reference's topological check,
// sle_engine.cu:684-753, on the device).
__global__ void k_island_init(DevNet net, int32_t* parent, int32_t* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < net.n_bus) parent[i] = i;
    if (i == 0) {
        out[0] = 0;
        out[1] = 0;
        out[3] = 0;
    }
}

__device__ __forceinline__ int island_root(const int32_t* parent, int x) {
    for (int guard = 0; guard < 64 && parent[x] != x; ++guard) x = parent[x];
    return x;
}

// out[3] = 1 when some branch joined two components this round
__global__ void k_island_hook(DevNet net, int32_t* parent, int32_t* out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= net.n_branch || !net.br_closed[k]) return;
    const int a = island_root(parent, net.br_from[k]);
    const int b = island_root(parent, net.br_to[k]);
    if (a == b) return;
    atomicMin(parent + max(a, b), min(a, b));
    out[3] = 1;
}

__global__ void k_island_jump(DevNet net, int32_t* parent) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= net.n_bus) return;
    int p = parent[i];
    for (int guard = 0; guard < 64 && parent[p] != p; ++guard) p = parent[p];
    parent[i] = p;
}

__global__ void k_island_count(DevNet net, const int32_t* parent, int32_t* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < net.n_bus && parent[i] == i) atomicAdd(out + 0, 1);
    if (i < net.n_meas && net.m_active[i]) atomicAdd(out + 1, 1);
}

// Stream mode: grids with active[g] join the running batch.
__global__ void k_batch_activate(DevNet net, DevWork w, DevBatch b) {
    const int g = blockIdx.x;
    if (!b.active[g]) return;
    if (threadIdx.x == 0) {
        b.flags[g] = 0u;
        b.iters[g] = 0;
        b.mismatch[g] = 0.0;
    }
    if (!b.flat[g]) return;
    for (int i = b.bus_off[g] + threadIdx.x; i < b.bus_off[g + 1]; i += blockDim.x) {
        const int t = net.bus_type[i];
        w.v[i] = (t == 1 || t == 2) ? net.v_setpoint[i] : 1.0;
        w.th[i] = 0.0;
    }
}

__global__ void k_batch_retire(DevBatch b) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < b.n_grids && b.retire[g]) b.flags[g] = (b.flags[g] | FLAG_FROZEN | FLAG_INACTIVE) & ~FLAG_FINAL;
}

// Batch a13, spread over CTAs: each item applies the step to its buses and
// writes its max |dx| and whether a step entry was not finite; then one
// thread per grid combines its items and decides, exactly as the single-grid
// loop does after its step: a frozen grid takes no step; a grid whose
// factorisation flagged a non-positive pivot stops as singular without
// applying the step; otherwise it stops when max |dx| < tol (converged) or
// dx is not finite (diverged).
//
// The last CTA does the second part, and inside a device-run loop it also
// takes the decision of the host loop of Engine::batch_solve for the graph's
// while node (in_loop): the step's flags and the running count are final then.
template <typename V>
__global__ void __launch_bounds__(kBlock) k_batch_update(DevFactor f, DevWork w, DevBatch b, SolveParams sp,
                                                         const V* step, cudaGraphConditionalHandle h, int in_loop,
                                                         DevStatus* host, int32_t* host_running) {
    __shared__ double sh[32];
    if (blockIdx.x < b.n_bus_items) {
        const int2 it = b.bus_items[blockIdx.x];
        if (!(b.flags[it.x] & (FLAG_FROZEN | FLAG_SINGULAR))) {  // the whole CTA
            const int end = min(it.y + kBatchChunk, b.bus_off[it.x + 1]);
            double mx = 0.0;
            int bad = 0;
            for (int i = it.y + threadIdx.x; i < end; i += blockDim.x)
                mx = fmax(mx, update_bus(f, w, sp, step, i, bad));
            bad = __syncthreads_or(bad);
            const double m = block_max(mx, sh);
            if (threadIdx.x == 0) {
                b.part[blockIdx.x] = m;
                b.part_bad[blockIdx.x] = bad;
            }
        }
    }
    if (!last_block(&w.status->blocks_done)) return;
    int running = 0;
    for (int g0 = 0; g0 < b.n_grids; g0 += blockDim.x) {
        const int g = g0 + threadIdx.x;
        bool runs = false;
        const uint32_t fl = g < b.n_grids ? b.flags[g] : FLAG_FROZEN;
        if (!(fl & FLAG_FROZEN)) {
            b.iters[g] += 1;
            if (fl & FLAG_SINGULAR) {
                b.flags[g] = fl | FLAG_FROZEN;
            } else {
                double m = 0.0;
                int bad = 0;
                for (int k = b.bus_item_ptr[g]; k < b.bus_item_ptr[g + 1]; ++k) {
                    m = fmax(m, __ldcg(b.part + k));
                    bad |= __ldcg(b.part_bad + k);
                }
                b.mismatch[g] = bad ? __longlong_as_double(0x7ff8000000000000LL) : m;
                if (bad)
                    b.flags[g] = fl | FLAG_NONFINITE | FLAG_FROZEN;
                else if (m < sp.tol)
                    b.flags[g] = fl | FLAG_CONVERGED | FLAG_FROZEN;
                else
                    runs = true;
            }
        }
        running += __syncthreads_count(runs);
    }
    if (threadIdx.x == 0) {
        *b.running = running;
        if (host) {
            *host = *w.status;
            *host_running = running;
        }
        if (in_loop) {
            const int32_t steps = b.loop[0] + 1;
            b.loop[0] = steps;
            const bool timed_out = (w.status->flags & FLAG_TIMEOUT) != 0u;
            if (timed_out) b.loop[2] = 1;
            cudaGraphSetConditional(h, (!timed_out && running > 0 && steps < b.loop[1]) ? 1u : 0u);
        }
    }
}

// Objective sum w r^2 of each selected grid (not inactive, flags holding
// `need`): per item in row order, then per grid over its items in order.
__global__ void __launch_bounds__(kBlock) k_batch_objective_part(DevNet net, DevWork w, DevBatch b, uint32_t need) {
    __shared__ double sh[32];
    const int2 it = b.row_items[blockIdx.x];
    const uint32_t fl = b.flags[it.x];
    if ((fl & FLAG_INACTIVE) || (fl & need) != need) return;  // the whole CTA
    const int end = min(it.y + kBatchChunk, b.meas_off[it.x + 1]);
    double acc = 0.0;
    for (int q = it.y + threadIdx.x; q < end; q += blockDim.x)
        if (net.m_kind[q] != 5) acc += net.m_w[q] * w.r[q] * w.r[q];
    const double tot = block_sum(acc, sh);
    if (threadIdx.x == 0) b.part[blockIdx.x] = tot;
}

__global__ void k_batch_objective_fin(DevBatch b, uint32_t need) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= b.n_grids) return;
    const uint32_t fl = b.flags[g];
    if ((fl & FLAG_INACTIVE) || (fl & need) != need) return;
    double t = 0.0;
    for (int k = b.row_item_ptr[g]; k < b.row_item_ptr[g + 1]; ++k) t += b.part[k];
    b.objective[g] = t;
}

__global__ void k_batch_mark_final(DevBatch b) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < b.n_grids && b.retire[g]) b.flags[g] |= FLAG_FINAL;
}

__global__ void k_gn_loop_init(DevBatch b, int32_t limit) {
    b.loop[0] = 0;
    b.loop[1] = limit;
    b.loop[2] = 0;
}

inline int nblocks(int n) { return (n + kBlock - 1) / kBlock; }

}  // namespace

cudaError_t launch_batch_begin(const DevNet& net, const DevWork& w, const DevBatch& b, cudaStream_t st) {
    if (b.n_grids <= 0) return cudaSuccess;
    k_batch_begin<<<b.n_grids, kBlock, 0, st>>>(net, w, b);
    count_launches(1);
    return cudaGetLastError();
}

template <typename V>
cudaError_t launch_batch_update(const DevNet& net, const DevFactor& f, const DevWork& w, const DevBatch& b,
                                const SolveParams& sp, const V* step, const cudaGraphConditionalHandle* loop,
                                DevStatus* host, int32_t* host_running, cudaStream_t st) {
    if (b.n_grids <= 0) return cudaSuccess;
    k_batch_update<<<std::max(b.n_bus_items, 1), kBlock, 0, st>>>(f, w, b, sp, step,
                                                                  loop ? *loop : cudaGraphConditionalHandle{},
                                                                  loop ? 1 : 0, host, host_running);
    count_launches(1);
    return cudaGetLastError();
}
template cudaError_t launch_batch_update(const DevNet&, const DevFactor&, const DevWork&, const DevBatch&,
                                         const SolveParams&, const float*, const cudaGraphConditionalHandle*,
                                         DevStatus*, int32_t*, cudaStream_t);
template cudaError_t launch_batch_update(const DevNet&, const DevFactor&, const DevWork&, const DevBatch&,
                                         const SolveParams&, const double*, const cudaGraphConditionalHandle*,
                                         DevStatus*, int32_t*, cudaStream_t);

cudaError_t launch_islands(const DevNet& net, int32_t* parent, int32_t* out, int32_t max_rounds, cudaStream_t st) {
    const int nb = nblocks(std::max(net.n_bus, 1));
    k_island_init<<<nb, kBlock, 0, st>>>(net, parent, out);
    count_launches(1);
    int32_t rounds = 0, joined = 1;
    cudaError_t e = cudaSuccess;
    while (joined && e == cudaSuccess) {
        if (rounds == max_rounds) {
            rounds = -1;
            break;
        }
        e = cudaMemsetAsync(out + 3, 0, sizeof(int32_t), st);
        if (net.n_branch > 0 && e == cudaSuccess) {
            k_island_hook<<<nblocks(net.n_branch), kBlock, 0, st>>>(net, parent, out);
            count_launches(1);
        }
        k_island_jump<<<nb, kBlock, 0, st>>>(net, parent);
        count_launches(1);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&joined, out + 3, sizeof(int32_t), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        ++rounds;
    }
    if (e != cudaSuccess) return e;
    k_island_count<<<nblocks(std::max(std::max(net.n_bus, net.n_meas), 1)), kBlock, 0, st>>>(net, parent, out);
    count_launches(1);
    e = cudaMemcpyAsync(out + 2, &rounds, sizeof(int32_t), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e == cudaSuccess ? cudaGetLastError() : e;
}

cudaError_t launch_batch_activate(const DevNet& net, const DevWork& w, const DevBatch& b, cudaStream_t st) {
    if (b.n_grids <= 0) return cudaSuccess;
    k_batch_activate<<<b.n_grids, kBlock, 0, st>>>(net, w, b);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_batch_retire(const DevBatch& b, cudaStream_t st) {
    if (b.n_grids <= 0) return cudaSuccess;
    k_batch_retire<<<(b.n_grids + kBlock - 1) / kBlock, kBlock, 0, st>>>(b);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_gn_loop_init(const DevBatch& b, int32_t limit, cudaStream_t st) {
    k_gn_loop_init<<<1, 1, 0, st>>>(b, limit);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_batch_objective(const DevNet& net, const DevWork& w, const DevBatch& b, uint32_t need,
                                   cudaStream_t st) {
    if (b.n_grids <= 0) return cudaSuccess;
    if (b.n_row_items > 0) {
        k_batch_objective_part<<<b.n_row_items, kBlock, 0, st>>>(net, w, b, need);
        count_launches(1);
    }
    k_batch_objective_fin<<<nblocks(b.n_grids), kBlock, 0, st>>>(b, need);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_batch_mark_final(const DevBatch& b, cudaStream_t st) {
    if (b.n_grids <= 0) return cudaSuccess;
    k_batch_mark_final<<<nblocks(b.n_grids), kBlock, 0, st>>>(b);
    count_launches(1);
    return cudaGetLastError();
}

std::atomic<int64_t> g_kernel_launches{0};
thread_local int64_t t_kernel_launches = 0;

cudaError_t launch_admittance_and_ybus(const DevNet& net, cudaStream_t st) {
    if (net.n_branch > 0) {
        k_admittance<<<nblocks(net.n_branch), kBlock, 0, st>>>(net);
        count_launches(1);
    }
    k_ybus<<<nblocks(net.n_bus), kBlock, 0, st>>>(net);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_evaluate(const DevNet& net, const DevWork& w, const SolveParams& sp, cudaStream_t st) {
    if (net.n_meas <= 0) return cudaSuccess;
    k_bus_trig<<<nblocks(net.n_bus), kBlock, 0, st>>>(net, w, sp);
    // the unit list has as many units as rows when no row is paired
    const bool exact = sp.exact_jacobian != 0;
    if (net.n_units < net.n_meas)
        (exact ? k_evaluate_pairs<true> : k_evaluate_pairs<false>)<<<nblocks(net.n_units), kBlock, 0, st>>>(net, w, sp);
    else
        (exact ? k_evaluate_rows<true> : k_evaluate_rows<false>)<<<nblocks(net.n_meas), kBlock, 0, st>>>(net, w, sp);
    count_launches(2);
    if (sp.huber_objective) {
        k_huber_objective<<<1, 1024, 0, st>>>(w, nblocks(net.n_units));
        count_launches(1);
    }
    return cudaGetLastError();
}

cudaError_t launch_objective(const DevNet& net, const DevWork& w, double bad_threshold, cudaStream_t st) {
    const int nb = net.n_meas > 0 ? nblocks(net.n_meas) : 0;
    if (nb > 0) {
        k_objective_part<<<nb, kBlock, 0, st>>>(net, w, bad_threshold);
        count_launches(1);
    }
    k_objective<<<1, 1024, 0, st>>>(net, w, nb, net.n_units > 0 ? nblocks(net.n_units) : 0);
    count_launches(1);
    return cudaGetLastError();
}

template <typename V>
cudaError_t launch_update(const DevNet& net, const DevFactor& f, const DevWork& w, const SolveParams& sp,
                          const V* step, DevStatus* host, cudaStream_t st) {
    k_update<<<nblocks(net.n_bus), kBlock, 0, st>>>(net, f, w, sp, step, host);
    count_launches(1);
    return cudaGetLastError();
}
template cudaError_t launch_update(const DevNet&, const DevFactor&, const DevWork&, const SolveParams&, const float*,
                                   DevStatus*, cudaStream_t);
template cudaError_t launch_update(const DevNet&, const DevFactor&, const DevWork&, const SolveParams&, const double*,
                                   DevStatus*, cudaStream_t);

cudaError_t launch_refine_begin(const DevFactor& f, const DevWork& w, cudaStream_t st) {
    k_refine_begin<<<nblocks(f.n_state), kBlock, 0, st>>>(f, w);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_refine_residual(const DevNet& net, const DevFactor& f, const DevWork& w, cudaStream_t st) {
    if (net.n_meas > 0) {
        k_refine_spmv<<<nblocks(net.n_meas), kBlock, 0, st>>>(net, w);
        count_launches(1);
    }
    k_refine_rhs<<<nblocks(f.n_state), kBlock, 0, st>>>(net, f, w);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_refine_accumulate(const DevFactor& f, const DevWork& w, cudaStream_t st) {
    k_refine_accumulate<<<nblocks(f.n_state), kBlock, 0, st>>>(f, w);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_flat_start(const DevNet& net, const DevWork& w, cudaStream_t st) {
    k_flat_start<<<nblocks(net.n_bus), kBlock, 0, st>>>(net, w);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_results(const DevNet& net, const DevWork& w, cudaStream_t st) {
    k_injections<<<nblocks(net.n_bus), kBlock, 0, st>>>(net, w);
    count_launches(1);
    if (net.n_branch > 0) {
        k_flows<<<nblocks(net.n_branch), kBlock, 0, st>>>(net, w);
        count_launches(1);
    }
    return cudaGetLastError();
}

}  // namespace sle_gb300
