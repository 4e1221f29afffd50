// Level-scheduled multifrontal Cholesky of the gain matrix G = H^T W H and the
// forward / backward solves (replaces the reference's per-call
// cusolverSp csrlsvchol, sparse_matrix.cu:793-895, and its quadratic RHS
// kernel, kernels.cu:823-862).
//
// Front s (rows R_s, nc_s pivot columns, order f_s) is assembled from
//   - its gain entries, each a fixed-order sum of w_m H[m,a] H[m,b] over the
//     measurement rows m that couple the two states (gathered, no atomics), and
//   - its children's update matrices, extend-added through relative maps,
// then partially factorised: L11 = chol(F11), L21 = F21 L11^-T,
// U_s = F22 - L21 L21^T.
//
// Small fronts (little work) are one CTA each with the whole front in shared
// memory.  Big fronts live in place in an f x f region (L panel = first nc
// columns, update matrix = trailing block, both column-major with ld = f) and
// are processed for a whole level at once by work lists: an assembly kernel
// (one CTA per 32-column tile column and block of rows, so every entry has one
// writer), then per 32-column step a panel (each CTA factors the diagonal block
// and solves a chunk of rows against it) and the trailing update (one CTA per
// tile): FP64 in two launches a step, FP32 in one that does a step's update and
// the next step's panel, after a panel launch for the first.
// The factor type T is double for the FP64 pipeline and float for the
// mixed-precision one; the mixed pipeline forms the gain entries' sums in
// float (gain_acc32, the default) or in double.
#include "kernels.cuh"

#include <algorithm>
#include <mutex>

namespace sle_gb300 {
namespace {

constexpr int kThreads = 256;
constexpr int kSMs = 152;

struct SolveVecs {
    const void* rhs;  // [n_state] right-hand side, permuted (V)
    void* sol;        // [n_state] solution, permuted (V)
    void* su;         // solve update vectors (V)
};
// Entry r of front s's right-hand-side row: a pivot's in sol (y once it is
// eliminated), a row's below them in the front's solve update vector.
template <typename V>
__device__ __forceinline__ V* rhs_entry(const SolveVecs& sv, int c0, int nc, int64_t su_off, int r) {
    return r < nc ? static_cast<V*>(sv.sol) + c0 + r : static_cast<V*>(sv.su) + su_off + (r - nc);
}

// Terms of a sum whose loads are in flight together: index, then value, is a
// chain of two or three loads, and the sums below are bound by it.  The gain
// launch of 512 grids took 195 us a term at a time, 175 by fours, 202 by eights
// (mostly short sums, and more registers); of 200k buses 119, 111 and 117.
constexpr int kGather = 4;

// G entry = sum over its pairs (a, b) of (w h_a) h_b, the weighted entry
// hw[a] written by the evaluation (FP64: the same product, so the same sum),
// accumulated in ACC.
template <typename HV, typename ACC>
__device__ __forceinline__ ACC gain_entry(const DevFactor& F, const HV* hval, const HV* hw, int tg) {
    ACC acc = ACC(0);
    const int64_t p0 = F.tgt_pair_ptr[tg];
    const int n = static_cast<int>(F.tgt_pair_ptr[tg + 1] - p0);
    for (int p = 0; p < n; p += kGather) {
        int a[kGather], b[kGather];
        HV x[kGather], y[kGather];
#pragma unroll
        for (int k = 0; k < kGather; ++k) {
            a[k] = p + k < n ? F.pair_a[p0 + p + k] : 0;
            b[k] = p + k < n ? F.pair_b[p0 + p + k] : 0;
        }
#pragma unroll
        for (int k = 0; k < kGather; ++k) {
            x[k] = p + k < n ? hw[a[k]] : HV(0);
            y[k] = p + k < n ? hval[b[k]] : HV(0);
        }
#pragma unroll
        for (int k = 0; k < kGather; ++k)
            if (p + k < n) acc += static_cast<ACC>(x[k]) * static_cast<ACC>(y[k]);
    }
    return acc;
}

// a11: entry t of b = H^T (w r) in permuted state order (gather).
__device__ __forceinline__ void rhs_value(const DevFactor& F, const DevWork& W, const int32_t* h_row, int t) {
    if (F.ps_grid && (W.grid_flags[F.ps_grid[t]] & FLAG_FROZEN)) return;
    double acc = 0.0;
    const int x1 = F.rhs_ptr[t + 1];
    for (int x = F.rhs_ptr[t]; x < x1; x += kGather) {
        int h[kGather], row[kGather];
        double v[kGather], w[kGather];
#pragma unroll
        for (int k = 0; k < kGather; ++k) h[k] = x + k < x1 ? F.rhs_h[x + k] : 0;
#pragma unroll
        for (int k = 0; k < kGather; ++k) {
            row[k] = x + k < x1 ? h_row[h[k]] : 0;
            v[k] = x + k < x1 ? W.hval[h[k]] : 0.0;
        }
#pragma unroll
        for (int k = 0; k < kGather; ++k) w[k] = x + k < x1 ? W.wr[row[k]] : 0.0;
#pragma unroll
        for (int k = 0; k < kGather; ++k)
            if (x + k < x1) acc += v[k] * w[k];
    }
    W.rhs[t] = acc;
    if (W.rhs32) W.rhs32[t] = static_cast<float>(acc);
}

__global__ void k_rhs(DevFactor F, DevWork W, const int32_t* h_row, int begin) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (begin && t == 0) W.status->flags = 0u;
    if (t < F.n_state) rhs_value(F, W, h_row, t);
}

// Counters that a factorisation starts from zero.
struct ZeroLists {
    int* p[3];
    int n[3];
};

// All gain entries of the factorisation at once: fully parallel, so the
// dependent gathers are hidden by occupancy instead of sitting on the
// elimination tree's critical path.  The first rhs_blocks CTAs compute the
// right-hand side of a Gauss-Newton step meanwhile (it has the longest chain
// of gathers per thread and needs few threads), and all clear the counters:
// with this and the step's end in one kernel (k_update) a step has seven nodes
// fewer, which took 25 us of 727 at 10k buses (FP32) and 65 of the 573 us of a
// whole estimate at 14 buses (FP64).
template <typename T, typename HV, typename ACC = double>
__global__ void k_gain_values(DevFactor F, DevWork W, const HV* hval, const HV* hw, T* gv, int n_tgt,
                              const int32_t* h_row, int rhs_blocks, ZeroLists Z) {
    const int me = blockIdx.x * blockDim.x + threadIdx.x, all = gridDim.x * blockDim.x;
#pragma unroll
    for (int k = 0; k < 3; ++k)
        for (int i = me; i < Z.n[k]; i += all) Z.p[k][i] = 0;
    if (blockIdx.x < rhs_blocks) {
        if (me == 0) W.status->flags = 0u;
        if (me < F.n_state) rhs_value(F, W, h_row, me);
        return;
    }
    for (int tg = me - rhs_blocks * blockDim.x; tg < n_tgt; tg += (gridDim.x - rhs_blocks) * blockDim.x) {
        if (F.tgt_grid && (W.grid_flags[F.tgt_grid[tg]] & FLAG_FROZEN)) continue;
        gv[tg] = static_cast<T>(gain_entry<HV, ACC>(F, hval, hw, tg));
    }
}

// Where a non-positive pivot of front s is reported: the grid's own flags in
// a batch, the engine status otherwise.
__device__ __forceinline__ uint32_t* singular_flags(const DevFactor& F, const DevWork& W, int s) {
    return W.grid_flags ? W.grid_flags + F.sn_grid[s] : &W.status->flags;
}
// Batch: fronts of grids that take no further step are skipped.
__device__ __forceinline__ bool front_frozen(const DevFactor& F, const DevWork& W, int s) {
    return W.grid_flags && (W.grid_flags[F.sn_grid[s]] & FLAG_FROZEN);
}
__device__ __forceinline__ bool front_frozen(const DevWork& W, const FrontRec& R) {
    return W.grid_flags && (W.grid_flags[R.grid] & FLAG_FROZEN);
}

// Positive and finite?  FP64 by the bit pattern: an FP64 comparison or
// conversion is an FP64 instruction like any (60 cycles, 19 of the SM's pipe).
__device__ __forceinline__ bool pivot_ok(float d) { return d > 0.f && isfinite(d); }
__device__ __forceinline__ bool pivot_ok(double d) {
    const int hi = __double2hiint(d);
    return hi < 0x7ff00000 && (hi > 0 || (hi == 0 && __double2loint(d) != 0));
}

// FP32 value of the leading bits of a positive d within the FP32 range (test
// first), and the FP64 value of a positive FP32 one, by their bits.
__device__ __forceinline__ bool in_fp32_range(double d) {
    return static_cast<unsigned>((__double2hiint(d) >> 20) - (1023 - 100)) < 200u;
}
__device__ __forceinline__ float leading_fp32(double d) {
    return __uint_as_float((static_cast<unsigned>(__double2hiint(d) - ((1023 - 127) << 20)) << 3) |
                           (static_cast<unsigned>(__double2loint(d)) >> 29));
}
__device__ __forceinline__ double widen_fp32(float y) {
    const unsigned b = __float_as_uint(y);
    return __hiloint2double(static_cast<int>((b >> 3) + ((1023u - 127u) << 20)), static_cast<int>(b << 29));
}

// Pivot: L_kk = sqrt(d) and 1 / L_kk for a positive finite d (the callers
// flag a non-positive or non-finite d as a matrix that is not positive
// definite and go on with 1).  FP64: an FP32 reciprocal square root refined by
// one third-order Newton (Householder) step, y (1 + e / 2 + 3 e^2 / 8) with
// e = 1 - d y^2 (2^-22 -> 2^-66, then rounding): five FP64 instructions on
// the chain where two second-order steps take eight; the library routines are
// used outside the FP32 range.
__device__ __forceinline__ void pivot_value(float d, float* sq, float* inv) {
    const float y = rsqrtf(d);  // the FP32 factor is a preconditioner of FP64 steps
    *sq = d * y;
    *inv = y;
}
__device__ __noinline__ double slow_sqrt(double d) { return sqrt(d); }
__device__ __noinline__ double slow_div(double a, double b) { return a / b; }
__device__ __forceinline__ void pivot_value(double d, double* sq, double* inv) {
    if (in_fp32_range(d)) {
        const double y = widen_fp32(rsqrtf(leading_fp32(d)));
        const double e = fma(-(d * y), y, 1.0);
        const double z = fma(y * e, fma(0.375, e, 0.5), y);
        *sq = d * z;
        *inv = z;
    } else {
        *sq = slow_sqrt(d);
        *inv = slow_div(1.0, *sq);
    }
}

// Extend-add of every child of a single-CTA front with no barrier between
// children: warp w owns the front's columns t = w (mod warps) and walks its list of the children's columns (DevFactor::asm_ent, in child
// order), so no two warps touch the same entry and each entry's additions keep
// the children's order.  Bound: load latency.  The 32 list entries and child
// records of a round are fetched a lane each; columns go eight at a time, 32
// rows a step, the next step's loads in flight while this one is added (as a
// walk over the children, each warp selecting its columns, the chain of
// dependent loads per child made the assembly half of a front's time).  Columns
// of a step with the same target (from different children) are added one after
// the other; if any is longer than a step, the eight are cut before the second
// of the two.  The children's solve update vectors are added to the front's
// right-hand side (entry t at rhs[t * rhs_ld]) the same way.  The caller
// follows with a block barrier.  Measured on the longest chain of a 10k-bus
// grid (mixed): 19k -> 7.6k cycles for 4 children of a 73-row front, 97k -> 65k
// for the 40 children of the 217-row root (one SM's L2 bandwidth).
template <typename T>
__device__ __forceinline__ void extend_add_children(const DevFactor& F, const SolveVecs& sv, const T* lx,
                                                    const T* ubase, const FrontRec& R, T* dst, int ldd, T* rhs,
                                                    int rhs_ld) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int kB = 8;  // columns per step
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int e1 = F.asm_ptr[R.asm_slot + warp + 1];
    for (int eb = F.asm_ptr[R.asm_slot + warp]; eb < e1; eb += 32) {
        const int n = min(32, e1 - eb);
        const T* up = nullptr;
        const int* rel = nullptr;
        int len = 0, t = 0;  // rows from the diagonal down, target column
        T bv = T(0);
        if (lane < n) {
            const int2 en = F.asm_ent[eb + lane];
            const ChildRec c = F.child_rec[en.x];
            const int j = en.y & 0xffff;
            t = en.y >> 16;
            len = c.m - j;
            up = (c.big ? lx : ubase) + c.u_off + (int64_t)j * c.ld + j;
            rel = F.sn_relmap + c.su_off + j;
            bv = __ldcg(static_cast<const T*>(sv.su) + c.su_off + j);
        }
        // the entry before with the same target (-1: none of this round)
        const unsigned before = __match_any_sync(kAll, lane < n ? t : -1 - lane) & ((1u << lane) - 1u);
        const int prev = 31 - __clz(before);
        // the batch from column q0: its columns, its longest one, shared targets
        struct Batch {
            int q0, cnt, longest;
            bool dup;
        };
        auto batch = [&](int q0) {
            Batch z;
            z.q0 = q0;
            z.cnt = min(kB, n - q0);
            const bool in = lane >= q0 && lane < q0 + z.cnt;
            z.longest = __reduce_max_sync(kAll, in ? len : 0);
            const unsigned cut = __ballot_sync(kAll, in && prev >= q0);
            z.dup = cut != 0u;
            if (z.dup && z.longest > 32) {
                z.cnt = __ffs(cut) - 1 - q0;
                z.dup = false;
            }
            return z;
        };
        T u[kB], un[kB];
        int ri[kB], rn[kB];
        auto load = [&](const Batch& z, int ib, T (&x)[kB], int (&r)[kB]) {
#pragma unroll
            for (int k = 0; k < kB; ++k) {
                const int q = z.q0 + k, row = ib + lane;
                const T* p = reinterpret_cast<const T*>(__shfl_sync(kAll, reinterpret_cast<unsigned long long>(up), q));
                const int* rp =
                    reinterpret_cast<const int*>(__shfl_sync(kAll, reinterpret_cast<unsigned long long>(rel), q));
                const bool ok = row < __shfl_sync(kAll, len, q) && k < z.cnt;
                x[k] = ok ? __ldcg(p + row) : T(0);
                r[k] = ok ? rp[row] : -1;
            }
        };
        Batch z = batch(0);
        load(z, 0, u, ri);
        int ib = 0;
        for (;;) {
            Batch zn = z;
            int nib = ib + 32;
            bool more = true;
            if (nib >= z.longest) {
                nib = 0;
                more = z.q0 + z.cnt < n;
                if (more) zn = batch(z.q0 + z.cnt);
            }
            if (more) load(zn, nib, un, rn);
            int to[kB];
#pragma unroll
            for (int k = 0; k < kB; ++k) to[k] = ri[k] + __shfl_sync(kAll, t, z.q0 + k) * ldd;
            if (!z.dup) {
                if (ib == 0 && lane >= z.q0 && lane < z.q0 + z.cnt) rhs[t * rhs_ld] += bv;
                T cur[kB];
#pragma unroll
                for (int k = 0; k < kB; ++k) cur[k] = ri[k] >= 0 ? dst[to[k]] : T(0);
#pragma unroll
                for (int k = 0; k < kB; ++k) {
                    if (k >= z.cnt) break;
                    if (ri[k] >= 0) dst[to[k]] = cur[k] + u[k];
                }
            } else {
#pragma unroll
                for (int k = 0; k < kB; ++k) {
                    if (k >= z.cnt) break;
                    if (lane == z.q0 + k) rhs[t * rhs_ld] += bv;  // a batch of one step
                    if (ri[k] >= 0) dst[to[k]] += u[k];
                    __syncwarp();
                }
            }
            __syncwarp();
            if (!more) break;
            z = zn;
            ib = nib;
#pragma unroll
            for (int k = 0; k < kB; ++k) {
                u[k] = un[k];
                ri[k] = rn[k];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Small fronts: one CTA per front, front held in shared memory.
//
// Layout: column-major with a leading dimension padded to 16 bytes
// (front_ld), so four consecutive rows of a column are one or two aligned
// vector loads.  The FP32 partial factorisation runs over panels (FP64: see
// front_factor):
//   (1) warp 0 factors the diagonal block (warp_potrf) and leaves L11^T and
//       1/diag in shared memory;
//   (2) warp 0 inverts the block (warp_trinv) while every other thread solves
//       one row of the panel below it, x = a L11^-T, by forward substitution
//       (row_trsm);
//   (3) the trailing lower triangle is updated by 4x4 register tiles,
//       A22 -= X X^T, two vector loads and sixteen FMAs per panel column.
// ---------------------------------------------------------------------------
constexpr int kPanel = 32;  // widest panel of the in-shared-memory factorisation
static_assert(kThreads - 32 >= kSmallFrontMax32, "one thread per front row besides warp 0");

__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
    *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(p);
}
__device__ __forceinline__ void store4(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = *reinterpret_cast<const float4*>(v);
}

// FP32 factors store L11^-1 in each diagonal block's slot, so that the solves
// multiply by it (independent dot products) instead of sweeping the triangle
// one column at a time.  FP64 keeps L11 there: at this GPU's FP64 rate the
// inversion costs the factorisation more than the solves save.
template <typename T>
constexpr bool kInvDiag = sizeof(T) == 4;

// FP32 diagonal blocks, one warp, kb <= 32 columns in blocks of eight.  An
// outer step takes the updates of the columns before it (each lane's row against
// the block's eight, read as two broadcast vectors) and then works the eight in
// registers; every entry gets the operations of the plain right-looking order in
// the same order.  As straight code for 32 columns they were some 600
// instructions each and held 32 entries a lane (128 registers for the wide
// fronts' kernel, 99 now); rolled over blocks of eight they take about the same
// time on a whole block (6.5k, 3.1k and 4.0k cycles) and less on the narrow
// panels that most fronts have: phase A 300 -> 284 us and phase B 157 -> 132 us
// a call at 200k buses (mixed).
//
// Cholesky: lane i owns row i; get(j) is its entry of column j <= i (else
// anything finite).  L goes to lt[c * ld + r] (16-byte aligned rows, ld > kb),
// which may be where get reads.  *inv_out = 1 / L_ii of the lane's row; returns
// true if a pivot was not positive and finite (then replaced by 1).
constexpr int kBlk = 8;
template <typename Get>
__device__ __forceinline__ bool warp_potrf(int kb, int lane, float* lt, int ld, float* inv_out, Get&& get) {
    bool bad = false;
    float my_inv = 0.f;
#pragma unroll 1
    for (int b0 = 0; b0 < kb; b0 += kBlk) {
        float a[kBlk];
#pragma unroll
        for (int q = 0; q < kBlk; ++q) a[q] = (lane < kb && b0 + q <= lane) ? get(b0 + q) : 0.f;
#pragma unroll 2
        for (int k = 0; k < b0; ++k) {
            const float lk = lt[k * ld + lane];
            float w[kBlk];
            *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(lt + k * ld + b0);
            *reinterpret_cast<float4*>(w + 4) = *reinterpret_cast<const float4*>(lt + k * ld + b0 + 4);
#pragma unroll
            for (int q = 0; q < kBlk; ++q) a[q] = a[q] - lk * w[q];
        }
        float d = __shfl_sync(0xffffffffu, a[0], b0);
#pragma unroll
        for (int q = 0; q < kBlk; ++q) {
            const int k = b0 + q;
            if (k < kb) {
                const bool ok = pivot_ok(d);
                bad |= !ok;
                d = ok ? d : 1.f;
                float sq, inv;
                pivot_value(d, &sq, &inv);
                const float lk = (lane == k) ? sq : (lane > k ? a[q] * inv : a[q]);
                my_inv = (lane == k) ? inv : my_inv;
                if (q + 1 < kBlk) {
                    // the next pivot first: lane k + 1 has its own l to update it
                    d = __shfl_sync(0xffffffffu, a[q + 1] - lk * lk, (k + 1) & 31);
                }
                if (lane < ld) lt[k * ld + lane] = lk;
                if (q + 1 < kBlk) {
                    __syncwarp();
                    float w[kBlk];
                    if (q < 3) *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(lt + k * ld + b0);
                    *reinterpret_cast<float4*>(w + 4) = *reinterpret_cast<const float4*>(lt + k * ld + b0 + 4);
#pragma unroll
                    for (int t = q + 1; t < kBlk; ++t) a[t] = a[t] - lk * w[t];
                }
            }
        }
        __syncwarp();
    }
    *inv_out = my_inv;
    return bad;
}

// L^-1, one column per lane (L^-1 e_j by right-looking substitution, lane j):
// rows i >= j to dst[i + j * dld].  rinv: the reciprocal diagonal.
__device__ __forceinline__ void load_row8(const float* p, float (&w)[kBlk]) {
    *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(p);
    *reinterpret_cast<float4*>(w + 4) = *reinterpret_cast<const float4*>(p + 4);
}
__device__ __forceinline__ void warp_trinv(const float* __restrict__ lt, int ld, const float* __restrict__ rinv, int kb,
                                           int lane, float* __restrict__ dst, int dld) {
    float* const mine = dst + lane * dld;
#pragma unroll 1
    for (int b0 = 0; b0 < kb; b0 += kBlk) {
        float x[kBlk], ri[kBlk], w[kBlk][kBlk];
#pragma unroll
        for (int q = 0; q < kBlk; ++q) {
            x[q] = (b0 + q == lane) ? 1.f : 0.f;
            ri[q] = b0 + q < kb ? rinv[b0 + q] : 0.f;
        }
#pragma unroll 4
        for (int c = 0; c < b0; ++c) {
            const float xc = (lane < kb && c >= lane) ? mine[c] : 0.f;
            float v[kBlk];
            load_row8(lt + c * ld + b0, v);
#pragma unroll
            for (int q = 0; q < kBlk; ++q) x[q] -= xc * v[q];
        }
#pragma unroll
        for (int q = 0; q + 1 < kBlk; ++q) load_row8(lt + min(b0 + q, kb - 1) * ld + b0, w[q]);
#pragma unroll
        for (int q = 0; q < kBlk; ++q) {
            x[q] *= ri[q];
#pragma unroll
            for (int t = q + 1; t < kBlk; ++t) x[t] -= x[q] * w[q][t];
        }
#pragma unroll
        for (int q = 0; q < kBlk; ++q)
            if (b0 + q < kb && b0 + q >= lane) mine[b0 + q] = x[q];
    }
}

// One row of X = A L^-T by substitution, in place: entry c at row[c * rld].
__device__ __forceinline__ void row_trsm(const float* __restrict__ lt, int ld, const float* __restrict__ rinv, int kb,
                                         float* __restrict__ row, int rld) {
#pragma unroll 1
    for (int b0 = 0; b0 < kb; b0 += kBlk) {
        float x[kBlk], ri[kBlk];
#pragma unroll
        for (int q = 0; q < kBlk; ++q) {
            x[q] = b0 + q < kb ? row[(b0 + q) * rld] : 0.f;
            ri[q] = b0 + q < kb ? rinv[b0 + q] : 0.f;
        }
#pragma unroll 4
        for (int c = 0; c < b0; ++c) {
            const float xc = row[c * rld];
            float v[kBlk];
            load_row8(lt + c * ld + b0, v);
#pragma unroll
            for (int q = 0; q < kBlk; ++q) x[q] -= xc * v[q];
        }
#pragma unroll
        for (int q = 0; q < kBlk; ++q) {
            x[q] *= ri[q];
            float v[kBlk];
            if (q + 1 < kBlk) load_row8(lt + min(b0 + q, kb - 1) * ld + b0, v);
#pragma unroll
            for (int t = q + 1; t < kBlk; ++t) x[t] -= x[q] * v[t];
        }
#pragma unroll
        for (int q = 0; q < kBlk; ++q)
            if (b0 + q < kb) row[(b0 + q) * rld] = x[q];
    }
}

constexpr int kWarpsPerCta = kThreads / 32;
constexpr int kWtLd = kWarpFrontMax + 1;

template <typename T>
struct WarpTile {
    T a[kWarpFrontMax * kWtLd];  // a[c * kWtLd + r] = front entry (r, c)
    T rinv[kWarpFrontMax];
    T v[kWarpFrontMax];          // right-hand side of the front's rows
};

__device__ __forceinline__ int warp_claim(int* counter) {
    int item = 0;
    if ((threadIdx.x & 31) == 0) item = atomicAdd(counter, 1);
    return __shfl_sync(0xffffffffu, item, 0);
}

// Counts a finished front into its parent when the parent belongs to the same
// phase (R.up_n > 0); returns the parent when this completed its last child.
// One thread, after the barrier that ends the front.
__device__ __forceinline__ int count_up(const FrontRec& R, int* cnt) {
    if (R.up_n <= 0) return -1;
    int seen;
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    asm volatile("atom.add.relaxed.gpu.global.s32 %0, [%1], 1;" : "=r"(seen) : "l"(cnt + R.parent) : "memory");
    if (seen + 1 != R.up_n) return -1;
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    return R.parent;
}
__device__ __forceinline__ int warp_continue_up(const FrontRec& R, int* cnt) {
    __syncwarp();
    int nxt = -1;
    if ((threadIdx.x & 31) == 0) nxt = count_up(R, cnt);
    nxt = __shfl_sync(0xffffffffu, nxt, 0);
    __syncwarp();
    return nxt;
}
// The forward sweep's counts go by its own children numbers.
__device__ __forceinline__ int warp_continue_up(const DevFactor& F, const int8_t* phase, int ph, const int32_t* nchild,
                                                int* cnt, int s) {
    __syncwarp();
    int nxt = -1;
    if ((threadIdx.x & 31) == 0) {
        const int p = F.sn_parent[s];
        if (p >= 0 && phase[p] == ph) {
            __threadfence();
            if (atomicAdd(cnt + p, 1) + 1 == nchild[p]) {
                __threadfence();
                nxt = p;
            }
        }
    }
    nxt = __shfl_sync(0xffffffffu, nxt, 0);
    __syncwarp();
    return nxt;
}

// One warp: assembly in its tile, then the partial factorisation column by
// column (left-looking): a pivot column takes the updates of the columns
// before it in one accumulator a lane, and the trailing columns take theirs at
// the end, four at a time, straight into the update matrix.  Every entry gets
// the operations of the right-looking order in the same order, without its
// read-modify-write of the tile per pivot (one shared-memory round trip per
// entry and pivot was three quarters of a front's time).  FP64 packs the
// trailing triangle into whole warps: an FP64 instruction costs the same
// whatever its lanes do.  Measured on a 301-bus grid's chain of six warp fronts:
// 73 -> 46 us (mixed), on a 30k-bus grid's 172 -> 108 us (FP64).
template <typename T>
__device__ void warp_front_factor(const DevFactor& F, const DevWork& W, const SolveVecs& sv, const T* gv, T* lx, T* ub,
                                  const FrontRec& R, int s, WarpTile<T>& t) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int kB = 8;  // a child's columns per step
    const int lane = threadIdx.x & 31;
    const int f = R.f, c0 = R.c0, nc = R.nc;
    // original entries, four per lane in flight while the tile is cleared
    const T b0 = lane < nc ? static_cast<const T*>(sv.rhs)[c0 + lane] : T(0);
    for (int tb = R.tgt0; tb < R.tgt1 || tb == R.tgt0; tb += 128) {
        T g[4];
        int l[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int tg = tb + lane + 32 * q;
            l[q] = tg < R.tgt1 ? F.tgt_local[tg] : -1;  // row + col * f
            g[q] = tg < R.tgt1 ? gv[tg] : T(0);
        }
        if (tb == R.tgt0) {
            for (int c = 0; c < f; ++c) t.a[c * kWtLd + lane] = T(0);
            t.v[lane] = b0;
            __syncwarp();
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (l[q] >= 0) {
                const int c = l[q] / f;
                t.a[c * kWtLd + (l[q] - c * f)] = g[q];
            }
    }
    __syncwarp();
    for (int cb = R.ch0; cb < R.ch1; cb += 32) {
        const int n = min(32, R.ch1 - cb);
        const T* up = nullptr;
        long long so = 0;
        int m = 0, ld = 0;
        if (lane < n) {
            const ChildRec c = F.child_rec[cb + lane];
            up = (c.big ? lx : ub) + c.u_off;
            so = c.su_off;
            m = c.m;
            ld = c.ld;
        }
        // steps of kB columns of a child, the next step's loads in flight
        T u[kB], un[kB], bv, bn;
        int ri, rn;
        auto load = [&](int ch, int j0, T (&x)[kB], int& r, T& b) {
            const T* p = reinterpret_cast<const T*>(__shfl_sync(kAll, reinterpret_cast<unsigned long long>(up), ch));
            const long long o = __shfl_sync(kAll, so, ch);
            const int mm = __shfl_sync(kAll, m, ch), ll = __shfl_sync(kAll, ld, ch);
            r = lane < mm ? F.sn_relmap[o + lane] : 0;
            b = lane < mm && j0 == 0 ? __ldcg(static_cast<const T*>(sv.su) + o + lane) : T(0);
#pragma unroll
            for (int k = 0; k < kB; ++k)
                x[k] = (j0 + k < mm && lane >= j0 + k && lane < mm) ? __ldcg(p + lane + (int64_t)(j0 + k) * ll) : T(0);
        };
        load(0, 0, u, ri, bv);
        int ch = 0, j0 = 0;
        for (;;) {
            const int mm = __shfl_sync(kAll, m, ch);
            int nch = ch, nj = j0 + kB;
            if (nj >= mm) {
                nch = ch + 1;
                nj = 0;
            }
            const bool more = nch < n;
            if (more) load(nch, nj, un, rn, bn);
            if (j0 == 0 && lane < mm) t.v[ri] += bv;
            T cur[kB];
            int to[kB];
#pragma unroll
            for (int k = 0; k < kB; ++k) {
                to[k] = __shfl_sync(kAll, ri, (j0 + k) & 31) * kWtLd + ri;
                if (!(j0 + k < mm && lane >= j0 + k && lane < mm)) to[k] = -1;
                cur[k] = to[k] >= 0 ? t.a[to[k]] : T(0);
            }
#pragma unroll
            for (int k = 0; k < kB; ++k) {
                if (j0 + k >= mm) break;
                if (to[k] >= 0) t.a[to[k]] = cur[k] + u[k];
            }
            __syncwarp();
            if (!more) break;
            ch = nch;
            j0 = nj;
            ri = rn;
            bv = bn;
#pragma unroll
            for (int k = 0; k < kB; ++k) u[k] = un[k];
        }
    }
    T my_inv = T(0);
    // FP64: the forward substitution rides along, row i's right-hand side in
    // lane i.  FP32 applies L11^-1 below, as the forward sweep does.
    T vi = t.v[lane];
    bool bad = false;
    for (int k = 0; k < nc; ++k) {
        T a = t.a[k * kWtLd + lane];
#pragma unroll 4
        for (int p = 0; p < k; ++p) a -= t.a[p * kWtLd + lane] * t.a[p * kWtLd + k];
        T d = __shfl_sync(kAll, a, k);
        const bool badk = !pivot_ok(d);
        bad |= badk;
        d = badk ? T(1) : d;
        T sq, inv;
        pivot_value(d, &sq, &inv);
        const bool below = lane > k && lane < f;
        const T lik = a * inv;
        if constexpr (!kInvDiag<T>) {
            const T yk = __shfl_sync(kAll, vi, k) * inv;
            vi = lane == k ? yk : (below ? vi - lik * yk : vi);
        }
        if (lane == k) {
            t.a[k * kWtLd + k] = sq;
            my_inv = inv;
        }
        if (below) t.a[k * kWtLd + lane] = lik;
        __syncwarp();
    }
    if (bad && lane == 0) atomicOr(singular_flags(F, W, s), FLAG_SINGULAR);
    if (lane < nc) reinterpret_cast<T*>(W.rdiag)[c0 + lane] = my_inv;
    T* L = lx + R.lx_off;
    const int row0 = kInvDiag<T> ? nc : 0;  // FP32 writes its diagonal block as L11^-1 below
    if (lane < f)
        for (int c = 0; c < nc; ++c)
            if (lane >= c && lane >= row0) L[lane + c * f] = t.a[c * kWtLd + lane];
    const int m = f - nc;
    T* Uo = ub + R.u_off;
    if constexpr (kInvDiag<T>) {
        for (int j = nc; j < f; j += 4) {
            T a[4];
            int jq[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                jq[q] = min(j + q, f - 1);
                a[q] = t.a[jq[q] * kWtLd + lane];
            }
#pragma unroll 2
            for (int p = 0; p < nc; ++p) {
                const T li = t.a[p * kWtLd + lane];
#pragma unroll
                for (int q = 0; q < 4; ++q) a[q] -= li * t.a[p * kWtLd + jq[q]];
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (j + q < f && lane >= j + q && lane < f) Uo[(lane - nc) + (j + q - nc) * m] = a[q];
        }
        // column j of L11^-1 by forward substitution, lane j; its entries
        // x_i (i > j) are kept transposed in the tile's free upper triangle,
        // at (row j, column i)
        if (lane < nc) t.rinv[lane] = my_inv;
        __syncwarp();
        if (lane < nc) {
            const int j = lane;
            for (int i = j + 1; i < nc; ++i) {
                T acc = -t.a[j * kWtLd + i] * my_inv;  // L_ij x_j with x_j = 1 / L_jj
#pragma unroll 4
                for (int k = j + 1; k < i; ++k) acc -= t.a[k * kWtLd + i] * t.a[k * kWtLd + j];
                t.a[i * kWtLd + j] = acc * t.rinv[i];
            }
        }
        __syncwarp();
        // L11^-1 into the diagonal block: lane i writes row i; y = L11^-1 v1
        T y = T(0);
        if (lane < nc) {
#pragma unroll 4
            for (int j = 0; j <= lane; ++j) {
                const T l = (j == lane) ? my_inv : t.a[lane * kWtLd + j];
                L[lane + j * f] = l;
                y += l * t.v[j];
            }
        }
        __syncwarp();
        if (lane < nc) {
            t.v[lane] = y;
            vi = y;
        }
        __syncwarp();
        if (lane >= nc) {
#pragma unroll 4
            for (int k = 0; k < nc; ++k) vi -= t.a[k * kWtLd + lane] * t.v[k];
        }
    } else {
        // the lower triangle folded (column p with column m - 1 - p) into rows of m + 1 entries
        const int total = m * (m + 1) / 2;
        for (int e = lane; e < total; e += 32) {
            const int pr = e / (m + 1), pos = e - pr * (m + 1);
            const bool first = pos < m - pr;
            const int j = nc + (first ? pr : m - 1 - pr);
            const int i = j + (first ? pos : pos - (m - pr));
            T a = t.a[j * kWtLd + i];
#pragma unroll 4
            for (int p = 0; p < nc; ++p) a -= t.a[p * kWtLd + i] * t.a[p * kWtLd + j];
            Uo[(i - nc) + (j - nc) * m] = a;
        }
    }
    if (lane < f) *rhs_entry<T>(sv, c0, nc, R.su_off, lane) = vi;
}

// u / d of an entry u and its column's pivot d: u times the reciprocal by the
// same means (y (1 + e + e^2), e = 1 - d y).  Outside the FP32 range a division:
// the reciprocal of a pivot below 2^-1024 is infinite.  A d that is not positive
// and finite is replaced by 1 and reported.
__device__ __forceinline__ double over_pivot(double u, double& d, bool& bad) {
    if (in_fp32_range(d)) {
        float yf;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(leading_fp32(d)));
        const double y = widen_fp32(yf);
        const double e = fma(-d, y, 1.0);
        return u * fma(y, fma(e, e, e), y);
    }
    if (!pivot_ok(d)) {
        bad = true;
        d = 1.0;
    }
    return slow_div(u, d);
}

// Column counters of an elimination within one CTA: a column's owner raises
// the counter after writing the column to shared memory, the other warps wait
// for it (the CTA's warps are all resident, so the owner always runs; the wait
// is bounded all the same).  A post is a store, so posts have to come in order:
// one warp makes them all, or a warp makes its own before it lets the next owner
// go on (a maximum instead costs the tiled panels' chain 2.5 % of a 10k- to
// 60k-bus pass).
__device__ __forceinline__ int wait_column(int* ready, int k, uint32_t* status) {
    const unsigned at = static_cast<unsigned>(__cvta_generic_to_shared(ready));
    int v;
    for (int spins = 0;; ++spins) {
        asm volatile("ld.acquire.cta.shared.b32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
        if (v >= k) break;
        if (spins > (1 << 22)) {
            atomicOr(status, FLAG_TIMEOUT);
            break;
        }
    }
    __syncwarp();
    return v;
}
__device__ __forceinline__ void post_column(int* ready, int k) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
        const unsigned at = static_cast<unsigned>(__cvta_generic_to_shared(ready));
        asm volatile("st.release.cta.shared.b32 [%0], %1;" ::"r"(at), "r"(k) : "memory");
    }
}

// Hand-over of one column between two warps on the chain, by a named barrier
// of 64 threads (about 35 cycles; the counter above takes about 140).
__device__ __forceinline__ void hand_over(int k) {
    asm volatile("bar.arrive %0, 64;" ::"r"(1 + (k & 7)) : "memory");
}
__device__ __forceinline__ void take_over(int k) { asm volatile("bar.sync %0, 64;" ::"r"(1 + (k & 7)) : "memory"); }

// Shared-memory scratch of one front besides the front itself.
template <typename T, int KP>
struct FrontSmem;
template <int KP>
struct FrontSmem<float, KP> {
    static constexpr int kLd = KP + 4;
    __align__(16) float lt[KP * kLd];  // lt[c * kLd + r] = L11[r][c] of the current panel
    float li[KP * (KP + 1)];        // L11^-1, column c at li + c * (KP + 1)
    float rinv[KP];                 // 1 / L11[c][c]
    float v[kSmallFrontMax32];      // right-hand side of the front's rows
};
template <int KP>
struct FrontSmem<double, KP> {
    double ms[KP][kPanel];      // column k of the current panel's block, unscaled, over its pivot
    double dk[KP];              // pivots, then 1 / sqrt
    int ready, ready_x;         // columns published: first 32 rows, rows below
};

// Front s with its gain entries and its children's update matrices, in shared
// memory (Fm holds front_ld(f) x f values), and its right-hand side (entry r at
// rhs[r * rhs_ld]): the factorisation carries the forward substitution along.
// The forward sweep of its own follows the same chain of the elimination tree
// as the factorisation, reading every L panel back: 1.04 ms of a 4.4 ms step at
// 200k buses (mixed), 0.56 of 7.1 at 60k (FP64); carried along, y costs each
// front a few hundred cycles.  FP32 keeps the sweep's order of operations
// (y = L11^-1 v per panel, then the rows below column by column): same bits.
template <typename T>
__device__ __forceinline__ void front_assemble(const DevFactor& F, const SolveVecs& sv, const T* gv, const T* lx,
                                               const T* ub, const FrontRec& R, T* Fm, T* rhs, int rhs_ld) {
    const int f = R.f, c0 = R.c0, nc = R.nc;
    const int ldf = front_ld<T>(f);
    const int tid = threadIdx.x, nth = blockDim.x;
    // the first targets in flight while the front is cleared
    const bool has = R.tgt0 + tid < R.tgt1;
    const int l0 = has ? F.tgt_local[R.tgt0 + tid] : 0;  // row + col * f
    const T g0 = has ? gv[R.tgt0 + tid] : T(0);
    if constexpr (sizeof(T) == 4) {
        for (int x = 4 * tid; x < ldf * f; x += 4 * nth) *reinterpret_cast<float4*>(Fm + x) = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
        for (int x = 2 * tid; x < ldf * f; x += 2 * nth) *reinterpret_cast<double2*>(Fm + x) = make_double2(0.0, 0.0);
    }
    __syncthreads();
    auto at = [&](int l) {
        const int c = l / f;
        return (l - c * f) + c * ldf;
    };
    if (has) Fm[at(l0)] = g0;
    for (int tg = R.tgt0 + tid + nth; tg < R.tgt1; tg += nth) Fm[at(F.tgt_local[tg])] = gv[tg];
    for (int r = tid; r < f; r += nth) rhs[r * rhs_ld] = r < nc ? static_cast<const T*>(sv.rhs)[c0 + r] : T(0);
    __syncthreads();
    extend_add_children<T>(F, sv, lx, ub, R, Fm, ldf, rhs, rhs_ld);
    __syncthreads();
}

// The finished front's L panel, update matrix and right-hand side to the factor
// and solve arrays.
template <typename T>
__device__ __forceinline__ void front_store(const SolveVecs& sv, T* lx, T* ub, const FrontRec& R, const T* Fm,
                                            const T* rhs, int rhs_ld) {
    const int f = R.f, c0 = R.c0, nc = R.nc;
    const int ldf = front_ld<T>(f);
    const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, warp = tid >> 5;
    for (int r = tid; r < f; r += nth) *rhs_entry<T>(sv, c0, nc, R.su_off, r) = rhs[r * rhs_ld];
    const int nwarp = nth >> 5, m = f - nc;
    T* L = lx + R.lx_off;
    for (int c = warp; c < nc; c += nwarp)
        for (int r = (c & ~31) + lane; r < f; r += 32) L[r + c * f] = Fm[r + c * ldf];
    T* U = ub + R.u_off;
    for (int j = warp; j < m; j += nwarp)
        for (int i = (j & ~31) + lane; i < m; i += 32) U[i + j * m] = Fm[(nc + i) + (nc + j) * ldf];
}

// Assembles and partially factorises front s in shared memory, FP64, with
// panels of KP columns.  Bound: the FP64 pipe (a warp instruction per 19
// cycles of the SM) and the pivots' chain, as in k_big_panel64, whose elimination
// the panels use: warp w owns the panel's columns w (mod 8), a lane per row,
// in registers; a column's unscaled rows are published in its place in Fm and
// its block's rows over the pivot in ms; the rows past the first 32 follow one
// column behind.  The trailing update takes one entry per thread, the lower
// triangle folded (column p with column m - 1 - p) into rows of m + 1 entries
// (then the right-hand side, which is row f of the front),
// so that no lane idles.  Measured on a 30k-bus grid, against one warp's
// factorisation of the block, a thread per row below it and 4 x 4 tiles in the
// update: phase B 337 -> 202 us, phase A 261 -> 159, synchronous levels 82 -> 50.
// An FP64 instruction costs the same with every lane off, so row groups and
// columns that a panel does not have are left by branches, not by predicates
// (2003 buses: phase A 137 -> 122 us, synchronous levels 97 -> 64).
template <int KP>
__device__ void front_factor(const DevFactor& F, const DevWork& W, const SolveVecs& sv, const double* gv, double* lx,
                             double* ub, const FrontRec& R, int s, double* Fm, FrontSmem<double, KP>& sm) {
    static_assert(KP <= kPanel && kThreads == 256, "columns over eight warps");
    constexpr int kW = kThreads / 32, kQ = KP / kW;
    constexpr int kG = ((KP == kPanel ? kSmallFrontMax : kFlowSmallFMax) + 1 + 31) / 32;  // row groups of 32
    const int f = R.f, c0 = R.c0, nc = R.nc;
    const int ldf = front_ld<double>(f);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    front_assemble<double>(F, sv, gv, lx, ub, R, Fm, Fm + f, ldf);
    double* rdg = reinterpret_cast<double*>(W.rdiag) + c0;
    uint32_t* status = &W.status->flags;
#pragma unroll 1
    for (int k0 = 0; k0 < nc; k0 += KP) {
        const int kb = min(KP, nc - k0);
        const int nrow = f + 1 - k0;  // with the right-hand-side row
        const int ng = (nrow + 31) >> 5;  // <= kG
        double* P = Fm + k0 + (int64_t)k0 * ldf;  // P[r + c * ldf]: row k0 + r, column k0 + c
        if (tid == 0) sm.ready = sm.ready_x = -1;
        double a[kQ][kG];
#pragma unroll
        for (int q = 0; q < kQ; ++q)
#pragma unroll
            for (int g = 0; g < kG; ++g) {
                const int c = w + kW * q, r = 32 * g + lane;
                a[q][g] = (c < kb && r < nrow) ? P[r + c * ldf] : 0.0;
            }
        __syncthreads();
        bool bad = false;
        auto publish = [&](double& aq, int k) {
            double d = __shfl_sync(0xffffffffu, aq, k);
            if (lane < nrow) P[lane + k * ldf] = aq;
            sm.ms[k][lane] = over_pivot(aq, d, bad);
            post_column(&sm.ready, k);  // before the next owner can post its own
            if (k + 1 < kb) hand_over(k);
            if (lane == k) aq = d;
            if (lane == 0) sm.dk[k] = d;
        };
        if (w == 0) publish(a[0][0], 0);
#pragma unroll
        for (int qq = 0; qq < kQ; ++qq) {
#pragma unroll 1
            for (int kk = 0; kk < kW; ++kk) {
                const int k = kW * qq + kk;
                if (k >= kb) break;
                const bool next = w == ((kk + 1) & (kW - 1)) && k + 1 < kb;
                if (next) take_over(k);
                else wait_column(&sm.ready, k, status);
                const double ub0 = lane < nrow ? P[lane + k * ldf] : 0.0;
                int done = k;
                if (next) {
                    const double m = sm.ms[k][k + 1];
                    if (kk + 1 < kW) {
                        a[qq][0] = fma(-ub0, m, a[qq][0]);
                        publish(a[qq][0], k + 1);
                    } else if (qq + 1 < kQ) {
                        const int qn = qq + 1 < kQ ? qq + 1 : kQ - 1;
                        a[qn][0] = fma(-ub0, m, a[qn][0]);
                        publish(a[qn][0], k + 1);
                    }
                    done = k + 1;
                }
#pragma unroll
                for (int q = qq; q < kQ; ++q) {
                    const int c = w + kW * q;
                    if (c > done && c < kb) a[q][0] = fma(-ub0, sm.ms[k][c], a[q][0]);
                }
                if (ng > 1) {
                    // the rows past the first 32: columns behind k - 1 by column k - 1, then column k is final
                    if (k > 0) {
                        wait_column(&sm.ready_x, k - 1, status);
#pragma unroll
                        for (int g = 1; g < kG; ++g) {
                            if (g >= ng) break;
                            const double u = (32 * g + lane < nrow) ? P[32 * g + lane + (k - 1) * ldf] : 0.0;
#pragma unroll
                            for (int q = qq; q < kQ; ++q) {
                                const int c = w + kW * q;
                                if (c >= kb) break;
                                if (c >= k) a[q][g] = fma(-u, sm.ms[k - 1][c], a[q][g]);
                            }
                            if (w == kk && 32 * g + lane < nrow) P[32 * g + lane + k * ldf] = a[qq][g];
                        }
                        if (w == kk) post_column(&sm.ready_x, k);
                    } else if (w == 0) {
                        post_column(&sm.ready_x, 0);  // column 0 is in place
                    }
                }
            }
        }
        if (bad && lane == 0) atomicOr(singular_flags(F, W, s), FLAG_SINGULAR);
        __syncthreads();
        if (w == 0 && lane < kb) {
            double sq, rs;
            pivot_value(sm.dk[lane], &sq, &rs);
            sm.dk[lane] = rs;
            rdg[k0 + lane] = rs;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
            const int c = w + kW * q;
            if (c >= kb) break;
            const double rs = sm.dk[c];
#pragma unroll
            for (int g = 0; g < kG; ++g) {
                if (g >= ng) break;
                if (32 * g + lane < nrow) P[32 * g + lane + c * ldf] = a[q][g] * rs;
            }
        }
        __syncthreads();
        const int q0 = k0 + kb, m = f - q0;
        const int tri = m * (m + 1) / 2;
        const double* X = Fm + k0 * ldf;
        for (int t = tid; t < tri + m; t += kThreads) {  // the last m: the right-hand-side row
            const int pr = t / (m + 1), pos = t - pr * (m + 1);
            const bool first = pos < m - pr;
            const int j = q0 + (t >= tri ? t - tri : first ? pr : m - 1 - pr);
            const int i = t >= tri ? f : j + (first ? pos : pos - (m - pr));
            double acc = Fm[i + j * ldf];
#pragma unroll 8
            for (int k = 0; k < kb; ++k) acc = fma(-X[i + k * ldf], X[j + k * ldf], acc);
            Fm[i + j * ldf] = acc;
        }
        __syncthreads();
    }
    front_store<double>(sv, lx, ub, R, Fm, Fm + f, ldf);
}

// FP32, with panels of KP <= kPanel columns.
template <int KP>
__device__ void front_factor(const DevFactor& F, const DevWork& W, const SolveVecs& sv, const float* gv, float* lx,
                             float* ub, const FrontRec& R, int s, float* Fm, FrontSmem<float, KP>& sm) {
    using T = float;
    static_assert(KP <= kPanel && KP <= 32, "panel wider than a warp");
    const int f = R.f, c0 = R.c0, nc = R.nc;
    const int ldf = front_ld<T>(f);
    const int tid = threadIdx.x, nth = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5;
    front_assemble<T>(F, sv, gv, lx, ub, R, Fm, sm.v, 1);
    // v_i -= L_i,k0.. y of a finished panel, by threads [t0, t0 + nt)
    auto rhs_below = [&](int k0, int kb, int t0, int nt) {
        for (int i = k0 + kb + tid - t0; tid >= t0 && i < f; i += nt) {
            float acc = sm.v[i];
            for (int k = 0; k < kb; ++k) acc -= Fm[i + (k0 + k) * ldf] * sm.v[k0 + k];
            sm.v[i] = acc;
        }
    };
    T* rdg = reinterpret_cast<T*>(W.rdiag) + c0;
#pragma unroll 1
    for (int k0 = 0; k0 < nc; k0 += KP) {
        const int kb = min(KP, nc - k0);
        // (1) diagonal block, one warp
        if (warp == 0) {
            constexpr int kLd = FrontSmem<float, KP>::kLd;
            float* P = Fm + k0 + k0 * ldf;
            float my_inv;
            const bool bad = warp_potrf(kb, lane, sm.lt, kLd, &my_inv, [&](int j) { return P[lane + j * ldf]; });
            if (lane < kb) {
                sm.rinv[lane] = my_inv;
                rdg[k0 + lane] = my_inv;
            }
            if (bad && lane == 0) atomicOr(singular_flags(F, W, s), FLAG_SINGULAR);
        } else if (k0 > 0) {
            rhs_below(k0 - KP, KP, 32, nth - 32);  // the other warps meanwhile: the previous panel's y
        }
        __syncthreads();
        // (2) warp 0 inverts the diagonal block, which then goes into its slot;
        // the other threads: rows below the block, x = a L11^-T, one row per
        // thread (f - q0 < kThreads - 32)
        const int q0 = k0 + kb;
        if (warp == 0) {
            constexpr int kLd = FrontSmem<float, KP>::kLd;
            warp_trinv(sm.lt, kLd, sm.rinv, kb, lane, sm.li, KP + 1);
            __syncwarp();
            for (int j = 0; j < kb; ++j)
                if (lane >= j && lane < kb) Fm[k0 + lane + (k0 + j) * ldf] = sm.li[lane + j * (KP + 1)];
        } else {
            const int r = q0 + tid - 32;
            if (r < f) row_trsm(sm.lt, FrontSmem<float, KP>::kLd, sm.rinv, kb, Fm + r + k0 * ldf, ldf);
        }
        __syncthreads();
        // y = L11^-1 v of the panel's rows, a lane per row (as in the forward sweep)
        if (warp == 0) {
            float y = 0.f;
            if (lane < kb)
                for (int j = 0; j <= lane; ++j) y += sm.li[lane + j * (KP + 1)] * sm.v[k0 + j];
            __syncwarp();
            if (lane < kb) sm.v[k0 + lane] = y;
        }
        // (3) trailing update of the lower triangle, 4x4 tiles on 4-aligned
        // rows; tiles are numbered down each tile column so that neighbouring
        // threads touch neighbouring rows (conflict-free vector accesses)
        if (q0 < f) {
            const int R0 = q0 & ~3;
            const int nt = (f - R0 + 3) >> 2;
            const int ntiles = nt * (nt + 1) / 2;
            const float b2 = 2.f * nt + 1.f;
#pragma unroll 1
            for (int t = tid; t < ntiles; t += nth) {
                // column bj holds tiles bi = bj..nt-1 and starts at bj*nt - bj*(bj-1)/2
                int bj = static_cast<int>((b2 - sqrtf(b2 * b2 - 8.f * t)) * 0.5f);
                bj = max(0, min(bj, nt - 1));
                while (bj > 0 && bj * nt - bj * (bj - 1) / 2 > t) --bj;
                while (bj + 1 < nt && (bj + 1) * nt - (bj + 1) * bj / 2 <= t) ++bj;
                const int bi = bj + (t - (bj * nt - bj * (bj - 1) / 2));
                const int i0 = R0 + 4 * bi, j0 = R0 + 4 * bj;
                T acc[4][4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int v = 0; v < 4; ++v) acc[u][v] = T(0);
#pragma unroll 2
                for (int c = 0; c < kb; ++c) {
                    const T* col = Fm + (k0 + c) * ldf;
                    T av[4], bv[4];
                    load4(col + i0, av);
                    load4(col + j0, bv);
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll
                        for (int v = 0; v < 4; ++v) acc[u][v] += av[u] * bv[v];
                }
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const int j = j0 + v;
                    if (j < q0 || j >= f) continue;
                    T* dst = Fm + i0 + j * ldf;
                    T cur[4];
                    load4(dst, cur);
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (i0 + u >= j && i0 + u < f) cur[u] -= acc[u][v];
                    store4(dst, cur);
                }
            }
        }
        __syncthreads();
    }
    const int kl = (nc - 1) / KP * KP;  // the last panel (nc > 0)
    rhs_below(kl, nc - kl, 0, nth);
    __syncthreads();
    front_store<T>(sv, lx, ub, R, Fm, sm.v, 1);
}

// Panel widths: fronts of dataflow phase A (f <= kFlowSmallFMax) use 16-column
// panels and a register budget for several CTAs per SM; the rest use 32-column
// panels and the full register file (one CTA per SM anyway).  A launch's CTAs
// take the shared memory of its widest front (FP64, 128 rows: 135 KB, one CTA
// per SM), so the budget pays where a phase's fronts are narrow: 64 grids of 30
// to 5000 buses FP64 8.49 ms a pass with it, 8.87 without; single grids of 2000
// to 60k buses the same either way.
constexpr int kPanelSmall = kPanelFlowA;
template <typename T>
constexpr int kMinBlocksA = sizeof(T) == 4 ? 3 : 2;

// Threads of a front's CTA: the wide FP32 fronts (phase B, synchronous levels)
// have an SM to themselves, and sixteen warps keep twice the children's loads
// and update tiles in flight that eight do.
template <typename T, int KP>
constexpr int kFrontThreads = 32 * asm_warps(sizeof(T) == 4, KP == kPanel);

template <typename T>
__global__ void __launch_bounds__(kFrontThreads<T, kPanel>, 1) k_front_small(DevFactor F, DevWork W, SolveVecs sv, const T* gv, T* lx,
                                                             T* ub, const int* fronts) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ FrontSmem<T, kPanel> sm;
    const int s = fronts[blockIdx.x];
    const FrontRec R = F.rec[s];
    if (front_frozen(W, R)) return;
    front_factor<kPanel>(F, W, sv, gv, lx, ub, R, s, reinterpret_cast<T*>(smem_raw), sm);
}

// ---------------------------------------------------------------------------
// Dataflow scheduling: a persistent grid claims work items in order from an
// atomic counter; an item waits (bounded) until the items it depends on have
// published their completion flag.  Items are ordered so that every
// dependency is claimed earlier, and a CTA only waits on items already
// claimed by running CTAs, so progress never depends on CTAs that have not
// started.  Data produced inside the pass is read with L1-bypassing loads.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void wait_done(const int* flag, uint32_t* status, long long limit) {
    for (long long spins = 0;;) {
        int v;
        asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
        if (v != 0) return;
        if (++spins > limit) {
            atomicOr(status, FLAG_TIMEOUT);
            return;
        }
        __nanosleep(32);
    }
}

__device__ __forceinline__ void publish_done(int* flag) {
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    asm volatile("st.relaxed.gpu.global.b32 [%0], 1;" ::"l"(flag) : "memory");
}

// Thread 0 alone claims, waits and publishes; each such step is followed by
// __syncwarp() so that warp 0 is converged again before the block barrier
// (the single-warp phases of a front rely on a converged warp 0).
__device__ __forceinline__ int claim(int* counter, int* slot) {
    __syncthreads();
    if (threadIdx.x == 0) *slot = atomicAdd(counter, 1);
    __syncwarp();
    __syncthreads();
    return *slot;
}

// Forward sweep, after front s is complete (all threads past a barrier): thread 0
// counts s into its parent's completed children; the CTA that completes the
// last child of a parent continues with that parent.  Returns the next front
// or -1.
__device__ __forceinline__ int continue_up(const DevFactor& F, const int32_t* nchild, int* cnt, int s, int* slot) {
    if (threadIdx.x == 0) {
        int nxt = -1;
        const int p = F.sn_parent[s];
        if (p >= 0) {
            __threadfence();
            if (atomicAdd(cnt + p, 1) + 1 == nchild[p]) {
                __threadfence();
                nxt = p;
            }
        }
        *slot = nxt;
    }
    __syncwarp();
    __syncthreads();
    return *slot;
}

template <typename T, int KP, int kMinBlocks>
__global__ void __launch_bounds__(kFrontThreads<T, KP>, kMinBlocks) k_front_flow(DevFactor F, DevWork W, SolveVecs sv, const T* gv,
                                                                     T* lx, T* ub, const int* ready, const int* n_ready,
                                                                     int* counter, int* cnt) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ FrontSmem<T, KP> sm;
    __shared__ int slot;
    const int nr = *n_ready;
    for (;;) {
        const int item = claim(counter, &slot);
        if (item >= nr) break;
        int s = ready[item];
        while (s >= 0) {
            const FrontRec R = F.rec[s];
            if (!front_frozen(W, R)) front_factor<KP>(F, W, sv, gv, lx, ub, R, s, reinterpret_cast<T*>(smem_raw), sm);
            __syncthreads();
            if (threadIdx.x == 0) slot = count_up(R, cnt);
            __syncwarp();
            __syncthreads();
            s = slot;
        }
    }
}

// ---------------------------------------------------------------------------
// Big fronts, in place (L panel and update matrix share the f x f region at
// sn_lx_off with ld = f).  Work lists: LevelSchedule.
// ---------------------------------------------------------------------------
// Assembly of a tiled front, one CTA per (tile column tj, block rb of
// kAsmRows rows from the tile's first column down): the block's G entries, then
// the update-matrix entries of the children that land in it, child by child (a
// barrier between children keeps every entry's sum in child order, as in the
// single-CTA fronts).  The block's target range and its contributing children
// with their column and row ranges come from the host schedule (AsmItem /
// AsmChild).  Bound: load latency, child after child, and the instructions
// of the columns and rows that a child does not have (four columns a warp, four
// rows a lane; most children have fewer): a warp leaves both loops at the
// child's end.  The block is summed in shared memory and written once.  A level
// at 60k buses FP64 20 us as read-modify-writes of the front, 18.5 in shared
// memory, 12.3 without the empty columns and rows; at 200k mixed 18.0 -> 11.9
// (two children in flight: 12.1 and 13.5, more registers).
// Row block 0 also assembles the tile column's right-hand-side entries: it
// holds the diagonal, so its list has every child with a column here.
template <typename T>
__global__ void __launch_bounds__(kThreads) k_big_assemble(DevFactor F, DevWork W, SolveVecs sv, const T* gv, T* lx,
                                                           T* ub, const AsmItem* work, const AsmChild* kids) {
    static_assert(kThreads == 256 && kTile == 32 && kAsmRows == 128, "four columns a warp, four rows a lane");
    constexpr int kKids = 32;
    __shared__ T tile[kTile * kAsmRows];  // [c][r]
    __shared__ T vv[kTile];
    __shared__ AsmChild ks[kKids];
    const AsmItem wk = work[blockIdx.x];
    const int s = wk.s, tj = wk.tj, rb = wk.rb;
    const FrontRec R = F.rec[s];
    if (front_frozen(W, R)) return;  // the whole CTA, before any barrier
    const int f = R.f, nc = R.nc;
    T* B = lx + R.lx_off;
    const int c0 = tj * kTile, c1 = min(c0 + kTile, f);
    const int R0 = c0 + rb * kAsmRows, R1 = min(R0 + kAsmRows, f);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int nwarp = kThreads / 32;
    if (rb == 0 && tid < kTile) vv[tid] = c0 + tid < nc ? static_cast<const T*>(sv.rhs)[R.c0 + c0 + tid] : T(0);
    for (int x = tid; x < kTile * kAsmRows; x += kThreads) tile[x] = T(0);
    __syncthreads();
    for (int tg = wk.tg_lo + tid; tg < wk.tg_hi; tg += kThreads) {
        const int l = F.tgt_local[tg];
        const int c = l / f, r = l - c * f;
        if (r >= R0 && r < R1) tile[(c - c0) * kAsmRows + r - R0] = gv[tg];
    }
    // one child's part, loaded while the one before is waited for
    struct Part {
        T u[4][4], b;
        int ri[4], pj[4], pb;
    };
    auto load = [&](const AsmChild& ch, Part& x) {
        const int* rel = F.sn_relmap + ch.su_off;
        const T* U = (ch.big ? lx : ub) + ch.u_off;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int i = ch.ilo + lane + 32 * t;
            x.ri[t] = i < ch.ihi ? rel[i] - R0 : -1;
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int j = ch.j0 + warp + nwarp * a;
            if (j >= ch.j1) break;  // the whole warp
            x.pj[a] = rel[j] - c0;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int i = ch.ilo + lane + 32 * t;
                x.u[a][t] = (i >= j && i < ch.ihi) ? U[(int64_t)j * ch.ld + i] : T(0);
            }
        }
        x.pb = -1;
        x.b = T(0);
        if (rb == 0 && warp == nwarp - 1 && ch.j0 + lane < ch.j1) {
            x.pb = rel[ch.j0 + lane] - c0;
            x.b = static_cast<const T*>(sv.su)[ch.su_off + ch.j0 + lane];
        }
    };
    for (int cb = wk.ch_lo; cb < wk.ch_hi; cb += kKids) {
        const int n = min(kKids, wk.ch_hi - cb);
        constexpr int kW16 = sizeof(AsmChild) / 16;
        static_assert(kKids * kW16 <= kThreads, "one 16-byte word per thread");
        if (tid < n * kW16) reinterpret_cast<int4*>(ks)[tid] = reinterpret_cast<const int4*>(kids + cb)[tid];
        __syncthreads();
        Part x;
        load(ks[0], x);
        for (int q = 0; q < n; ++q) {
            const AsmChild& ch = ks[q];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const int j = ch.j0 + warp + nwarp * a;
                if (j >= ch.j1) break;  // the whole warp
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const int i = ch.ilo + 32 * t;
                    if (i >= ch.ihi) break;
                    if (x.ri[t] >= 0 && i + lane >= j) tile[x.pj[a] * kAsmRows + x.ri[t]] += x.u[a][t];
                }
            }
            if (x.pb >= 0) vv[x.pb] += x.b;
            if (q + 1 < n) load(ks[q + 1], x);
            __syncthreads();
        }
    }
    __syncthreads();
    for (int c = warp; c < c1 - c0; c += nwarp)
        for (int r = lane; r < R1 - R0; r += 32)
            if (R0 + r >= c0 + c) B[R0 + r + (int64_t)(c0 + c) * f] = tile[c * kAsmRows + r];
    if (rb == 0 && tid < c1 - c0) *rhs_entry<T>(sv, R.c0, nc, R.su_off, c0 + tid) = vv[tid];
}

// FP64 panel step p of the tiled fronts: the diagonal block's factorisation
// and the rows below it, one CTA per kPanelRows64 rows (each factors the
// block itself; the CTA that reads the block last writes it back, so no CTA
// reads an overwritten block and none waits for another).
//
// Bound: an FP64 warp instruction has a latency of 60 cycles and an SM finishes
// one in 19, however many lanes are active.  So what counts is the serial chain
// of the pivots, the number of FP64 instructions beside it, and that few of them
// are in flight at a time: with more than three, each one on the chain waits.  The
// elimination is a_ij -= u_i (u_j / d) with the unscaled column u, so a pivot's
// chain is one update, a reciprocal (3 instructions; a square root takes 10) and
// the product u / d; the square roots of all pivots come together at the end.
// Warp roles:
//  - one warp runs the chain, alone on its scheduler: it takes column k + 2 as
//    the others left it (updated by the pivots before k), applies the pivots k
//    and k + 1 itself and publishes u and u / d, a lane per row;
//  - four warps bring the columns to that point, each a column from its first
//    pivot to its last in the order the chain needs them (columns from 16 on in
//    pairs, 16 rows each);
//  - two warps solve the chunk, eight rows each, four columns an instruction, so
//    that they wait for the chain only.
// Columns reach the chain over named barriers (a flag cost it 170 cycles).  With
// the columns dealt round eight warps, each in turn on the chain, a pivot took
// about 1000 cycles and a full step 37k; with this 650 to 700 (alone on the SM the
// chain takes 600) and 25k.  On average over a 60k-bus grid's steps 18.1 -> 13.5
// us (47 + 22 us as one warp's factorisation and a launch of one-warp row solves);
// two warps for the columns or one for the chunk are slower (20 to 33 us against
// 18 with the launch).  A second CTA of an SM has its chain on another scheduler.
__global__ void __launch_bounds__(kPanelThreads64, 2) k_big_panel64(DevFactor F, DevWork W, SolveVecs sv, double* lx,
                                                                 const int4* work, int p, int* step_cnt) {
    static_assert(kPanelThreads64 == 256 && kPanelRows64 == 16 && kTile == 32, "warp roles below");
    constexpr int kW = kPanelThreads64 / 32;
    __shared__ double us[kTile][kTile];  // column k as eliminated so far, then final (u)
    __shared__ double ms[kTile][kTile];  // u / d
    __shared__ double dk[kTile];         // pivots, then 1 / sqrt
    __shared__ int ready;                // pivots published
    __shared__ int last;
    const int4 wk = work[blockIdx.x];
    const int s = wk.x, chunk = wk.y;
    if (front_frozen(F, W, s)) return;  // the whole CTA, before any barrier
    const int f = F.sn_f[s];
    const int c0 = F.sn_c0[s];
    const int nc = F.sn_c0[s + 1] - c0;
    double* B = lx + F.sn_lx_off[s];
    const int p0 = p * kTile;
    const int pb = min(kTile, nc - p0);
    const int r0 = p0 + pb + chunk * kPanelRows64;
    const int nr = min(kPanelRows64, f + 1 - r0);  // row f: the right-hand side
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int role = (w - static_cast<int>(blockIdx.x / kSMs)) & (kW - 1);
    // chunk: entry (r0 + xr, p0 + c), column stride 1 in the right-hand-side row
    const int xr = 8 * (role & 1) + (lane & 7), xg = lane >> 3;
    const bool solves = role == 5 || role == 6, in = solves && xr < nr;
    double* const xb = r0 + xr == f ? static_cast<double*>(sv.sol) + c0 + p0 : B + (r0 + xr) + (int64_t)p0 * f;
    const int64_t xld = r0 + xr == f ? 1 : f;
    if (threadIdx.x == 0) ready = -1;
    double x[kTile / 4];  // columns 4 i + xg
#pragma unroll
    for (int i = 0; i < kTile / 4; ++i) x[i] = (in && 4 * i + xg < pb) ? xb[(4 * i + xg) * xld] : 0.0;
    {
        double a[kTile / kW];
#pragma unroll
        for (int q = 0; q < kTile / kW; ++q) {
            const int c = w + kW * q;
            a[q] = (c < pb && lane >= c && lane < pb) ? B[(p0 + lane) + (int64_t)(p0 + c) * f] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < kTile / kW; ++q) us[w + kW * q][lane] = a[q];
    }
    __syncthreads();
    bool bad = false;
    uint32_t* status = &W.status->flags;
    int seen = -1;  // pivots known to be published
    if (role == 0) {
        double cur = us[0][lane], next = us[1][lane];
#pragma unroll 1
        for (int k = 0; k < pb; ++k) {
            double d = __shfl_sync(0xffffffffu, cur, k);
            const double m = over_pivot(cur, d, bad);
            us[k][lane] = lane == k ? d : cur;
            ms[k][lane] = m;
            if (lane == 0) dk[k] = d;
            post_column(&ready, k);
            double after = 0.0;
            if (k + 2 < pb) {
                if (k > 0) take_over(k + 2);
                after = us[k + 2][lane];
            }
            const double m1 = __shfl_sync(0xffffffffu, m, k + 1), m2 = __shfl_sync(0xffffffffu, m, k + 2);
            const double u = cur;
            cur = fma(-u, m1, next);
            next = fma(-u, m2, after);
        }
    } else if (solves) {
#pragma unroll
        for (int k = 0; k < kTile; ++k) {
            constexpr int kG = kTile / 4;
            if (k >= pb) break;
            if (seen < k) seen = wait_column(&ready, k, status);
            const double u = __shfl_sync(0xffffffffu, x[k / 4], 8 * (k & 3) + (lane & 7));
            if ((k & 3) < 3) {
                const double xn = fma(-u, ms[k][4 * (k / 4) + xg], x[k / 4]);
                if (xg > (k & 3)) x[k / 4] = xn;
            }
#pragma unroll
            for (int i = k / 4 + 1; i < kG; ++i) x[i] = fma(-u, ms[k][4 * i + xg], x[i]);
        }
    } else if (role == 4) {
        // shares the chain's scheduler and stays out of its way; this CTA has read the block
        if (lane == 0) last = atomicAdd(step_cnt + wk.w, 1) == wk.z - 1;
    } else {
        constexpr unsigned kOwner = 0x273173u;
        // entry (row, c) by the pivots up to k1
        auto eliminate = [&](double& a, int row, int c, int k, int k1) {
            while (k <= k1) {
                if (seen < k) seen = wait_column(&ready, k, status);
                const int hi = min(k1, max(seen, k));
#pragma unroll 4
                for (; k <= hi; ++k) a = fma(-us[k][row], ms[k][c], a);
            }
        };
        // columns 3..15, then the pairs from 16 on; roles 3 and 7, whose scheduler has no
        // solver, take two of three
        for (int i = 0; i < 13 + 8; ++i) {
            if (static_cast<int>((kOwner >> (4 * (i % 6))) & 15u) != role) continue;
            const int c = i < 13 ? 3 + i : 16 + 2 * (i - 13);
            if (c >= pb) break;
            if (c < 16) {
                double a = us[c][lane];
                eliminate(a, lane, c, 0, c - 3);
                us[c][lane] = a;
                hand_over(c);
            } else {
                const int row = 16 + (lane & 15), h = lane >> 4;
                double a = us[c + h][row];
                eliminate(a, row, c + h, 0, c - 3);
                if (h == 0) us[c][row] = a;
                __syncwarp();
                hand_over(c);
                if (c + 1 >= pb) break;
                eliminate(a, row, c + h, c - 2, c - 2);
                if (h == 1) us[c + 1][row] = a;
                __syncwarp();
                hand_over(c + 1);
            }
        }
    }
    __syncthreads();  // every pivot is in dk
    if (bad && lane == 0 && chunk == 0) atomicOr(singular_flags(F, W, s), FLAG_SINGULAR);
    if (w == 0 && lane < pb) {
        double sq, rs;
        pivot_value(dk[lane], &sq, &rs);
        dk[lane] = rs;
        if (chunk == 0) reinterpret_cast<double*>(W.rdiag)[c0 + p0 + lane] = rs;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kTile / 4; ++i) {
        const int c = 4 * i + xg;
        if (in && c < pb) xb[c * xld] = x[i] * dk[c];
    }
    if (last) {
#pragma unroll
        for (int q = 0; q < kTile / kW; ++q) {
            const int c = w + kW * q;
            if (c < pb && lane >= c && lane < pb) B[(p0 + lane) + (int64_t)(p0 + c) * f] = us[c][lane] * dk[c];
        }
    }
}

// Loads of front entries in the tiled-front kernels.  kL2: the entry may have
// been written by another CTA of the same launch (the dataflow kernel), so
// the load bypasses L1.
template <bool kL2, typename T>
__device__ __forceinline__ T ld_entry(const T* p) {
    if constexpr (kL2) return __ldcg(p);
    else return *p;
}

// FP32 panel step p of the tiled fronts.  The rows below the diagonal block
// are cut into chunks of kPanelRows, one CTA each.  Every CTA stages the block
// and its chunk, factors the 32 x 32 diagonal block itself and inverts it (warp
// 0), and solves the chunk as X = A L_dd^-T = A (L_dd^-1)^T, a register-tiled
// product with 4 x 4 outputs per thread.  The CTA that reads the diagonal
// tile last (a counter per front and step) writes L_dd^-1 into it for the
// solves: no CTA reads an overwritten tile, and none waits for another.
template <bool kL2>
__device__ __forceinline__ void big_panel32_item(const DevFactor& F, const DevWork& W, const SolveVecs& sv, float* lx,
                                                 int s, int p, int chunk, int nchunk, int pair, int* step_cnt) {
    static_assert(kThreads == 256 && kPanelRows == 128 && kTile == 32, "thread tiling below");
    constexpr int ld = kTile + 4;          // 16-byte aligned rows
    constexpr int lt_ld = kTile + 4;       // 16-byte aligned rows
    constexpr int as_ld = kPanelRows + 4;  // 16-byte aligned rows
    __shared__ __align__(16) float D[kTile * ld];  // D[i + j * ld]: the block, then L_dd
    __shared__ float rdiag[kTile];
    __shared__ __align__(16) float Lt[kTile * lt_ld];  // Lt[k][c] = L_dd^-1[c][k]
    __shared__ __align__(16) float As[kTile * as_ld];  // As[k][r] = A[r0 + r][k], then X
    __shared__ int last;
    const int f = F.sn_f[s];
    const int nc = F.sn_c0[s + 1] - F.sn_c0[s];
    float* B = lx + F.sn_lx_off[s];
    const int p0 = p * kTile;
    const int pb = min(kTile, nc - p0);
    const int r0 = p0 + pb + chunk * kPanelRows;     // first row of the chunk
    const int nr = max(0, min(kPanelRows, f - r0));  // its rows
    const int tid = threadIdx.x;
    // From the second step on, the previous step's trailing update has already
    // factored and inverted this diagonal block: its slot holds L_dd^-1, the
    // pivots are checked and rdiag is written.
    const bool pre = p > 0;
    {
        // all staging loads in flight before the first shared-memory store:
        // thread (j, i) with i = tid % 32 reads column j = tid / 32 + 8 q of
        // the diagonal tile and rows i + 32 u of the chunk's column
        constexpr int kQ = kTile / (kThreads / 32);  // columns per thread
        const int i = tid & 31, j0 = tid >> 5;
        float dv[kQ], av[kQ][kPanelRows / 32];
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
            const int j = j0 + q * (kThreads / 32);
            const float* col = B + (int64_t)(p0 + j) * f;
            dv[q] = (j < pb && i < pb && i >= j) ? ld_entry<kL2>(col + p0 + i) : 0.f;
#pragma unroll
            for (int u = 0; u < kPanelRows / 32; ++u) {
                const int r = i + 32 * u;
                av[q][u] = (j < pb && r < nr) ? ld_entry<kL2>(col + r0 + r) : 0.f;
            }
        }
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
            const int j = j0 + q * (kThreads / 32);
            D[i + j * ld] = pre ? 0.f : dv[q];
            Lt[j * lt_ld + i] = pre ? dv[q] : 0.f;  // Lt[j][i] = L_dd^-1[i][j]
#pragma unroll
            for (int u = 0; u < kPanelRows / 32; ++u) As[j * as_ld + i + 32 * u] = av[q][u];
        }
    }
    __syncthreads();
    if (tid == 0) last = !pre && (atomicAdd(step_cnt + pair, 1) == nchunk - 1);  // this CTA's tile reads are done
    if (tid < 32 && !pre) {
        const int i = tid;
        float inv;
        const bool bad = warp_potrf(pb, i, D, ld, &inv, [&](int j) { return D[i + j * ld]; });
        if (bad && i == 0 && chunk == 0) atomicOr(singular_flags(F, W, s), FLAG_SINGULAR);
        if (i < pb) rdiag[i] = inv;
        if (chunk == 0 && i < pb) reinterpret_cast<float*>(W.rdiag)[F.sn_c0[s] + p0 + i] = inv;
        __syncwarp();
        warp_trinv(D, ld, rdiag, pb, i, Lt, lt_ld);
    }
    __syncthreads();
    if (chunk == 0 && tid < 32) {
        // y = L_dd^-1 v of the block's right-hand-side entries, a lane per row
        float* yv = static_cast<float*>(sv.sol) + F.sn_c0[s] + p0;
        const float v = tid < pb ? ld_entry<kL2>(yv + tid) : 0.f;
        float y = 0.f;
#pragma unroll
        for (int j = 0; j < kTile; ++j) {
            const float vj = __shfl_sync(0xffffffffu, v, j);
            if (j <= tid && j < pb) y += Lt[j * lt_ld + tid] * vj;
        }
        if (tid < pb) yv[tid] = y;
    }
    {
        // thread (rg, cg): rows 4rg..4rg+3, columns 4cg..4cg+3 of the chunk
        const int cg = tid & 7, rg = tid >> 3;
        float acc[4][4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[u][v] = 0.f;
#pragma unroll 8
        for (int k = 0; k < kTile; ++k) {
            const float4 a4 = *reinterpret_cast<const float4*>(&As[k * as_ld + 4 * rg]);
            const float4 l4 = *reinterpret_cast<const float4*>(&Lt[k * lt_ld + 4 * cg]);
            const float av[4] = {a4.x, a4.y, a4.z, a4.w}, lv[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[u][v] += av[u] * lv[v];
        }
        __syncthreads();  // every read of A is done
#pragma unroll
        for (int v = 0; v < 4; ++v)
            *reinterpret_cast<float4*>(&As[(4 * cg + v) * as_ld + 4 * rg]) =
                make_float4(acc[0][v], acc[1][v], acc[2][v], acc[3][v]);
    }
    __syncthreads();
    for (int x = tid; x < kTile * kPanelRows; x += kThreads) {
        const int r = x % kPanelRows, k = x / kPanelRows;
        if (r < nr && k < pb) B[(r0 + r) + (int64_t)(p0 + k) * f] = As[k * as_ld + r];
    }
    if (last) {
        for (int x = tid; x < kTile * kTile; x += kThreads) {
            const int i = x % kTile, j = x / kTile;
            if (i < pb && j <= i) B[(p0 + i) + (int64_t)(p0 + j) * f] = Lt[j * lt_ld + i];
        }
    }
}

__global__ void __launch_bounds__(kThreads) k_big_panel32(DevFactor F, DevWork W, SolveVecs sv, float* lx,
                                                          const int4* work, int p, int* step_cnt) {
    const int4 wk = work[blockIdx.x];
    if (front_frozen(F, W, wk.x)) return;  // the whole CTA, before any barrier
    big_panel32_item<false>(F, W, sv, lx, wk.x, p, wk.y, wk.z, wk.w, step_cnt);
}

// FP32 trailing update of step p as a dataflow item: tile (ti, tj) -= A_i A_j^T
// over the panel's columns, restricted to rows >= cols >= p0 + pb.  The two
// row blocks of the panel are staged k-major in shared memory; thread
// (tr, tc) accumulates rows tr + 16u and columns tc + 16v (u, v < 2) in
// registers, four shared loads per four FMAs (a thread per output needed
// two per FMA), and its read-modify-writes of a column touch 16 consecutive
// rows per half warp.
__device__ __forceinline__ void big_update_item(const DevFactor& F, const DevWork& W, const SolveVecs& sv, float* lx,
                                                int s, int p, int ti, int tj) {
    using T = float;
    constexpr bool kL2 = true;
    static_assert(kThreads == 256 && kUpdTile == 32, "thread tiling below");
    constexpr int ld = kUpdTile + 1;
    __shared__ T Ai[kTile * ld];  // Ai[k * ld + r] = A(R0 + r, p0 + k)
    __shared__ T Aj[kTile * ld];
    const int f = F.sn_f[s];
    const int nc = F.sn_c0[s + 1] - F.sn_c0[s];
    T* B = lx + F.sn_lx_off[s];
    const int p0 = p * kTile;
    const int pb = min(kTile, nc - p0);
    const int q0 = p0 + pb;
    const int R0 = ti * kUpdTile, C0 = tj * kUpdTile;
    for (int x = threadIdx.x; x < kUpdTile * kTile; x += kThreads) {
        const int r = x % kUpdTile, k = x / kUpdTile;
        const T* col = B + (int64_t)(p0 + k) * f;
        Ai[k * ld + r] = (k < pb && R0 + r < f) ? ld_entry<kL2>(col + R0 + r) : T(0);
        Aj[k * ld + r] = (k < pb && C0 + r < f) ? ld_entry<kL2>(col + C0 + r) : T(0);
    }
    __syncthreads();
    if (ti == tj && threadIdx.x >= kThreads - 32) {
        // the last warp of a diagonal tile: the tile's right-hand-side entries,
        // a lane per column
        const int c = threadIdx.x & 31, gc = C0 + c;
        if (gc >= q0 && gc < f) {
            const T* y = static_cast<const T*>(sv.sol) + F.sn_c0[s] + p0;
            T* v = rhs_entry<T>(sv, F.sn_c0[s], nc, F.sn_su_off[s], gc);
            T acc = ld_entry<kL2>(v);
#pragma unroll 8
            for (int k = 0; k < pb; ++k) acc -= Aj[k * ld + c] * ld_entry<kL2>(y + k);
            *v = acc;
        }
    }
    const int tr = threadIdx.x & 15, tc = threadIdx.x >> 4;
    T acc[2][2] = {{T(0), T(0)}, {T(0), T(0)}};
#pragma unroll 4
    for (int k = 0; k < pb; ++k) {
        const T a0 = Ai[k * ld + tr], a1 = Ai[k * ld + tr + 16];
        const T b0 = Aj[k * ld + tc], b1 = Aj[k * ld + tc + 16];
        acc[0][0] += a0 * b0;
        acc[0][1] += a0 * b1;
        acc[1][0] += a1 * b0;
        acc[1][1] += a1 * b1;
    }
#pragma unroll
    for (int v = 0; v < 2; ++v) {
        const int gc = C0 + tc + 16 * v;
        if (gc < q0 || gc >= f) continue;
        T* dst = B + (int64_t)gc * f;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int gr = R0 + tr + 16 * u;
            if (gr >= gc && gr < f) dst[gr] = ld_entry<kL2>(dst + gr) - acc[u][v];
        }
    }
    // Look-ahead (FP32 tiled fronts): the tile that is the next step's
    // diagonal block comes first in the step's work list; after its own
    // update its CTA factors the block (L_dd) and inverts it in warp 0
    // while the step's other tiles are still updating, and leaves L_dd^-1
    // in the block's slot, the pivots' reciprocals in rdiag and the pivot
    // check done, so that the next panel step only applies L_dd^-1.  The
    // arithmetic is that of the panel kernel's own factorisation.
    if (ti == tj && R0 == q0 && q0 < nc) {
        constexpr int dld = kTile + 4, lt_ld = kTile + 4;  // 16-byte aligned rows
        __shared__ __align__(16) float D[kTile * dld];
        __shared__ float rdiag[kTile];
        __shared__ float Lt[kTile * lt_ld];
        __syncthreads();  // every update of this tile is written
        const int pb2 = min(kTile, nc - q0);
        if (threadIdx.x < 32) {
            const int i = threadIdx.x;
            float inv;
            const bool bad = warp_potrf(pb2, i, D, dld, &inv,
                                        [&](int j) { return ld_entry<kL2>(B + (q0 + i) + (int64_t)(q0 + j) * f); });
            if (bad && i == 0) atomicOr(singular_flags(F, W, s), FLAG_SINGULAR);
            if (i < pb2) {
                rdiag[i] = inv;
                reinterpret_cast<float*>(W.rdiag)[F.sn_c0[s] + q0 + i] = inv;
            }
            __syncwarp();
            warp_trinv(D, dld, rdiag, pb2, i, Lt, lt_ld);
            __syncwarp();
            for (int c = 0; c < pb2; ++c)
                if (i >= c && i < pb2) B[(q0 + i) + (int64_t)(q0 + c) * f] = Lt[c * lt_ld + i];
        }
    }
}

// FP32 step p of the tiled fronts in one launch: the trailing update of step p
// and the panel of step p + 1.  A chunk's CTA of the next panel updates its own
// rows of the panel's columns and, for itself, the diagonal block, which warp 0
// then factors and inverts while the other warps update the chunk; then the
// chunk is solved against the inverse.  No CTA waits for another: the diagonal
// block is updated and factored by every chunk's CTA, and the one that has read
// it last (a counter per front and step) writes L_dd^-1 into its slot.  The
// other tiles are plain updates.  Bound: the chain of load latency, the block's
// 32 pivots and its inverse.  Measured at 200k buses: 9.9 us a step, where the
// update (with the next diagonal block's factorisation in it) and the next panel
// as two launches took 11.3 + 4.7 us and two gaps.  (64 registers and 24 bytes of
// spills a thread.)
constexpr int kStepLd = kTile + 4, kStepRows = kPanelRows + 4;  // 16-byte aligned rows
struct StepPanelSmem {
    float xd[kTile * kStepLd];    // [k][r]: panel p, rows of the next diagonal block
    float d[kTile * kStepLd];     // [j][i]: the diagonal block, then L_dd
    float lt[kTile * kStepLd];    // [k][c] = L_dd^-1[c][k]
    float xc[kTile * kStepRows];  // [k][r]: panel p, the chunk's rows
    float as[kTile * kStepRows];  // [j][r]: the chunk, then X
    float rdiag[kTile], v[kTile];
    int last;
};
struct StepTileSmem {
    float ai[kTile * (kUpdTile + 1)], aj[kTile * (kUpdTile + 1)];
};
__device__ __forceinline__ void step_panel(const DevFactor& F, const DevWork& W, const SolveVecs& sv, float* lx,
                                           const StepItem& it, int p, int* step_cnt, StepPanelSmem& sm) {
    static_assert(kThreads == 256 && kPanelRows == 128 && kTile == 32, "thread tiling below");
    constexpr int kQ = kTile / (kThreads / 32), kU = kPanelRows / 32;
    const int f = it.f, nc = it.nc, chunk = it.a;
    float* B = lx + it.lx_off;
    const int p0 = p * kTile, q0 = p0 + kTile;  // panel p is whole: there is a next one
    const int pb = min(kTile, nc - q0);         // columns of the next panel
    const int r0 = q0 + pb + chunk * kPanelRows, nr = max(0, min(kPanelRows, f - r0));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* const y = static_cast<float*>(sv.sol) + it.c0;
    {
        // thread (i, j0): columns j0 + 8 q; rows i of the block, i + 32 u of the chunk
        const int i = lane, j0 = warp;
        float xd[kQ], dv[kQ], xc[kQ][kU], av[kQ][kU];
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
            const int j = j0 + q * (kThreads / 32);
            const float* xcol = B + (int64_t)(p0 + j) * f;
            const float* acol = B + (int64_t)(q0 + j) * f;
            const bool in = q0 + j < f;
            xd[q] = q0 + i < f ? xcol[q0 + i] : 0.f;
            dv[q] = (j < pb && i < pb && i >= j) ? acol[q0 + i] : 0.f;
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int r = i + 32 * u;
                xc[q][u] = r < nr ? xcol[r0 + r] : 0.f;
                av[q][u] = (in && r < nr && r0 + r >= q0 + j) ? acol[r0 + r] : 0.f;
            }
        }
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
            const int j = j0 + q * (kThreads / 32);
            sm.xd[j * kStepLd + i] = xd[q];
            sm.d[j * kStepLd + i] = dv[q];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                sm.xc[j * kStepRows + i + 32 * u] = xc[q][u];
                sm.as[j * kStepRows + i + 32 * u] = av[q][u];
            }
        }
    }
    __syncthreads();
    if (tid == 0) sm.last = atomicAdd(step_cnt + it.pair, 1) == it.b - 1;  // this CTA's block reads are done
    {
        // the diagonal block's update: rows tr + 16 u, columns tc + 16 v
        const int tr = tid & 15, tc = tid >> 4;
        float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 8
        for (int k = 0; k < kTile; ++k) {
            const float a0 = sm.xd[k * kStepLd + tr], a1 = sm.xd[k * kStepLd + tr + 16];
            const float b0 = sm.xd[k * kStepLd + tc], b1 = sm.xd[k * kStepLd + tc + 16];
            acc[0][0] += a0 * b0;
            acc[0][1] += a0 * b1;
            acc[1][0] += a1 * b0;
            acc[1][1] += a1 * b1;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                float* e = &sm.d[(tc + 16 * v) * kStepLd + tr + 16 * u];
                *e = *e - acc[u][v];
            }
    }
    __syncthreads();
    if (warp == 0) {
        const int i = lane;
        for (int j = 0; j < kTile; ++j) sm.lt[j * kStepLd + i] = 0.f;
        float inv;
        const bool bad = warp_potrf(pb, i, sm.d, kStepLd, &inv, [&](int j) { return sm.d[i + j * kStepLd]; });
        if (bad && i == 0 && chunk == 0) atomicOr(singular_flags(F, W, it.s), FLAG_SINGULAR);
        if (i < pb) sm.rdiag[i] = inv;
        if (chunk == 0 && i < pb) reinterpret_cast<float*>(W.rdiag)[it.c0 + q0 + i] = inv;
        __syncwarp();
        warp_trinv(sm.d, kStepLd, sm.rdiag, pb, i, sm.lt, kStepLd);
    } else {
        // the chunk's update, 4 x 4 entries a turn
        for (int t = tid - 32; t < kThreads; t += kThreads - 32) {
            const int cg = t & 7, rg = t >> 3;
            float acc[4][4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[u][v] = 0.f;
#pragma unroll 8
            for (int k = 0; k < kTile; ++k) {
                float av[4], bv[4];
                load4(&sm.xc[k * kStepRows + 4 * rg], av);
                load4(&sm.xd[k * kStepLd + 4 * cg], bv);
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int v = 0; v < 4; ++v) acc[u][v] += av[u] * bv[v];
            }
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                float cur[4];
                load4(&sm.as[(4 * cg + v) * kStepRows + 4 * rg], cur);
#pragma unroll
                for (int u = 0; u < 4; ++u) cur[u] = cur[u] - acc[u][v];
                store4(&sm.as[(4 * cg + v) * kStepRows + 4 * rg], cur);
            }
        }
        if (chunk == 0 && warp == 1) {
            // the right-hand side of the panel's tile column (entries past pb belong to rows below)
            const int gc = q0 + lane;
            float acc = 0.f;
            if (gc < f) {
                float* v = rhs_entry<float>(sv, it.c0, nc, it.su_off, gc);
                acc = *v;
#pragma unroll 8
                for (int k = 0; k < kTile; ++k) acc -= sm.xd[k * kStepLd + lane] * y[p0 + k];
                if (lane >= pb) *v = acc;
            }
            sm.v[lane] = acc;
        }
    }
    __syncthreads();
    if (chunk == 0 && warp == 0) {
        // y = L_dd^-1 v, a lane per row
        float yv = 0.f;
        for (int j = 0; j < pb; ++j)
            if (j <= lane) yv += sm.lt[j * kStepLd + lane] * sm.v[j];
        if (lane < pb) y[q0 + lane] = yv;
    }
    {
        // X = A (L_dd^-1)^T: rows 4 rg.., columns 4 cg..; columns past pb stay updated entries
        const int cg = tid & 7, rg = tid >> 3;
        float acc[4][4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[u][v] = 0.f;
#pragma unroll 8
        for (int k = 0; k < kTile; ++k) {
            float av[4], lv[4];
            load4(&sm.as[k * kStepRows + 4 * rg], av);
            load4(&sm.lt[k * kStepLd + 4 * cg], lv);
            if (k >= pb) {
#pragma unroll
                for (int u = 0; u < 4; ++u) av[u] = 0.f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[u][v] += av[u] * lv[v];
        }
        __syncthreads();  // every read of A is done
#pragma unroll
        for (int v = 0; v < 4; ++v)
            if (4 * cg + v < pb)
                *reinterpret_cast<float4*>(&sm.as[(4 * cg + v) * kStepRows + 4 * rg]) =
                    make_float4(acc[0][v], acc[1][v], acc[2][v], acc[3][v]);
    }
    __syncthreads();
    for (int x = tid; x < kTile * kPanelRows; x += kThreads) {
        const int r = x % kPanelRows, k = x / kPanelRows;
        if (r < nr && q0 + k < f && r0 + r >= q0 + k) B[(r0 + r) + (int64_t)(q0 + k) * f] = sm.as[k * kStepRows + r];
    }
    if (sm.last) {
        for (int x = tid; x < kTile * kTile; x += kThreads) {
            const int i = x % kTile, j = x / kTile;
            if (i < pb && j <= i) B[(q0 + i) + (int64_t)(q0 + j) * f] = sm.lt[j * kStepLd + i];
        }
    }
}

__global__ void __launch_bounds__(kThreads) k_big_step32(DevFactor F, DevWork W, SolveVecs sv, float* lx,
                                                         const StepItem* work, int p, int* step_cnt) {
    __shared__ __align__(16) union {
        StepPanelSmem panel;
        StepTileSmem tile;
    } sm;
    const StepItem it = work[blockIdx.x];
    if (W.grid_flags && front_frozen(F, W, it.s)) return;  // the whole CTA, before any barrier
    if (it.pair >= 0) {
        step_panel(F, W, sv, lx, it, p, step_cnt, sm.panel);
        return;
    }
    constexpr int ld = kUpdTile + 1;
    float* B = lx + it.lx_off;
    const int f = it.f, nc = it.nc, ti = it.a, tj = it.b;
    const int p0 = p * kTile, pb = min(kTile, nc - p0), q0 = p0 + pb;
    const int R0 = ti * kUpdTile, C0 = tj * kUpdTile;
    const int tid = threadIdx.x, tr = tid & 15, tc = tid >> 4;
    // every load of the CTA in flight at once
    float cur[2][2], xi[4], xj[4];
#pragma unroll
    for (int v = 0; v < 2; ++v)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int gc = C0 + tc + 16 * v, gr = R0 + tr + 16 * u;
            cur[u][v] = (gc >= q0 && gc < f && gr >= gc && gr < f) ? B[(int64_t)gc * f + gr] : 0.f;
        }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r = tid & 31, k = (tid >> 5) + 8 * q;
        const float* col = B + (int64_t)(p0 + k) * f;
        xi[q] = (k < pb && R0 + r < f) ? col[R0 + r] : 0.f;
        xj[q] = (k < pb && C0 + r < f) ? col[C0 + r] : 0.f;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r = tid & 31, k = (tid >> 5) + 8 * q;
        sm.tile.ai[k * ld + r] = xi[q];
        sm.tile.aj[k * ld + r] = xj[q];
    }
    __syncthreads();
    if (ti == tj && tid >= kThreads - 32) {
        // the last warp of a diagonal tile: the tile's right-hand-side entries, a lane per column
        const int c = tid & 31, gc = C0 + c;
        if (gc >= q0 && gc < f) {
            const float* y = static_cast<const float*>(sv.sol) + it.c0 + p0;
            float* v = rhs_entry<float>(sv, it.c0, nc, it.su_off, gc);
            float acc = *v;
#pragma unroll 8
            for (int k = 0; k < pb; ++k) acc -= sm.tile.aj[k * ld + c] * y[k];
            *v = acc;
        }
    }
    float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 4
    for (int k = 0; k < pb; ++k) {
        const float a0 = sm.tile.ai[k * ld + tr], a1 = sm.tile.ai[k * ld + tr + 16];
        const float b0 = sm.tile.aj[k * ld + tc], b1 = sm.tile.aj[k * ld + tc + 16];
        acc[0][0] += a0 * b0;
        acc[0][1] += a0 * b1;
        acc[1][0] += a1 * b0;
        acc[1][1] += a1 * b1;
    }
#pragma unroll
    for (int v = 0; v < 2; ++v)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int gc = C0 + tc + 16 * v, gr = R0 + tr + 16 * u;
            if (gc >= q0 && gc < f && gr >= gc && gr < f) B[(int64_t)gc * f + gr] = cur[u][v] - acc[u][v];
        }
}

// FP64 trailing update of step p, one CTA per kUpdTile64 x kUpdTile64 tile
// and one entry per thread.  Bound: FP64 issue (two FMAs a cycle per SM), so
// the tile is small: a 32 x 32 tile kept its SM for 16k cycles while a step
// of a single grid has fewer such tiles than the GPU has SMs (30k-bus grid:
// 12.5 us a step with 32 x 32 tiles, 5.8 us with 16 x 16).
__global__ void __launch_bounds__(kUpdTile64 * kUpdTile64) k_big_update64(DevFactor F, DevWork W, SolveVecs sv,
                                                                          double* lx, const int4* work, int p) {
    constexpr int kN = kUpdTile64, kAll = kN * kN;
    __shared__ double Ai[kTile][kN + 1], Aj[kTile][kN + 1];  // [k][row]; Ai's last column: y
    const int4 wk = work[blockIdx.x];
    const int s = wk.x;
    if (front_frozen(F, W, s)) return;  // the whole CTA, before any barrier
    const int f = F.sn_f[s];
    const int nc = F.sn_c0[s + 1] - F.sn_c0[s];
    double* B = lx + F.sn_lx_off[s];
    const int p0 = p * kTile;
    const int pb = min(kTile, nc - p0);
    const int q0 = p0 + pb;
    const int R0 = wk.y * kN, C0 = wk.z * kN;
    const int tr = threadIdx.x % kN, tc = threadIdx.x / kN;
    const int gr = R0 + tr, gc = C0 + tc;
    // A diagonal tile's right-hand-side entries v_j -= sum y_k X_jk fall to
    // threads above the diagonal: (j, j + 1), and (0, last) for the last column.
    const bool diag = wk.y == wk.z;
    const bool rhs = diag && (tc == tr + 1 || (tr == 0 && tc == kN - 1));
    const int jv = (tc == tr + 1) ? tr : kN - 1;
    bool mine = gc >= q0 && gc < f && gr >= gc && gr < f;
    double* dst = B + gr + (int64_t)gc * f;
    if (rhs) {
        mine = C0 + jv >= q0 && C0 + jv < f;
        if (mine) dst = rhs_entry<double>(sv, F.sn_c0[s], nc, F.sn_su_off[s], C0 + jv);
    }
    double acc = mine ? *dst : 0.0;
#pragma unroll
    for (int k = tc; k < kTile; k += kAll / kN) {
        const double* col = B + (int64_t)(p0 + k) * f;
        Ai[k][tr] = (k < pb && R0 + tr < f) ? col[R0 + tr] : 0.0;
        Aj[k][tr] = (k < pb && C0 + tr < f) ? col[C0 + tr] : 0.0;
        if (diag && tr == 0) Ai[k][kN] = k < pb ? static_cast<const double*>(sv.sol)[F.sn_c0[s] + p0 + k] : 0.0;
    }
    __syncthreads();
    const double* ai = &Ai[0][rhs ? kN : tr];
    const double* aj = &Aj[0][rhs ? jv : tc];
#pragma unroll 8
    for (int k = 0; k < pb; ++k) acc = fma(-ai[k * (kN + 1)], aj[k * (kN + 1)], acc);
    if (mine) *dst = acc;
}

// Bounded wait of the tiled-front dataflow (one lane per dependency): true
// once the flag is set; false when the wait runs out (it then raises
// FLAG_TIMEOUT) or when another wait of the pass has run out, so that a
// failed pass ends in about one spin limit instead of one per item.
__device__ __forceinline__ bool wait_tile(const int* flag, uint32_t* status, long long limit) {
    long long spins = 0;
    for (;;) {
        int v;
        asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
        if (v != 0) return true;
        if (++spins > limit) {
            atomicOr(status, FLAG_TIMEOUT);
            return false;
        }
        if ((spins & 63) == 0 && (atomicOr(status, 0u) & FLAG_TIMEOUT)) return false;
        __nanosleep(32);
    }
}

// FP32 tiled fronts of one synchronous level in one launch: a persistent grid
// claims the level's TileTask items in order, waits (bounded) for each
// item's dependencies and publishes its completion; the items run the same
// arithmetic as the per-step kernels.  Dependencies are always claimed
// earlier, so the smallest unfinished item is always running and progress
// never depends on CTAs that have not started (the grid need not be
// co-resident; a CTA holds at most the item it runs and the next one it has
// claimed).  Per item: the next claim and its 64-byte task load are issued
// while the current item runs, and warp 0 polls the dependencies in
// parallel, one lane each.  Entries written during the launch are read past
// L1 (ld_entry<true>).  Items of frozen grids, and every item once a wait has
// timed out, publish without computing.
constexpr int kTileFlowBlocks = 3;
__global__ void __launch_bounds__(kThreads, kTileFlowBlocks)
    k_big_flow32(DevFactor F, DevWork W, SolveVecs sv, float* lx, const TileTask* tasks, int n, int* done, int* counter,
                 int* step_cnt) {
    constexpr int kWords = sizeof(TileTask) / sizeof(int);
    static_assert(kWords <= 32, "one lane per task word");
    __shared__ TileTask task[2];
    __shared__ int next[2];
    __shared__ int skip;
    const int tid = threadIdx.x, lane = tid & 31;
    uint32_t* status = &W.status->flags;
    int buf = 0;
    if (tid < 32) {
        int item = 0;
        if (lane == 0) item = atomicAdd(counter, 1);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (lane == 0) next[0] = item;
        if (item < n && lane < kWords)
            reinterpret_cast<int*>(&task[0])[lane] = __ldg(reinterpret_cast<const int*>(tasks + item) + lane);
    }
    __syncthreads();
    for (;;) {
        const int item = next[buf];
        if (item >= n) break;
        // warp 1 claims and loads the next item; warp 0 waits for this one's inputs
        if (tid >= 32 && tid < 64) {
            int nx = 0;
            if (lane == 0) nx = atomicAdd(counter, 1);
            nx = __shfl_sync(0xffffffffu, nx, 0);
            if (lane == 0) next[buf ^ 1] = nx;
            if (nx < n && lane < kWords)
                reinterpret_cast<int*>(&task[buf ^ 1])[lane] =
                    __ldg(reinterpret_cast<const int*>(tasks + nx) + lane);
        }
        const TileTask& t = task[buf];
        if (tid < 32) {
            const bool ok = lane < t.ndep ? wait_tile(done + t.dep[lane], status, W.spin_limit) : true;
            const bool all = __all_sync(0xffffffffu, ok);
            if (lane == 0) skip = !all || front_frozen(F, W, t.s) || (atomicOr(status, 0u) & FLAG_TIMEOUT) != 0u;
            __syncwarp();
        }
        __syncthreads();
        if (!skip) {
            if (t.kind == 0)
                big_panel32_item<true>(F, W, sv, lx, t.s, t.p, t.a, t.b, t.aux, step_cnt);
            else
                big_update_item(F, W, sv, lx, t.s, t.p, t.a, t.b);
        }
        __syncthreads();
        if (tid == 0) publish_done(done + item);
        __syncwarp();
        buf ^= 1;
    }
}

// ---------------------------------------------------------------------------
// Solves.  Forward (bottom-up): v = [b of own columns; 0] + children's update
// vectors; y = L11^-1 v1; update vector = v2 - L21 y.
// Backward (top-down): x1 = L11^-T (y - L21^T x_rows).
// Blocked by columns: each diagonal block is staged in shared memory and
// applied by one warp (FP32: a mat-vec with the stored L11^-1, one lane per
// row; FP64: a column sweep); the rectangular update below (forward) or the
// dot products against the solved rows (backward) use every thread with
// coalesced reads of the column-major panel.
// ---------------------------------------------------------------------------
// Forward step of a warp front: v = [b of own columns; 0] + children's update
// vectors (in child order), y = L11^-1 v1, update vector v2 - L21 y.
template <typename T, typename V>
__device__ void warp_front_fwd(const DevFactor& F, const T* lx, const T* rdiag, const SolveVecs& sv, int s, V* v) {
    const V* rhs = reinterpret_cast<const V*>(sv.rhs);
    V* sol = reinterpret_cast<V*>(sv.sol);
    V* sub = reinterpret_cast<V*>(sv.su);
    const int lane = threadIdx.x & 31;
    const int f = F.sn_f[s];
    const int c0 = F.sn_c0[s];
    const int nc = F.sn_c0[s + 1] - c0;
    const T* L = lx + F.sn_lx_off[s];
    const V rd = (!kInvDiag<T> && lane < nc) ? static_cast<V>(rdiag[c0 + lane]) : V(0);
    v[lane] = (lane < nc) ? rhs[c0 + lane] : V(0);
    __syncwarp();
    const int cp0 = F.sn_child_ptr[s], cp1 = F.sn_child_ptr[s + 1];
    for (int cb = cp0; cb < cp1; cb += 8) {
        V val[8];
        int row[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            row[u] = -1;
            val[u] = V(0);
            if (cb + u < cp1) {
                const int c = F.sn_child[cb + u];
                const int m = F.sn_f[c] - (F.sn_c0[c + 1] - F.sn_c0[c]);
                if (lane < m) {
                    const int64_t o = F.sn_su_off[c];
                    val[u] = __ldcg(sub + o + lane);
                    row[u] = F.sn_relmap[o + lane];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (row[u] >= 0) v[row[u]] += val[u];
            __syncwarp();
        }
    }
    V y = V(0);
    if constexpr (kInvDiag<T>) {
        if (lane < nc)
            for (int j = 0; j <= lane; ++j) y += static_cast<V>(L[lane + j * f]) * v[j];
        __syncwarp();
        if (lane < nc) v[lane] = y;
    } else {
        for (int k = 0; k < nc; ++k) {
            const V yk = v[k] * __shfl_sync(0xffffffffu, rd, k);
            __syncwarp();
            if (lane > k && lane < nc) v[lane] -= static_cast<V>(L[lane + k * f]) * yk;
            if (lane == 0) v[k] = yk;
            __syncwarp();
        }
        y = lane < nc ? v[lane] : V(0);
    }
    __syncwarp();
    if (lane < nc) {
        sol[c0 + lane] = y;
    } else if (lane < f) {
        V acc = v[lane];
        for (int k = 0; k < nc; ++k) acc -= static_cast<V>(L[lane + k * f]) * v[k];
        sub[F.sn_su_off[s] + (lane - nc)] = acc;
    }
    __syncwarp();
}

template <typename T, typename V>
__device__ void front_fwd(const DevFactor& F, const T* lx, const T* rdiag, const SolveVecs& sv, int s, V* v, T* D) {
    const V* rhs = reinterpret_cast<const V*>(sv.rhs);
    V* sol = reinterpret_cast<V*>(sv.sol);
    V* sub = reinterpret_cast<V*>(sv.su);
    const int f = F.sn_f[s];
    const int c0 = F.sn_c0[s];
    const int nc = F.sn_c0[s + 1] - c0;
    const int tid = threadIdx.x, nth = blockDim.x;
    const T* L = lx + F.sn_lx_off[s];
    for (int i = tid; i < f; i += nth) v[i] = (i < nc) ? rhs[c0 + i] : V(0);
    __syncthreads();
    // children's update vectors, eight children at a time: every thread issues
    // its loads for all eight before the ordered adds (one barrier per child
    // keeps the sum order fixed)
    const int cp0 = F.sn_child_ptr[s], cp1 = F.sn_child_ptr[s + 1];
    for (int cb = cp0; cb < cp1; cb += 8) {
        V val[8];
        int row[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            row[u] = -1;
            val[u] = V(0);
            if (cb + u < cp1) {
                const int c = F.sn_child[cb + u];
                const int m = F.sn_f[c] - (F.sn_c0[c + 1] - F.sn_c0[c]);
                if (tid < m) {
                    const int64_t o = F.sn_su_off[c];
                    val[u] = __ldcg(sub + o + tid);
                    row[u] = F.sn_relmap[o + tid];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (cb + u < cp1) {
                if (row[u] >= 0) v[row[u]] += val[u];
                const int c = F.sn_child[cb + u];
                const int m = F.sn_f[c] - (F.sn_c0[c + 1] - F.sn_c0[c]);
                const int64_t o = F.sn_su_off[c];
                for (int i = tid + nth; i < m; i += nth) v[F.sn_relmap[o + i]] += __ldcg(sub + o + i);
                __syncthreads();
            }
        }
    }
    // blocks of the factor's panel width (FP32: the diagonal slots hold
    // L11^-1) or of kTile (FP64: L11 with its reciprocal diagonal)
    const int bw = kInvDiag<T> ? (F.sn_pw ? F.sn_pw[s] : kTile) : kTile;
    constexpr int ld = kTile + 1;
    for (int k0 = 0; k0 < nc; k0 += bw) {
        const int kb = min(bw, nc - k0);
        for (int x = tid; x < kb * kb; x += nth) {
            const int i = x % kb, j = x / kb;
            if constexpr (kInvDiag<T>)
                D[i + j * ld] = (i >= j) ? L[(k0 + i) + (int64_t)(k0 + j) * f] : T(0);
            else
                D[i + j * ld] = (i == j) ? rdiag[c0 + k0 + i] : L[(k0 + i) + (int64_t)(k0 + j) * f];
        }
        __syncthreads();
        if (tid < 32) {
            if constexpr (kInvDiag<T>) {
                // y = L11^-1 v: one lane per row, independent dot products
                V y = V(0);
                if (tid < kb)
                    for (int j = 0; j <= tid; ++j) y += static_cast<V>(D[tid + j * ld]) * v[k0 + j];
                __syncwarp();
                if (tid < kb) v[k0 + tid] = y;
            } else {
                // column sweep, lane i updating row k + 1 + i
                for (int k = 0; k < kb; ++k) {
                    const V yk = v[k0 + k] * static_cast<V>(D[k + k * ld]);
                    __syncwarp();
                    const int i = k + 1 + tid;
                    if (i < kb) v[k0 + i] -= static_cast<V>(D[i + k * ld]) * yk;
                    if (tid == 0) v[k0 + k] = yk;
                    __syncwarp();
                }
            }
        }
        __syncthreads();
        for (int i = k0 + kb + tid; i < f; i += nth) {
            V acc = v[i];
            for (int k = 0; k < kb; ++k) acc -= static_cast<V>(L[i + (int64_t)(k0 + k) * f]) * v[k0 + k];
            v[i] = acc;
        }
        __syncthreads();
    }
    for (int k = tid; k < nc; k += nth) sol[c0 + k] = v[k];
    V* su = sub + F.sn_su_off[s];
    for (int i = tid; i < f - nc; i += nth) su[i] = v[nc + i];
}

// Asynchronous copy of one factor entry to shared memory.
template <typename T>
__device__ __forceinline__ void copy_async(T* to, const T* from) {
    const unsigned at = static_cast<unsigned>(__cvta_generic_to_shared(to));
    if constexpr (sizeof(T) == 4)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(at), "l"(from) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(at), "l"(from) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Four columns' sums over a warp: v[u] the lane's part of column u.  FP32: lane
// 0 ends with each sum, added in the order of a shuffle-down tree.  FP64: the
// columns fold into one another, six additions instead of twenty; sum u ends in
// lane 8 u.  `apply` takes (u, sum).
template <typename F>
__device__ __forceinline__ void warp_sum4(float (&v)[4], F&& apply) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] += __shfl_down_sync(0xffffffffu, v[u], o);
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int u = 0; u < 4; ++u) apply(u, v[u]);
    }
}
template <typename F>
__device__ __forceinline__ void warp_sum4(double (&v)[4], F&& apply) {
    const int lane = threadIdx.x & 31;
    const bool h = lane & 16, q = lane & 8;
    double a = (h ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, h ? v[0] : v[2], 16);
    double b = (h ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, h ? v[1] : v[3], 16);
    double c = (q ? b : a) + __shfl_xor_sync(0xffffffffu, q ? a : b, 8);
    for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((lane & 7) == 0) apply(lane >> 3, c);
}

// Backward step of a single-CTA or tiled front, x1 = L11^-T (y - L21^T x2), by
// column blocks of the factor's panels, last first.  Bound: latency, front
// after front down the tree.  Everything that does not depend on the parent --
// the record, the row indices, y, the last two blocks' factor entries -- is on
// its way before `wait` waits for the parent, and each further block is copied
// to shared memory while the one before it is applied.  A block whose rows do
// not fit the stage (cap entries) reads them from memory.
// FP32: the diagonal slots hold L11^-1 (a lane per column, rows in order);
// FP64: a column sweep on entries scaled by the reciprocal diagonal
// beforehand, so that each step of the chain is one FMA and one shuffle.
// Measured per call: 200k buses mixed 600 -> 312 us, 60k FP64 520 -> 306 us.
constexpr int kStageD = kTile * (kTile + 1) + kTile;  // diagonal block (ld 33), reciprocal diagonal
template <typename T>
constexpr size_t bwd_smem(int maxf, int cap) {
    return sizeof(T) * ((size_t)(maxf + 3) / 4 * 4 + 2 * ((size_t)kStageD + cap));
}
// Stage capacities.  The narrow fronts' launch wants many CTAs per SM (their
// blocks hold a few hundred entries; the line is flat: with 1024 or 4096 whole
// passes at 10k, 60k and 200k buses and of batches take the same within 0.5 %, or
// within the spread of runs, 1.3 % for 512 grids); the wide fronts' one, few and
// long, takes what shared memory holds, up to a whole 32-column block.
constexpr int kBwdCap = 2048;
constexpr size_t kBwdSmemMax = 200 * 1024;
template <typename T>
int bwd_top_cap(int maxf) {
    const int64_t room = ((int64_t)(kBwdSmemMax / sizeof(T)) - (maxf + 3) / 4 * 4) / 2 - kStageD;
    return (int)std::max<int64_t>(0, std::min<int64_t>(room, (int64_t)maxf * kTile));
}
template <typename T, typename Wait>
__device__ void front_bwd(const DevFactor& F, const FrontRec& R, const T* lx, const T* rdiag, const SolveVecs& sv, T* x,
                          T* stages, int cap, Wait&& wait) {
    constexpr int ld = kTile + 1, kIdx = 4;
    T* sol = static_cast<T*>(sv.sol);
    const int f = R.f, c0 = R.c0, nc = R.nc;
    const int* rows = F.sn_rows + R.rows_off;
    const T* L = lx + R.lx_off;
    const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarp = nth >> 5;
    const int bw = kInvDiag<T> ? R.pw : kTile;
    const int nblk = (nc + bw - 1) / bw;
    auto issue = [&](int b) {
        if (b >= 0) {
            const int k0 = b * bw, kb = min(bw, nc - k0), q0 = k0 + kb, n = f - q0;
            T* D = stages + (b & 1) * (kStageD + cap);
            T* S = D + kStageD;
            const bool staged = n * kb <= cap;
            for (int j = warp; j < kb; j += nwarp) {
                const T* col = L + (int64_t)(k0 + j) * f;
                if (lane < kb && lane >= j) copy_async(D + lane + j * ld, col + k0 + lane);
                if (staged)
                    for (int r = lane; r < n; r += 32) copy_async(S + r + j * n, col + q0 + r);
            }
            if (!kInvDiag<T> && tid < kb) copy_async(D + kTile * ld + tid, rdiag + c0 + k0 + tid);
        }
        copies_commit();
    };
    issue(nblk - 1);
    issue(nblk - 2);
    for (int r = tid; r < nc; r += nth) x[r] = __ldcg(sol + c0 + r);
    int idx[kIdx];
#pragma unroll
    for (int u = 0; u < kIdx; ++u) idx[u] = nc + tid + u * nth < f ? rows[nc + tid + u * nth] : -1;
    wait();  // the parent is done; a block barrier
#pragma unroll
    for (int u = 0; u < kIdx; ++u)
        if (idx[u] >= 0) x[nc + tid + u * nth] = __ldcg(sol + idx[u]);
    for (int r = nc + tid + kIdx * nth; r < f; r += nth) x[r] = __ldcg(sol + rows[r]);
    for (int b = nblk - 1; b >= 0; --b) {
        const int k0 = b * bw, kb = min(bw, nc - k0), q0 = k0 + kb, n = f - q0;
        T* D = stages + (b & 1) * (kStageD + cap);
        const T* S = D + kStageD;
        copies_wait<1>();  // this block's copies (the next block's may still run)
        __syncthreads();
        // t_k = x_k - sum over the rows below of L[r][k] x_r: four columns per warp, rows over the lanes
        T acc[4] = {T(0), T(0), T(0), T(0)};
        if (warp < kb) {
            if (n * kb <= cap) {
                int co[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) co[u] = min(warp + nwarp * u, kb - 1) * n;
#pragma unroll 2
                for (int r = lane; r < n; r += 32) {
                    const T xr = x[q0 + r];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (warp + nwarp * u < kb) acc[u] += S[co[u] + r] * xr;
                }
            } else {
                const T* Lq[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) Lq[u] = L + (int64_t)(k0 + min(warp + nwarp * u, kb - 1)) * f + q0;
#pragma unroll 4
                for (int r = lane; r < n; r += 32) {
                    const T xr = x[q0 + r];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (warp + nwarp * u < kb) acc[u] += Lq[u][r] * xr;
                }
            }
            warp_sum4(acc, [&](int u, T sum) {
                if (warp + nwarp * u < kb) x[k0 + warp + nwarp * u] -= sum;
            });
        }
        if constexpr (!kInvDiag<T>) {
            const T* rd = D + kTile * ld;
            for (int j = warp; j < kb; j += nwarp)
                if (lane > j && lane < kb) D[lane + j * ld] *= rd[lane];
        }
        __syncthreads();
        if (warp == 0) {
            if constexpr (kInvDiag<T>) {
                // x = (L11^-1)^T t: one lane per column of L11^-1
                T val = T(0);
#pragma unroll 8
                for (int i = 0; i < kb; ++i)
                    if (i >= lane) val += D[i + lane * ld] * x[k0 + i];
                __syncwarp();
                if (lane < kb) x[k0 + lane] = val;
            } else {
                T t = lane < kb ? x[k0 + lane] : T(0);
                for (int k = kb - 1; k > 0; --k) {
                    const T tk = __shfl_sync(0xffffffffu, t, k);
                    if (lane < k) t -= D[k + lane * ld] * tk;
                }
                if (lane < kb) x[k0 + lane] = t * D[kTile * ld + lane];
            }
        }
        __syncthreads();
        issue(b - 2);
    }
    for (int k = tid; k < nc; k += nth) sol[c0 + k] = x[k];
}

template <typename T, typename V>
__global__ void __launch_bounds__(kThreads) k_fwd(DevFactor F, DevWork W, const T* lx, const T* rdiag, SolveVecs sv,
                                                  const int* fronts) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ T D[kTile * (kTile + 1)];
    const int s = fronts[blockIdx.x];
    if (front_frozen(F, W, s)) return;
    front_fwd<T, V>(F, lx, rdiag, sv, s, reinterpret_cast<V*>(smem_raw), D);
}

// A frozen grid's sol holds its last solution, not y: the factorisation has
// left its fronts out.
template <typename T>
__global__ void __launch_bounds__(kThreads) k_bwd(DevFactor F, DevWork W, const T* lx, const T* rdiag, SolveVecs sv,
                                                  int maxf, int cap, const int* fronts) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* x = reinterpret_cast<T*>(smem_raw);
    const FrontRec R = F.rec[fronts[blockIdx.x]];
    if (front_frozen(W, R)) return;
    front_bwd<T>(F, R, lx, rdiag, sv, x, x + (maxf + 3) / 4 * 4, cap, [] { __syncthreads(); });
}

// Forward sweep by continuation from the leaves (see continue_up).
template <typename T, typename V>
__global__ void __launch_bounds__(kThreads) k_fwd_flow(DevFactor F, DevWork W, const T* lx, const T* rdiag,
                                                       SolveVecs sv, const int* ready, const int* n_ready,
                                                       const int32_t* nchild, int* counter, int* cnt) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ T D[kTile * (kTile + 1)];
    __shared__ int slot;
    const int nr = *n_ready;
    for (;;) {
        const int item = claim(counter, &slot);
        if (item >= nr) break;
        int s = ready[item];
        while (s >= 0) {
            if (!front_frozen(F, W, s)) front_fwd<T, V>(F, lx, rdiag, sv, s, reinterpret_cast<V*>(smem_raw), D);
            __syncthreads();
            s = continue_up(F, nchild, cnt, s, &slot);
        }
    }
}

// Backward sweep as dataflow: order = fronts top-down, waits on the parent.
template <typename T>
__global__ void __launch_bounds__(kThreads) k_bwd_flow(DevFactor F, DevWork W, const T* lx, const T* rdiag,
                                                       SolveVecs sv, int maxf, int cap, const int* order,
                                                       const int* n_items, int* counter, int* done) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int slot;
    T* x = reinterpret_cast<T*>(smem_raw);
    const int ni = *n_items;
    for (;;) {
        const int item = claim(counter, &slot);
        if (item >= ni) break;
        const int s = order[item];
        const FrontRec R = F.rec[s];
        if (!front_frozen(W, R)) {
            front_bwd<T>(F, R, lx, rdiag, sv, x, x + (maxf + 3) / 4 * 4, cap, [&] {
                if (threadIdx.x == 0 && R.parent >= 0) wait_done(done + R.parent, &W.status->flags, W.spin_limit);
                __syncwarp();
                __syncthreads();
            });
            __syncthreads();
        }
        if (threadIdx.x == 0 && s != W.hold_front) publish_done(done + s);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Warp fronts: a front whose whole subtree is at most kWarpFrontMax wide is
// handled by one warp (eight fronts per CTA, no block barriers).  Factor: the
// front is assembled in the warp's tile in shared memory (original entries,
// then the children's update matrices in child order) and partially factorised
// there, left-looking (warp_front_factor); L (FP32: with L11^-1 in its diagonal
// block) and the update matrix are written out.  Solves: the forward steps of
// the same fronts, a lane per row, and the backward ones, a lane per column.
// A warp continues with the parent when it completes the parent's last child
// in the same phase, as the CTA sweeps do.
// ---------------------------------------------------------------------------
template <typename T>
constexpr int kMinBlocksW = sizeof(T) == 4 ? 4 : 2;

template <typename T>
__global__ void __launch_bounds__(kThreads, kMinBlocksW<T>) k_front_warp(DevFactor F, DevWork W, SolveVecs sv, const T* gv,
                                                                         T* lx, T* ub, const int* ready, const int* n_ready,
                                                                         int* counter, int* cnt) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WarpTile<T>& t = reinterpret_cast<WarpTile<T>*>(smem_raw)[threadIdx.x >> 5];
    const int nr = *n_ready;
    for (;;) {
        const int item = warp_claim(counter);
        if (item >= nr) break;
        int s = ready[item];
        while (s >= 0) {
            const FrontRec R = F.rec[s];
            if (!front_frozen(W, R)) warp_front_factor<T>(F, W, sv, gv, lx, ub, R, s, t);
            s = warp_continue_up(R, cnt);
        }
    }
}

template <typename T, typename V>
__global__ void __launch_bounds__(kThreads) k_fwd_warp(DevFactor F, DevWork W, const T* lx, const T* rdiag,
                                                       SolveVecs sv, const int* ready, const int* n_ready,
                                                       const int8_t* phase, int ph, const int32_t* nchild,
                                                       int* counter, int* cnt) {
    __shared__ V vw[kWarpsPerCta][kWarpFrontMax];
    V* v = vw[threadIdx.x >> 5];
    const int nr = *n_ready;
    for (;;) {
        const int item = warp_claim(counter);
        if (item >= nr) break;
        int s = ready[item];
        while (s >= 0) {
            if (!front_frozen(F, W, s)) warp_front_fwd<T, V>(F, lx, rdiag, sv, s, v);
            s = warp_continue_up(F, phase, ph, nchild, cnt, s);
        }
    }
}

// Backward steps of the warp fronts in top-down order, each waiting (bounded)
// on its parent's flag; parents outside the warp phase finished in the CTA
// sweep before this launch.  t = y - L21^T x2, x1 = L11^-T t, a lane per column.
// The panel is copied to shared memory (odd leading dimension) and y and the
// row indices are loaded before the wait.  FP64: the rows of t are split over
// the groups of lanes that the columns leave free, and the column sweep works
// on entries scaled by the reciprocal diagonal, as in front_bwd.  Measured: 60k
// buses FP64 119 -> 49 us, 10k mixed 36 -> 20 us.
template <typename T>
struct WarpPanel {
    T l[kWarpFrontMax * kWtLd];
    T x[kWarpFrontMax];
};
template <typename T>
__global__ void __launch_bounds__(kThreads) k_bwd_warp(DevFactor F, DevWork W, const T* lx, const T* rdiag,
                                                       SolveVecs sv, const int* order, const int* n_items,
                                                       int* counter, int* done) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr unsigned kAll = 0xffffffffu;
    WarpPanel<T>& t = reinterpret_cast<WarpPanel<T>*>(smem_raw)[threadIdx.x >> 5];
    T* sol = static_cast<T*>(sv.sol);
    const int lane = threadIdx.x & 31;
    const int ni = *n_items;
    for (;;) {
        const int item = warp_claim(counter);
        if (item >= ni) break;
        const int s = order[item];
        const FrontRec R = F.rec[s];
        if (!front_frozen(W, R)) {
            const int f = R.f, c0 = R.c0, nc = R.nc;
            const T* L = lx + R.lx_off;
            for (int c = 0; c < nc; ++c)
                if (lane >= c && lane < f) copy_async(t.l + lane + c * kWtLd, L + lane + c * f);
            copies_commit();
            const int at = lane < nc ? c0 + lane : lane < f ? F.sn_rows[R.rows_off + lane] : 0;
            const T rd = (!kInvDiag<T> && lane < nc) ? rdiag[c0 + lane] : T(0);
            T v = lane < nc ? __ldcg(sol + at) : T(0);
            copies_wait<0>();
            __syncwarp();
            if constexpr (!kInvDiag<T>) {
                for (int k = 1; k < nc; ++k) {
                    const T rk = __shfl_sync(kAll, rd, k);
                    if (lane < k) t.l[k + lane * kWtLd] *= rk;
                }
            }
            if (lane == 0 && R.parent >= 0) wait_done(done + R.parent, &W.status->flags, W.spin_limit);
            __syncwarp();
            if (lane >= nc && lane < f) v = __ldcg(sol + at);
            t.x[lane] = v;
            __syncwarp();
            if constexpr (kInvDiag<T>) {
                if (lane < nc) {
#pragma unroll 4
                    for (int r = nc; r < f; ++r) v -= t.l[r + lane * kWtLd] * t.x[r];
                }
                __syncwarp();
                if (lane < nc) t.x[lane] = v;
                __syncwarp();
                v = T(0);
                if (lane < nc) {
#pragma unroll 4
                    for (int i = lane; i < nc; ++i) v += t.l[i + lane * kWtLd] * t.x[i];
                }
            } else {
                const int w2 = nc <= 1 ? 1 : 1 << (32 - __clz(nc - 1));  // lanes per group
                const int c = lane & (w2 - 1), step = 32 / w2;
                T a = T(0);
                if (c < nc)
                    for (int r = nc + lane / w2; r < f; r += step) a += t.l[r + c * kWtLd] * t.x[r];
                for (int o = w2; o < 32; o <<= 1) a += __shfl_xor_sync(kAll, a, o);
                v -= a;
                for (int k = nc - 1; k > 0; --k) {
                    const T vk = __shfl_sync(kAll, v, k);
                    if (lane < k) v -= t.l[k + lane * kWtLd] * vk;
                }
                v *= rd;
            }
            if (lane < nc) sol[c0 + lane] = v;
            __syncwarp();
        }
        if (lane == 0 && s != W.hold_front) publish_done(done + s);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Claim-list compaction for a batch.  The claim lists (LevelSchedule::src_lists)
// are cut into chunks of kCompactChunk entries, one CTA each.  Pass 1 counts each chunk's fronts whose grid is not
// frozen; pass 2 offsets a chunk by the counts of the chunks before it in
// the same list and writes its kept entries in their original order (the
// claim order carries the critical-path priority and, for the backward
// sweep, parents before children).  A frozen grid's fronts form whole trees
// of their own, so no kept front has a dropped child or parent.
// ---------------------------------------------------------------------------
struct ReadyLists {
    const int* src[kReadyLists];
    int* dst[kReadyLists];
    int n[kReadyLists];
    int chunk0[kReadyLists + 1];  // first chunk of each list; the last entry = all chunks
};

__device__ __forceinline__ int list_of_chunk(const ReadyLists& R, int b) {
    int l = 0;
    while (l < kReadyLists - 1 && b >= R.chunk0[l + 1]) ++l;
    return l;
}

__device__ __forceinline__ bool claim_kept(const DevFactor& F, const DevWork& W, const ReadyLists& R, int l, int i) {
    return i < R.n[l] && !(W.grid_flags[F.sn_grid[R.src[l][i]]] & FLAG_FROZEN);
}

constexpr int kCompactThreads = 256;
static_assert(kCompactChunk % kCompactThreads == 0, "whole rounds per chunk");

__global__ void __launch_bounds__(kCompactThreads) k_ready_count(DevFactor F, DevWork W, ReadyLists R, int* chunk_cnt) {
    const int b = blockIdx.x;
    const int l = list_of_chunk(R, b);
    const int base = (b - R.chunk0[l]) * kCompactChunk;
    int total = 0;
    for (int r = 0; r < kCompactChunk; r += kCompactThreads)
        total += __syncthreads_count(claim_kept(F, W, R, l, base + r + threadIdx.x));
    if (threadIdx.x == 0) chunk_cnt[b] = total;
}

__global__ void __launch_bounds__(kCompactThreads) k_ready_compact(DevFactor F, DevWork W, ReadyLists R,
                                                                    const int* chunk_cnt, int* counts) {
    __shared__ int warp_n[kCompactThreads / 32];
    __shared__ int s_off;
    const int b = blockIdx.x;
    const int l = list_of_chunk(R, b);
    const int base = (b - R.chunk0[l]) * kCompactChunk;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // offset of this chunk: kept entries of the list's earlier chunks
    int part = 0;
    for (int q = R.chunk0[l] + threadIdx.x; q < b; q += kCompactThreads) part += chunk_cnt[q];
    for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
    if (lane == 0) warp_n[warp] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int w = 0; w < kCompactThreads / 32; ++w) t += warp_n[w];
        s_off = t;
    }
    __syncthreads();
    int off = s_off;
    for (int r = 0; r < kCompactChunk; r += kCompactThreads) {
        const int i = base + r + threadIdx.x;
        const bool keep = claim_kept(F, W, R, l, i);
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        __syncthreads();  // warp_n of the previous round has been read
        if (lane == 0) warp_n[warp] = __popc(m);
        __syncthreads();
        int before = 0, all = 0;
        for (int w = 0; w < kCompactThreads / 32; ++w) {
            before += (w < warp) ? warp_n[w] : 0;
            all += warp_n[w];
        }
        if (keep) R.dst[l][off + before + __popc(m & ((1u << lane) - 1u))] = R.src[l][i];
        off += all;
    }
    if (threadIdx.x == 0 && b == R.chunk0[l + 1] - 1) counts[l] = off;
}


template <typename HV>
__global__ void k_gain_export(DevFactor F, const HV* hval, const HV* hw, int n_tgt, double* out) {
    for (int tg = blockIdx.x * blockDim.x + threadIdx.x; tg < n_tgt; tg += gridDim.x * blockDim.x)
        out[tg] = gain_entry<HV, double>(F, hval, hw, tg);
}

inline int grid_for(int64_t n, int threads) {
    int64_t g = (n + threads - 1) / threads;
    if (g > kSMs * 16) g = kSMs * 16;
    return (int)(g < 1 ? 1 : g);
}

template <typename V>
size_t solve_smem(int maxf) {
    return (size_t)(maxf + 2) * sizeof(V);
}

template <typename T, typename HV>
cudaError_t prepare_impl() {
    cudaError_t e = cudaFuncSetAttribute(k_front_small<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)front_smem<T>(small_front_max<T>()));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_front_flow<T, kPanel, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)front_smem<T>(small_front_max<T>()));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_front_flow<T, kPanelSmall, kMinBlocksA<T>>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)front_smem<T>(kFlowSmallFMax));
    const int mx = (int)solve_smem<double>(16384), mb = (int)kBwdSmemMax;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_fwd<T, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_bwd<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, mb);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_fwd_flow<T, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_bwd_flow<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, mb);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_bwd_warp<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(WarpPanel<T>) * kWarpsPerCta));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_front_warp<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(WarpTile<T>) * kWarpsPerCta));

    return e;
}

template <typename T, typename HV>
cudaError_t factor_impl(const DevNet& net, const DevFactor& F, const DevWork& W, const LevelSchedule& ls, const HV* hval,
                        const HV* hw, T* lx, T* ub, SolveVecs sv, bool begin, cudaStream_t st) {
    T* gv = reinterpret_cast<T*>(W.gvals);
    const bool tile_flow = sizeof(T) == 4 && ls.n_tt > 0;
    {
        // the flags and counters of the factorisation and of the backward sweep after it
        const ZeroLists Z{{W.flow, ls.d_pot_cnt, ls.d_tt_done},
                          {3 * F.n_super + 16, ls.n_pot_pairs, tile_flow ? ls.n_tt + ls.n_levels : 0}};
        const int nr = begin ? (F.n_state + kThreads - 1) / kThreads : 0, nb = nr + grid_for(ls.n_tgt, kThreads);
        if (sizeof(T) == 4 && ls.gain_acc32)
            k_gain_values<T, HV, float><<<nb, kThreads, 0, st>>>(F, W, hval, hw, gv, ls.n_tgt, net.h_row, nr, Z);
        else
            k_gain_values<T, HV, double><<<nb, kThreads, 0, st>>>(F, W, hval, hw, gv, ls.n_tgt, net.h_row, nr, Z);
        count_launches(1);
    }
    if (ls.flow_a_n + ls.flow_b_n + ls.flow_w_n > 0) {
        int* counters = W.flow + F.n_super;
        if (ls.flow_w_n > 0) {
            k_front_warp<T><<<ls.flow_w_grid, kThreads, sizeof(WarpTile<T>) * kWarpsPerCta, st>>>(
                F, W, sv, gv, lx, ub, ls.d_flow_w, ls.d_ready_n + 4, counters + 2, W.flow);
            count_launches(1);
        }
        if (ls.flow_a_n > 0) {
            const int mf = ls.flow_a_maxf;
            k_front_flow<T, kPanelSmall, kMinBlocksA<T>><<<ls.flow_a_grid, kThreads, front_smem<T>(mf), st>>>(
                F, W, sv, gv, lx, ub, ls.d_flow_a, ls.d_ready_n + 0, counters + 0, W.flow);
            count_launches(1);
        }
        if (ls.flow_b_n > 0) {
            const int mf = ls.flow_b_maxf;
            k_front_flow<T, kPanel, 1><<<ls.flow_b_grid, kFrontThreads<T, kPanel>, front_smem<T>(mf), st>>>(
                F, W, sv, gv, lx, ub, ls.d_flow_b, ls.d_ready_n + 1, counters + 1, W.flow);
            count_launches(1);
        }
    }
    for (int l = 0; l < ls.n_levels; ++l) {
        const int ns = ls.h_small_ptr[l + 1] - ls.h_small_ptr[l];
        const int na = ls.h_asm_ptr[l + 1] - ls.h_asm_ptr[l];
        const int nt = tile_flow ? ls.h_tt_ptr[l + 1] - ls.h_tt_ptr[l] : 0;
        // The fronts of a level do not depend on each other: its single-CTA ones
        // run on the side stream beside the tiled ones' steps, which leave most
        // SMs idle (60k buses FP64 26.1 -> 23.8 ms, 64 grids 13.7 -> 12.3).  Not
        // beside the tile dataflow kernel, whose CTAs fill the GPU and wait for
        // one another.
        const bool beside = ns > 0 && na > 0 && nt == 0;
        if (beside) {
            cudaError_t e = cudaEventRecord(ls.fork, st);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(ls.side, ls.fork, 0);
            if (e != cudaSuccess) return e;
        }
        if (ns > 0) {
            const int mf = ls.h_small_maxf[l];
            k_front_small<T><<<ns, kFrontThreads<T, kPanel>, front_smem<T>(mf), beside ? ls.side : st>>>(
                F, W, sv, gv, lx, ub, ls.d_small + ls.h_small_ptr[l]);
            count_launches(1);
        }
        if (beside) {
            cudaError_t e = cudaEventRecord(ls.join, ls.side);
            if (e != cudaSuccess) return e;
        }
        if (na > 0) {
            k_big_assemble<T><<<na, kThreads, 0, st>>>(F, W, sv, gv, lx, ub, ls.d_asm + ls.h_asm_ptr[l],
                                                   ls.d_asm_child);
            count_launches(1);
            if constexpr (sizeof(T) == 4) {
                if (nt > 0) {
                    k_big_flow32<<<std::min(nt, ls.tt_grid), kThreads, 0, st>>>(
                        F, W, sv, lx, ls.d_tt + ls.h_tt_ptr[l], nt, ls.d_tt_done + ls.h_tt_ptr[l],
                        ls.d_tt_done + ls.n_tt + l, ls.d_pot_cnt);
                    count_launches(1);
                }
            }
            for (int p = 0; nt == 0 && p < ls.h_lvl_panels[l]; ++p) {
                const int slot = ls.h_step_ptr[l] + p;
                const int npot = ls.h_pot_ptr[slot + 1] - ls.h_pot_ptr[slot];
                const int nupd = ls.h_upd_ptr[slot + 1] - ls.h_upd_ptr[slot];
                if (npot > 0) {
                    const int4* work = ls.d_pot + ls.h_pot_ptr[slot];
                    if constexpr (sizeof(T) == 4)
                        k_big_panel32<<<npot, kThreads, 0, st>>>(F, W, sv, lx, work, p, ls.d_pot_cnt);
                    else
                        k_big_panel64<<<npot, kPanelThreads64, 0, st>>>(F, W, sv, lx, work, p, ls.d_pot_cnt);
                    count_launches(1);
                }
                if (nupd > 0) {
                    if constexpr (sizeof(T) == 4)
                        k_big_step32<<<nupd, kThreads, 0, st>>>(F, W, sv, lx, ls.d_step + ls.h_upd_ptr[slot], p,
                                                                ls.d_pot_cnt);
                    else
                        k_big_update64<<<nupd, kUpdTile64 * kUpdTile64, 0, st>>>(F, W, sv, lx,
                                                                                 ls.d_upd + ls.h_upd_ptr[slot], p);
                    count_launches(1);
                }
            }
        }
        if (beside) {
            cudaError_t e = cudaStreamWaitEvent(st, ls.join, 0);
            if (e != cudaSuccess) return e;
        }
    }
    return cudaGetLastError();
}

// Forward and backward sweeps (forward), or the backward sweep alone after a
// factorisation that carried the right-hand side along (factor_impl, which
// also cleared the flags).
template <typename T>
cudaError_t solve_impl(const DevFactor& F, const DevWork& W, const LevelSchedule& ls, const T* lx, const T* rdiag,
                       SolveVecs sv, bool forward, cudaStream_t st) {
    if (ls.solve_flow) {
        // flags: [0, n_super) forward, [n_super, 2 n_super) backward, then counters
        const int ns = F.n_super;
        int* fwd_done = W.flow + ns + 8;
        int* bwd_done = fwd_done + ns;
        int* counters = bwd_done + ns;
        const size_t smem = solve_smem<T>(ls.solve_maxf);
        // warp fronts first going up, last coming down
        if (forward) {
            cudaError_t e = cudaMemsetAsync(fwd_done, 0, sizeof(int) * (size_t)(2 * ns + 8), st);
            if (e != cudaSuccess) return e;
            if (ls.flow_w_n > 0) {
                k_fwd_warp<T, T><<<ls.solve_w_grid, kThreads, 0, st>>>(F, W, lx, rdiag, sv, ls.d_flow_w,
                                                                       ls.d_ready_n + 4, ls.d_phase, 3,
                                                                       ls.d_phase_nchild, counters + 2, fwd_done);
                count_launches(1);
            }
            if (ls.up_n > 0) {
                k_fwd_flow<T, T><<<ls.up_grid, kThreads, smem, st>>>(F, W, lx, rdiag, sv, ls.d_up, ls.d_ready_n + 2,
                                                                     ls.d_nchild, counters + 0, fwd_done);
                count_launches(1);
            }
        }
        if (ls.down_top_n > 0) {
            const int cap = bwd_top_cap<T>(ls.solve_maxf);
            k_bwd_flow<T><<<ls.down_top_grid, kThreads, bwd_smem<T>(ls.solve_maxf, cap), st>>>(
                F, W, lx, rdiag, sv, ls.solve_maxf, cap, ls.d_down_top, ls.d_ready_n + 6, counters + 4, bwd_done);
            count_launches(1);
        }
        if (ls.down_n > 0) {
            k_bwd_flow<T><<<ls.down_grid, kThreads, bwd_smem<T>(ls.down_maxf, kBwdCap), st>>>(
                F, W, lx, rdiag, sv, ls.down_maxf, kBwdCap, ls.d_down, ls.d_ready_n + 3, counters + 1, bwd_done);
            count_launches(1);
        }
        if (ls.down_w_n > 0) {
            k_bwd_warp<T><<<ls.down_w_grid, kThreads, sizeof(WarpPanel<T>) * kWarpsPerCta, st>>>(
                F, W, lx, rdiag, sv, ls.d_down_w, ls.d_ready_n + 5, counters + 3, bwd_done);
            count_launches(1);
        }
        return cudaGetLastError();
    }
    for (int l = 0; forward && l < ls.n_levels; ++l) {
        const int n = ls.h_all_ptr[l + 1] - ls.h_all_ptr[l];
        if (n > 0) {
            k_fwd<T, T><<<n, kThreads, solve_smem<T>(ls.h_lvl_maxf[l]), st>>>(F, W, lx, rdiag, sv,
                                                                               ls.d_all + ls.h_all_ptr[l]);
            count_launches(1);
        }
    }
    for (int l = ls.n_levels - 1; l >= 0; --l) {
        const int n = ls.h_all_ptr[l + 1] - ls.h_all_ptr[l];
        if (n > 0) {
            const int mf = ls.h_lvl_maxf[l];
            k_bwd<T><<<n, kThreads, bwd_smem<T>(mf, kBwdCap), st>>>(F, W, lx, rdiag, sv, mf, kBwdCap,
                                                                   ls.d_all + ls.h_all_ptr[l]);
            count_launches(1);
        }
    }
    return cudaGetLastError();
}

template <typename T>
FlowGrids flow_grids_impl(int32_t maxf_a, int32_t maxf_b, int32_t solve_maxf, int32_t down_maxf) {
    FlowGrids g{0, 0, 0, 0, 0, 0, 0, 0, 0};
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return g;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return g;
    auto resident = [&](const void* fn, size_t smem, int threads = kThreads) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem) != cudaSuccess) return 0;
        return per_sm * sms;
    };
    g.a = resident((const void*)k_front_flow<T, kPanelSmall, kMinBlocksA<T>>, front_smem<T>(maxf_a));
    g.b = resident((const void*)k_front_flow<T, kPanel, 1>, front_smem<T>(maxf_b), kFrontThreads<T, kPanel>);
    if (solve_maxf <= 16384) g.solve = resident((const void*)k_fwd_flow<T, T>, solve_smem<T>(solve_maxf));
    g.w = resident((const void*)k_front_warp<T>, sizeof(WarpTile<T>) * kWarpsPerCta);
    g.wsolve = resident((const void*)k_fwd_warp<T, T>, 0);
    g.down = resident((const void*)k_bwd_flow<T>, bwd_smem<T>(down_maxf, kBwdCap));
    if (solve_maxf <= 16384)
        g.down_top = resident((const void*)k_bwd_flow<T>, bwd_smem<T>(solve_maxf, bwd_top_cap<T>(solve_maxf)));
    g.down_w = resident((const void*)k_bwd_warp<T>, sizeof(WarpPanel<T>) * kWarpsPerCta);
    g.tile = sizeof(T) == 4 ? resident((const void*)k_big_flow32, 0) : 0;
    cudaGetLastError();
    return g;
}

}  // namespace

cudaError_t launch_ready_compact(const DevFactor& F, const DevWork& W, const LevelSchedule& ls, cudaStream_t st) {
    ReadyLists R;
    R.chunk0[0] = 0;
    for (int l = 0; l < kReadyLists; ++l) {
        R.src[l] = ls.src_lists[l];
        R.dst[l] = ls.cmp_lists[l];
        R.n[l] = ls.src_n[l];
        R.chunk0[l + 1] = R.chunk0[l] + (R.n[l] + kCompactChunk - 1) / kCompactChunk;
    }
    const int nb = R.chunk0[kReadyLists];
    if (nb == 0 || !W.grid_flags) return cudaSuccess;
    k_ready_count<<<nb, kCompactThreads, 0, st>>>(F, W, R, ls.d_chunk_cnt);
    k_ready_compact<<<nb, kCompactThreads, 0, st>>>(F, W, R, ls.d_chunk_cnt, ls.d_ready_n);
    count_launches(2);
    return cudaGetLastError();
}

FlowGrids flow_grids(bool mixed, int32_t maxf_a, int32_t maxf_b, int32_t solve_maxf, int32_t down_maxf) {
    return mixed ? flow_grids_impl<float>(maxf_a, maxf_b, solve_maxf, down_maxf)
                 : flow_grids_impl<double>(maxf_a, maxf_b, solve_maxf, down_maxf);
}

cudaError_t prepare_factor_kernels() {
    cudaError_t e = prepare_impl<double, double>();
    if (e == cudaSuccess) e = prepare_impl<float, float>();
    return e;
}

namespace {
SolveVecs vecs32(const DevWork& W) { return SolveVecs{W.rhs32, W.sol32, W.su32}; }
SolveVecs vecs64(const DevWork& W) { return SolveVecs{W.rhs, W.sol, W.su}; }
}  // namespace

cudaError_t launch_rhs(const DevNet& net, const DevFactor& F, const DevWork& W, bool begin, cudaStream_t st) {
    k_rhs<<<(F.n_state + kThreads - 1) / kThreads, kThreads, 0, st>>>(F, W, net.h_row, begin ? 1 : 0);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_factor32(const DevNet& net, const DevFactor& F, const DevWork& W, const LevelSchedule& ls,
                            bool begin, cudaStream_t st) {
    return factor_impl<float, float>(net, F, W, ls, W.hval32, W.hw32, W.lx32, W.u32, vecs32(W), begin, st);
}

cudaError_t launch_solve32(const DevFactor& F, const DevWork& W, const LevelSchedule& ls, bool forward,
                           cudaStream_t st) {
    return solve_impl<float>(F, W, ls, W.lx32, reinterpret_cast<const float*>(W.rdiag), vecs32(W), forward, st);
}

cudaError_t launch_factor(const DevNet& net, const DevFactor& F, const DevWork& W, const LevelSchedule& ls, bool begin,
                          cudaStream_t st) {
    return factor_impl<double, double>(net, F, W, ls, W.hval, W.hw, W.lx, W.u, vecs64(W), begin, st);
}

cudaError_t launch_solve(const DevFactor& F, const DevWork& W, const LevelSchedule& ls, bool forward,
                         cudaStream_t st) {
    return solve_impl<double>(F, W, ls, W.lx, reinterpret_cast<const double*>(W.rdiag), vecs64(W), forward, st);
}

cudaError_t launch_gain_export(const DevNet& net, const DevFactor& F, const DevWork& W, int32_t n_tgt, double* out,
                               cudaStream_t st) {
    if (n_tgt > 0) {
        k_gain_export<double><<<grid_for(n_tgt, 256), 256, 0, st>>>(F, W.hval, W.hw, n_tgt, out);
        count_launches(1);
    }
    return cudaGetLastError();
}


// ---------------------------------------------------------------------------
// Allocation-free factor/solve.  One call's scratch -- right-hand side and
// solution staging in state order, the dataflow flags, the solve update
// vectors and the small fronts' update matrices -- lives in one file-scope
// device array of kNoAllocScratchBytes.  The address is looked up once per
// device (cudaGetSymbolAddress, with that device current); every call on a
// device shares the array, so calls that overlap in time race.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

namespace {
constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
unsigned char* g_noalloc_ptr[kNoAllocMaxDevices] = {};

size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

struct NoAllocLayout {
    size_t rhs, x, flow, su, u, total;  // byte offsets into the scratch array
};

NoAllocLayout noalloc_layout(const NoAllocShape& sh) {
    NoAllocLayout l{};
    size_t off = 0;
    l.rhs = off;
    off = align256(off + sizeof(double) * (size_t)sh.n_state);
    l.x = off;
    off = align256(off + sizeof(double) * (size_t)sh.n_state);
    l.flow = off;
    off = align256(off + sizeof(int) * (3 * (size_t)sh.n_super + 16));
    l.su = off;
    off = align256(off + sizeof(double) * (size_t)sh.su_elems);
    l.u = off;
    off = align256(off + sizeof(double) * (size_t)sh.u_elems);
    l.total = off;
    return l;
}

// state index -> permuted position (theta of every bus but the slack, then |V|)
__device__ __forceinline__ int ps_of_state(const DevNet& net, const DevFactor& F, int st) {
    const int nth = net.n_bus - 1;
    if (st < nth) return F.bus_ps_theta[st < net.slack ? st : st + 1];
    return F.bus_ps_v[st - nth];
}

__global__ void k_state_to_ps(DevNet net, DevFactor F, const double* in, double* out) {
    const int st = blockIdx.x * blockDim.x + threadIdx.x;
    if (st < F.n_state) out[ps_of_state(net, F, st)] = in[st];
}

__global__ void k_ps_to_state(DevNet net, DevFactor F, const double* in, double* out) {
    const int st = blockIdx.x * blockDim.x + threadIdx.x;
    if (st < F.n_state) out[st] = in[ps_of_state(net, F, st)];
}
}  // namespace

size_t noalloc_scratch_need(const NoAllocShape& sh) { return noalloc_layout(sh).total; }

cudaError_t noalloc_scratch_setup(void** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kNoAllocMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_noalloc_ptr[dev] = static_cast<unsigned char*>(p);
    }
    *out = g_noalloc_ptr[dev];
    return cudaSuccess;
}

cudaError_t launch_factor_solve_noalloc(const DevNet& net, const DevFactor& F, const DevWork& W,
                                        const LevelSchedule& ls, const NoAllocShape& sh, const double* rhs_host,
                                        double* x_host, cudaStream_t st) {
    const NoAllocLayout l = noalloc_layout(sh);
    if (l.total > kNoAllocScratchBytes) return cudaErrorInvalidValue;  // callers check the size first
    void* base = nullptr;
    cudaError_t e = noalloc_scratch_setup(&base);
    if (e != cudaSuccess) return e;
    unsigned char* b = static_cast<unsigned char*>(base);
    double* d_rhs = reinterpret_cast<double*>(b + l.rhs);
    double* d_x = reinterpret_cast<double*>(b + l.x);
    DevWork W2 = W;
    W2.flow = reinterpret_cast<int*>(b + l.flow);  // cleared at the start of each pass
    W2.su = reinterpret_cast<double*>(b + l.su);
    W2.u = reinterpret_cast<double*>(b + l.u);
    const int n = F.n_state;
    e = cudaMemcpyAsync(d_rhs, rhs_host, sizeof(double) * (size_t)n, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    if (n > 0) {
        k_state_to_ps<<<grid_for(n, 256), 256, 0, st>>>(net, F, d_rhs, W2.rhs);
        count_launches(1);
    }
    e = launch_factor(net, F, W2, ls, false, st);
    if (e == cudaSuccess) e = launch_solve(F, W2, ls, false, st);
    if (e != cudaSuccess) return e;
    if (n > 0) {
        k_ps_to_state<<<grid_for(n, 256), 256, 0, st>>>(net, F, W2.sol, d_x);
        count_launches(1);
    }
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(x_host, d_x, sizeof(double) * (size_t)n, cudaMemcpyDeviceToHost, st);
    return e;
}

}  // namespace sle_gb300
