// SDF value and gradient point queries on sm_100a.
//
// Recipes (src/field_engine/ikarus_v1/eval_warp.py:478-488 eval_batch, :718-733 gradient_batch):
//   k_eval_points evaluates the compiled program at float32 points (thread per point).  With a
//   built field's culling lists (the lists a classification left in its scratch) k_query_warp (few
//   points) and k_query_sorted (many) cull the superblock's list once more to the points at hand --
//   exact, by the same strict-domination argument as the build -- instead of walking the whole chain.
//   k_gradient_points: central differences with step h along each axis, the six offset points
//   formed in float64 and rounded to float32 as the reference does.  By sizes (by_items, short_chain)
//   the offset points of an accelerated query go as points of their own, and short chains whole.
// Per-block pitch fields (src/field_engine/faltkarna_v1_multires.py:84-104, :384-459):
//   k_multires_tiles fills each active brick's (B*2^l + 1)^3 lattice at pitch h/2^l;
//   k_multires_value answers avstand (trilinear at the brick's own pitch, +-margin outside active
//   bricks) and k_multires_gradient the brick-clamped central difference.
#include "common.cuh"
#include "cull.cuh"
#include "prims.cuh"
#include <algorithm>
#include <cmath>
#include <type_traits>

namespace {

// Program value at a float32 world point.  chain_mode 1: `list` (entries chain index << 2 | mode)
// over the chain; chain_mode 0: the postfix program with a float32 stack.
__device__ float eval_point(const PrimF* __restrict__ primf, const FbInsn* __restrict__ chain, int n_chain,
                            int chain_mode, const uint32_t* __restrict__ list, int len, float x, float y, float z) {
    if (chain_mode) {
        float acc = 0.f;
        for (int i = 0; i < len; ++i) {
            const uint32_t e = list ? list[i] : (uint32_t)i << 2;
            const FbInsn I = chain[e >> 2];
            const uint32_t mode = e & 3u;
            const int op = mode == 1u ? CH_SET : (mode == 2u ? CH_SETNEG : I.op);
            const float v = op == CH_OFFSET ? 0.f : primf_world(primf[I.arg], x, y, z);
            acc = chain_apply(op, acc, v, (float)I.k);
        }
        return acc;
    }
    float st[32];
    int sp = 0;
    for (int i = 0; i < n_chain; ++i) {
        const FbInsn I = chain[i];
        if (I.op == OP_PUSH) {
            if (sp < 32) st[sp++] = primf_world(primf[I.arg], x, y, z);
        } else if (I.op == OP_OFFSET) {
            if (sp > 0) st[sp - 1] -= (float)I.k;
        } else if (sp > 1) {
            const float b = st[--sp];
            const int op = I.op == OP_UNION ? CH_UNION : (I.op == OP_INTERSECT ? CH_INTERSECT : CH_SUBTRACT);
            st[sp - 1] = combine_f(op, st[sp - 1], b, (float)I.k);
        }
    }
    return sp == 1 ? st[0] : __int_as_float(0x7fc00000);
}

struct Accel {  // a built field's culling lists (nullptr pool: walk the whole chain)
    const uint32_t* pool;
    const int64_t* sb_off;
    const int32_t* sb_len;
    // per-block lists (nullable): used where kind == 0, or for every block when blk_all
    const int32_t* kind;
    const int32_t* blk_off;
    const int32_t* blk_len;
    const uint32_t* blk_pool;
    int64_t blk_cap;
    int blk_all;
    double x0, y0, z0, pitch;
    int nx, ny, nz, B, S, nsx, nsy, nsz, nbx, nby, nbz;
    float eps;  // slack of the bounds beside the primitives' own rounding, from the grid's coordinates
};

// The list a point at (x, y, z) walks on its own: its block's where the classification kept one, its
// superblock's elsewhere inside the grid, the whole chain (nullptr) outside.
__device__ __forceinline__ void accel_list(const Accel& A, int n_chain, float x, float y, float z,
                                           const uint32_t*& list, int& len) {
    {
        // the voxel cell containing the point, inside the grid's block range
        const double fx = ((double)x - A.x0) / A.pitch, fy = ((double)y - A.y0) / A.pitch,
                     fz = ((double)z - A.z0) / A.pitch;
        const double ex = (double)A.nbx * A.B, ey = (double)A.nby * A.B, ez = (double)A.nbz * A.B;
        if (fx >= 0 && fy >= 0 && fz >= 0 && fx <= ex && fy <= ey && fz <= ez) {
            const int bi = min((int)(fx / A.B), A.nbx - 1), bj = min((int)(fy / A.B), A.nby - 1),
                      bk = min((int)(fz / A.B), A.nbz - 1);
            if (A.blk_len) {  // the block's own list: culled for a region holding the whole block
                const int64_t b = ((int64_t)bi * A.nby + bj) * A.nbz + bk;
                if (A.blk_all || A.kind[b] == 0) {
                    const int n = A.blk_len[b];
                    const int64_t off = n >= 0 ? (int64_t)A.blk_off[b] : -1;
                    if (n >= 0 && off >= 0 && off + n <= A.blk_cap) {
                        list = A.blk_pool + off;
                        len = n;
                        return;
                    }
                }
            }
            const int64_t s = ((int64_t)(bi / A.S) * A.nsy + bj / A.S) * A.nsz + bk / A.S;
            list = A.pool + A.sb_off[s];
            len = A.sb_len[s];
            return;
        }
    }
    list = nullptr;
    len = n_chain;
}

__global__ void k_eval_points(const PrimF* __restrict__ primf, const FbInsn* __restrict__ chain, int n_chain,
                              int chain_mode, const float* __restrict__ pts, int64_t n, float* __restrict__ out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = eval_point(primf, chain, n_chain, chain_mode, nullptr, n_chain, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]);
}

// Central difference with step h: (f(p + h e_a) - f(p - h e_a)) / (2h) in float32, the offset
// points formed in float64 and rounded to float32 (eval_warp.py:718-733).  `value` (nullable)
// also receives f(p).
__global__ void k_gradient_points(const PrimF* __restrict__ primf, const FbInsn* __restrict__ chain, int n_chain,
                                  int chain_mode, const float* __restrict__ pts, int64_t n, double h,
                                  float* __restrict__ grad, float* __restrict__ value) {
    const float inv = (float)(2.0 * h);
    auto eval = [&](float x, float y, float z) {
        return eval_point(primf, chain, n_chain, chain_mode, nullptr, n_chain, x, y, z);
    };
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double p[3] = {pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]};
        for (int a = 0; a < 3; ++a) {
            float q[2][3];
            for (int s = 0; s < 2; ++s)
                for (int c = 0; c < 3; ++c) q[s][c] = (float)(c == a ? p[c] + (s ? -h : h) : p[c]);
            grad[3 * i + a] = (eval(q[0][0], q[0][1], q[0][2]) - eval(q[1][0], q[1][1], q[1][2])) / inv;
        }
        if (value) value[i] = eval((float)p[0], (float)p[1], (float)p[2]);
    }
}

// ------------------------------------------------------------------------------------ queries near a field
// A point has NV evaluations: variant 0 the point itself and, with a gradient (NV = 7), 1 + 2a + s the
// offset along axis a (s = 0: +h, 1: -h), formed in float64 and rounded to float32 as
// k_gradient_points forms them.  A superblock's list holds for its whole bounding ball (that is what
// the build culled it for), so the variants of one or of many points of a superblock that lie in the
// ball share the list -- and a warp first culls it once more, to the ball around just those points
// (warp_walk_once, the build's own exact rule), before anything is evaluated.  Points outside every ball
// (beyond the grid's edge) have the whole chain culled to the ball around them in the same way.  What
// is left -- an offset that leaves its point's ball, non-finite coordinates -- walks its own list
// (accel_list).  Values are independent of the list they come from, so all paths give the whole
// chain's values bit for bit.
constexpr int kQueryWarps = 4;
constexpr int kQueryCap = 192;  // survivors kept per warp; a longer list is walked as it is

struct Variants {
    float p[3], plus[3], minus[3];
    __device__ __forceinline__ float at(int v, int axis) const {
        float q = p[axis];
        if (v == 1 + 2 * axis) q = plus[axis];
        if (v == 2 + 2 * axis) q = minus[axis];
        return q;
    }
};

__device__ __forceinline__ Variants load_variants(const float* __restrict__ pts, int64_t i, double h) {
    Variants V;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float x = pts[3 * i + a];
        V.p[a] = (float)(double)x;
        V.plus[a] = (float)((double)x + h);
        V.minus[a] = (float)((double)x - h);
    }
    return V;
}

// What a query's item is: point i itself with its variants, or (kItems) one evaluation, variant i % 7 of point
// i / 7.
template <bool kItems>
__device__ __forceinline__ Variants load_query(const float* __restrict__ pts, int64_t i, double h) {
    if (!kItems) return load_variants(pts, i, h);
    const int64_t at = i / 7;
    const int v = (int)(i - 7 * at);
    Variants V = load_variants(pts, at, h);
#pragma unroll
    for (int a = 0; a < 3; ++a) V.p[a] = V.at(v, a);
    return V;
}

// The superblock nearest a point, the bit mask of the point's variants inside that superblock's ball
// (0 when the point itself is not), and the point's sorting cell: C^3 cells per superblock.
struct Place {
    int s, cell;
    unsigned inside, beyond;  // beyond: outside that ball and outside the grid (the whole chain's)
};

template <int NV>
__device__ __forceinline__ Place place_of(const Accel& A, const Variants& V, int C) {
    const double edge = (double)A.S * A.B, inv = 1.0 / (A.pitch * edge);
    const double o[3] = {A.x0, A.y0, A.z0};
    const int ns[3] = {A.nsx, A.nsy, A.nsz};
    int si[3], ci[3];
    double ctr[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double f = ((double)V.p[a] - o[a]) * inv;  // in superblocks
        const double g = fmin(fmax(f, 0.0), (double)ns[a] - 0.5);  // NaN: 0
        si[a] = (int)g;
        ci[a] = min((int)((g - si[a]) * C), C - 1);
        ctr[a] = o[a] + (si[a] + 0.5) * edge * A.pitch;
    }
    const double R = 0.5 * 1.7320508 * edge * A.pitch, R2 = R * R * (1.0 - 1e-5);
    Place P;
    P.s = (si[0] * A.nsy + si[1]) * A.nsz + si[2];
    // boustrophedon inside the superblock: consecutive cells touch, so a warp's points stay close
    const int y = (ci[0] & 1) ? C - 1 - ci[1] : ci[1];
    P.cell = (P.s * C + ci[0]) * C * C + y * C + (((ci[0] * C + y) & 1) ? C - 1 - ci[2] : ci[2]);
    double d2[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double d = (double)V.p[a] - ctr[a];
        d2[a] = d * d;
    }
    const double sum = d2[0] + d2[1] + d2[2];
    P.inside = sum <= R2 ? 1u : 0u;  // false for NaN
    P.beyond = 0u;
    if (NV > 1 && P.inside) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double dp = (double)V.plus[a] - ctr[a], dm = (double)V.minus[a] - ctr[a];
            if (sum - d2[a] + dp * dp <= R2) P.inside |= 2u << (2 * a);
            if (sum - d2[a] + dm * dm <= R2) P.inside |= 4u << (2 * a);
        }
    }
    const unsigned all = (1u << NV) - 1u;
    if (P.inside != all) {
        const int nb[3] = {A.nbx, A.nby, A.nbz};
        auto out = [&](int a, float x) {
            const double f = ((double)x - o[a]) * inv * A.S;  // in blocks
            return !(f >= 0.0 && f <= (double)nb[a]);
        };
        unsigned off[3];  // per axis: bit 0 the point, 1 +h, 2 -h beyond the grid along it
#pragma unroll
        for (int a = 0; a < 3; ++a)
            off[a] = out(a, V.p[a]) | (NV > 1 ? out(a, V.plus[a]) << 1 | out(a, V.minus[a]) << 2 : 0);
        const unsigned any = (off[0] | off[1] | off[2]) & 1u;
        P.beyond = any;
        if (NV > 1) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const unsigned rest = (off[(a + 1) % 3] | off[(a + 2) % 3]) & 1u;
                P.beyond |= ((off[a] >> 1 & 1u) | rest) << (1 + 2 * a) | ((off[a] >> 2) | rest) << (2 + 2 * a);
            }
        }
        P.beyond &= ~P.inside & all;
    }
    return P;
}

// The largest coordinate of a point's variants where all are finite and far from overflow, else -1.
template <int NV>
__device__ __forceinline__ float finite_reach(const Variants& V) {
    float m = 0.f;
    bool ok = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        m = fmaxf(m, fabsf(V.p[a]));
        ok &= fabsf(V.p[a]) < 1.0e15f;
        if (NV > 1) {
            m = fmaxf(m, fmaxf(fabsf(V.plus[a]), fabsf(V.minus[a])));
            ok &= fabsf(V.plus[a]) < 1.0e15f && fabsf(V.minus[a]) < 1.0e15f;
        }
    }
    return ok ? m : -1.f;
}

// A warp's survivors in shared memory.
struct Survivors {
    uint32_t ent[kQueryCap];
    float lo[kQueryCap], hi[kQueryCap];
};

// `list` (nullptr: the whole chain) culled to the ball (c, R) of points whose coordinates reach `reach`;
// left as it is where the survivors do not fit.
template <bool kStretches>
__device__ __forceinline__ void cull_to(const uint32_t*& list, int& len, const FbInsn* __restrict__ chain,
                                        const PrimF* __restrict__ primf, const float* c, float R, float reach,
                                        float eps, Survivors& out) {
    const float e = fmaxf(eps, 16.f * 1.2e-7f * reach);  // 16 float32 ulps
    const int m = warp_walk_once<kStretches>(list, len, chain, primf, c[0], c[1], c[2], R, e, out.ent, out.lo, out.hi, kQueryCap);
    if (m <= kQueryCap) {
        list = out.ent;
        len = m;
    }
}

// eval_point out of line: the rare paths' copy.
static __device__ __noinline__ float eval_list(const PrimF* __restrict__ primf, const FbInsn* __restrict__ chain,
                                               const uint32_t* list, int len, float x, float y, float z) {
    return eval_point(primf, chain, len, 1, list, len, x, y, z);
}

static __device__ __noinline__ float canon_rare(const PrimF& P, float x, float y, float z) {
    return canon_f(P.type, P.p, x, y, z);
}

// Two values of one kind, canon_f's operations on primf_world's coordinates.
template <int T>
__device__ __forceinline__ void canon_pair(const PrimF& P, const float* x, const float* y, const float* z, float* v) {
#pragma unroll
    for (int k = 0; k < 2; ++k) v[k] = canon_f(T, P.p, x[k], y[k], z[k]);
}

__device__ __forceinline__ void eval_pair(const PrimF& P, const float* qx, const float* qy, const float* qz, float* v) {
    float x[2], y[2], z[2];
    if (P.ident) {  // products with 1 and 0 are exact: the sums with the translation are all that rounds
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            x[k] = qx[k] + P.A[3];
            y[k] = qy[k] + P.A[7];
            z[k] = qz[k] + P.A[11];
        }
    } else {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            x[k] = fmaf(P.A[0], qx[k], fmaf(P.A[1], qy[k], fmaf(P.A[2], qz[k], P.A[3])));
            y[k] = fmaf(P.A[4], qx[k], fmaf(P.A[5], qy[k], fmaf(P.A[6], qz[k], P.A[7])));
            z[k] = fmaf(P.A[8], qx[k], fmaf(P.A[9], qy[k], fmaf(P.A[10], qz[k], P.A[11])));
        }
    }
    switch (P.type) {
    case P_SPHERE: canon_pair<P_SPHERE>(P, x, y, z, v); break;
    case P_BOX: canon_pair<P_BOX>(P, x, y, z, v); break;
    case P_CAPSULE: canon_pair<P_CAPSULE>(P, x, y, z, v); break;
    case P_TORUS: canon_pair<P_TORUS>(P, x, y, z, v); break;
    default:
#pragma unroll
        for (int k = 0; k < 2; ++k) v[k] = canon_rare(P, x[k], y[k], z[k]);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) v[k] = fmaf(P.s, v[k], -P.off);
}

// The chain's list at the variants of a lane's point, eval_point's values.  Each element is read once;
// its variants go in pairs through one copy of the code, the accumulators rotating through registers:
// with the seven variants unrolled inside every kind the loop missed the instruction cache.
template <int NV>
__device__ __forceinline__ void eval_variants(const PrimF* __restrict__ primf, const FbInsn* __restrict__ chain,
                                              const uint32_t* list, int len, const Variants& V, float* acc) {
    constexpr int kPairs = (NV + 1) / 2;  // pair 0 the point itself (twice), pair 1 + a the offsets along axis a
    float r[2 * kPairs];
#pragma unroll
    for (int k = 0; k < 2 * kPairs; ++k) r[k] = 0.f;
    for (int i = 0; i < len; ++i) {
        const uint32_t e = list ? list[i] : (uint32_t)i << 2;
        const FbInsn I = chain[e >> 2];
        const int op = effective_op(e, I.op);
        const float kk = (float)I.k;
        if (op == CH_OFFSET) {
#pragma unroll
            for (int k = 0; k < 2 * kPairs; ++k) r[k] -= kk;
            continue;
        }
        const PrimF& P = primf[I.arg];
#pragma unroll 1
        for (int j = 0; j < kPairs; ++j) {
            float qx[2], qy[2], qz[2], v[2];
            qx[0] = j == 1 ? V.plus[0] : V.p[0];
            qy[0] = j == 2 ? V.plus[1] : V.p[1];
            qz[0] = j == 3 ? V.plus[2] : V.p[2];
            qx[1] = j == 1 ? V.minus[0] : V.p[0];
            qy[1] = j == 2 ? V.minus[1] : V.p[1];
            qz[1] = j == 3 ? V.minus[2] : V.p[2];
            eval_pair(P, qx, qy, qz, v);
            float a0 = r[0], a1 = r[1];
            if (kk == 0.f && op == CH_UNION) {
                a0 = sel_min(a0, v[0]);
                a1 = sel_min(a1, v[1]);
            } else {
                a0 = chain_apply(op, a0, v[0], kk);
                a1 = chain_apply(op, a1, v[1], kk);
            }
#pragma unroll
            for (int k = 0; k + 2 < 2 * kPairs; ++k) r[k] = r[k + 2];
            r[2 * kPairs - 2] = a0;
            r[2 * kPairs - 1] = a1;
        }
    }
    acc[0] = r[0];
#pragma unroll
    for (int k = 1; k < NV; ++k) acc[k] = r[k + 1];
}

__device__ __forceinline__ void write_point(int64_t i, const float* v, float inv, float* __restrict__ grad,
                                            float* __restrict__ value) {
    if (grad) {
#pragma unroll
        for (int a = 0; a < 3; ++a) grad[3 * i + a] = (v[1 + 2 * a] - v[2 + 2 * a]) / inv;
    }
    if (value) value[i] = v[0];
}

// A warp per point, for few points: no sorting passes.  The superblock's list is culled to the ball
// around the point's variants (a handful of elements remain), and lane v evaluates variant v.  Bound by
// the latency of the culling's loads and reductions: 1000 points of a 64^3 field in 9 us, against 55 us
// in eight kernels when all 7000 evaluations were sorted by the list that each walked.
template <int NV, bool kStretches, bool kItems = false>
__global__ void __launch_bounds__(32 * kQueryWarps) k_query_warp(const PrimF* __restrict__ primf,
                                                                 const FbInsn* __restrict__ chain, int n_chain,
                                                                 Accel A, const float* __restrict__ pts, int64_t n,
                                                                 double h, float* __restrict__ grad,
                                                                 float* __restrict__ value) {
    __shared__ Survivors s_list[kQueryWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float inv = (float)(2.0 * h);
    const int64_t nwarps = (int64_t)gridDim.x * kQueryWarps;
    for (int64_t i = blockIdx.x * (int64_t)kQueryWarps + warp; i < n; i += nwarps) {
        const Variants V = load_query<kItems>(pts, i, h);
        const Place P = place_of<NV>(A, V, 1);
        const uint32_t* list = A.pool + A.sb_off[P.s];
        int len = A.sb_len[P.s];
        const float reach = finite_reach<NV>(V);
        // else the whole chain, culled to the ball around all variants
        const bool ball = (P.inside & 1u) && !P.beyond;
        if (ball || reach >= 0.f) {
            float R = 0.f;
            if (NV > 1) {
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    if (!ball || (P.inside & (2u << (2 * a)))) R = fmaxf(R, fabsf(V.plus[a] - V.p[a]));
                    if (!ball || (P.inside & (4u << (2 * a)))) R = fmaxf(R, fabsf(V.minus[a] - V.p[a]));
                }
            }
            R *= 1.00001f;
            if (!ball) {
                list = nullptr;
                len = n_chain;
            }
            cull_to<kStretches>(list, len, chain, primf, V.p, R, ball ? 0.f : reach, A.eps, s_list[warp]);
        }
        __syncwarp();
        float r = 0.f;
        if (lane < NV) {
            const float x = V.at(lane, 0), y = V.at(lane, 1), z = V.at(lane, 2);
            if (ball ? !((P.inside >> lane) & 1u) : reach < 0.f) accel_list(A, n_chain, x, y, z, list, len);
            r = eval_list(primf, chain, list, len, x, y, z);
        }
        float v[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) v[k] = __shfl_sync(0xffffffffu, r, k);
        if (lane == 0) write_point(i, v, inv, NV > 1 ? grad : nullptr, value);
        __syncwarp();
    }
}

// A point's sorting cell and its rank among the cell's points; outside the grid the nearest cell, or (outside >= 0)
// that key for all that lie more than half a superblock's edge beyond it.
template <bool kItems>
__global__ void k_query_keys(Accel A, const float* __restrict__ pts, int64_t n, double h, int C, int outside,
                             int2* __restrict__ keys, int32_t* __restrict__ count) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const Variants V = load_query<kItems>(pts, i, h);
        int32_t key = place_of<1>(A, V, C).cell;
        if (outside >= 0) {
            const double inv = 1.0 / ((double)A.S * A.B * A.pitch);
            const double x = (V.p[0] - A.x0) * inv, y = (V.p[1] - A.y0) * inv, z = (V.p[2] - A.z0) * inv;
            if (!(x >= -0.5 && y >= -0.5 && z >= -0.5 && x <= A.nsx + 0.5 && y <= A.nsy + 0.5 && z <= A.nsz + 0.5))
                key = outside;
        }
        keys[i] = make_int2(key, atomicAdd(&count[key], 1));
    }
}

// Exclusive scan of count[0, n) in place: tiles of kScanTile per CTA, then the tile sums, then the
// tile offsets added back.
constexpr int kScanThreads = 1024, kScanItems = 4, kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ int32_t block_exclusive_scan(int32_t v, int32_t* warp_sums, int32_t& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t t = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += t;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int32_t w = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        warp_sums[lane] = w;
    }
    __syncthreads();
    total = warp_sums[(blockDim.x >> 5) - 1];
    const int32_t before = warp > 0 ? warp_sums[warp - 1] : 0;
    __syncthreads();
    return before + x - v;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(int32_t* __restrict__ data, int64_t n,
                                                             int32_t* __restrict__ tile_sums) {
    __shared__ int32_t warp_sums[32];
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    int32_t v[kScanItems], sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < n ? data[base + k] : 0;
        sum += v[k];
    }
    int32_t total;
    int32_t run = block_exclusive_scan(sum, warp_sums, total);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) data[base + k] = run;
        run += v[k];
    }
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// One CTA scans the tile sums (at most kScanTile of them) in place.
__global__ void __launch_bounds__(kScanThreads) k_scan_sums(int32_t* __restrict__ tile_sums, int ntiles) {
    __shared__ int32_t warp_sums[32];
    const int base = threadIdx.x * kScanItems;
    int32_t v[kScanItems], sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < ntiles ? tile_sums[base + k] : 0;
        sum += v[k];
    }
    int32_t total;
    int32_t run = block_exclusive_scan(sum, warp_sums, total);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < ntiles) tile_sums[base + k] = run;
        run += v[k];
    }
}

__global__ void k_scan_add(int32_t* __restrict__ data, int64_t n, const int32_t* __restrict__ tile_sums) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        data[i] += tile_sums[i / kScanTile];
}

// start[key] is the key's first sorted position.
__global__ void k_query_scatter(const int2* __restrict__ keys, int64_t n, const int32_t* __restrict__ start,
                                int32_t* __restrict__ order) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int2 k = keys[i];
        order[start[k.x] + k.y] = (int32_t)i;
    }
}

// Values alone: lists up to this are walked by the lane itself (a block's own list mostly), longer ones culled for
// the group: one evaluation a point does not repay the cull of a short list.  10^6 values with 12, 24 and 48
// here (us): 256^3 field of 576 elements 196, 179, 196 (no lane by itself 243), 300 blends 355, 298, 282 (476), 512^3
// of 3000 419, 384, 347 (405).
constexpr int kDirectList = 24;

// Centre and radius of the ball around a warp's variants: a lane's are those of `mask`.
template <int NV>
__device__ __forceinline__ float ball_of(const Variants& V, unsigned mask, float* c) {
    float d = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const unsigned fixed = mask & ~(6u << (2 * a));  // variants at the point's own coordinate a
        float lo = fixed ? V.p[a] : 3.0e38f, hi = fixed ? V.p[a] : -3.0e38f;
        if (NV > 1) {
            if (mask & (2u << (2 * a))) { lo = fminf(lo, V.plus[a]); hi = fmaxf(hi, V.plus[a]); }
            if (mask & (4u << (2 * a))) { lo = fminf(lo, V.minus[a]); hi = fmaxf(hi, V.minus[a]); }
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        c[a] = 0.5f * lo + 0.5f * hi;
        const float e = fmaxf(hi - c[a], c[a] - lo);
        d = fmaf(e, e, d);
    }
    return sqrtf(d) * 1.00001f;
}

// What the groups in the superblocks' balls leave of a warp's points (lane: item i, nearest superblock s):
// `beyond` the variants outside the grid, `left` the others; their values in vals[NV * lane + variant].
// Rare, and out of line: the groups' loop keeps its registers.
// Variants beyond the grid go by the superblock nearest to their point, the whole chain culled to the ball
// around the group.  Groups of which that keeps too much (scattered points) are put together: many points
// evaluate the whole chain side by side, few go one after another, each culled to a ball of its own as in
// k_query_warp.  The lines between them are measured costs in issue slots: about 100 for one evaluation of an
// element by the warp, 45 for one element's part in a cull (its record is gathered from L2).
// The rest are handed out to the lanes, each on its own list.
template <int NV, bool kStretches, bool kItems>
static __device__ __noinline__ void eval_rest(const PrimF* __restrict__ primf, const FbInsn* __restrict__ chain,
                                              int n_chain, const Accel& A, const float* __restrict__ pts, int64_t i,
                                              double h, int s, unsigned beyond, unsigned left, Survivors& survivors,
                                              uint8_t* items, float* vals) {
    const int lane = threadIdx.x & 31;
    const Variants V = load_query<kItems>(pts, i, h);
    const float reach = finite_reach<NV>(V);
    const int whole_cost = 100 * (NV + 1), point_cost = 45 * n_chain + 1500;
    unsigned scattered = 0u;
    for (unsigned todo = __ballot_sync(0xffffffffu, beyond != 0u); todo;) {
        const int group_s = __shfl_sync(0xffffffffu, s, __ffs(todo) - 1);
        const bool in = beyond != 0u && s == group_s;
        const unsigned group = __ballot_sync(0xffffffffu, in), mask = in ? beyond : 0u;
        todo &= ~group;
        float c[3], far = in ? reach : 0.f;
        const float R = ball_of<NV>(V, mask, c);
        for (int o = 16; o > 0; o >>= 1) far = fmaxf(far, __shfl_xor_sync(0xffffffffu, far, o));
        const uint32_t* list = nullptr;  // the whole chain
        int len = n_chain;
        cull_to<kStretches>(list, len, chain, primf, c, R, far, A.eps, survivors);
        if ((int64_t)len * whole_cost > (int64_t)__popc(group) * point_cost) {
            scattered |= group;
        } else {
            float acc[NV];
            eval_variants<NV>(primf, chain, list, len, V, acc);
#pragma unroll
            for (int k = 0; k < NV; ++k)
                if ((mask >> k) & 1u) vals[lane * NV + k] = acc[k];
        }
        __syncwarp();
    }
    if ((int64_t)n_chain * whole_cost <= (int64_t)__popc(scattered) * point_cost) {
        const unsigned mask = (scattered >> lane) & 1u ? beyond : 0u;
        if (NV == 1) {
            if (mask) vals[lane] = eval_list(primf, chain, nullptr, n_chain, V.p[0], V.p[1], V.p[2]);
        } else {
            float acc[NV];
            eval_variants<NV>(primf, chain, nullptr, n_chain, V, acc);
#pragma unroll
            for (int k = 0; k < NV; ++k)
                if ((mask >> k) & 1u) vals[lane * NV + k] = acc[k];
        }
        scattered = 0u;
    }
    __syncwarp();
    for (; scattered; scattered &= scattered - 1) {
        const int o = __ffs(scattered) - 1;
        const unsigned his = __shfl_sync(0xffffffffu, beyond, o);
        const int64_t at = __shfl_sync(0xffffffffu, i, o);
        const float far = __shfl_sync(0xffffffffu, reach, o);
        const Variants W = load_query<kItems>(pts, at, h);
        float r = 0.f;
        if (NV > 1) {
#pragma unroll
            for (int a = 0; a < 3; ++a) r = fmaxf(r, fmaxf(fabsf(W.plus[a] - W.p[a]), fabsf(W.minus[a] - W.p[a])));
        }
        const uint32_t* list = nullptr;
        int len = n_chain;
        cull_to<kStretches>(list, len, chain, primf, W.p, r * 1.00001f, far, A.eps, survivors);
        __syncwarp();
        if (lane < NV && ((his >> lane) & 1u))
            vals[o * NV + lane] = eval_list(primf, chain, list, len, W.at(lane, 0), W.at(lane, 1), W.at(lane, 2));
        __syncwarp();
    }
    int before = __popc(left);
    const int mine = before;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += y;
    }
    const int total = __shfl_sync(0xffffffffu, before, 31);
    before -= mine;
    for (unsigned b = left; b; b &= b - 1) items[before++] = (uint8_t)(lane * 8 + __ffs(b) - 1);
    __syncwarp();
    for (int t = 0; t < total; t += 32) {
        const int item = t + lane < total ? items[t + lane] : 0;
        const int own = item >> 3, v = item & 7;
        const int64_t at = __shfl_sync(0xffffffffu, i, own);
        if (t + lane < total) {
            const Variants W = load_query<kItems>(pts, at, h);
            const float x = W.at(v, 0), y = W.at(v, 1), z = W.at(v, 2);
            const uint32_t* list;
            int len;
            accel_list(A, n_chain, x, y, z, list, len);
            vals[own * NV + v] = eval_list(primf, chain, list, len, x, y, z);
        }
    }
    __syncwarp();
}

// A thread per point in sorted order.  The warp's points of one superblock form a group: its list is
// culled to the ball around the group's variants, then every lane evaluates its NV variants on what is
// left.  Variants outside the ball follow in eval_rest.
// Bound by instruction issue and the latencies of 20 warps per SM (52 % of issue slots, 30 of 32
// lanes): 10^6 points with gradients on a 256^3 field of 576 elements in 445 us, against 2680 us for
// 7 10^6 sorted evaluations on the whole superblock lists (and 1100 us for their keys and scatter, which
// go by points now: 24 us).  Groups are kept to one superblock: one group of far points in a warp, whose
// ball nothing is culled from, took 600 us by itself.
template <int NV, bool kStretches, bool kItems = false>
__global__ void __launch_bounds__(32 * kQueryWarps, 5) k_query_sorted(const PrimF* __restrict__ primf,
                                                                   const FbInsn* __restrict__ chain, int n_chain,
                                                                   const __grid_constant__ Accel A,
                                                                   const float* __restrict__ pts, int64_t n, double h,
                                                                   const int32_t* __restrict__ order,
                                                                   const int32_t* __restrict__ inside,
                                                                   float* __restrict__ grad,
                                                                   float* __restrict__ value) {
    if (inside) n = *inside;  // the rest is k_query_outside's
    __shared__ Survivors s_list[kQueryWarps];
    __shared__ uint8_t s_item[kQueryWarps][32 * NV];
    __shared__ float s_val[kQueryWarps][32 * NV];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float inv = (float)(2.0 * h);
    const int64_t nwarps = (int64_t)gridDim.x * kQueryWarps;
    for (int64_t w = blockIdx.x * (int64_t)kQueryWarps + warp; w * 32 < n; w += nwarps) {
        const bool live = w * 32 + lane < n;
        const int64_t i = live ? order[w * 32 + lane] : 0;
        const Variants V = load_query<kItems>(pts, i, h);
        const Place P = place_of<NV>(A, V, 1);
        float r[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) r[k] = 0.f;
        bool open = live;  // not evaluated yet
        if (NV == 1) {
            const uint32_t* list;
            int len;
            accel_list(A, n_chain, V.p[0], V.p[1], V.p[2], list, len);
            if (live && len <= kDirectList) {
                r[0] = eval_list(primf, chain, list, len, V.p[0], V.p[1], V.p[2]);
                open = false;
            }
            __syncwarp();
        }
        const bool ball = open && (P.inside & 1u);
        for (unsigned todo = __ballot_sync(0xffffffffu, ball); todo;) {  // groups: the variants in one superblock's ball
            const int s = __shfl_sync(0xffffffffu, P.s, __ffs(todo) - 1);
            const bool in = ball && P.s == s;
            todo &= ~__ballot_sync(0xffffffffu, in);
            // a lone variant is inside where its lane is in (written so: from `in ? P.inside : 0u` nvcc 12.9 made
            // 0 for NV = 1 with both set)
            const unsigned mask = in ? (NV == 1 ? 1u : P.inside) : 0u;
            float c[3];
            const float R = ball_of<NV>(V, mask, c);
            const uint32_t* list = A.pool + A.sb_off[s];
            int len = A.sb_len[s];
            cull_to<kStretches>(list, len, chain, primf, c, R, 0.f, A.eps, s_list[warp]);
            float acc[NV];
            eval_variants<NV>(primf, chain, list, len, V, acc);
#pragma unroll
            for (int k = 0; k < NV; ++k)
                if ((mask >> k) & 1u) r[k] = acc[k];
            __syncwarp();
        }
        const unsigned rest = open ? ~P.inside & ((1u << NV) - 1u) : 0u;
        if (__any_sync(0xffffffffu, rest != 0u)) {
            const unsigned beyond = finite_reach<NV>(V) >= 0.f ? rest & P.beyond : 0u;
            eval_rest<NV, kStretches, kItems>(primf, chain, n_chain, A, pts, i, h, P.s, beyond, rest & ~beyond, s_list[warp],
                                              s_item[warp], s_val[warp]);
#pragma unroll
            for (int k = 0; k < NV; ++k)
                if ((rest >> k) & 1u) r[k] = s_val[warp][lane * NV + k];
            __syncwarp();
        }
        if (live) write_point(i, r, inv, NV > 1 ? grad : nullptr, value);
    }
}

// The sorted points from *inside on, which lie far outside the grid, on the whole chain: a thread each.
template <bool kItems>
__global__ void __launch_bounds__(256) k_query_outside(const PrimF* __restrict__ primf, const FbInsn* __restrict__ chain,
                                                       int n_chain, const float* __restrict__ pts, int64_t n, double h,
                                                       const int32_t* __restrict__ order,
                                                       const int32_t* __restrict__ inside, float* __restrict__ value) {
    for (int64_t t = *inside + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = order[t];
        const Variants V = load_query<kItems>(pts, i, h);
        value[i] = eval_point(primf, chain, n_chain, 1, nullptr, n_chain, V.p[0], V.p[1], V.p[2]);
    }
}

// Chains longer than this (about what L1 holds of their records) are not culled for points far outside the grid
// where each is one evaluation: 100 000 of them scattered around a 512^3 field of 3000 elements 8600 us with the groups'
// and points' culls, 2200 a thread each.
constexpr int kCulledOutside = 1024;

// From the seven values of every point: the value and the gradient, k_gradient_points' arithmetic.
__global__ void k_query_combine(const float* __restrict__ vals, int64_t n, double h, float* __restrict__ grad,
                                float* __restrict__ value) {
    const float inv = (float)(2.0 * h);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        write_point(i, vals + 7 * i, inv, grad, value);
}

// Up to warp_points points go a warp per point, without scratch; more are sorted first.  Values and
// gradients, a warp per point against sorted points: 32 000 points 94 / 93 us (64^3 field of 54
// elements), 143 / 204 us (256^3, 576) and 151 / 249 us (300^3, 787); 64 000 points 179 / 84, 260 / 193
// and 265 / 240 us: the lines cross between 32 000 and 64 000.
// Values alone leave a warp 31 idle lanes, so their lines cross sooner, and the later the more superblocks
// the points are spread over (a sorted warp then culls for several of them): 64^3 field (64 superblocks)
// 46 / 52 us at 16 384 points and 66 / 50 at 24 576; 256^3 (512) 81 / 93 at 20 480 and 120 / 89 at 32 768;
// 300^3 (1000) 93 / 99 and 120 / 97 at 24 576 and 32 768; 512^3 (4096) 136 / 140 at 40 960.
constexpr int64_t kWarpPoints = 40960;

int64_t warp_points(int64_t nsuper, bool grad) {
    return grad ? kWarpPoints : std::min<int64_t>(kWarpPoints, 19000 + 6 * nsuper);
}

// Gradient queries as 7 n points of their own -- the points and their offsets sorted together, values combined
// at the end -- against a thread per point with its seven variants (us, steps of 1 and 4 voxels):
//   64^3 field of 60 elements     41 000 points  87, 103 / 118, 194    200 000  263, 310 / 151, 290
//   256^3, 576                    41 000  99, 142 / 419, 534    400 000  384, 462 / 421, 665    10^6  824, 998 / 630, 1029
//   512^3, 3000                   41 000  196, 368 / 1064, 1381    400 000  742, 1064 / 982, 1562    10^6  1599, 2177 / 1291, 2369
//   256^3, 300 blends             41 000  146, 175 / 577, 699    400 000  658, 753 / 646, 984
// Seven variants in one lane are a long chain of evaluations in few warps; with enough points the groups' culls,
// seven times as many, outweigh it, the later the more superblocks there are, the longer the step (which takes
// variants out of their point's ball) and the longer the lists (100 000 points, 16 elements: 97 / 65).  Few points go by the warp (20 480 points of the 64^3 field 64,
// 32 768 95), except for steps over a quarter of a superblock's edge.
bool by_items(int64_t nsuper, int64_t n_chain, int64_t n, double edges) {  // edges: the step in superblock edges
    if (n <= std::min<int64_t>(40960, 24000 + 4 * nsuper)) return edges > 0.25;
    const double most = 30000.0 + std::min(std::min(400.0 * nsuper, 1000.0 * n_chain), 500000.0);
    return edges >= 1.0 || (double)n <= most * (1.0 + 8.0 * edges);
}

// Chains this short are evaluated whole, a thread per point, where the points are many for them (both sides
// measured on 2 to 64 parts, 1000 to 10^6 points: 4 parts 9 us against 36 for 40 000 values, 19 against 76 with
// gradients; 12 parts 41 against 88; 8 parts 10^6 with gradients 272 against 183).
bool short_chain(int n_chain, int64_t n, int64_t warp_most, bool grad) {
    if (grad) return n <= warp_most ? n > 1700 * (int64_t)n_chain : n_chain <= 12 && n * n_chain <= 3500000;
    return n <= warp_most ? n > 650 * (int64_t)n_chain : n_chain <= 32 && n * n_chain <= 32000000;
}

// How a query on an accelerated grid runs and where its scratch lies.
struct QueryPlan {
    int64_t nsuper, n;  // n: points, or their evaluations
    bool items, sorted;
    int64_t nbins, ntiles;
    int C;  // sorting cells per superblock edge
    int64_t vals, keys, order, count, tiles, total;
};

constexpr int64_t kMaxBins = int64_t(kScanTile) * kScanTile;  // one tile-sum CTA covers them (one for points outside)
constexpr int64_t kMaxSortedPoints = int64_t(1) << 31;        // sorted positions are int32

// edges: the step in superblock edges; negative where it is not known.  n_chain: kAnyChain for the most scratch.
constexpr int64_t kAnyChain = int64_t(1) << 31;

QueryPlan query_plan(const int32_t* dims, int64_t n_chain, int64_t n, bool grad, double edges) {
    QueryPlan p{};
    const int B = dims[3];
    const int64_t nbx = (dims[0] + B - 1) / B, nby = (dims[1] + B - 1) / B, nbz = (dims[2] + B - 1) / B;
    const int64_t S = std::max(1, fb_super_edge(dims[0], dims[1], dims[2]) / B);
    p.nsuper = ((nbx + S - 1) / S) * ((nby + S - 1) / S) * ((nbz + S - 1) / S);
    p.items = grad && edges >= 0.0 && n < kMaxSortedPoints / 7 && by_items(p.nsuper, n_chain, n, edges);
    p.n = p.items ? 7 * n : n;
    for (p.C = 4; p.C > 1 && p.nsuper * p.C * p.C * p.C >= kMaxBins; p.C /= 2) {
    }
    p.nbins = p.nsuper * p.C * p.C * p.C;
    p.ntiles = (p.nbins + 1 + kScanTile - 1) / kScanTile;
    p.sorted = p.nsuper >= 1 && p.nbins < kMaxBins && p.n < kMaxSortedPoints &&
               p.n > warp_points(p.nsuper, grad && !p.items);
    auto al = [](int64_t b) { return (b + 255) / 256 * 256; };
    int64_t at = 0;
    p.vals = at; at += p.items ? al(p.n * 4) : 0;
    if (p.sorted) {
        p.keys = at; at += al(p.n * 8);
        p.order = at; at += al(p.n * 4);
        p.count = at; at += al((p.nbins + 1) * 4);
        p.tiles = at; at += al(p.ntiles * 4);
    }
    p.total = at;
    return p;
}

double step_edges(const double* grid, const int32_t* dims, double h) {
    const int S = std::max(1, fb_super_edge(dims[0], dims[1], dims[2]) / dims[3]);
    return std::fabs(h) / (S * dims[3] * grid[3]);
}

// ------------------------------------------------------------------------------------ multires
struct Multi {
    double lx, ly, lz;   // world origin of the brick lattice
    double h;            // coarse pitch
    int B, bx, by, bz;   // brick edge in coarse voxels, brick grid
    double margin;       // +-margin answers outside active bricks (float64, as the reference)
};

// Samples of brick b at level l: (B*2^l + 1)^3 float32 at pitch h/2^l from the brick origin.
// Warp per active brick.  The brick's culled list (its classification block's, whose culling
// region is the brick's closed box) is localised to the brick origin once in shared memory, the
// lattice is evaluated in block-local float32, and values inside the guard band are recomputed in
// float64 -- the leaf kernel's scheme.
constexpr int kTileWarps = 4, kTileCap = 48;

__global__ void __launch_bounds__(32 * kTileWarps) k_multires_tiles(
    const PrimF* __restrict__ primf, const FbInsn* __restrict__ chain, int n_chain, int chain_mode,
    const FbPrim* __restrict__ prims, Multi M, const int32_t* __restrict__ bricks, const int8_t* __restrict__ levels,
    const int64_t* __restrict__ offsets, int64_t nbricks, const int32_t* __restrict__ blk_off,
    const int32_t* __restrict__ blk_len, const uint32_t* __restrict__ blk_pool, float guard, float* __restrict__ pool) {
    __shared__ LocalPrim s_prim[kTileWarps][kTileCap];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t gwarp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    LocalPrim* sp = s_prim[warp];
    for (int64_t k = gwarp; k < nbricks; k += nwarps) {
        const int64_t b = bricks[k];
        const int l = levels[k];
        const int bk = (int)(b % M.bz), bj = (int)((b / M.bz) % M.by), bi = (int)(b / ((int64_t)M.bz * M.by));
        const int m = (M.B << l) + 1;
        const double pitch = M.h / (double)(1 << l);
        const float fpitch = (float)pitch;
        // every float64 operation rounded once, as NumPy does (no contraction)
        const double ox = rn_add(M.lx, rn_mul((double)(bi * M.B), M.h)), oy = rn_add(M.ly, rn_mul((double)(bj * M.B), M.h)),
                     oz = rn_add(M.lz, rn_mul((double)(bk * M.B), M.h));
        const bool listed = blk_len && blk_len[b] >= 0;
        const uint32_t* list = listed ? blk_pool + blk_off[b] : nullptr;
        const int len = listed ? blk_len[b] : n_chain;
        const bool staged = chain_mode && listed && len <= kTileCap;
        if (staged) {
            for (int i = lane; i < len; i += 32) {
                const uint32_t e = list[i];
                const FbInsn I = chain[e >> 2];
                const uint32_t mode = e & 3u;
                const int op = mode == 1u ? CH_SET : (mode == 2u ? CH_SETNEG : I.op);
                if (op == CH_OFFSET) {
                    sp[i].op = op;
                    sp[i].k = (float)I.k;
                } else {
                    localise(prims[I.arg], primf[I.arg], ox, oy, oz, op, (float)I.k, sp[i]);
                }
            }
        }
        __syncwarp();
        float* out = pool + offsets[k];
        const int64_t total = (int64_t)m * m * m;
        for (int64_t v = lane; v < total; v += 32) {
            const int iz = (int)(v % m), iy = (int)((v / m) % m), ix = (int)(v / ((int64_t)m * m));
            const double x = rn_add(ox, rn_mul((double)ix, pitch)), y = rn_add(oy, rn_mul((double)iy, pitch)),
                         z = rn_add(oz, rn_mul((double)iz, pitch));
            float val;
            if (!chain_mode) {
                val = (float)program_eval_d(prims, chain, n_chain, x, y, z);
            } else {
                if (staged) {
                    const float dx = ix * fpitch, dy = iy * fpitch, dz = iz * fpitch;
                    float acc = 0.f;
                    for (int i = 0; i < len; ++i) {
                        const LocalPrim& P = sp[i];
                        acc = P.op == CH_OFFSET ? acc - P.k : chain_apply(P.op, acc, local_eval(P, dx, dy, dz), P.k);
                    }
                    val = acc;
                } else {
                    val = eval_point(primf, chain, n_chain, 1, list, len, (float)x, (float)y, (float)z);
                }
                if (!(fabsf(val) >= guard) || !staged) {  // float64 inside the guard band (and when unstaged)
                    double acc = 0.0;
                    for (int i = 0; i < len; ++i) {
                        const uint32_t e = list ? list[i] : (uint32_t)i << 2;
                        const FbInsn I = chain[e >> 2];
                        const uint32_t mode = e & 3u;
                        const int op = mode == 1u ? CH_SET : (mode == 2u ? CH_SETNEG : I.op);
                        const double pv = op == CH_OFFSET ? 0.0 : prim_world_d(prims[I.arg], x, y, z);
                        acc = chain_apply_d(op, acc, pv, I.k);
                    }
                    val = (float)acc;
                }
            }
            out[v] = val;
        }
        __syncwarp();
    }
}

// Brick of a world point, preferring an active brick when the point lies exactly on a face
// (faltkarna_v1_multires.py:384-402).  Returns false when the point is outside the lattice.
__device__ bool brick_of(const Multi& M, const int8_t* __restrict__ kind, double px, double py, double pz, int b[3]) {
    const double L = rn_mul((double)M.B, M.h);
    const double rel[3] = {rn_div(rn_sub(px, M.lx), L), rn_div(rn_sub(py, M.ly), L), rn_div(rn_sub(pz, M.lz), L)};
    const int shp[3] = {M.bx, M.by, M.bz};
    bool outside = false;
    for (int a = 0; a < 3; ++a) {
        const double f = floor(rel[a]);
        long long v = (long long)f;
        outside |= v < 0 || v >= shp[a];
        b[a] = (int)min(max(v, 0ll), (long long)shp[a] - 1);
    }
    auto kind_at = [&](int x, int y, int z) { return kind[((int64_t)x * M.by + y) * M.bz + z]; };
    bool inactive = kind_at(b[0], b[1], b[2]) != 0;
    for (int a = 0; a < 3; ++a) {
        const bool on_plane = rel[a] == floor(rel[a]) && b[a] > 0 && inactive && !outside;
        if (!on_plane) continue;
        int c[3] = {b[0], b[1], b[2]};
        c[a] -= 1;
        if (kind_at(c[0], c[1], c[2]) == 0) b[a] -= 1;
        inactive = kind_at(b[0], b[1], b[2]) != 0;
    }
    return !outside;
}

// scipy.ndimage.map_coordinates(tile, coords, order=1, mode='nearest') at one point of a cubic
// (m x m x m) float32 tile: each coordinate clamped into [0, m-1], weights (1-t, t) per axis,
// sum over the eight corners in C order of value x w0 x w1 x w2 in float64.
__device__ double tile_trilinear(const float* __restrict__ t, int m, double cx, double cy, double cz) {
    const double c[3] = {fmin(fmax(cx, 0.0), (double)(m - 1)), fmin(fmax(cy, 0.0), (double)(m - 1)),
                         fmin(fmax(cz, 0.0), (double)(m - 1))};
    int s[3];
    double f[3];
    for (int a = 0; a < 3; ++a) {
        const double fl = floor(c[a]);
        s[a] = (int)fl;
        f[a] = __dsub_rn(c[a], fl);
    }
    double acc = 0.0;
    for (int h = 0; h < 8; ++h) {
        const int a = (h >> 2) & 1, b = (h >> 1) & 1, d = h & 1;
        const int X = min(s[0] + a, m - 1), Y = min(s[1] + b, m - 1), Z = min(s[2] + d, m - 1);
        double coeff = (double)t[((int64_t)X * m + Y) * m + Z];
        coeff = __dmul_rn(coeff, a ? f[0] : __dsub_rn(1.0, f[0]));
        coeff = __dmul_rn(coeff, b ? f[1] : __dsub_rn(1.0, f[1]));
        coeff = __dmul_rn(coeff, d ? f[2] : __dsub_rn(1.0, f[2]));
        acc = __dadd_rn(acc, coeff);
    }
    return acc;
}

__device__ double multires_value(const Multi& M, const int8_t* __restrict__ kind, const int8_t* __restrict__ level,
                                 const int64_t* __restrict__ tile_off, const float* __restrict__ pool, double px,
                                 double py, double pz) {
    int b[3];
    const bool inside = brick_of(M, kind, px, py, pz, b);
    const int64_t lin = ((int64_t)b[0] * M.by + b[1]) * M.bz + b[2];
    const int kd = kind[lin];
    if (!inside) return M.margin;
    if (kd != 0) return kd < 0 ? -M.margin : M.margin;
    const int l = level[lin];
    const double pitch = rn_div(M.h, (double)(1 << l));
    const double L = rn_mul((double)M.B, M.h);
    const double ox = rn_add(M.lx, rn_mul((double)b[0], L)), oy = rn_add(M.ly, rn_mul((double)b[1], L)),
                 oz = rn_add(M.lz, rn_mul((double)b[2], L));
    const int m = (M.B << l) + 1;
    // map_coordinates returns the tile's dtype: one float32 rounding
    return (double)__double2float_rn(
        tile_trilinear(pool + tile_off[lin], m, rn_div(rn_sub(px, ox), pitch), rn_div(rn_sub(py, oy), pitch),
                       rn_div(rn_sub(pz, oz), pitch)));
}

__global__ void k_multires_value(Multi M, const int8_t* __restrict__ kind, const int8_t* __restrict__ level,
                                 const int64_t* __restrict__ tile_off, const float* __restrict__ pool,
                                 const double* __restrict__ pts, int64_t n, double* __restrict__ out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = multires_value(M, kind, level, tile_off, pool, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]);
}

// Central difference at the point's brick pitch, both probes clamped into the brick
// (faltkarna_v1_multires.py:437-459).
__global__ void k_multires_gradient(Multi M, const int8_t* __restrict__ kind, const int8_t* __restrict__ level,
                                    const int64_t* __restrict__ tile_off, const float* __restrict__ pool,
                                    const double* __restrict__ pts, int64_t n, double* __restrict__ out) {
    const double L = rn_mul((double)M.B, M.h);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double p[3] = {pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]};
        int b[3];
        brick_of(M, kind, p[0], p[1], p[2], b);
        const int lv = level[((int64_t)b[0] * M.by + b[1]) * M.bz + b[2]];
        const double h = rn_div(M.h, (double)(1 << max(lv, 0)));
        const double o[3] = {rn_add(M.lx, rn_mul((double)b[0], L)), rn_add(M.ly, rn_mul((double)b[1], L)),
                             rn_add(M.lz, rn_mul((double)b[2], L))};
        for (int a = 0; a < 3; ++a) {
            double pa[3] = {p[0], p[1], p[2]}, pb[3] = {p[0], p[1], p[2]};
            pa[a] = fmin(rn_add(p[a], rn_mul(0.5, h)), rn_add(o[a], L));
            pb[a] = fmax(rn_sub(p[a], rn_mul(0.5, h)), o[a]);
            for (int c = 0; c < 3; ++c)
                if (c != a) {
                    pa[c] = fmin(p[c], rn_add(o[c], L));
                    pb[c] = fmax(p[c], o[c]);
                }
            const double step = rn_sub(pa[a], pb[a]);
            const double va = multires_value(M, kind, level, tile_off, pool, pa[0], pa[1], pa[2]);
            const double vb = multires_value(M, kind, level, tile_off, pool, pb[0], pb[1], pb[2]);
            out[3 * i + a] = rn_div(rn_sub(va, vb), fmax(step, 1e-12));
        }
    }
}

// Overlap band (faltkarna_v1_multires.py:211-251): every face of a fine brick whose neighbour is an
// active brick of a coarser level takes the trilinear sample of the neighbour's lattice at the face's
// own sample points.  One CTA per brick of the launch's level, its six faces in the reference's order
// (axis 0..2, side -1 then +1; a later face overwrites the edges it shares with an earlier one).  The
// reference walks the bricks in ascending id and overwrites lattices in place, so a neighbour of level
// >= 1 is read as overwritten when its id is smaller than this brick's and as built otherwise: the
// host launches level 1, 2, 3 in turn and passes `orig`, a copy of the pool taken before the band.
__global__ void __launch_bounds__(256) k_multires_band(Multi M, const int8_t* __restrict__ kind,
                                                       const int8_t* __restrict__ level,
                                                       const int64_t* __restrict__ tile_off, float* __restrict__ pool,
                                                       const float* __restrict__ orig,
                                                       const int32_t* __restrict__ bricks, int n_bricks, int lvl,
                                                       int* __restrict__ faces) {
    const int idx = blockIdx.x;
    if (idx >= n_bricks) return;
    const int lin = bricks[idx];
    const int b[3] = {lin / (M.by * M.bz), (lin / M.bz) % M.by, lin % M.bz};
    const double L = rn_mul((double)M.B, M.h);
    const double lo[3] = {M.lx, M.ly, M.lz};
    const int shp[3] = {M.bx, M.by, M.bz};
    const int n_l = M.B << lvl, m = n_l + 1;
    const double h_f = rn_div(M.h, (double)(1 << lvl));
    double bo[3];
    for (int a = 0; a < 3; ++a) bo[a] = rn_add(lo[a], rn_mul((double)b[a], L));
    float* tile = pool + tile_off[lin];
    for (int ax = 0; ax < 3; ++ax) {
        for (int sida = -1; sida <= 1; sida += 2) {
            int nb[3] = {b[0], b[1], b[2]};
            nb[ax] += sida;
            if (nb[ax] < 0 || nb[ax] >= shp[ax]) continue;
            const int64_t nlin = ((int64_t)nb[0] * M.by + nb[1]) * M.bz + nb[2];
            if (kind[nlin] != 0) continue;
            const int lvl_n = level[nlin];
            if (lvl_n < 0 || lvl_n >= lvl) continue;
            const float* src = (lvl_n >= 1 && nlin < lin ? pool : orig) + tile_off[nlin];
            const int m_n = (M.B << lvl_n) + 1;
            const double h_n = rn_div(M.h, (double)(1 << lvl_n));
            double no[3];
            for (int a = 0; a < 3; ++a) no[a] = rn_add(lo[a], rn_mul((double)nb[a], L));
            const int u = ax == 0 ? 1 : 0, w = ax == 2 ? 1 : 2;  // the face's free axes, ascending
            const int fixed = sida < 0 ? 0 : n_l;
            for (int k = threadIdx.x; k < m * m; k += blockDim.x) {
                int g[3];
                g[ax] = fixed;
                g[u] = k / m;
                g[w] = k % m;
                double c[3];
                for (int a = 0; a < 3; ++a) {
                    const double pt = rn_add(rn_mul((double)g[a], h_f), bo[a]);
                    c[a] = rn_div(rn_sub(pt, no[a]), h_n);
                }
                tile[((int64_t)g[0] * m + g[1]) * m + g[2]] = (float)tile_trilinear(src, m_n, c[0], c[1], c[2]);
            }
            if (threadIdx.x == 0) atomicAdd(faces, 1);
            __syncthreads();
        }
    }
}

Multi make_multi(const double* lo, double h, int B, const int32_t* bshape, double margin) {
    Multi M;
    M.lx = lo[0];
    M.ly = lo[1];
    M.lz = lo[2];
    M.h = h;
    M.B = B;
    M.bx = bshape[0];
    M.by = bshape[1];
    M.bz = bshape[2];
    M.margin = margin;
    return M;
}

// Many (leaf A, leaf B) gridfield pairs in one launch (src/field_engine/ikarus_v1/eval_warp.py:521-564):
// thread per point, pair = pair_of_point[i], value max(sample(A), sample(B)) with the gridfield
// sampler.  params: 12 floats per leaf (the gridfield record layout: origin, pitch, iso, is_sdf, nx,
// ny, nz, -, table address halves).  An index outside its table reads NaN.
__global__ void k_grid_pairs(const float* __restrict__ params, int n_leaves, const float* __restrict__ pts,
                             const int32_t* __restrict__ pair, int64_t n, const int32_t* __restrict__ la,
                             const int32_t* __restrict__ lb, int n_pairs, float* __restrict__ out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int pid = pair[i];
        float v = __int_as_float(0x7fc00000);
        if (pid >= 0 && pid < n_pairs) {
            const int a = la[pid], b = lb[pid];
            if (a >= 0 && a < n_leaves && b >= 0 && b < n_leaves) {
                const float x = pts[3 * i], y = pts[3 * i + 1], z = pts[3 * i + 2];
                v = fmaxf(grid_sample_f(params + 12 * a, x, y, z), grid_sample_f(params + 12 * b, x, y, z));
            }
        }
        out[i] = v;
    }
}

}  // namespace

extern "C" {

// Overlap band of a per-block-pitch field (k_multires_band): d_orig is caller scratch the size of
// the pool (its state before the band); d_bricks lists the active bricks of level >= 1 sorted by
// level (n_of_level[l] of level l = 1..3 after n_of_level[0] = 0); d_faces (one int) counts the faces
// written.  Stream-ordered.
int fb_multires_band_device(const double* lo, double h, int32_t B, const int32_t* bshape, const int8_t* d_kind,
                            const int8_t* d_level, const int64_t* d_tile_off, float* d_pool, int64_t pool_len,
                            float* d_orig, const int32_t* d_bricks, const int32_t* n_of_level, int32_t* d_faces,
                            void* stream) noexcept {
    if (!lo || !bshape || !d_kind || !d_level || !d_tile_off || !d_pool || !d_orig || !n_of_level || !d_faces ||
        B < 1 || !(h > 0) || pool_len < 0)
        return FB_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const Multi M = make_multi(lo, h, B, bshape, 0.0);
    FB_CUDA(cudaMemsetAsync(d_faces, 0, sizeof(int32_t), st));
    FB_CUDA(cudaMemcpyAsync(d_orig, d_pool, pool_len * 4, cudaMemcpyDeviceToDevice, st));
    int at = 0;
    for (int l = 1; l <= 3; ++l) {
        const int n = n_of_level[l];
        if (n < 0) return FB_INVALID;
        if (n > 0) {
            if (!d_bricks) return FB_INVALID;
            k_multires_band<<<n, 256, 0, st>>>(M, d_kind, d_level, d_tile_off, d_pool, d_orig, d_bricks + at, n, l,
                                               d_faces);
            FB_LAUNCH();
        }
        at += n;
    }
    return FB_OK;
}

// The multi-pair gridfield sweep (k_grid_pairs); all pointers on the device, stream-ordered.
int fb_grid_pairs_device(const float* d_params, int32_t n_leaves, const float* d_pts, const int32_t* d_pair,
                         int64_t n, const int32_t* d_leaf_a, const int32_t* d_leaf_b, int32_t n_pairs, float* d_out,
                         void* stream) noexcept {
    if (n < 0 || n_leaves < 1 || n_pairs < 1 || !d_params ||
        (n > 0 && (!d_pts || !d_pair || !d_leaf_a || !d_leaf_b || !d_out)))
        return FB_INVALID;
    if (n == 0) return FB_OK;
    k_grid_pairs<<<(int)std::min<int64_t>((n + 255) / 256, (int64_t)fb_sm_count() * 16), 256, 0,
                   static_cast<cudaStream_t>(stream)>>>(d_params, n_leaves, d_pts, d_pair, n, d_leaf_a, d_leaf_b,
                                                        n_pairs, d_out);
    FB_LAUNCH();
    return FB_OK;
}


// Values (and gradients) of a compiled recipe at float32 points, device pointers.  d_primf is the
// float32 primitive mirror a field build prepared (fb_query_prepare fills one).  accel_* (all
// nullable) are a built field's superblock lists and grid; without them every point walks the
// whole chain / program.
int fb_query_prepare(const FbPrim* d_prims, int32_t n_prims, void* d_primf, void* stream) noexcept;

// Scratch bytes of a query of n points (with_grad: gradients, a thread or a warp per point whatever the step)
// on an accelerated grid of dims (nx, ny, nz, B); 0 where it takes a path without scratch, -1 for
// invalid arguments.
int64_t fb_query_scratch_bytes(const int32_t* accel_dims, int64_t n, int32_t with_grad) noexcept {
    if (!accel_dims || accel_dims[3] < 1 || n < 0) return -1;
    return query_plan(accel_dims, kAnyChain, n, with_grad != 0, -1.0).total;
}

// The same for gradients of step h on a grid of x0, y0, z0, pitch (accel_grid).
int64_t fb_query_scratch_bytes_h(const double* accel_grid, const int32_t* accel_dims, int64_t n, int32_t with_grad,
                                 double h) noexcept {
    if (!accel_grid || !accel_dims || accel_dims[3] < 1 || n < 0) return -1;
    return query_plan(accel_dims, kAnyChain, n, with_grad != 0, step_edges(accel_grid, accel_dims, h)).total;
}

int fb_query_points_device(const void* d_primf, const FbInsn* d_chain, int32_t n_chain, int32_t mode,
                           const void* accel_pool, const int64_t* accel_off, const int32_t* accel_len,
                           const double* accel_grid /* x0,y0,z0,pitch */, const int32_t* accel_dims /* nx,ny,nz,B */,
                           const int32_t* d_kind, const int32_t* blk_off, const int32_t* blk_len,
                           const uint32_t* blk_pool, int64_t blk_cap, int32_t blk_all, const float* d_points, int64_t n,
                           double h, float* d_value, float* d_grad, void* d_scratch, int64_t scratch_len,
                           void* stream) noexcept {
    if (!d_primf || !d_chain || n_chain < 1 || !d_points || n < 0 || (!d_value && !d_grad)) return FB_INVALID;
    if (n == 0) return FB_OK;
    Accel A{};
    if (accel_pool && accel_off && accel_len && accel_grid && accel_dims && (mode == 1 || mode == 3) && accel_dims[3] >= 1) {
        A.pool = static_cast<const uint32_t*>(accel_pool);
        A.sb_off = accel_off;
        A.sb_len = accel_len;
        A.x0 = accel_grid[0]; A.y0 = accel_grid[1]; A.z0 = accel_grid[2]; A.pitch = accel_grid[3];
        A.nx = accel_dims[0]; A.ny = accel_dims[1]; A.nz = accel_dims[2]; A.B = accel_dims[3];
        A.nbx = (A.nx + A.B - 1) / A.B; A.nby = (A.ny + A.B - 1) / A.B; A.nbz = (A.nz + A.B - 1) / A.B;
        A.S = std::max(1, fb_super_edge(A.nx, A.ny, A.nz) / A.B);
        A.nsx = (A.nbx + A.S - 1) / A.S;
        A.nsy = (A.nby + A.S - 1) / A.S;
        A.nsz = (A.nbz + A.S - 1) / A.S;
        if (blk_off && blk_len && blk_pool && blk_cap > 0 && (blk_all || d_kind)) {
            A.kind = d_kind;
            A.blk_off = blk_off;
            A.blk_len = blk_len;
            A.blk_pool = blk_pool;
            A.blk_cap = blk_cap;
            A.blk_all = blk_all ? 1 : 0;
        }
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const PrimF* primf = static_cast<const PrimF*>(d_primf);
    QueryPlan P{};
    bool whole = !A.pool;
    if (A.pool) {
        P = query_plan(accel_dims, n_chain, n, d_grad != nullptr, step_edges(accel_grid, accel_dims, h));
        // scratch that was sized without the step, or none: its points in place of their evaluations
        if (P.items && (!d_scratch || scratch_len < P.total)) P = query_plan(accel_dims, n_chain, n, true, -1.0);
        whole = short_chain(n_chain, n, warp_points(P.nsuper, d_grad != nullptr), d_grad != nullptr);
    }
    if (!whole) {
        // 16 float32 ulps of the largest coordinate a superblock's ball reaches: the default guard's slack
        float far = 0.f;
        const double reach = (A.S * A.B + 1) * A.pitch;
        const double lo[3] = {A.x0, A.y0, A.z0};
        const int ext[3] = {A.nbx * A.B, A.nby * A.B, A.nbz * A.B};
        for (int a = 0; a < 3; ++a)
            far = std::max(far, (float)std::max(std::fabs(lo[a] - reach), std::fabs(lo[a] + ext[a] * A.pitch + reach)));
        A.eps = 16.f * (std::nextafter(far, 3.4e38f) - far);
        const bool sorted = P.sorted && d_scratch;
        if (sorted && scratch_len < P.total) return FB_INVALID;
        char* b = static_cast<char*>(d_scratch);
        float* out = P.items ? reinterpret_cast<float*>(b + P.vals) : d_value;
        int32_t* order = nullptr;
        const int32_t* inside = nullptr;
        if (sorted) {
            int2* keys = reinterpret_cast<int2*>(b + P.keys);
            order = reinterpret_cast<int32_t*>(b + P.order);
            int32_t* count = reinterpret_cast<int32_t*>(b + P.count);
            int32_t* tiles = reinterpret_cast<int32_t*>(b + P.tiles);
            const int ge = (int)std::min<int64_t>((P.n + 255) / 256, (int64_t)fb_sm_count() * 16);
            const bool apart = n_chain > kCulledOutside && (P.items || !d_grad);
            if (apart) inside = count + P.nbins;
            const int outside = apart ? (int)P.nbins : -1;
            FB_CUDA(cudaMemsetAsync(count, 0, (P.nbins + 1) * 4, st));
            if (P.items) k_query_keys<true><<<ge, 256, 0, st>>>(A, d_points, P.n, h, P.C, outside, keys, count);
            else k_query_keys<false><<<ge, 256, 0, st>>>(A, d_points, P.n, 0.0, P.C, outside, keys, count);
            FB_LAUNCH();
            k_scan_tiles<<<(unsigned)P.ntiles, kScanThreads, 0, st>>>(count, P.nbins + 1, tiles);
            FB_LAUNCH();
            k_scan_sums<<<1, kScanThreads, 0, st>>>(tiles, (int)P.ntiles);
            FB_LAUNCH();
            k_scan_add<<<(int)std::min<int64_t>((P.nbins + 256) / 256, (int64_t)fb_sm_count() * 16), 256, 0, st>>>(
                count, P.nbins + 1, tiles);
            FB_LAUNCH();
            k_query_scatter<<<ge, 256, 0, st>>>(keys, P.n, count, order);
            FB_LAUNCH();
        }
        const int per = sorted ? 32 * kQueryWarps : kQueryWarps;  // points a CTA takes at a time
        const int gs = (int)std::min<int64_t>((P.n + per - 1) / per, (int64_t)fb_sm_count() * 64);
        auto run = [&](auto nv, auto stretches, auto items) {
            constexpr int NV = decltype(nv)::value;
            constexpr bool kS = decltype(stretches)::value, kI = decltype(items)::value;
            const double step = NV > 1 || kI ? h : 0.0;
            float* grad = NV > 1 ? d_grad : nullptr;
            if (sorted)
                k_query_sorted<NV, kS, kI><<<gs, 32 * kQueryWarps, 0, st>>>(primf, d_chain, n_chain, A, d_points, P.n, step,
                                                                            order, inside, grad, out);
            else
                k_query_warp<NV, kS, kI><<<gs, 32 * kQueryWarps, 0, st>>>(primf, d_chain, n_chain, A, d_points, P.n, step,
                                                                          grad, out);
        };
        const std::integral_constant<int, 1> one;
        const std::integral_constant<int, 7> seven;
        const std::true_type yes;
        const std::false_type no;
        if (P.items) {
            if (mode == 3) run(one, yes, yes);
            else run(one, no, yes);
        } else if (d_grad) {
            if (mode == 3) run(seven, yes, no);
            else run(seven, no, no);
        } else {
            if (mode == 3) run(one, yes, no);
            else run(one, no, no);
        }
        FB_LAUNCH();
        if (inside) {
            const int go = (int)std::min<int64_t>((P.n + 255) / 256, (int64_t)fb_sm_count() * 16);
            if (P.items)
                k_query_outside<true><<<go, 256, 0, st>>>(primf, d_chain, n_chain, d_points, P.n, h, order, inside, out);
            else
                k_query_outside<false><<<go, 256, 0, st>>>(primf, d_chain, n_chain, d_points, P.n, 0.0, order, inside, out);
            FB_LAUNCH();
        }
        if (P.items) {
            k_query_combine<<<(int)std::min<int64_t>((n + 255) / 256, (int64_t)fb_sm_count() * 16), 256, 0, st>>>(
                out, n, h, d_grad, d_value);
            FB_LAUNCH();
        }
        return FB_OK;
    }
    const int grid = (int)std::min<int64_t>((n + 127) / 128, (int64_t)fb_sm_count() * 16);
    if (d_grad) {
        k_gradient_points<<<grid, 128, 0, st>>>(primf, d_chain, n_chain, mode, d_points, n, h, d_grad, d_value);
    } else {
        k_eval_points<<<grid, 128, 0, st>>>(primf, d_chain, n_chain, mode, d_points, n, d_value);
    }
    return cudaGetLastError() == cudaSuccess ? FB_OK : FB_RUNTIME;
}

// Fill the (B*2^l+1)^3 lattices of the listed active bricks (device pointers).  levels[k] in 0..3,
// offsets[k] = start of brick k's lattice in d_pool.  blk_* (nullable) are the per-block culled
// lists of a classification of the same recipe on the brick grid.
int fb_multires_tiles_device(const void* d_primf, const FbInsn* d_chain, int32_t n_chain, int32_t mode,
                             const FbPrim* d_prims, const double* lo, double h, int32_t B, const int32_t* bshape,
                             const int32_t* d_bricks, const int8_t* d_levels, const int64_t* d_offsets,
                             int64_t nbricks, const int32_t* d_blk_off, const int32_t* d_blk_len,
                             const uint32_t* d_blk_pool, float guard, float* d_pool, void* stream) noexcept {
    if (!d_primf || !d_chain || !d_prims || !lo || !bshape || !d_pool || nbricks < 0 || B < 1 || !(h > 0))
        return FB_INVALID;
    if (nbricks == 0) return FB_OK;
    const Multi M = make_multi(lo, h, B, bshape, 0.0);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    k_multires_tiles<<<fb_sm_count() * 8, 32 * kTileWarps, 0, st>>>(static_cast<const PrimF*>(d_primf), d_chain, n_chain, mode,
                                                       d_prims, M, d_bricks, d_levels, d_offsets, nbricks, d_blk_off,
                                                       d_blk_len, d_blk_pool, guard, d_pool);
    return cudaGetLastError() == cudaSuccess ? FB_OK : FB_RUNTIME;
}

// avstand / gradient of a per-block-pitch field at float64 points (device pointers); d_grad
// (nullable) gets (n, 3) when requested, d_value (nullable) the values.
int fb_multires_query_device(const double* lo, double h, int32_t B, const int32_t* bshape, double margin,
                             const int8_t* d_kind, const int8_t* d_level, const int64_t* d_tile_off,
                             const float* d_pool, const double* d_points, int64_t n, double* d_value,
                             double* d_grad, void* stream) noexcept {
    if (!lo || !bshape || !d_kind || !d_level || !d_tile_off || !d_pool || !d_points || n < 0 || B < 1 || !(h > 0))
        return FB_INVALID;
    if (n == 0) return FB_OK;
    const Multi M = make_multi(lo, h, B, bshape, margin);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int grid = (int)std::min<int64_t>((n + 127) / 128, (int64_t)fb_sm_count() * 16);
    if (d_value) k_multires_value<<<grid, 128, 0, st>>>(M, d_kind, d_level, d_tile_off, d_pool, d_points, n, d_value);
    if (d_grad) k_multires_gradient<<<grid, 128, 0, st>>>(M, d_kind, d_level, d_tile_off, d_pool, d_points, n, d_grad);
    return cudaGetLastError() == cudaSuccess ? FB_OK : FB_RUNTIME;
}

}  // extern "C"
