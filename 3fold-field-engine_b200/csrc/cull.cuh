// Exact culling of a CSG chain for a region: interval bounds of its elements and the warp-cooperative
// walk that keeps only the elements that can influence the region (shared by the field build and the
// point queries; each source includes its own copy).
#pragma once
#include "prims.cuh"

namespace {

// One interval step of the chain walk.  Returns 0 skip, 1 keep, 2 reset to "set", 3 reset to
// "set negated".  [alo, ahi] bounds the accumulator over the region.
__device__ __forceinline__ int interval_step(int op, float k, float plo, float phi, float& alo, float& ahi) {
    switch (op) {
    case CH_SET:
        alo = plo; ahi = phi;
        return 2;
    case CH_SETNEG:
        alo = -phi; ahi = -plo;
        return 3;
    case CH_UNION:
        if (plo > ahi + k) return 0;
        if (phi < alo - k) { alo = plo; ahi = phi; return 2; }
        alo = fminf(alo, plo) - 0.25f * k;
        ahi = fminf(ahi, phi);
        return 1;
    case CH_INTERSECT:
        if (phi < alo - k) return 0;
        if (plo > ahi + k) { alo = plo; ahi = phi; return 2; }
        alo = fmaxf(alo, plo);
        ahi = fmaxf(ahi, phi) + 0.25f * k;
        return 1;
    case CH_SUBTRACT:
        if (-plo < alo - k) return 0;
        if (-phi > ahi + k) { alo = -phi; ahi = -plo; return 3; }
        alo = fmaxf(alo, -phi);
        ahi = fmaxf(ahi, -plo) + 0.25f * k;
        return 1;
    default:  // offset
        alo -= k; ahi -= k;
        return 1;
    }
}

__device__ __forceinline__ int effective_op(uint32_t entry, int op) {
    const uint32_t mode = entry & 3u;
    return mode == 1u ? CH_SET : (mode == 2u ? CH_SETNEG : op);
}

// primf_world with the rarely used kinds out of line: the culling walks have several copies of it, and
// with every kind inlined in each they missed the instruction cache.
static __device__ __noinline__ float canon_out_of_line(const PrimF& P, float x, float y, float z) {
    return canon_f(P.type, P.p, x, y, z);
}

__device__ __forceinline__ float primf_world_common(const PrimF& P, float x, float y, float z) {
    const float lx = fmaf(P.A[0], x, fmaf(P.A[1], y, fmaf(P.A[2], z, P.A[3])));
    const float ly = fmaf(P.A[4], x, fmaf(P.A[5], y, fmaf(P.A[6], z, P.A[7])));
    const float lz = fmaf(P.A[8], x, fmaf(P.A[9], y, fmaf(P.A[10], z, P.A[11])));
    float c;
    switch (P.type) {
    case P_SPHERE: c = canon_f(P_SPHERE, P.p, lx, ly, lz); break;
    case P_BOX: c = canon_f(P_BOX, P.p, lx, ly, lz); break;
    case P_CAPSULE: c = canon_f(P_CAPSULE, P.p, lx, ly, lz); break;
    case P_TORUS: c = canon_f(P_TORUS, P.p, lx, ly, lz); break;
    default: c = canon_out_of_line(P, lx, ly, lz);
    }
    return fmaf(P.s, c, -P.off);
}

// A region's radius for element_interval, widened so that the bound also covers the float32 rounding that
// comes with the coordinates (32 u |A| |x|_1 of PrimF.err's rule; |A|_1 is at most sqrt(3) of the norm in
// `lip`).  What comes with a primitive's own frame is PrimF.err: a sphere of radius 300 through a unit
// grid rounds by 4e-5 there, twenty times the grid's own 16 ulps.
__device__ __forceinline__ float bounds_radius(float cx, float cy, float cz, float R) {
    return fmaf(3.4e-6f, fabsf(cx) + fabsf(cy) + fabsf(cz) + 2.f * R, R);
}

// Interval of one chain element's primitive around (cx, cy, cz) with radius R (bounds_radius): holds every
// value of it there, exact or computed in float32.
__device__ __forceinline__ void element_interval(const PrimF& P, float cx, float cy, float cz, float R, float eps,
                                                 float& lo, float& hi) {
    const float v = primf_world_common(P, cx, cy, cz);
    const float r = fmaf(P.lip, R, eps + P.err + 1e-6f * fabsf(v));
    lo = v - r;
    hi = v + r;
}

// A hard (k == 0) union / intersection / subtraction: consecutive ones of the same kind form a
// run whose result is an order-free min or max of the accumulator and the run's elements.
__device__ __forceinline__ bool runnable(int op, float k) {
    return k == 0.f && (op == CH_UNION || op == CH_INTERSECT || op == CH_SUBTRACT);
}

struct Elem {
    uint32_t ent;
    int op;
    float k;
    float lo, hi;  // bounds of the value the combine sees (-p for a subtraction)
};

// A primitive's bounding ball by itself (PrimF.ball, ball_k, off, p[8..11]): what the coarse level reads
// of every element.  32 consecutive bytes: gathered from the 128-byte records, 32 lanes' loads took 32
// cache lines each and the records of 4096 elements did not stay in L1.
struct __align__(16) Ball {
    float x, y, z, r;
    float k, off, has, err;  // value scale and offset; has != 0: the ball holds; PrimF.err
};

// The enclosure from the bounding ball: no evaluation of the primitive, a few loads -- looser by up to
// the ball's diameter.
__device__ __forceinline__ void element_interval_ball(const Ball& P, float cx, float cy, float cz, float R, float eps,
                                                      float& lo, float& hi) {
    const float dx = cx - P.x, dy = cy - P.y, dz = cz - P.z;
    const float d = sqrt_rn(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
    const float m = eps + P.err + 1e-6f * (P.k * (d + R + P.r) + fabsf(P.off));
    lo = fmaf(P.k, d - R - P.r, -P.off) - m;
    hi = fmaf(P.k, d + R + P.r, -P.off) + m;
}

__device__ __forceinline__ Elem load_elem(const uint32_t* __restrict__ in, int e, const FbInsn* __restrict__ chain,
                                          const PrimF* __restrict__ primf, float cx, float cy, float cz, float R,
                                          float eps, bool with_bounds, const Ball* __restrict__ balls = nullptr) {
    Elem E;
    E.ent = in ? in[e] : (uint32_t)e << 2;  // a null list is the whole chain in order
    const FbInsn I = chain[E.ent >> 2];
    E.op = effective_op(E.ent, I.op);
    E.k = E.op == CH_OFFSET ? (float)I.k : fmaxf((float)I.k, 0.f);  // a negative blend width is a hard boolean
    E.lo = E.hi = 0.f;
    if (with_bounds && E.op != CH_OFFSET) {
        float lo, hi;
        Ball b;
        b.has = 0.f;
        if (balls) b = balls[I.arg];
        if (b.has != 0.f) element_interval_ball(b, cx, cy, cz, R, eps, lo, hi);
        else element_interval(primf[I.arg], cx, cy, cz, R, eps, lo, hi);
        if (E.op == CH_SUBTRACT || E.op == CH_SETNEG) { E.lo = -hi; E.hi = -lo; }
        else { E.lo = lo; E.hi = hi; }
    }
    return E;
}

// Run decision.  union: result = min(acc, run); an element whose lower bound exceeds
// H = min(acc_hi, min run hi) is never the minimum and is dropped; when min run hi < acc_lo the
// accumulator so far is dominated everywhere and dropped (the run restarts the list).
// intersection / subtraction: the mirror image with max.  All comparisons are strict, so every
// decision is exact for the float values the bounds enclose.
struct RunState {
    float bound;   // H (union) or L (max kinds)
    bool reset;
};

__device__ __forceinline__ RunState run_decide(int op, float agg, float alo, float ahi) {
    RunState r;
    if (op == CH_UNION) {
        r.reset = agg < alo;
        r.bound = r.reset ? agg : fminf(ahi, agg);
    } else {
        r.reset = agg > ahi;
        r.bound = r.reset ? agg : fmaxf(alo, agg);
    }
    return r;
}

__device__ __forceinline__ bool run_keep(int op, const Elem& E, float bound) {
    return op == CH_UNION ? !(E.lo > bound) : !(E.hi < bound);
}

// One element that is no part of a run: interval_step on its primitive's own bounds.
__device__ __forceinline__ int single_step(const Elem& E, float& alo, float& ahi) {
    const bool neg = E.op == CH_SUBTRACT || E.op == CH_SETNEG;
    return interval_step(E.op, E.k, neg ? -E.hi : E.lo, neg ? -E.lo : E.hi, alo, ahi);
}

// The accumulator's bounds after a run whose kept elements have bounds [klo, khi] (a warp's lanes each
// hold their part).
__device__ __forceinline__ void end_run(int op, const RunState& rs, float klo, float khi, float& alo, float& ahi) {
    for (int o = 16; o > 0; o >>= 1) {
        klo = fminf(klo, __shfl_xor_sync(0xffffffffu, klo, o));
        khi = fmaxf(khi, __shfl_xor_sync(0xffffffffu, khi, o));
    }
    if (op == CH_UNION) {
        alo = rs.reset ? klo : fminf(alo, klo);
        ahi = rs.bound;
    } else {
        alo = rs.bound;
        ahi = rs.reset ? khi : fmaxf(ahi, khi);
    }
}

// Warp-cooperative chain walk over `in` for the region centred at (cx, cy, cz) with radius R.
// Hard runs are decided with two warp-parallel passes (aggregate bound, then keep/drop with
// ballot compaction); other elements (offsets, smooth booleans, sets) step one at a time.
// Returns the kept count (may exceed cap: then the output is incomplete and must not be used).
__device__ int warp_walk(const uint32_t* __restrict__ in, int n_in, const FbInsn* __restrict__ chain,
                         const PrimF* __restrict__ primf, float cx, float cy, float cz, float R, float eps,
                         uint32_t* __restrict__ out, int cap) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    R = bounds_radius(cx, cy, cz, R);
    float alo = 0.f, ahi = 0.f;
    int n = 0;
    int i = 0;
    while (i < n_in) {
        const Elem head = load_elem(in, i, chain, primf, cx, cy, cz, R, eps, false);
        if (!runnable(head.op, head.k)) {
            const Elem E = load_elem(in, i, chain, primf, cx, cy, cz, R, eps, true);
            const int act = single_step(E, alo, ahi);
            if (act) {
                uint32_t rec = E.ent;
                if (act == 2) { n = 0; rec = (E.ent & ~3u) | 1u; }
                if (act == 3) { n = 0; rec = (E.ent & ~3u) | 2u; }
                if (n < cap && lane == 0) out[n] = rec;
                ++n;
            }
            ++i;
            continue;
        }
        const int op = head.op;
        // pass 1, 32 elements at a time: the run's end (the first element of another kind) and the
        // aggregate bound of the elements before it
        float agg = op == CH_UNION ? 3.0e38f : -3.0e38f;
        int j = n_in;
        for (int b = i; b < n_in; b += 32) {
            const int e = b + lane;
            bool same = false;
            Elem E;
            if (e < n_in) {
                E = load_elem(in, e, chain, primf, cx, cy, cz, R, eps, true);
                same = e == i || (E.op == op && runnable(E.op, E.k));
            }
            const unsigned stop = __ballot_sync(0xffffffffu, e < n_in && !same);
            const int end = stop ? b + __ffs(stop) - 1 : min(b + 32, n_in);
            if (e < end) agg = op == CH_UNION ? fminf(agg, E.hi) : fmaxf(agg, E.lo);
            if (stop) {
                j = end;
                break;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const float t = __shfl_xor_sync(0xffffffffu, agg, o);
            agg = op == CH_UNION ? fminf(agg, t) : fmaxf(agg, t);
        }
        const RunState rs = run_decide(op, agg, alo, ahi);
        float klo = 3.0e38f, khi = -3.0e38f;
        if (rs.reset) n = 0;
        bool first = rs.reset;
        // pass 2: keep / drop, ballot compaction in chain order
        for (int b = i; b < j; b += 32) {
            const int e = b + lane;
            bool keep = false;
            Elem E;
            if (e < j) {
                E = load_elem(in, e, chain, primf, cx, cy, cz, R, eps, true);
                keep = run_keep(op, E, rs.bound);
                if (keep) { klo = fminf(klo, E.lo); khi = fmaxf(khi, E.hi); }
            }
            const unsigned kept = __ballot_sync(0xffffffffu, keep);
            if (keep) {
                const int pos = n + __popc(kept & below);
                uint32_t rec = E.ent;
                if (first && pos == 0) rec = (E.ent & ~3u) | (op == CH_SUBTRACT ? 2u : 1u);
                if (pos < cap) out[pos] = rec;
            }
            if (kept) first = false;
            n += __popc(kept);
        }
        end_run(op, rs, klo, khi, alo, ahi);
        i = j;
    }
    return n;
}

// The same walk of the whole chain (the coarse level, where every region walks it), bounding
// primitives by their bounding balls where they have one.  Pass 1 of a run also writes its candidates:
// elements not beaten by the bound so far, a superset of those the final bound keeps (every other
// element provably loses, so the run's result is the candidates' result); the exact bounds of the
// candidates alone give the run's decision, and they are compacted in place with it.  Few warps walk
// here (a region each), so a warp keeps the loads of kBallChunks chunks in flight.  4096 regions of 4096
// elements: 541 -> 318 us with the balls in a table of their own.  Returns the kept count, or cap + 1 where
// the list does not fit.
constexpr int kBallChunks = 4;

__device__ int warp_walk_ball(int n_in, const FbInsn* __restrict__ chain, const PrimF* __restrict__ primf,
                              const Ball* __restrict__ balls, float cx, float cy, float cz, float R, float eps,
                              uint32_t* __restrict__ out, int cap, float* klo_of, float* khi_of, int n_of) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    R = bounds_radius(cx, cy, cz, R);
    float alo = 0.f, ahi = 0.f;
    int n = 0;
    int i = 0;
    while (i < n_in) {
        const Elem head = load_elem(nullptr, i, chain, primf, cx, cy, cz, R, eps, false);
        if (!runnable(head.op, head.k)) {
            const Elem E = load_elem(nullptr, i, chain, primf, cx, cy, cz, R, eps, true);
            const int act = single_step(E, alo, ahi);
            if (act) {
                uint32_t rec = E.ent;
                if (act == 2) { n = 0; rec = (E.ent & ~3u) | 1u; }
                if (act == 3) { n = 0; rec = (E.ent & ~3u) | 2u; }
                if (n < cap && lane == 0) out[n] = rec;
                ++n;
            }
            ++i;
            continue;
        }
        const int op = head.op;
        float agg = op == CH_UNION ? 3.0e38f : -3.0e38f;
        int j = n_in;
        const int n0 = n;
        for (int b = i, chunks = 1; b < n_in; b += 32 * chunks, chunks = kBallChunks) {  // a short run loads one
            Elem E[kBallChunks];
#pragma unroll
            for (int c = 0; c < kBallChunks; ++c) {
                const int e = b + 32 * c + lane;
                E[c].op = -1;
                E[c].k = E[c].lo = E[c].hi = 0.f;
                E[c].ent = 0u;
                if (c < chunks && e < n_in) E[c] = load_elem(nullptr, e, chain, primf, cx, cy, cz, R, eps, true, balls);
            }
            int end = min(b + 32 * chunks, n_in);
            bool stopped = false;
#pragma unroll
            for (int c = 0; c < kBallChunks; ++c) {
                const int e = b + 32 * c + lane;
                const bool same = e == i || (E[c].op == op && runnable(E[c].op, E[c].k));
                const unsigned stop = __ballot_sync(0xffffffffu, c < chunks && e < n_in && !same);
                if (stop && !stopped) {
                    stopped = true;
                    end = b + 32 * c + __ffs(stop) - 1;
                }
            }
            float run = agg;
#pragma unroll
            for (int c = 0; c < kBallChunks; ++c)
                if (b + 32 * c + lane < end) run = op == CH_UNION ? fminf(run, E[c].hi) : fmaxf(run, E[c].lo);
            for (int o = 16; o > 0; o >>= 1) {
                const float t = __shfl_xor_sync(0xffffffffu, run, o);
                run = op == CH_UNION ? fminf(run, t) : fmaxf(run, t);
            }
            agg = run;
#pragma unroll
            for (int c = 0; c < kBallChunks; ++c) {
                const bool keep = b + 32 * c + lane < end && run_keep(op, E[c], run);
                const unsigned kept = __ballot_sync(0xffffffffu, keep);
                if (keep) {
                    const int pos = n + __popc(kept & below);
                    if (pos < cap) out[pos] = E[c].ent;
                }
                n += __popc(kept);
            }
            if (stopped) {
                j = end;
                break;
            }
        }
        const int nc = n - n0;  // candidates at out[n0, n)
        // overflowed: the bounds after this run are not known, so nothing later may be decided by them
        if (n > cap) return cap + 1;
        __syncwarp();  // the candidates are read by other lanes
        float agg2 = op == CH_UNION ? 3.0e38f : -3.0e38f;
        for (int b = 0; b < nc; b += 32) {
            if (b + lane < nc) {
                const Elem E = load_elem(out + n0, b + lane, chain, primf, cx, cy, cz, R, eps, true);
                if (b + lane < n_of) {  // kept for the decisions below (a lane reads what it wrote)
                    klo_of[b + lane] = E.lo;
                    khi_of[b + lane] = E.hi;
                }
                agg2 = op == CH_UNION ? fminf(agg2, E.hi) : fmaxf(agg2, E.lo);
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const float t = __shfl_xor_sync(0xffffffffu, agg2, o);
            agg2 = op == CH_UNION ? fminf(agg2, t) : fmaxf(agg2, t);
        }
        const RunState rs = run_decide(op, agg2, alo, ahi);
        float klo = 3.0e38f, khi = -3.0e38f;
        n = rs.reset ? 0 : n0;  // compaction target: positions never above the ones being read
        bool first = rs.reset;
        for (int b = 0; b < nc; b += 32) {
            bool keep = false;
            Elem E;
            if (b + lane < nc) {
                if (b + lane < n_of) {
                    E.ent = out[n0 + b + lane];
                    E.lo = klo_of[b + lane];
                    E.hi = khi_of[b + lane];
                } else {
                    E = load_elem(out + n0, b + lane, chain, primf, cx, cy, cz, R, eps, true);
                }
                keep = run_keep(op, E, rs.bound);
                if (keep) { klo = fminf(klo, E.lo); khi = fmaxf(khi, E.hi); }
            }
            const unsigned kept = __ballot_sync(0xffffffffu, keep);  // every read precedes the writes
            if (keep) {
                const int pos = n + __popc(kept & below);
                uint32_t rec = E.ent;
                if (first && pos == 0) rec = (E.ent & ~3u) | (op == CH_SUBTRACT ? 2u : 1u);
                out[pos] = rec;
            }
            if (kept) first = false;
            n += __popc(kept);
            __syncwarp();
        }
        end_run(op, rs, klo, khi, alo, ahi);
        i = j;
    }
    return n;
}

// x -> min(max(x + c, a), b) with a <= b: what a boolean does to a bound of the accumulator.  Closed under
// composition, so the bounds before each element of a stretch come from one scan over the warp.
struct Clamp {
    float c, a, b;
    __device__ __forceinline__ float operator()(float x) const { return fminf(fmaxf(x + c, a), b); }
};

// g applied to f's result.
__device__ __forceinline__ Clamp then(const Clamp& f, const Clamp& g) { return Clamp{f.c + g.c, g(f.a), g(f.b)}; }

__device__ __forceinline__ Clamp shfl_up(const Clamp& f, int o) {
    return Clamp{__shfl_up_sync(0xffffffffu, f.c, o), __shfl_up_sync(0xffffffffu, f.a, o),
                 __shfl_up_sync(0xffffffffu, f.b, o)};
}

// Booleans that form no run of kRunLeast go by the stretch from kStretch of them on: one at a time a step is a
// chain of shuffles and comparisons of about 40 instructions, a stretch of up to 32 takes about 250.
constexpr int kRunLeast = 9, kStretch = 5;

struct Walk {  // accumulator's bounds, kept entries, elements taken (0: no stretch here)
    float alo, ahi;
    int n, taken;
};

// The warp's elements E from `pos` on in one stretch, up to where a run of kRunLeast starts, or one that
// reaches the end of a full 32, or an offset or set: every element decides by interval_step on the bounds
// before it.
__device__ __forceinline__ Walk walk_stretch(uint32_t entry, int op, float width, float elo, float ehi, int cnt,
                                                 int pos, float alo, float ahi, int n, uint32_t* ent, int cap) {
    const int lane = threadIdx.x & 31;
    const bool hard = runnable(op, width);
    const int next = __shfl_down_sync(0xffffffffu, hard ? op : -1, 1);
    const unsigned pairs = __ballot_sync(0xffffffffu, lane < 31 && hard && next == op);
    const unsigned hards = __ballot_sync(0xffffffffu, hard);
    unsigned stops = pairs & pairs >> 1;
    stops &= stops >> 2;
    stops &= stops >> 4;
    static_assert(kRunLeast == 9, "eight pairs in a row");
    if (cnt == 32 && hards >> 31) stops |= 1u << (31 - __clz(~(pairs << 1)));
    stops |= __ballot_sync(0xffffffffu, lane >= cnt || op == CH_OFFSET || op == CH_SET || op == CH_SETNEG);
    stops >>= pos;
    const int length = stops ? __ffs(stops) - 1 : 32 - pos;
    if (length < kStretch) return Walk{alo, ahi, n, 0};
    const bool mine = lane >= pos && lane < pos + length;
    const float q = 0.2500025f * width;  // the blend's deepest, a little widened for the sums' rounding
    constexpr float kInf = 3.0e38f;
    Clamp lo{0.f, -kInf, kInf}, hi{0.f, -kInf, kInf};
    if (mine && op == CH_UNION) {
        lo = Clamp{-q, -kInf, elo - q};
        hi.b = ehi;
    } else if (mine) {
        lo.a = elo;
        hi = Clamp{q, ehi + q, kInf};
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const Clamp a = shfl_up(lo, o), b = shfl_up(hi, o);
        if (lane >= o) {
            lo = then(a, lo);
            hi = then(b, hi);
        }
    }
    const Clamp lo_before = shfl_up(lo, 1), hi_before = shfl_up(hi, 1);
    float l = lane > pos ? lo_before(alo) : alo, h = lane > pos ? hi_before(ahi) : ahi;
    int act = 0;
    const bool neg = op == CH_SUBTRACT;  // back to the primitive's own bounds
    if (mine) act = interval_step(op, width, neg ? -ehi : elo, neg ? -elo : ehi, l, h);
    unsigned kept = __ballot_sync(0xffffffffu, act != 0);
    const unsigned resets = __ballot_sync(0xffffffffu, act >= 2);
    if (resets) {  // what lies before the last reset is dominated
        n = 0;
        kept &= ~0u << (31 - __clz(resets));
    }
    if (n + __popc(kept) <= cap && ((kept >> lane) & 1u))
        ent[n + __popc(kept & ((1u << lane) - 1u))] = act >= 2 ? (entry & ~3u) | (unsigned)(act - 1) : entry;
    __syncwarp();
    return Walk{__shfl_sync(0xffffffffu, lo(alo), pos + length - 1), __shfl_sync(0xffffffffu, hi(ahi), pos + length - 1),
                n + __popc(kept), length};
}

// The same walk with every element bounded once, for lists that fit shared memory: candidates of a run
// (elements not beaten by the bound so far) are kept with their bounds in `ent`, `blo`, `bhi` (shared,
// `cap` each) and compacted in place when the run ends and its bound is final.  One copy of the code:
// inlined at each call it missed the instruction cache.  kStretches: also by the stretch, for chains that
// are no few long runs (in the usual chains' walk it cost 10^6 queries on a 256^3 field 3 %, through the
// registers that a caller spills around it).  Returns the kept count, or cap + 1 where the
// candidates did not fit; every lane of the warp calls it, and the list is readable after it.
template <bool kStretches>
static __device__ __noinline__ int warp_walk_once(const uint32_t* in, int n_in, const FbInsn* __restrict__ chain,
                                                  const PrimF* __restrict__ primf, float cx, float cy, float cz,
                                                  float R, float eps, uint32_t* ent, float* blo, float* bhi, int cap) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    R = bounds_radius(cx, cy, cz, R);
    float alo = 0.f, ahi = 0.f, agg = 0.f;
    int n = 0, n0 = 0, run = -1;  // entries; where the open run's start; its operation (-1: none)
    auto finish = [&]() {
        const RunState rs = run_decide(run, agg, alo, ahi);
        const int end = n;
        float klo = 3.0e38f, khi = -3.0e38f;
        bool first = rs.reset;
        n = rs.reset ? 0 : n0;
        __syncwarp();
        for (int b = n0; b < end; b += 32) {
            bool keep = false;
            Elem E;
            if (b + lane < end) {
                E.ent = ent[b + lane];
                E.lo = blo[b + lane];
                E.hi = bhi[b + lane];
                keep = run_keep(run, E, rs.bound);
                if (keep) { klo = fminf(klo, E.lo); khi = fmaxf(khi, E.hi); }
            }
            const unsigned kept = __ballot_sync(0xffffffffu, keep);  // every read precedes the writes
            if (keep) {
                const int pos = n + __popc(kept & below);
                ent[pos] = first && pos == 0 ? (E.ent & ~3u) | (run == CH_SUBTRACT ? 2u : 1u) : E.ent;
                blo[pos] = E.lo;
                bhi[pos] = E.hi;
            }
            if (kept) first = false;
            n += __popc(kept);
            __syncwarp();
        }
        end_run(run, rs, klo, khi, alo, ahi);
        run = -1;
    };
    for (int b = 0; b < n_in; b += 32) {
        const int cnt = min(32, n_in - b);
        Elem E;
        E.ent = 0u;
        E.op = CH_OFFSET;
        E.k = E.lo = E.hi = 0.f;
        if (lane < cnt) E = load_elem(in, b + lane, chain, primf, cx, cy, cz, R, eps, true);
        const bool hard = runnable(E.op, E.k);
        int pos = 0;
        while (pos < cnt) {
            const int op = __shfl_sync(0xffffffffu, E.op, pos);
            const bool same = hard && E.op == op && lane >= pos && lane < cnt;
            const unsigned run_mask = __ballot_sync(0xffffffffu, same);
            if (run >= 0 && (run != op || !((run_mask >> pos) & 1u))) finish();
            const unsigned gap = ~(run_mask >> pos);
            const int end = gap ? min(pos + __ffs(gap) - 1, cnt) : cnt;  // of the run here, if any
            if (kStretches && run < 0 && end - pos < kRunLeast && cnt - pos >= kStretch && op >= CH_UNION &&
                op <= CH_SUBTRACT) {
                const Walk w = walk_stretch(E.ent, E.op, E.k, E.lo, E.hi, cnt, pos, alo, ahi, n, ent, cap);
                if (w.n > cap) return cap + 1;
                if (w.taken) {
                    alo = w.alo;
                    ahi = w.ahi;
                    n = w.n;
                    pos += w.taken;
                    continue;
                }
            }
            if (!((run_mask >> pos) & 1u)) {  // offsets, sets, smooth booleans: one at a time
                const float lo = __shfl_sync(0xffffffffu, E.lo, pos), hi = __shfl_sync(0xffffffffu, E.hi, pos);
                const float k = __shfl_sync(0xffffffffu, E.k, pos);
                const bool neg = op == CH_SUBTRACT || op == CH_SETNEG;  // back to the primitive's own bounds
                const int act = interval_step(op, k, neg ? -hi : lo, neg ? -lo : hi, alo, ahi);
                if (act) {
                    if (act >= 2) n = 0;
                    if (n >= cap) return cap + 1;
                    if (lane == pos) ent[n] = act >= 2 ? (E.ent & ~3u) | (unsigned)(act - 1) : E.ent;
                    ++n;
                    __syncwarp();
                }
                ++pos;
                continue;
            }
            if (run < 0) {
                run = op;
                n0 = n;
                agg = op == CH_UNION ? 3.0e38f : -3.0e38f;
            }
            const bool mine = lane >= pos && lane < end;
            float a = mine ? (op == CH_UNION ? E.hi : E.lo) : agg;
            for (int o = 16; o > 0; o >>= 1) {
                const float t = __shfl_xor_sync(0xffffffffu, a, o);
                a = op == CH_UNION ? fminf(a, t) : fmaxf(a, t);
            }
            agg = op == CH_UNION ? fminf(agg, a) : fmaxf(agg, a);
            const bool keep = mine && run_keep(op, E, agg);
            const unsigned kept = __ballot_sync(0xffffffffu, keep);
            if (n + __popc(kept) > cap) return cap + 1;
            if (keep) {
                const int at = n + __popc(kept & below);
                ent[at] = E.ent;
                blo[at] = E.lo;
                bhi[at] = E.hi;
            }
            n += __popc(kept);
            pos = end;
        }
    }
    if (run >= 0) finish();
    __syncwarp();
    return n;
}

}  // namespace
