// Exact integer squared Euclidean distance transform and the paired signed distance, sm_100a.
//
// Algorithm (a from-scratch design, not the reference's one-thread-per-line envelope):
//   1. k_edt_bits  : the uint8 mask becomes one 32-bit word per 32 z-samples of every (x, y) line
//                    (1 B read + 1/8 B written per voxel, four bytes per SWAR step); the validating
//                    form also checks the mask (values 0/1, both classes present) with
//                    warp-aggregated counters.
//   2. k_edt_zy    : one CTA per (32-wide z chunk, x plane, polarity).  A lane per y line fills the
//                    chunk's squared z distances from the line's bit words into shared memory; then,
//                    lanes = z columns, the y pass g(y,z) = min_y' dz(y',z)^2 + (y-y')^2 as an exact
//                    minimum over groups of rows, most of them ruled out by a bound (below).  Writes
//                    float32 g (integers below 2^22; 4 B/voxel); a plane without a site is filled.
//   3. k_edt_x     : one CTA per (z chunk, y row, polarity): stages the nx x 32 column block of g in
//                    shared memory with cp.async (every load in flight at once), runs the same pass
//                    along x and writes the final int32 (4 B/voxel); the paired form runs both
//                    polarities, then k_edt_signed turns the two squared distances into the correctly
//                    rounded signed float32.
// Global traffic per voxel and polarity: 1 (mask) + 4 + 4 (g round trip) + 4 (output) + 1/4 (bit
// words, mostly L2) bytes -- the 13 B/voxel algorithmic figure.
//
// Exactness: every pass computes the exact min-plus of its input, so the result equals the
// reference's separable definition bit for bit (sentinel sum((n-1)^2)+1 where no site reaches,
// src/field_engine/field_edt_integer_v1.py:14-26, edt_native_large_v1/edt.cu:33-61).
#include "common.cuh"
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <type_traits>
#include <new>

namespace {

constexpr int kMaxAxis = 512;  // the reference's bound; 512 rows of a column block fit three CTAs per SM

struct Counters {
    unsigned long long ones;     // mask bytes equal to 1
    unsigned long long invalid;  // mask bytes greater than 1
};

// Nonzero flags of the four bytes of q as bits 0..3 (byte i -> bit i).  The byte-wise OR folds
// every bit of a byte onto its bit 0; the multiply then gathers the four bit-0s: byte i's bit lands
// at bit 24 + i of the product and no partial products overlap, so nothing carries.
__device__ __forceinline__ uint32_t nonzero4(uint32_t q) {
    uint32_t t = q | (q >> 4);
    t |= t >> 2;
    t |= t >> 1;
    t &= 0x01010101u;
    return (t * 0x01020408u) >> 24;
}

// kCount: also count the mask bytes equal to 1 and flag bytes greater than 1.
template <bool kCount>
__global__ void __launch_bounds__(256) k_edt_bits(const uint8_t* __restrict__ mask, uint32_t* __restrict__ bits,
                                                  int64_t lines, int nz, int W, Counters* counters) {
    unsigned long long ones = 0;
    uint32_t bad = 0;
    const int64_t total = lines * W;
    const bool vec = (nz & 15) == 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t line = i / W;
        const int w = (int)(i - line * W);
        const int z0 = 32 * w;
        const int n = min(32, nz - z0);
        const uint8_t* src = mask + line * nz + z0;
        uint32_t word = 0;
        if (vec) {
            // 16-byte aligned: line*nz and z0 are multiples of 16; n is 16 or 32.
            for (int h = 0; h < n; h += 16) {
                const uint4 v = *reinterpret_cast<const uint4*>(src + h);
                const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    word |= nonzero4(q[j]) << (h + 4 * j);
                    if (kCount) {
                        ones += __popc(q[j] & 0x01010101u);
                        bad |= q[j] & 0xfefefefeu;
                    }
                }
            }
        } else {
            for (int b = 0; b < n; ++b) {
                const uint32_t byte = src[b];
                word |= (uint32_t)(byte != 0) << b;
                if (kCount) {
                    ones += byte & 1u;
                    bad |= byte & 0xfeu;
                }
            }
        }
        bits[i] = word;
    }
    if (kCount) {
        // a byte > 1 makes the mask invalid whatever `ones` says, so `ones` may count its low bit
        unsigned long long invalid = bad != 0;
        for (int o = 16; o > 0; o >>= 1) {
            ones += __shfl_xor_sync(0xffffffffu, ones, o);
            invalid += __shfl_xor_sync(0xffffffffu, invalid, o);
        }
        if ((threadIdx.x & 31) == 0) {
            if (ones) atomicAdd(&counters->ones, ones);
            if (invalid) atomicAdd(&counters->invalid, invalid);
        }
    }
}

void launch_bits(int grid, cudaStream_t stream, const uint8_t* mask, uint32_t* bits, int64_t lines, int nz, int W,
                 Counters* counters) {
    if (counters) k_edt_bits<true><<<grid, 256, 0, stream>>>(mask, bits, lines, nz, W, counters);
    else k_edt_bits<false><<<grid, 256, 0, stream>>>(mask, bits, lines, nz, W, nullptr);
}

// ------------------------------------------------------------------------------------------
// Exact 1-D min-plus along a column, out(q) = min_s f(s) + (q - s)^2, by pruned groups.
//
// A CTA owns 32 adjacent columns (lanes) over the whole axis, staged in shared memory as float32 rows
// (every value is an integer below 2^22, so float32 holds it and every sum below exactly).  Rows are
// taken kGroup at a time: `mins` keeps each group's smallest f per column and `low` over all columns,
// and a warp works out kGroup consecutive outputs (a strip) of its 32 columns at once.  A group at
// distance d (nearest row to nearest output) can lower an output of a column only where the column's
// min f + d^2 lies below the largest of its outputs so far, so every other group is passed over and the
// result is the full minimum.  The strip's own group comes first, the nearest kNear on each side next
// (one test per column and a vote each); of the rest, lanes take a group each and test it with `low`
// against the largest output of all columns, the lowest bound is evaluated first, and what remains
// below the new largest output follows -- a site hundreds of rows away costs a few groups, not all
// those in between.
//
// Inside a group, output k and site i (both counted in their group, D = first output - first site) meet
// at f + (D - i)^2 + 2 k (D - i) + k^2: per two sites one packed square and one FMA per output (FFMA2 on
// the pair of sites), whose two results and the running value go through one three-operand minimum.
// k^2 is added at the end.  76 instructions for 64 pairs; pairing the outputs instead of the sites,
// which needs every site's terms twice, issued about 175.
//
// Sites without a finite value carry the sentinel, which a finite value always beats and which stays
// the result where the whole column has none.
//
// Bound: instruction issue (70 % of the issue slots; the FMA and ALU pipes half busy each, DRAM a
// fifth).  A lower envelope built as a hull per column (one push, its pops and one walk step per voxel,
// band hulls joined pairwise) took 107 (x) and 149 (zy) warp instructions per 32 voxels of the 512^3
// obstacle grid (2000 boxes, 8 % filled), its loops diverging over the lanes; here it is 74 and 92, and
// the work depends on the data only through votes: x 638 -> 395 us, zy 851 -> 559 us, the transform
// 1515 -> 986 us (30 % random voxels 1640 -> 773, one box or ball far from most voxels 14 - 18 % less).
// The hulls remain faster where a smooth surface lies hundreds of voxels away from most of the grid along
// its diagonal (half-spaces of 512^3: x + y + z < 350 986 against 1273 us, < 700 1138 / 1414, z < 100
// 1058 / 1123; a shell of radius 240 1472 / 1560).
// ------------------------------------------------------------------------------------------
constexpr int kWarps = 8;
constexpr int kThreads = 32 * kWarps;
constexpr int kGroup = 8;              // rows per group, outputs per strip
constexpr int kNear = 2;               // groups on each side of a strip that are tested one by one
constexpr int kMaxGroups = kMaxAxis / kGroup;  // 64: two per lane
constexpr float kPadValue = 8.0e6f;    // rows past the axis and groups taken: above every bound
constexpr float kFar = 2048.f;         // z distance on a side of a row without a site
constexpr float kIntBias = 8388608.f;  // 2^23: adding it puts a non-negative integer into the mantissa bits

__host__ __device__ __forceinline__ int groups_of(int n) { return (n + kGroup - 1) / kGroup; }

// Shared memory of a pass over an axis of length n with rows of `ld` words: the rows, padded to whole
// groups, then the groups' minima per column and over all columns.
int pass_smem_bytes(int n, int ld) { return (groups_of(n) * (kGroup * ld + 32) + 2 * kNear * 32 + kMaxGroups) * 4; }

__device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// Extremes over the warp of non-negative floats (their bits order as unsigned integers).
__device__ __forceinline__ float warp_max(float v) {
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
}
__device__ __forceinline__ float warp_min(float v) {
    return __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(v)));
}

// A strip's outputs of one column: a[k] is output k less k^2.
struct Strip {
    float a[kGroup];

    __device__ __forceinline__ float value(int k) const { return a[k] + (float)(k * k); }
    __device__ __forceinline__ int integer(int k) const {  // value(k), exact: its bits above 2^23
        return __float_as_int(a[k] + (kIntBias + (float)(k * k))) - 0x4b000000;
    }
    // the sites of one group: col points at its first row's value of this column, e = (D, D - 1),
    // back2 = (-2, -2); output k + 1's terms are output k's plus 2 (D - i), so no constants are held
    template <int LD, bool kFirst = false>
    __device__ __forceinline__ void group(const float* __restrict__ col, float2 e, float2 back2) {
#pragma unroll
        for (int i = 0; i < kGroup; i += 2) {
            const float2 step = __fadd2_rn(e, e);
            float2 c = __ffma2_rn(e, e, make_float2(col[i * LD], col[(i + 1) * LD]));
#pragma unroll
            for (int k = 0; k < kGroup; ++k) {
                a[k] = kFirst && i == 0 ? fminf(c.x, c.y) : min3(a[k], c.x, c.y);
                if (k + 1 < kGroup) c = __fadd2_rn(c, step);
            }
            e = __fadd2_rn(e, back2);
        }
    }
    // Largest value of the strip (past the axis's end its outputs count too: a last strip may then look
    // at a group more than it needs).
    __device__ __forceinline__ float largest() const {
        return max3(max3(value(0), value(1), value(2)), max3(value(3), value(4), value(5)), fmaxf(value(6), value(7)));
    }
};

// Minima of a warp's own groups [g0, g1).
template <int LD>
__device__ __forceinline__ void group_minima(const float* __restrict__ rows, float* __restrict__ mins,
                                             float* __restrict__ low, int g0, int g1) {
    const int lane = threadIdx.x & 31;
    for (int g = g0; g < g1; ++g) {
        const float* col = rows + g * kGroup * LD + lane;
        float m = col[0];
#pragma unroll
        for (int i = 1; i + 1 < kGroup; i += 2) m = min3(m, col[i * LD], col[(i + 1) * LD]);
        m = fminf(m, col[(kGroup - 1) * LD]);
        mins[g * 32 + lane] = m;
        m = warp_min(m);
        if (lane == 0) low[g] = m;
    }
}

// The strips [g0, g1) of one warp, an axis of n rows: store(strip, g) for each, columns
// inside the grid.  All rows and minima of the CTA are in place (the caller has synchronised); `mins`
// holds kNear groups of kPadValue before the first and after the last group, which therefore fail every
// test.  Columns outside the grid hold kPadValue in every row and take no part in the decisions.
//
// Far from every site the minimum lies groups away and moves less than a group per strip: a strip that
// ended there hands the place to the next one, which begins with that group instead of its own.  The
// site of an output never lies before the previous output's, so groups before the least such place of
// the columns are left out, and groups beyond a column's own are tested at the strip's last output.
// kLastFirst: the last strip goes before the others, whose groups then end at its first output's minimum, and
// groups that can only gain on a column's last or first output are tried on that output alone before they are
// taken.  Smooth masks far away leave tens of groups within the bounds of 32 columns; the x pass, 512^3:
// half-spaces x + y + z < 350 and < 700 968 -> 699 and 691 -> 584 us, z < 100 564 -> 450, boxes unchanged.  In
// the zy pass it gains a twelfth there and costs the boxes a twentieth (its registers spill).
template <int LD, bool kLastFirst, typename Store>
__device__ __forceinline__ void strips(const float* __restrict__ rows, const float* __restrict__ mins,
                                       const float* __restrict__ low, int n, int g0, int g1, bool in, Store store) {
    const int lane = threadIdx.x & 31;
    const int ng = groups_of(n);
    // packed constants, kept in registers (their values hidden from the compiler, which would rebuild
    // each from immediates at every use)
    float2 origin = make_float2(0.f, -1.f), back2 = make_float2(-2.f, -2.f);
    float2 ahead = make_float2((float)kGroup, (float)kGroup), behind = make_float2(-(float)kGroup, -(float)kGroup);
    asm volatile("" : "+f"(origin.x), "+f"(origin.y), "+f"(back2.x), "+f"(back2.y));
    asm volatile("" : "+f"(ahead.x), "+f"(ahead.y), "+f"(behind.x), "+f"(behind.y));
    const int middle = kLastFirst ? __popc(__ballot_sync(0xffffffffu, in)) >> 1 : 0;  // of the columns inside the grid
    int seed = 0;   // offset of the group to begin with
    int least = 0;  // groups before it hold no minimum of this and later strips
    int greatest = ng;  // groups behind it hold none of the strips before the last one
    const bool ends = kLastFirst && g1 - g0 > 5;  // worth it
    for (int t = ends ? g0 - 1 : g0; t < (ends ? g1 - 1 : g1); ++t) {
        const int g = kLastFirst && t < g0 ? g1 - 1 : t;
        const float* const own = rows + g * kGroup * LD + lane;
        const float* const near = mins + g * 32 + lane;
        Strip s;
        float most;  // largest output of this column
        if (seed == 0) {
            s.group<LD, true>(own, origin, back2);
            most = in ? s.largest() : 0.f;
            float2 left = origin, right = origin;
#pragma unroll
            for (int o = 1; o <= kNear; ++o) {
                const float d = (float)(kGroup * o - (kGroup - 1));
                left = __fadd2_rn(left, ahead);
                right = __fadd2_rn(right, behind);
                if (__any_sync(0xffffffffu, near[-o * 32] < most - d * d)) {
                    s.group<LD>(own - o * kGroup * LD, left, back2);
                    most = in ? s.largest() : 0.f;
                }
                if (__any_sync(0xffffffffu, near[o * 32] < most - d * d)) {
                    s.group<LD>(own + o * kGroup * LD, right, back2);
                    most = in ? s.largest() : 0.f;
                }
            }
        } else {
#pragma unroll
            for (int k = 0; k < kGroup; ++k) s.a[k] = kPadValue;
            most = in ? kPadValue : 0.f;
        }
        constexpr float kReach = (float)(kGroup * kNear + 1);
        if (seed != 0 || __any_sync(0xffffffffu, kReach * kReach < most)) {
            float top = warp_max(most);  // of all columns
            const int skip = seed == 0 ? kNear : -1;
            int at = seed == 0 ? -kNear : ng;  // a group no later than the last output's minimum, as an offset
            int first = seed == 0 ? kNear : -ng;  // and one no earlier than the first output's
            const int o0 = abs(lane - g), o1 = abs(lane + 32 - g);
            const float d0 = fmaxf((float)(kGroup * o0 - (kGroup - 1)), 0.f), d1 = fmaxf((float)(kGroup * o1 - (kGroup - 1)), 0.f);
            float b0 = o0 > skip && lane >= least && (!kLastFirst || lane <= greatest) && lane < ng ? fmaf(d0, d0, low[lane]) : kPadValue;
            float b1 = o1 > skip && lane + 32 >= least && (!kLastFirst || lane + 32 <= greatest) && lane + 32 < ng ? fmaf(d1, d1, low[lane + 32]) : kPadValue;
            int next = g + seed;
            bool begin = seed != 0;
            for (;;) {  // each turn takes one group out
                int j = next;
                if (!begin) {
                    const float b = fminf(b0, b1), best = warp_min(b);
                    if (!(best < top)) break;
                    const int who = __ffs(__ballot_sync(0xffffffffu, b == best)) - 1;
                    j = __shfl_sync(0xffffffffu, b0 <= b1 ? lane : lane + 32, who);
                }
                if (lane == j) b0 = kPadValue;
                if (lane + 32 == j) b1 = kPadValue;
                const int o = j - g;
                const float D = (float)(-kGroup * o);
                // distance to the nearest output, and from the last one where only that can gain
                const float d = fmaxf(fabsf(D) - (float)(kGroup - 1), 0.f);
                const float dl = o < 0 ? D : d;
                const bool beyond = o > at;
                const float e = beyond ? dl : d;
                const float lim = beyond && in ? s.value(kGroup - 1) : most;
                if (!begin && !__any_sync(0xffffffffu, near[o * 32] < fmaf(-e, e, lim))) continue;
                if (kLastFirst && !begin) {
                    const bool may = near[o * 32] < fmaf(-e, e, lim);
                    const bool before = o < first;
                    const float* const col = own + o * (kGroup * LD);
                    const float x = beyond ? D + (float)(kGroup - 1) : D, end = beyond ? s.value(kGroup - 1) : s.value(0);
                    float2 q = make_float2(x, x - 1.f);
                    float v = kPadValue;
#pragma unroll
                    for (int i = 0; i < kGroup; i += 2) {
                        const float2 c = __ffma2_rn(q, q, make_float2(col[i * LD], col[(i + 1) * LD]));
                        v = min3(v, c.x, c.y);
                        q = __fadd2_rn(q, back2);
                    }
                    if (!__any_sync(0xffffffffu, may && in && (!(beyond || before) || v < end))) continue;
                }
                begin = false;
                const float was = s.a[kGroup - 1];
                [[maybe_unused]] const float was0 = s.a[0];
                s.group<LD>(own + o * (kGroup * LD), make_float2(D, D - 1.f), back2);
                if (s.a[kGroup - 1] < was) at = o;
                if (kLastFirst && s.a[0] < was0) first = o;
                most = in ? s.largest() : 0.f;
                top = warp_max(most);
            }
            least = g + __reduce_min_sync(0xffffffffu, in ? at : ng);
            seed = __shfl_sync(0xffffffffu, at, middle) - 1;
            if (seed >= -kNear - 1 && seed <= kNear) seed = 0;
            if (kLastFirst && t < g0) greatest = g + __reduce_max_sync(0xffffffffu, in ? first : -ng);
        } else if (kLastFirst && t < g0) {
            greatest = g + kNear;
        }
        if (kLastFirst && t < g0) seed = least = 0;
        if (in) store(s, g);
    }
}

// Outputs of strip g of an axis of n rows, `stride` elements apart from `out` (row 0) on.
template <typename T>
__device__ __forceinline__ void put(const Strip& s, T* __restrict__ out, int64_t stride, int n, int g) {
    T* p = out + (int64_t)(g * kGroup) * stride;
    const int valid = n - g * kGroup;
    auto one = [&](int k) {
        if constexpr (std::is_same_v<T, int32_t>) *p = s.integer(k);
        else *p = s.value(k);
        p += stride;
    };
    if (valid >= kGroup) {
#pragma unroll
        for (int k = 0; k < kGroup; ++k) one(k);
    } else {
#pragma unroll
        for (int k = 0; k < kGroup; ++k)
            if (k < valid) one(k);
    }
}

// The padding groups of `mins` (strips).
__device__ __forceinline__ void pad_minima(float* __restrict__ mins, int ng) {
    for (int i = threadIdx.x; i < kNear * 32; i += blockDim.x) {
        mins[i - kNear * 32] = kPadValue;
        mins[ng * 32 + i] = kPadValue;
    }
}

// cp.async of `bytes` (4 or 16) to shared memory.
template <int bytes>
__device__ __forceinline__ void cp_async(float* smem_dst, const float* src) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// z pass (nearest set bit along z from the bit words) + y pass.  grid = (W, nx, polarities),
// block = kThreads, dynamic smem = pass_smem_bytes(ny, kZyLd).  Polarity p measures to set bits when
// (p ^ invert) == 0, to clear bits otherwise.
//
// z: a lane owns a row.  It reads the row's words once, keeps the last nonzero word before and the
// first one after its own, and fills the row's 32 distances by a forward and a backward count over the
// own word's bits, two instructions a voxel each -- where a lane per voxel spent ballots, shuffles and
// bit searches on every one.  Rows are 33 words apart so that these stores, one row per lane, and the
// y pass's reads, one column per lane, are both free of bank conflicts.
constexpr int kZyLd = 33;

// Squared z distances of a row's 32 voxels to the set bits of `own` and to the nearest sites outside the
// word, `from` and `to` voxels before its first and after its last neighbour.  Out of line: its counts
// stay out of the registers of the y pass.
__device__ __noinline__ void fill_row(float* __restrict__ row, uint32_t own, float from, float to) {
    float up[32], d = from;
#pragma unroll
    for (int z = 0; z < 32; ++z) {
        d = (own >> z) & 1u ? 0.f : d + 1.f;
        up[z] = d;
    }
    d = to;
#pragma unroll
    for (int z = 31; z >= 0; --z) {
        d = (own >> z) & 1u ? 0.f : d + 1.f;
        const float m = fminf(d, up[z]);
        row[z] = m * m;
    }
}

__global__ void __launch_bounds__(kThreads, 3) k_edt_zy(const uint32_t* __restrict__ bits, float* __restrict__ g,
                                                        int nx, int ny, int nz, int W, int invert, float sentinel) {
    extern __shared__ __align__(16) float smem[];
    const int w = blockIdx.x, x = blockIdx.y, pol = blockIdx.z;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ng = groups_of(ny);
    float* const rows = smem;
    float* const mins = smem + ng * kGroup * kZyLd + kNear * 32;
    float* const low = mins + (ng + kNear) * 32;
    pad_minima(mins, ng);
    const uint32_t flip = (pol ^ invert) != 0 ? 0xffffffffu : 0u;
    const int tail = nz & 31;
    const uint32_t last_valid = tail ? ((1u << tail) - 1u) : 0xffffffffu;
    const int live = min(32, nz - 32 * w);  // columns of this chunk inside the grid
    const int per = (ng + kWarps - 1) / kWarps;
    const int g0 = min(ng, warp * per), g1 = min(ng, g0 + per);
    // a plane without a site keeps the sentinel everywhere
    const uint32_t* const plane = bits + (int64_t)x * ny * W;
    bool some = false;
    for (int k = threadIdx.x; k < ny * W; k += kThreads) {
        uint32_t word = plane[k] ^ flip;
        if (tail && k % W == W - 1) word &= last_valid;
        some |= word != 0u;
    }
    float* const out = g + (int64_t)pol * nx * ny * nz + (int64_t)x * ny * nz + 32 * w + lane;
    const bool in = lane < live;
    if (!__syncthreads_or(some)) {
        if (in)
            for (int y = g0 * kGroup; y < min(ny, g1 * kGroup); ++y) out[(int64_t)y * nz] = sentinel;
        return;
    }
    for (int y0 = g0 * kGroup; y0 < g1 * kGroup; y0 += 32) {
        const int y = y0 + lane;
        if (y >= g1 * kGroup) continue;
        float* const row = rows + y * kZyLd;
        if (y >= ny) {  // padding to a whole group
#pragma unroll
            for (int z = 0; z < 32; ++z) row[z] = kPadValue;
            continue;
        }
        const uint32_t* const line = plane + y * W;
        uint32_t before = 0u, after = 0u;
        int bw = 0, aw = 0;
        for (int k = 0; k < w; ++k) {
            const uint32_t word = line[k] ^ flip;
            if (word) { before = word; bw = k; }
        }
        const uint32_t own = (line[w] ^ flip) & (w == W - 1 ? last_valid : 0xffffffffu);
        for (int k = W - 1; k > w; --k) {
            const uint32_t word = (line[k] ^ flip) & (k == W - 1 ? last_valid : 0xffffffffu);
            if (word) { after = word; aw = k; }
        }
        if (!(before | own | after)) {
#pragma unroll
            for (int z = 0; z < 32; ++z) row[z] = sentinel;
        } else {
            fill_row(row, own, before ? (float)(32 * (w - bw) - 1 - (31 - __clz(before))) : kFar,
                     after ? (float)(32 * (aw - w) - 32 + __ffs(after) - 1) : kFar);
        }
        for (int z = live; z < 32; ++z) row[z] = kPadValue;
    }
    __syncwarp();
    group_minima<kZyLd>(rows, mins, low, g0, g1);
    __syncthreads();
    strips<kZyLd, false>(rows, mins, low, ny, g0, g1, in, [&](const Strip& s, int gr) { put<float>(s, out, nz, ny, gr); });
}

// x pass.  grid = (W, ny, polarities), block = kThreads, dynamic smem = pass_smem_bytes(nx, 32).
// Reads g (polarity-major, `size` voxels each) and writes out with the same layout; out may be g
// itself (each CTA reads its whole column block before it writes any of it).  kVec: rows of g are
// 16-byte aligned (nz a multiple of 4 and g itself aligned), so one copy instruction moves four rows'
// segments of the block instead of one.
template <bool kVec>
__global__ void __launch_bounds__(kThreads, 3) k_edt_x(const float* g, int32_t* out, int nx, int ny, int nz) {
    extern __shared__ __align__(16) float smem[];
    const int w = blockIdx.x, y = blockIdx.y, pol = blockIdx.z;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ng = groups_of(nx);
    float* const rows = smem;
    float* const mins = smem + ng * kGroup * 32 + kNear * 32;
    float* const low = mins + (ng + kNear) * 32;
    pad_minima(mins, ng);
    const int64_t size = (int64_t)nx * ny * nz, stride = (int64_t)ny * nz;
    const int64_t col = (int64_t)pol * size + (int64_t)y * nz + 32 * w;
    const int live = min(32, nz - 32 * w);
    const int per = (ng + kWarps - 1) / kWarps;
    const int g0 = min(ng, warp * per), g1 = min(ng, g0 + per);
    const int x1 = min(nx, g1 * kGroup);
    // the warp's rows, 4 a copy instruction (kVec) or one; columns outside the grid are filled
    const int rstep = kVec ? 4 : 1, c = kVec ? 4 * (lane & 7) : lane;
    const int xa = g0 * kGroup + (kVec ? lane >> 3 : 0);
    if (c < live) {
        const float* src = g + col + xa * stride + c;
        float* to = rows + xa * 32 + c;
#pragma unroll 4
        for (int x = xa; x < x1; x += rstep) {
            cp_async<kVec ? 16 : 4>(to, src);
            src += rstep * stride;
            to += rstep * 32;
        }
    } else {
        for (int x = xa; x < x1; x += rstep)
            for (int k = 0; k < (kVec ? 4 : 1); ++k) rows[x * 32 + c + k] = kPadValue;
    }
    for (int x = max(nx, g0 * kGroup); x < g1 * kGroup; ++x) rows[x * 32 + lane] = kPadValue;
    cp_async_wait_all();
    __syncwarp();
    group_minima<32>(rows, mins, low, g0, g1);
    __syncthreads();
    int32_t* const dst = out + col + lane;
    const bool in = lane < live;
    strips<32, true>(rows, mins, low, nx, g0, g1, in, [&](const Strip& s, int gr) { put<int32_t>(s, dst, stride, nx, gr); });
}

// Correctly rounded signed distance of one voxel from its two squared distances, the reference's
// definition (src/field_engine/edt_persistent_pair_v1/edt.cu:36-42).
__device__ __forceinline__ float signed_from_pair(int32_t sq_out, int32_t sq_in, double pitch, float half) {
    const float outside = __double2float_rn(__dmul_rn(__dsqrt_rn((double)sq_out), pitch));
    const float inside = __double2float_rn(__dmul_rn(__dsqrt_rn((double)sq_in), pitch));
    const float delta = __fsub_rn(outside, inside);
    const float sign = delta > 0.f ? 1.f : (delta < 0.f ? -1.f : 0.f);
    return __fsub_rn(delta, __fmul_rn(sign, half));
}

// Signed float32 distance of every voxel from the two polarities' squared distances (sq[0]: to the
// nonzero voxels, sq[1]: to the zero voxels).
__global__ void __launch_bounds__(256) k_edt_signed(const int32_t* __restrict__ sq, float* __restrict__ out,
                                                    int64_t size, double pitch, float half) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < size; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = signed_from_pair(sq[i], sq[size + i], pitch, half);
}

bool shape_ok(int nx, int ny, int nz) {
    return nx >= 1 && ny >= 1 && nz >= 1 && nx <= kMaxAxis && ny <= kMaxAxis && nz <= kMaxAxis;
}

int32_t sentinel_of(int nx, int ny, int nz) {
    return (nx - 1) * (nx - 1) + (ny - 1) * (ny - 1) + (nz - 1) * (nz - 1) + 1;
}

int words_of(int nz) { return (nz + 31) / 32; }

void launch_x(const float* g, int32_t* out, int nx, int ny, int nz, int W, int npol, cudaStream_t stream) {
    const dim3 grid(W, ny, npol);
    const int smem = pass_smem_bytes(nx, 32);
    if (nz % 4 == 0 && (reinterpret_cast<uintptr_t>(g) & 15) == 0)
        k_edt_x<true><<<grid, kThreads, smem, stream>>>(g, out, nx, ny, nz);
    else
        k_edt_x<false><<<grid, kThreads, smem, stream>>>(g, out, nx, ny, nz);
}

// Scratch layout: [Counters (256 B)] [bit words] [g for up to two polarities].
int64_t scratch_bytes(int nx, int ny, int nz, int npol) {
    const int64_t size = (int64_t)nx * ny * nz;
    const int64_t bits = ((int64_t)nx * ny * words_of(nz) * 4 + 255) / 256 * 256;
    return 256 + bits + (int64_t)npol * size * 4;
}

// The column passes use more than 48 KB of dynamic shared memory at 512 rows, an opt-in that is a
// per-device function attribute: set once for every device that runs a transform (under a lock,
// since serving threads enqueue transforms concurrently).
constexpr int kMaxDevices = 64;
std::mutex g_configure_lock;
bool g_configured[kMaxDevices] = {};

int configure_device() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return FB_RUNTIME;
    std::lock_guard<std::mutex> guard(g_configure_lock);
    if (g_configured[dev]) return FB_OK;
    const auto most = cudaFuncAttributeMaxDynamicSharedMemorySize;
    FB_CUDA(cudaFuncSetAttribute(k_edt_zy, most, pass_smem_bytes(kMaxAxis, kZyLd)));
    FB_CUDA(cudaFuncSetAttribute(k_edt_x<true>, most, pass_smem_bytes(kMaxAxis, 32)));
    FB_CUDA(cudaFuncSetAttribute(k_edt_x<false>, most, pass_smem_bytes(kMaxAxis, 32)));
    g_configured[dev] = true;
    return FB_OK;
}

// Enqueue the whole transform on `stream`.  paired == 0: sites are the nonzero mask bytes when
// sites_nonzero, else the zero bytes; writes int32 to out_sq.  paired == 1: both polarities
// (polarity 0 to the nonzero voxels), signed float32 to out_signed, optional squared pair to out_sq.
int enqueue(const uint8_t* d_mask, int nx, int ny, int nz, int paired, int sites_nonzero, double pitch,
            int32_t* out_sq, float* out_signed, void* scratch, int64_t scratch_len, cudaStream_t stream,
            bool count) {
    if (int rc = configure_device()) return rc;
    const int npol = paired ? 2 : 1;
    if (scratch_len < scratch_bytes(nx, ny, nz, npol)) return FB_INVALID;
    const int W = words_of(nz);
    const int64_t lines = (int64_t)nx * ny;
    const int64_t size = lines * nz;
    char* base = static_cast<char*>(scratch);
    Counters* counters = reinterpret_cast<Counters*>(base);
    uint32_t* bits = reinterpret_cast<uint32_t*>(base + 256);
    float* g = reinterpret_cast<float*>(base + 256 + ((lines * W * 4 + 255) / 256 * 256));
    if (count) FB_CUDA(cudaMemsetAsync(counters, 0, sizeof(Counters), stream));
    const int sms = fb_sm_count();
    const int64_t words = lines * W;
    int grid0 = (int)std::min<int64_t>((words + 255) / 256, (int64_t)sms * 8);
    launch_bits(grid0, stream, d_mask, bits, lines, nz, W, count ? counters : nullptr);
    FB_LAUNCH();
    const int32_t sentinel = sentinel_of(nx, ny, nz);
    // Single polarity measuring to zero bytes = the set bits flipped.
    const int invert = paired ? 0 : (sites_nonzero ? 0 : 1);
    k_edt_zy<<<dim3(W, nx, npol), kThreads, pass_smem_bytes(ny, kZyLd), stream>>>(bits, g, nx, ny, nz, W, invert,
                                                                                  (float)sentinel);
    FB_LAUNCH();
    if (paired) {
        // both polarities' x passes into the squared output (or in place), then the signed values
        int32_t* sq = out_sq ? out_sq : reinterpret_cast<int32_t*>(g);
        launch_x(g, sq, nx, ny, nz, W, 2, stream);
        FB_LAUNCH();
        const int grid = (int)std::min<int64_t>((size + 255) / 256, (int64_t)sms * 16);
        k_edt_signed<<<grid, 256, 0, stream>>>(sq, out_signed, size, pitch, (float)(0.5 * pitch));
    } else {
        launch_x(g, out_sq, nx, ny, nz, W, 1, stream);
    }
    FB_LAUNCH();
    return FB_OK;
}

// Mask validity from the counters of k_edt_bits: 0 ok, 1 invalid (a byte > 1, or one class only).
int read_validity(const void* scratch, int64_t size, cudaStream_t stream) {
    Counters c;
    FB_CUDA(cudaMemcpyAsync(&c, scratch, sizeof(c), cudaMemcpyDeviceToHost, stream));
    FB_CUDA(cudaStreamSynchronize(stream));
    if (c.invalid) return FB_INVALID;
    if (c.ones == 0 || (int64_t)c.ones == size) return FB_INVALID;
    return FB_OK;
}

struct Pair {
    int nx, ny, nz;
    int64_t size;
    uint8_t* mask = nullptr;
    void* scratch = nullptr;
    int64_t scratch_len = 0;
    float* distance = nullptr;
    int32_t* squared = nullptr;
    cudaStream_t stream = nullptr;
    bool failed = false;
};

}  // namespace

// ---------------------------------------------------------------------------------------------
// Allocation-free EDT for callers that cannot allocate device memory.
//
// Some hosts own every byte of device memory themselves (an engine embedding this library behind
// its own pool allocator, a real-time loop that must never hit the implicit synchronisation of
// cudaMalloc/cudaFree, a plugin whose host forbids allocation calls); they can pass input and
// output buffers but not scratch.  For them the squared EDT below keeps its scratch (bit words
// and the float32 intermediate) in a fixed array compiled into this library.
//
// Limit: at most kNoAllocVoxels = 2^20 voxels and 512 per axis -- the reference's own EDT
// contract (src/field_engine/edt_native_large_v1/edt.cu:34-37).  Every GPU that loads this
// library holds the array (kNoAllocScratchBytes, about 5.1 MiB) until the process exits.
// ---------------------------------------------------------------------------------------------
constexpr int64_t kNoAllocVoxels = int64_t(1) << 20;
// bit words: nx*ny*ceil(nz/32) <= voxels/32 + nx*ny <= 2^15 + 512*512; plus 256 B of counters and
// one float32 intermediate per voxel
constexpr int64_t kNoAllocBitBytes = ((kNoAllocVoxels / 32 + 512 * 512) * 4 + 255) / 256 * 256;
constexpr int64_t kNoAllocScratchBytes = 256 + kNoAllocBitBytes + kNoAllocVoxels * 4;
static __device__ __align__(256) unsigned char g_edt_noalloc_scratch[kNoAllocScratchBytes];

namespace {

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_lock;
struct NoAllocEntry {
    void* context;  // the driver context the address belongs to
    void* ptr;
};
NoAllocEntry g_noalloc[kNoAllocMaxDevices] = {};

// The current driver context (CUcontext), through the runtime's driver entry point so the library
// does not link libcuda itself; nullptr when it cannot be had.
void* current_context() {
    using GetCurrent = int (*)(void**);
    static GetCurrent fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<GetCurrent>(f);
    }();
    void* ctx = nullptr;
    if (!fn || fn(&ctx) != 0) return nullptr;
    return ctx;
}

// Device address of the array on the current device, looked up once per device and context.  The
// name g_edt_noalloc_scratch in host code is a host-side stand-in, not a device address, so kernels
// get this pointer instead.  A context torn down and created again (cudaDeviceReset) maps the array
// at a new address: the lookup is keyed on the context and repeated for a new one.
int noalloc_scratch(void** out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices) return FB_RUNTIME;
    void* ctx = current_context();  // nullptr before the runtime has made a context current
    std::lock_guard<std::mutex> guard(g_noalloc_lock);
    NoAllocEntry& e = g_noalloc[dev];
    if (!e.ptr || !ctx || e.context != ctx) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_edt_noalloc_scratch) != cudaSuccess || !p) return FB_RUNTIME;
        e.ptr = p;
        e.context = ctx ? ctx : current_context();
    }
    *out = e.ptr;
    return FB_OK;
}

}  // namespace

extern "C" {

// Squared EDT exactly as fb_edt_squared_device, with no allocation and no caller scratch: the
// scratch is the library's fixed device array.  Inputs and outputs are the caller's device
// buffers.  Status 0 ok, 1 invalid arguments (a null pointer, an axis below 1), 2 CUDA failure,
// 7 grid beyond the fixed scratch (an axis above 512 or more than 2^20 voxels) -- both rejected
// before anything is enqueued.
// The first call on each device looks the array up (cudaGetSymbolAddress) with that device
// current; make that first call before any stream capture.  The array is shared by every call
// and keeps the last call's contents (nothing in it needs to start at zero: every word a call
// reads it writes first), so calls whose work overlaps on the GPU -- on different streams, or
// from different threads -- race on it and must be serialised by the caller.
int fb_edt_squared_device_noalloc(const uint8_t* d_mask, int nx, int ny, int nz, int sites_nonzero,
                                  int32_t* d_out, void* stream) noexcept {
    if (!d_mask || !d_out || nx < 1 || ny < 1 || nz < 1) return FB_INVALID;
    if (!shape_ok(nx, ny, nz) || (int64_t)nx * ny * nz > kNoAllocVoxels) return FB_NOALLOC_LIMIT;
    const int64_t need = scratch_bytes(nx, ny, nz, 1);
    if (need > kNoAllocScratchBytes) return FB_NOALLOC_LIMIT;
    void* scratch = nullptr;
    if (int rc = noalloc_scratch(&scratch)) return rc;
    return enqueue(d_mask, nx, ny, nz, 0, sites_nonzero, 1.0, d_out, nullptr, scratch, kNoAllocScratchBytes,
                   static_cast<cudaStream_t>(stream), false);
}

// Size in bytes of the fixed scratch array and the largest voxel count it serves.
int64_t fb_edt_noalloc_capacity(int64_t* max_voxels) noexcept {
    if (max_voxels) *max_voxels = kNoAllocVoxels;
    return kNoAllocScratchBytes;
}

}  // extern "C"

extern "C" {

// ---------------------------------------------------------------------------------------------
// Device-pointer forms (stream-ordered; nothing is allocated).
// ---------------------------------------------------------------------------------------------

int64_t fb_edt_scratch_bytes(int nx, int ny, int nz, int paired) {
    if (!shape_ok(nx, ny, nz)) return -1;
    return scratch_bytes(nx, ny, nz, paired ? 2 : 1);
}

int fb_edt_squared_device(const uint8_t* d_mask, int nx, int ny, int nz, int sites_nonzero, int32_t* d_out,
                          void* d_scratch, int64_t scratch_len, void* stream) noexcept {
    if (!d_mask || !d_out || !d_scratch || !shape_ok(nx, ny, nz)) return FB_INVALID;
    return enqueue(d_mask, nx, ny, nz, 0, sites_nonzero, 1.0, d_out, nullptr, d_scratch, scratch_len,
                   static_cast<cudaStream_t>(stream), false);
}

int fb_edt_pair_device(const uint8_t* d_mask, int nx, int ny, int nz, double pitch, float* d_signed,
                       int32_t* d_squared, void* d_scratch, int64_t scratch_len, void* stream) noexcept {
    if (!d_mask || !d_signed || !d_scratch || !shape_ok(nx, ny, nz)) return FB_INVALID;
    if (!std::isfinite(pitch) || pitch < 1e-12 || pitch > 1e12) return FB_INVALID;
    return enqueue(d_mask, nx, ny, nz, 1, 1, pitch, d_squared, d_signed, d_scratch, scratch_len,
                   static_cast<cudaStream_t>(stream), false);
}

// Mask check on the device: status 1 when a byte is > 1 or only one class is present.
int fb_edt_validate_device(const uint8_t* d_mask, int nx, int ny, int nz, void* d_scratch, int64_t scratch_len,
                           void* stream) noexcept {
    if (!d_mask || !d_scratch || !shape_ok(nx, ny, nz) || scratch_len < scratch_bytes(nx, ny, nz, 1))
        return FB_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int W = words_of(nz);
    const int64_t lines = (int64_t)nx * ny;
    char* base = static_cast<char*>(d_scratch);
    FB_CUDA(cudaMemsetAsync(base, 0, sizeof(Counters), s));
    int grid0 = (int)std::min<int64_t>((lines * W + 255) / 256, (int64_t)fb_sm_count() * 8);
    launch_bits(grid0, s, d_mask, reinterpret_cast<uint32_t*>(base + 256), lines, nz, W,
                reinterpret_cast<Counters*>(base));
    FB_LAUNCH();
    return read_validity(base, lines * nz, s);
}

// ---------------------------------------------------------------------------------------------
// Host-pointer forms with the reference's names, arguments and status codes.
// ---------------------------------------------------------------------------------------------

static int squared_host(const uint8_t* mask, int nx, int ny, int nz, int32_t* output) {
    const int64_t size = (int64_t)nx * ny * nz;
    uint8_t* d_mask = nullptr;
    int32_t* d_out = nullptr;
    void* scratch = nullptr;
    const int64_t sb = scratch_bytes(nx, ny, nz, 1);
    int status = FB_RUNTIME;
    cudaStream_t s = nullptr;
    do {
        if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) break;
        if (cudaMallocAsync(&d_mask, size, s) != cudaSuccess) break;
        if (cudaMallocAsync(&d_out, size * 4, s) != cudaSuccess) break;
        if (cudaMallocAsync(&scratch, sb, s) != cudaSuccess) break;
        if (cudaMemcpyAsync(d_mask, mask, size, cudaMemcpyHostToDevice, s) != cudaSuccess) break;
        int rc = enqueue(d_mask, nx, ny, nz, 0, 0, 1.0, d_out, nullptr, scratch, sb, s, true);
        if (rc) { status = rc; break; }
        rc = read_validity(scratch, size, s);
        if (rc) { status = rc; break; }
        if (cudaMemcpyAsync(output, d_out, size * 4, cudaMemcpyDeviceToHost, s) != cudaSuccess) break;
        if (cudaStreamSynchronize(s) != cudaSuccess) break;
        status = FB_OK;
    } while (0);
    if (d_mask) cudaFreeAsync(d_mask, s);
    if (d_out) cudaFreeAsync(d_out, s);
    if (scratch) cudaFreeAsync(scratch, s);
    if (s) {
        if (cudaStreamSynchronize(s) != cudaSuccess) status = FB_RUNTIME;
        cudaStreamDestroy(s);
    }
    return status;
}

// Replaces src/field_engine/edt_native_large_v1/edt.cu:33 (edt_squared_large).  Same arguments
// and statuses; the axis limit stays 512 and the voxel cap is lifted from 2^20 to 512^3.
int edt_squared_large(const uint8_t* mask, int nx, int ny, int nz, int32_t* output) noexcept {
    if (!mask || !output || !shape_ok(nx, ny, nz)) return FB_INVALID;
    return squared_host(mask, nx, ny, nz, output);
}

// Replaces src/field_engine/edt_native_v1/edt.cu:20 (edt_squared): <= 128 per axis, <= 262144
// voxels, exactly the reference's bound.
int edt_squared(const uint8_t* mask, int nx, int ny, int nz, int32_t* output) noexcept {
    if (!mask || !output || nx < 1 || ny < 1 || nz < 1 || nx > 128 || ny > 128 || nz > 128) return FB_INVALID;
    if ((int64_t)nx * ny * nz > 262144) return FB_INVALID;
    return squared_host(mask, nx, ny, nz, output);
}

// Replaces src/field_engine/edt_persistent_pair_v1/edt.cu:48 (edt_pair_create).  Persistent
// device buffers and a private stream; the voxel cap is lifted from 2^20 to 512^3.
void* edt_pair_create(int nx, int ny, int nz) noexcept {
    if (!shape_ok(nx, ny, nz)) return nullptr;
    Pair* p = new (std::nothrow) Pair;
    if (!p) return nullptr;
    p->nx = nx;
    p->ny = ny;
    p->nz = nz;
    p->size = (int64_t)nx * ny * nz;
    p->scratch_len = scratch_bytes(nx, ny, nz, 2);
    bool ok = cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking) == cudaSuccess &&
              cudaMalloc(&p->mask, p->size) == cudaSuccess &&
              cudaMalloc(&p->scratch, p->scratch_len) == cudaSuccess &&
              cudaMalloc(&p->distance, p->size * 4) == cudaSuccess &&
              cudaMalloc(&p->squared, p->size * 8) == cudaSuccess;
    if (!ok) {
        if (p->mask) cudaFree(p->mask);
        if (p->scratch) cudaFree(p->scratch);
        if (p->distance) cudaFree(p->distance);
        if (p->squared) cudaFree(p->squared);
        if (p->stream) cudaStreamDestroy(p->stream);
        delete p;
        return nullptr;
    }
    return p;
}

// Replaces src/field_engine/edt_persistent_pair_v1/edt.cu:59 (edt_pair_query).  Status 1 for
// invalid input (nothing written), 2 for a runtime failure, after which the handle stays failed.
int edt_pair_query(void* pointer, const uint8_t* mask, double pitch, float* output, int32_t* squared) noexcept {
    Pair* p = static_cast<Pair*>(pointer);
    if (!p || !mask || !output || !std::isfinite(pitch) || pitch < 1e-12 || pitch > 1e12) return FB_INVALID;
    if (p->failed) return FB_RUNTIME;
#define PAIR_CHECK(x)            \
    if ((x) != cudaSuccess) {    \
        p->failed = true;        \
        return FB_RUNTIME;       \
    }
    PAIR_CHECK(cudaMemcpyAsync(p->mask, mask, p->size, cudaMemcpyHostToDevice, p->stream));
    int rc = enqueue(p->mask, p->nx, p->ny, p->nz, 1, 1, pitch, p->squared, p->distance, p->scratch, p->scratch_len,
                     p->stream, true);
    if (rc) {
        p->failed = rc != FB_INVALID;
        return rc;
    }
    rc = read_validity(p->scratch, p->size, p->stream);
    if (rc == FB_INVALID) return FB_INVALID;
    if (rc) {
        p->failed = true;
        return rc;
    }
    PAIR_CHECK(cudaMemcpyAsync(output, p->distance, p->size * 4, cudaMemcpyDeviceToHost, p->stream));
    if (squared) PAIR_CHECK(cudaMemcpyAsync(squared, p->squared, p->size * 8, cudaMemcpyDeviceToHost, p->stream));
    PAIR_CHECK(cudaStreamSynchronize(p->stream));
#undef PAIR_CHECK
    return FB_OK;
}

// Replaces src/field_engine/edt_persistent_pair_v1/edt.cu:45 (edt_pair_destroy).
void edt_pair_destroy(void* pointer) noexcept {
    Pair* p = static_cast<Pair*>(pointer);
    if (!p) return;
    if (p->stream) cudaStreamSynchronize(p->stream);
    if (p->mask) cudaFree(p->mask);
    if (p->scratch) cudaFree(p->scratch);
    if (p->distance) cudaFree(p->distance);
    if (p->squared) cudaFree(p->squared);
    if (p->stream) cudaStreamDestroy(p->stream);
    delete p;
}

}  // extern "C"
