// Export step: the zero (or `level`) isosurface of a resident sparse field as a triangle mesh,
// straight from the leaf tiles -- the mesh that marching cubes gives on the dense reconstruction
// (tiles in active blocks, -BIG / +BIG elsewhere; src/field_engine/faltkarna_v1.py:302-350 followed
// by skimage.measure.marching_cubes, and faltvolym_v1.py:83-104 for the enclosed volume).
//
// Vertices: one per grid edge whose ends lie on opposite sides (inside = value < level, the
// classifier's convention that 0 counts as outside), at the linear interpolation
// t = g0 / (g0 - g1), g = value - level, in float64, stored as float32 world coordinates
// origin + pitch (index + t).  Each edge is owned by the active block of its lower end, else by the
// active block of its upper end; a block numbers its edges in slot order (inner edges
// ((lx B + ly) B + lz) 3 + axis, then the edges that enter it across its low faces), so vertex ids
// run block by block in ascending block id.  A bit word per 32 slots and the word's exclusive
// prefix turn an edge into its vertex id with one popcount.
//
// Faces: per cube, the crossing edges are joined on each of its six faces into segments that keep
// the inside on their left as seen from outside the cube; a face with four crossings is resolved by
// the asymptotic decider (the sign of the bilinear saddle value, evaluated from the face's own four
// values, so both cubes that share the face agree and the surface has no cracks).  The segments
// close into loops; a loop is fanned from its first vertex, in loop order from its lowest-numbered
// edge, that lies on no cube face the loop crosses twice (else from the lowest edge: possible only
// where the field changes sign several times across one cube, and then the fan can lay a flat
// zero-volume triangle into such a face), triangles wound so that their normals point to the
// outside (increasing value).  A cube is owned by the active block of its lowest
// corner, else by the first active block among its corners; triangles run block by block, cubes in
// lexicographic order inside a block's range, loops by lowest edge.  Cubes whose interior is
// ambiguous (two loops that the trilinear interior would join by a tunnel) keep the two loops.
#include "common.cuh"
#include "scan.cuh"
#include <algorithm>
#include <climits>

namespace {

constexpr int kMcThreads = 256;
constexpr int kMcMaxBlock = 32;

struct McField {
    const int32_t* kind;
    const int32_t* slot;
    const float* tiles;
    int64_t nx, ny, nz;
    int B, nby, nbz;
    double ox, oy, oz, pitch, level;
    float big;
};

__host__ __device__ inline int64_t mc_slots(int B) { return 3LL * B * B * B + 3LL * B * B; }
__host__ __device__ inline int64_t mc_words(int B) { return (mc_slots(B) + 31) / 32; }

// Corner c of a cube: bit 0 = +x, bit 1 = +y, bit 2 = +z.  Edge e = axis * 4 + w runs along
// `axis` from the corner whose other two bits are w (lower axis in bit 0).
__device__ __forceinline__ int edge_corner0(int e) {
    const int a = e >> 2, w = e & 3;
    if (a == 0) return ((w & 1) << 1) | ((w >> 1) << 2);
    if (a == 1) return (w & 1) | ((w >> 1) << 2);
    return (w & 1) | ((w >> 1) << 1);
}
__device__ __forceinline__ int edge_of(int ca, int cb) {  // corners that differ in one bit
    const int d = __ffs(ca ^ cb) - 1, c = ca & cb;
    int w;
    if (d == 0) w = ((c >> 1) & 1) | (((c >> 2) & 1) << 1);
    else if (d == 1) w = (c & 1) | (((c >> 2) & 1) << 1);
    else w = (c & 1) | (((c >> 1) & 1) << 1);
    return d * 4 + w;
}

// The loops of one cube: next[e] for every crossing edge e (cross bit e).  g: value - level at the
// eight corners, float64.
struct CubeLoops {
    unsigned cross;
    int8_t next[12];
};

__device__ CubeLoops cube_loops(const double g[8]) {
    CubeLoops L;
    unsigned in = 0;
    for (int c = 0; c < 8; ++c) in |= (unsigned)(g[c] < 0.0) << c;
    L.cross = 0;
    for (int e = 0; e < 12; ++e) L.next[e] = -1;
    if (in == 0 || in == 255) return L;
    for (int e = 0; e < 12; ++e) {
        const int c0 = edge_corner0(e), c1 = c0 | (1 << (e >> 2));
        L.cross |= (unsigned)(((in >> c0) & 1) != ((in >> c1) & 1)) << e;
    }
    for (int f = 0; f < 6; ++f) {
        const int a = f >> 1, s = f & 1, u = (a + 1) % 3, v = (a + 2) % 3;
        // corners in counter-clockwise order as seen from outside the face
        int q[4];
        const int b = s << a;
        q[0] = b;
        q[2] = b | (1 << u) | (1 << v);
        q[1] = b | (1 << (s ? u : v));
        q[3] = b | (1 << (s ? v : u));
        int E[4], inq[4];
        for (int i = 0; i < 4; ++i) {
            E[i] = edge_of(q[i], q[(i + 1) & 3]);
            inq[i] = (in >> q[i]) & 1;
        }
        const int k = (inq[0] != inq[1]) + (inq[1] != inq[2]) + (inq[2] != inq[3]) + (inq[3] != inq[0]);
        if (k == 2) {
            int st = -1, en = -1;
            for (int i = 0; i < 4; ++i) {
                if (inq[i] && !inq[(i + 1) & 3]) st = E[i];
                if (!inq[i] && inq[(i + 1) & 3]) en = E[i];
            }
            L.next[st] = (int8_t)en;
        } else if (k == 4) {
            // asymptotic decider on the (u, v)-ordered values: the saddle value's sign
            const double g00 = g[b], g10 = g[b | (1 << u)], g11 = g[b | (1 << u) | (1 << v)], g01 = g[b | (1 << v)];
            const double num = __dsub_rn(__dmul_rn(g00, g11), __dmul_rn(g10, g01));
            const bool connected = (g00 < 0.0) ? (num > 0.0) : (num < 0.0);  // inside corners joined
            for (int i = 0; i < 4; ++i)
                if (inq[i]) L.next[E[i]] = (int8_t)(connected ? E[(i + 1) & 3] : E[(i + 3) & 3]);
        }
    }
    return L;
}

// Bit mask of the two cube faces (axis * 2 + side) that contain edge e.
__device__ __forceinline__ unsigned edge_faces(int e) {
    const int c0 = edge_corner0(e), a = e >> 2;
    unsigned m = 0;
    for (int b = 0; b < 3; ++b)
        if (b != a) m |= 1u << (b * 2 + ((c0 >> b) & 1));
    return m;
}

// Next edge of a loop; every crossing edge starts exactly one face segment (the two faces through
// an edge walk it in opposite directions), so next is a permutation of the crossing edges.  The
// checks only keep a broken table inside the cube's 12 edges.
__device__ __forceinline__ int loop_next(const CubeLoops& L, int e) {
    const int n = L.next[e];
    return n >= 0 && n < 12 ? n : -1;
}

// Triangles of a cube's loops: sum over loops of (length - 2).
__device__ __forceinline__ int cube_triangles(const CubeLoops& L) {
    int loops = 0;
    unsigned todo = L.cross;
    while (todo) {
        const int e0 = __ffs(todo) - 1;
        int e = e0;
        for (int i = 0; i < 12; ++i) {
            todo &= ~(1u << e);
            e = loop_next(L, e);
            if (e < 0 || e == e0) break;
        }
        if (e != e0) return 0;
        ++loops;
    }
    return __popc(L.cross) - 2 * loops;
}

// World position of the vertex on edge (p, axis), p the edge's lower end.
__device__ __forceinline__ void edge_vertex(const McField& F, int64_t px, int64_t py, int64_t pz, int a, double g0,
                                            double g1, float* out) {
    const double t = __ddiv_rn(g0, __dsub_rn(g0, g1));
    double p[3] = {(double)px, (double)py, (double)pz};
    p[a] = __dadd_rn(p[a], t);
    out[0] = (float)__dadd_rn(F.ox, __dmul_rn(F.pitch, p[0]));
    out[1] = (float)__dadd_rn(F.oy, __dmul_rn(F.pitch, p[1]));
    out[2] = (float)__dadd_rn(F.oz, __dmul_rn(F.pitch, p[2]));
}

// Triangles of the cubes that need no face decision, by the eight corners' inside bits: the loops of
// cube_loops fanned as the emit pass fans them, three edges a triangle.  kAmbiguous marks the corner
// patterns with a face of four crossings, whose loops depend on the values.
constexpr int kAmbiguous = 255;
constexpr int kMaxTableTris = 4;  // 12 crossing edges in four loops of three; any other split has fewer loops to fan

struct CubeTable {
    uint8_t ntri[256];
    uint8_t edge[256][16];
};

constexpr int c_edge_corner0(int e) {
    const int a = e >> 2, w = e & 3;
    return a == 0 ? ((w & 1) << 1) | ((w >> 1) << 2) : (a == 1 ? (w & 1) | ((w >> 1) << 2) : (w & 1) | ((w >> 1) << 1));
}

constexpr int c_edge_of(int ca, int cb) {
    const int x = ca ^ cb, d = x == 1 ? 0 : (x == 2 ? 1 : 2), c = ca & cb;
    const int w = d == 0 ? ((c >> 1) & 1) | (((c >> 2) & 1) << 1)
                         : (d == 1 ? (c & 1) | (((c >> 2) & 1) << 1) : (c & 1) | (((c >> 1) & 1) << 1));
    return d * 4 + w;
}

constexpr unsigned c_edge_faces(int e) {
    unsigned m = 0;
    for (int b = 0; b < 3; ++b)
        if (b != (e >> 2)) m |= 1u << (b * 2 + ((c_edge_corner0(e) >> b) & 1));
    return m;
}

constexpr CubeTable make_cube_table() {
    CubeTable T{};
    for (int in = 0; in < 256; ++in) {
        int next[12] = {-1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1};
        unsigned cross = 0;
        bool ambiguous = false;
        for (int e = 0; e < 12; ++e) {
            const int c0 = c_edge_corner0(e), c1 = c0 | (1 << (e >> 2));
            cross |= (unsigned)(((in >> c0) & 1) != ((in >> c1) & 1)) << e;
        }
        for (int f = 0; f < 6; ++f) {
            const int a = f >> 1, s = f & 1, u = (a + 1) % 3, v = (a + 2) % 3, b = s << a;
            const int q[4] = {b, b | (1 << (s ? u : v)), b | (1 << u) | (1 << v), b | (1 << (s ? v : u))};
            int k = 0, st = -1, en = -1;
            for (int i = 0; i < 4; ++i) {
                const int i0 = (in >> q[i]) & 1, i1 = (in >> q[(i + 1) & 3]) & 1;
                k += i0 != i1;
                if (i0 && !i1) st = c_edge_of(q[i], q[(i + 1) & 3]);
                if (!i0 && i1) en = c_edge_of(q[i], q[(i + 1) & 3]);
            }
            if (k == 2) next[st] = en;
            ambiguous |= k == 4;
        }
        if (ambiguous) {
            T.ntri[in] = kAmbiguous;
            continue;
        }
        int n = 0;
        unsigned todo = cross;
        while (todo) {
            int e0 = 0;
            while (!((todo >> e0) & 1u)) ++e0;
            int el[12] = {}, len = 0, e = e0;
            do {
                todo &= ~(1u << e);
                el[len++] = e;
                e = next[e];
            } while (e != e0 && len < 12);
            unsigned seen = 0, twice = 0;
            for (int i = 0; i < len; ++i) {
                const unsigned f = c_edge_faces(el[i]) & c_edge_faces(el[i + 1 < len ? i + 1 : 0]);
                twice |= seen & f;
                seen |= f;
            }
            int c = 0;
            while (c < len && (c_edge_faces(el[c]) & twice)) ++c;
            if (c == len) c = 0;
            for (int i = 1; i + 1 < len; ++i, ++n) {
                T.edge[in][3 * n] = (uint8_t)el[c];
                T.edge[in][3 * n + 1] = (uint8_t)el[(c + i + 1) % len];
                T.edge[in][3 * n + 2] = (uint8_t)el[(c + i) % len];
            }
        }
        T.ntri[in] = (uint8_t)n;
    }
    return T;
}

constexpr CubeTable kCubeTable = make_cube_table();
constexpr bool table_fits() {
    for (int in = 0; in < 256; ++in)
        if (kCubeTable.ntri[in] != kAmbiguous && kCubeTable.ntri[in] > kMaxTableTris) return false;
    return true;
}
static_assert(table_fits(), "five triangles need a face decision");
__device__ const CubeTable d_cube_table = kCubeTable;

// Where a local vertex coordinate lies along one axis: the block below (0), this one (1), the next (2).
__device__ __forceinline__ int block_side(int q, int B) { return q < 0 ? 0 : (q >= B ? 2 : 1); }

// A block's place and surroundings, in shared memory.
struct McBlock {
    int slot[27];    // leaf slots of the 3^3 neighbourhood (13: the block); -1 inactive, -2 outside the grid
    float fill[27];  // an inactive neighbour's value
};

// Vertex id of edge (p, axis), p in the block's own coordinates (-1 .. B): owner block, slot, popcount
// below the slot.  -1 if the edge has no vertex (never for the edges of a cube's loops).
__device__ __forceinline__ int64_t vertex_id(const McBlock& N, int B, const int* p, int a,
                                             const uint32_t* __restrict__ bits, const int32_t* __restrict__ wpre,
                                             const int32_t* __restrict__ voff, int W) {
    int o[3] = {block_side(p[0], B), block_side(p[1], B), block_side(p[2], B)};
    int s = N.slot[o[0] * 9 + o[1] * 3 + o[2]];
    int sl;
    if (s >= 0) {
        sl = (((p[0] - (o[0] - 1) * B) * B + p[1] - (o[1] - 1) * B) * B + p[2] - (o[2] - 1) * B) * 3 + a;
    } else {
        o[a] = block_side(p[a] + 1, B);
        s = N.slot[o[0] * 9 + o[1] * 3 + o[2]];
        if (s < 0) return -1;
        const int u = a == 0 ? 1 : 0, v = a == 2 ? 1 : 2;
        sl = 3 * B * B * B + a * B * B + (p[u] - (o[u] - 1) * B) * B + p[v] - (o[v] - 1) * B;
    }
    if (voff[s] == voff[s + 1]) return -1;  // a block without a crossing has no bit words
    const int64_t at = (int64_t)s * W + (sl >> 5);
    const uint32_t word = bits[at];
    if (!((word >> (sl & 31)) & 1u)) return -1;
    return (int64_t)voff[s] + wpre[at] + __popc(word & ((1u << (sl & 31)) - 1u));
}

// Block-wide exclusive scan of one int per thread (kMcThreads); returns the prefix, *total the sum.
__device__ __forceinline__ int block_scan(int v, int* s_warp, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    int before = inc - v, sum = 0;
#pragma unroll
    for (int w = 0; w < kMcThreads / 32; ++w) {
        if (w < warp) before += s_warp[w];
        sum += s_warp[w];
    }
    *total = sum;
    __syncthreads();
    return before;
}

// Triangle (f0, f1, f2) with positions q0, q1, q2, before the end of its block's range: its signed volume
// term v0 . (v1 x v2).  A field that changed since the count pass may have more triangles than were counted.
__device__ __forceinline__ double write_triangle(int64_t at, int64_t end, const int64_t* vid, const float (*q)[3],
                                                 int32_t* __restrict__ faces, int32_t* __restrict__ err) {
    if (at >= end) return 0.0;
    if (vid[0] < 0 || vid[1] < 0 || vid[2] < 0) atomicAdd(err, 1);
    faces[3 * at] = (int32_t)vid[0];
    faces[3 * at + 1] = (int32_t)vid[1];
    faces[3 * at + 2] = (int32_t)vid[2];
    const double ax = q[0][0], ay = q[0][1], az = q[0][2], bx = q[1][0], by = q[1][1], bz = q[1][2];
    const double cx = q[2][0], cy = q[2][1], cz = q[2][2];
    return ax * (by * cz - bz * cy) + ay * (bz * cx - bx * cz) + az * (bx * cy - by * cx);
}

// One CTA per active block (grid-stride).  kEmit = false: edge bits, word prefixes, vertex and
// triangle counts.  kEmit = true: vertices, triangles and the block's volume term.  kB: the block edge
// (0: any, read from the field).
// Bound by the latency of its passes over a block, so what a block does not need is left out: most
// active blocks lie in the margin's shell and hold no crossing (the count pass ends after the staged
// signs, the emit pass at the counts); index arithmetic is 32-bit with the block edge a constant;
// corner signs are bytes; loops come from a table except where a face needs its decision; and the emit
// pass hands out triangles, not cubes, to the threads.  27 balls on 256 x 256 x 250: count 301 -> 61 us,
// emit 414 -> 60 us.  Blocks of more than kMcDense triangles, or two a cube, have enough for all threads either
// way: a cube then goes to one thread, which forms each vertex of its loops once instead of once a triangle
// (128^3 noise, blocks of 8: emit 1759 -> 750 us, 1256 when every cube went to one; of 16 2464 -> 1047, 1302).
constexpr int kMcDense = 1024;
constexpr int kMcItems = 1024;  // triangles (or undecided cubes) handed out at a time
constexpr size_t kMcStatic = kMcItems * sizeof(uint2) + 1024;  // k_mc's static shared memory is below it
static_assert(kMcItems >= kMcThreads * kMaxTableTris, "one round of cubes must fit");

template <int kB, bool kEmit>
__global__ void __launch_bounds__(kMcThreads) k_mc(McField F, const int32_t* __restrict__ active, int64_t n_active,
                                                   uint32_t* __restrict__ bits, int32_t* __restrict__ wpre,
                                                   int32_t* __restrict__ vcount, int32_t* __restrict__ tcount,
                                                   float* __restrict__ verts, int64_t* __restrict__ vkey,
                                                   int32_t* __restrict__ faces, double* __restrict__ vol_part,
                                                   int32_t* __restrict__ err, unsigned long long* __restrict__ totals) {
    extern __shared__ float s_val[];  // (B + 2)^3 values of the block and its low/high shell, then their signs
    __shared__ McBlock s_nb;
    __shared__ int s_warp[kMcThreads / 32];
    __shared__ int s_sum;
    __shared__ double s_vol[kMcThreads / 32];
    __shared__ uint2 s_item[kEmit ? kMcItems : 1];  // emit: cube | triangle << 16, offset in the block's range
    const int B = kB ? kB : F.B, R = B + 2, R3 = R * R * R;
    const int S = 3 * B * B * B + 3 * B * B, W = (S + 31) / 32;
    uint8_t* s_in = reinterpret_cast<uint8_t*>(s_val + R3);  // value < level
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t nbx = (F.nx + B - 1) / B;
    for (int64_t sa = blockIdx.x; sa < n_active; sa += gridDim.x) {
        if (kEmit && vcount[sa + 1] == vcount[sa] && tcount[sa + 1] == tcount[sa]) {
            if (threadIdx.x == 0) vol_part[sa] = 0.0;
            continue;
        }
        const int64_t id = active[sa];
        const int64_t bx = id / ((int64_t)F.nby * F.nbz), by = (id / F.nbz) % F.nby, bz = id % F.nbz;
        const int64_t o[3] = {bx * B, by * B, bz * B};
        // vertices the block's region has inside the grid, along each axis: local 0 (or -1) up to top
        const int top[3] = {(int)min((int64_t)B, F.nx - 1 - o[0]), (int)min((int64_t)B, F.ny - 1 - o[1]),
                            (int)min((int64_t)B, F.nz - 1 - o[2])};
        const int bot[3] = {o[0] > 0 ? -1 : 0, o[1] > 0 ? -1 : 0, o[2] > 0 ? -1 : 0};
        if (threadIdx.x < 27) {
            const int64_t nx_ = bx + threadIdx.x / 9 - 1, ny_ = by + (threadIdx.x / 3) % 3 - 1, nz_ = bz + threadIdx.x % 3 - 1;
            int v = -2;  // outside the grid
            float fill = 0.f;
            if (nx_ >= 0 && nx_ < nbx && ny_ >= 0 && ny_ < F.nby && nz_ >= 0 && nz_ < F.nbz) {
                const int64_t n = (nx_ * F.nby + ny_) * F.nbz + nz_;
                v = F.slot[n];
                fill = F.kind[n] < 0 ? -F.big : F.big;
            }
            s_nb.slot[threadIdx.x] = v;
            s_nb.fill[threadIdx.x] = fill;
        }
        if (threadIdx.x == 0) s_sum = 0;
        __syncthreads();
        int seen = 0;  // bit 0: a value inside, bit 1: one outside
        for (int r = threadIdx.x; r < R3; r += kMcThreads) {
            const int p[3] = {r / (R * R) - 1, (r / R) % R - 1, r % R - 1};
            float v = 0.f;
            bool in = false;
            if (p[0] >= bot[0] && p[0] <= top[0] && p[1] >= bot[1] && p[1] <= top[1] && p[2] >= bot[2] && p[2] <= top[2]) {
                const int s0 = block_side(p[0], B), s1 = block_side(p[1], B), s2 = block_side(p[2], B);
                const int nb = s0 * 9 + s1 * 3 + s2, s = s_nb.slot[nb];
                v = s < 0 ? s_nb.fill[nb]
                          : F.tiles[(int64_t)s * (B * B * B) + ((p[0] - (s0 - 1) * B) * B + p[1] - (s1 - 1) * B) * B +
                                    p[2] - (s2 - 1) * B];
                in = __dsub_rn((double)v, F.level) < 0.0;
                seen |= in ? 1 : 2;
            }
            s_val[r] = v;
            s_in[r] = in;
        }
        const bool crossed = __syncthreads_or(seen & 1) && __syncthreads_or(seen & 2);
        if (!kEmit && !crossed) {
            if (threadIdx.x == 0) {
                vcount[sa] = 0;
                tcount[sa] = 0;
            }
            __syncthreads();
            continue;
        }
        auto at = [&](const int* p) { return ((p[0] + 1) * R + p[1] + 1) * R + p[2] + 1; };
        auto val = [&](int r) { return __dsub_rn((double)s_val[r], F.level); };
        const int step[3] = {R * R, R, 1};
        // ---- edges: a warp per bit word ----
        int verts_here = 0;
        for (int w = warp; w < W; w += kMcThreads / 32) {
            const int sl = w * 32 + lane;
            uint32_t word = 0;
            if (kEmit) {
                word = bits[sa * W + w];
                if (!word) continue;
            }
            bool hit = kEmit && ((word >> lane) & 1u);
            int p[3] = {0, 0, 0}, a = 0;
            if (kEmit ? hit : sl < S) {
                if (sl < 3 * B * B * B) {
                    a = sl % 3;
                    const int lin = sl / 3;
                    p[0] = lin / (B * B);
                    p[1] = (lin / B) % B;
                    p[2] = lin % B;
                } else {
                    const int r = sl - 3 * B * B * B;
                    a = r / (B * B);
                    const int u = a == 0 ? 1 : 0, v = a == 2 ? 1 : 2;
                    p[u] = (r % (B * B)) / B;
                    p[v] = r % B;
                    p[a] = -1;
                }
                const int r = at(p);
                if (kEmit) {
                    const int64_t vid = (int64_t)vcount[sa] + wpre[sa * W + w] + __popc(word & ((1u << lane) - 1u));
                    const int64_t g[3] = {o[0] + p[0], o[1] + p[1], o[2] + p[2]};
                    edge_vertex(F, g[0], g[1], g[2], a, val(r), val(r + step[a]), verts + 3 * vid);
                    if (vkey) vkey[vid] = ((g[0] * F.ny + g[1]) * F.nz + g[2]) * 3 + a;
                } else {
                    bool ok = p[0] <= top[0] && p[1] <= top[1] && p[2] <= top[2] && p[a] >= bot[a] && p[a] + 1 <= top[a];
                    // an entering edge is ours only when its lower block is inactive
                    if (sl >= 3 * B * B * B) ok = ok && s_nb.slot[a == 0 ? 4 : (a == 1 ? 10 : 12)] < 0;
                    hit = ok && s_in[r] != s_in[r + step[a]];
                }
            }
            if (!kEmit) {
                const unsigned ball = __ballot_sync(0xffffffffu, hit);
                if (lane == 0) {
                    bits[sa * W + w] = ball;
                    wpre[sa * W + w] = __popc(ball);  // its prefix below
                }
            }
        }
        if (!kEmit) {
            __syncthreads();
            if (warp == 0) {  // exclusive prefixes of the words' counts
                for (int w0 = 0; w0 < W; w0 += 32) {
                    const int c = w0 + lane < W ? wpre[sa * W + w0 + lane] : 0;
                    int inc = c;
                    for (int d = 1; d < 32; d <<= 1) {
                        const int y = __shfl_up_sync(0xffffffffu, inc, d);
                        if (lane >= d) inc += y;
                    }
                    if (w0 + lane < W) wpre[sa * W + w0 + lane] = verts_here + inc - c;
                    verts_here += __shfl_sync(0xffffffffu, inc, 31);
                }
                if (lane == 0) {
                    vcount[sa] = verts_here;
                    if (verts_here) atomicAdd(&totals[0], (unsigned long long)verts_here);
                }
            }
        }
        // ---- cubes: lowest corners -1 .. B - 1 per axis, lexicographic ----
        const int C = B + 1, ncube = C * C * C;
        int run = 0, items = 0, tri_sum = 0;
        double vol = 0.0;
        const bool whole_cubes = kEmit && tcount[sa + 1] - tcount[sa] > min(kMcDense, 2 * ncube);
        auto corners = [&](int r, double* g) {
#pragma unroll
            for (int c = 0; c < 8; ++c) g[c] = val(r + ((c & 1) ? R * R : 0) + ((c & 2) ? R : 0) + ((c & 4) ? 1 : 0));
        };
        auto edge_point = [&](const int* m, int e, int64_t& vid, float* q) {
            const int c0 = edge_corner0(e), a = e >> 2;
            const int p[3] = {m[0] + (c0 & 1), m[1] + ((c0 >> 1) & 1), m[2] + ((c0 >> 2) & 1)};
            vid = vertex_id(s_nb, B, p, a, bits, wpre, vcount, W);
            const int r = at(p);
            edge_vertex(F, o[0] + p[0], o[1] + p[1], o[2] + p[2], a, val(r), val(r + step[a]), q);
        };
        auto flush = [&]() {  // the threads take the handed-out items
            __syncthreads();
            const int64_t base = tcount[sa], end = tcount[sa + 1];
            for (int i = threadIdx.x; i < items; i += kMcThreads) {
                const uint2 it = s_item[i];
                const int ci = it.x & 0xffff, t = it.x >> 16;
                const int m[3] = {ci / (C * C) - 1, (ci / C) % C - 1, ci % C - 1};
                const int r = at(m);
                if (t < kMaxTableTris) {
                    int in = 0;
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        in |= s_in[r + ((c & 1) ? R * R : 0) + ((c & 2) ? R : 0) + ((c & 4) ? 1 : 0)] << c;
                    int64_t vid[3];
                    float q[3][3];
                    for (int k = 0; k < 3; ++k) edge_point(m, d_cube_table.edge[in][3 * t + k], vid[k], q[k]);
                    vol += write_triangle(base + it.y, end, vid, q, faces, err);
                    continue;
                }
                double g[8];
                corners(r, g);
                const CubeLoops L = cube_loops(g);
                int64_t to = base + it.y;
                unsigned todo = L.cross;
                while (todo) {
                    const int e0 = __ffs(todo) - 1;
                    int el[12];
                    int len = 0, e = e0;
                    do {  // a permutation cycle of at most 12 edges (cube_triangles counted it)
                        todo &= ~(1u << e);
                        el[len++] = e;
                        e = loop_next(L, e);
                    } while (e >= 0 && e != e0 && len < 12);
                    // fan centre: the first vertex on no face that the loop crosses twice (a fan
                    // from such a face would lay a flat triangle into it), else the lowest edge
                    unsigned faces_seen = 0, twice = 0;
                    for (int i2 = 0; i2 < len; ++i2) {
                        const unsigned f = edge_faces(el[i2]) & edge_faces(el[i2 + 1 < len ? i2 + 1 : 0]);
                        twice |= faces_seen & f;
                        faces_seen |= f;
                    }
                    int c = 0;
                    while (c < len && (edge_faces(el[c]) & twice)) ++c;
                    if (c == len) c = 0;
                    int64_t vid[3];
                    float q[3][3];
                    edge_point(m, el[c], vid[0], q[0]);
                    edge_point(m, el[c + 1 < len ? c + 1 : c + 1 - len], vid[2], q[2]);
                    for (int i2 = 2; i2 < len; ++i2) {  // each vertex of the loop once
                        const int j = c + i2 < len ? c + i2 : c + i2 - len;
                        edge_point(m, el[j], vid[1], q[1]);
                        vol += write_triangle(to++, end, vid, q, faces, err);
                        vid[2] = vid[1];
#pragma unroll
                        for (int a = 0; a < 3; ++a) q[2][a] = q[1][a];
                    }
                }
            }
            __syncthreads();
            items = 0;
        };
        for (int c0 = 0; c0 < ncube; c0 += kMcThreads) {
            const int ci = c0 + threadIdx.x;
            int ntri = 0, n_items = 0;
            if (ci < ncube) {
                const int m[3] = {ci / (C * C) - 1, (ci / C) % C - 1, ci % C - 1};
                bool ok = true;
#pragma unroll
                for (int a = 0; a < 3; ++a) ok &= m[a] >= bot[a] && m[a] + 1 <= top[a];
                int in = 0;
                const int r = at(m);
                if (ok) {
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        in |= s_in[r + ((c & 1) ? R * R : 0) + ((c & 2) ? R : 0) + ((c & 4) ? 1 : 0)] << c;
                    ok = in != 0 && in != 255;
                }
                if (ok && (m[0] < 0 || m[1] < 0 || m[2] < 0)) {
                    // a cube reaching into the low shell: ours if its first corner in an active block is here
                    int first = -1;
                    for (int c = 0; c < 8 && first < 0; ++c) {
                        const int nb = block_side(m[0] + (c & 1), B) * 9 + block_side(m[1] + ((c >> 1) & 1), B) * 3 +
                                       block_side(m[2] + ((c >> 2) & 1), B);
                        if (s_nb.slot[nb] >= 0) first = nb;
                    }
                    ok = first == 13;
                }
                if (ok) {
                    ntri = n_items = d_cube_table.ntri[in];
                    if (ntri == kAmbiguous) {
                        double g[8];
                        corners(r, g);
                        ntri = cube_triangles(cube_loops(g));
                        n_items = ntri ? kMaxTableTris + 1 : 0;  // marks one item for the whole cube
                    } else if (kEmit && whole_cubes && ntri) {
                        n_items = kMaxTableTris + 1;
                    }
                }
            }
            if (!kEmit) {
                tri_sum += ntri;
                continue;
            }
            const int put = n_items > kMaxTableTris ? 1 : n_items;
            int total;
            const int before = block_scan(put << 16 | ntri, s_warp, &total);  // at most 1024 items, 3072 triangles
            if (items + (total >> 16) > kMcItems) flush();
            for (int t = 0; t < put; ++t)
                s_item[items + (before >> 16) + t] =
                    make_uint2((uint32_t)ci | (uint32_t)(n_items > kMaxTableTris ? kMaxTableTris : t) << 16,
                               (uint32_t)(run + (before & 0xffff) + t));
            items += total >> 16;
            run += total & 0xffff;
        }
        if (!kEmit) {
            for (int d = 16; d > 0; d >>= 1) tri_sum += __shfl_xor_sync(0xffffffffu, tri_sum, d);
            if (lane == 0 && tri_sum) atomicAdd(&s_sum, tri_sum);
            __syncthreads();
            if (threadIdx.x == 0) {
                tcount[sa] = s_sum;
                if (s_sum) atomicAdd(&totals[1], (unsigned long long)s_sum);
            }
        } else {
            flush();
            if (threadIdx.x == 0 && run != tcount[sa + 1] - tcount[sa]) atomicAdd(err, 1);
            for (int d = 16; d > 0; d >>= 1) vol += __shfl_xor_sync(0xffffffffu, vol, d);
            if (lane == 0) s_vol[warp] = vol;
            __syncthreads();
            if (threadIdx.x == 0) {
                double t = 0.0;
                for (int w = 0; w < kMcThreads / 32; ++w) t += s_vol[w];
                vol_part[sa] = t;
            }
        }
        __syncthreads();
    }
}

// Sum of the blocks' volume terms in block order (one CTA, fixed tree): deterministic.
__global__ void k_mc_volume(const double* __restrict__ part, int64_t n, double* __restrict__ out) {
    __shared__ double s[kMcThreads];
    double t = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += kMcThreads) t += part[i];
    s[threadIdx.x] = t;
    __syncthreads();
    for (int o = kMcThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = s[0] / 6.0;
}

__global__ void k_mc_slot_map(const int32_t* __restrict__ active, int64_t n_active, int32_t* __restrict__ slot) {
    const int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (a < n_active) slot[active[a]] = (int32_t)a;
}

int mc_field(McField& F, const int32_t* d_kind, const float* d_tiles, int64_t nx, int64_t ny, int64_t nz, int32_t block,
             double ox, double oy, double oz, double pitch, double level, float big, const int32_t* d_slot) {
    if (!d_kind || !d_slot || nx < 1 || ny < 1 || nz < 1 || block < 1 || block > kMcMaxBlock ||
        !(pitch > 0) || !(level == level) || level > 1e300 || level < -1e300)
        return FB_INVALID;
    F = McField{d_kind, d_slot, d_tiles, nx, ny, nz, block, (int)((ny + block - 1) / block),
                (int)((nz + block - 1) / block), ox, oy, oz, pitch, level, big};
    return FB_OK;
}

size_t mc_smem(int B) { return (size_t)(B + 2) * (B + 2) * (B + 2) * (sizeof(float) + 1); }

template <int kB, bool kEmit>
int mc_launch_block(const McField& F, const int32_t* d_active, int64_t n_active, uint32_t* bits, int32_t* wpre,
              int32_t* vcount, int32_t* tcount, float* verts, int64_t* vkey, int32_t* faces, double* vol_part,
              int32_t* err, unsigned long long* totals, cudaStream_t st) {
    if (n_active == 0) return FB_OK;
    const size_t smem = mc_smem(F.B);
    // the limit without the opt-in is on the static and the dynamic part together
    if (smem + kMcStatic > 48 * 1024) FB_CUDA(cudaFuncSetAttribute(k_mc<kB, kEmit>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int grid = (int)std::min<int64_t>(n_active, (int64_t)fb_sm_count() * 8);
    k_mc<kB, kEmit><<<grid, kMcThreads, smem, st>>>(F, d_active, n_active, bits, wpre, vcount, tcount, verts, vkey,
                                                   faces, vol_part, err, totals);
    FB_LAUNCH();
    return FB_OK;
}

template <bool kEmit>
int mc_launch(const McField& F, const int32_t* d_active, int64_t n_active, uint32_t* bits, int32_t* wpre,
              int32_t* vcount, int32_t* tcount, float* verts, int64_t* vkey, int32_t* faces, double* vol_part,
              int32_t* err, unsigned long long* totals, cudaStream_t st) {
#define FB_MC(BB) mc_launch_block<BB, kEmit>(F, d_active, n_active, bits, wpre, vcount, tcount, verts, vkey, faces, \
                                             vol_part, err, totals, st)
    switch (F.B) {
    case 4: return FB_MC(4);
    case 8: return FB_MC(8);
    case 16: return FB_MC(16);
    default: return FB_MC(0);
    }
#undef FB_MC
}

// ---- connected components of the exported mesh (faltvolym_v1.py:95-101 keeps the largest) ----
// Union-find over the vertices, a thread per triangle; a root is always linked under the smaller
// root, so parent[v] <= v, every chain ends, and a component's final root is its smallest vertex id
// whatever the order of the unions.  Reads go through volatile pointers (other threads link and
// halve paths meanwhile); path halving only writes ancestors into non-roots.
constexpr int kUnionTries = 1 << 16;

__device__ __forceinline__ int32_t cc_find(volatile int32_t* parent, int32_t x) {
    while (true) {  // strictly decreasing ids: at most x steps
        const int32_t p = parent[x];
        if (p == x) return x;
        const int32_t gp = parent[p];
        if (gp != p) parent[x] = gp;
        x = gp;
    }
}

__device__ __forceinline__ void cc_union(int32_t* parent, int32_t a, int32_t b, int32_t* err) {
    for (int it = 0; it < kUnionTries; ++it) {
        a = cc_find(parent, a);
        b = cc_find(parent, b);
        if (a == b) return;
        if (a < b) {
            const int32_t t = a;
            a = b;
            b = t;
        }
        const int32_t old = atomicCAS(parent + a, a, b);
        if (old == a) return;
        a = old;  // linked meanwhile: continue from its new parent
    }
    atomicAdd(err, 1);
}

__global__ void k_cc_init(int32_t* __restrict__ parent, double* __restrict__ vol, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) {
        parent[i] = (int32_t)i;
        vol[i] = 0.0;
    }
}

__global__ void k_cc_union(const int32_t* __restrict__ faces, int64_t nf, int32_t* parent, int32_t* err) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nf) return;
    cc_union(parent, faces[3 * t], faces[3 * t + 1], err);
    cc_union(parent, faces[3 * t], faces[3 * t + 2], err);
}

__global__ void k_cc_label(int32_t* parent, int64_t n, int32_t* __restrict__ count) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t r = cc_find(parent, (int32_t)i);
    if (r == (int32_t)i) atomicAdd(count, 1);
}

__global__ void k_cc_flatten(const int32_t* __restrict__ parent, int64_t n, int32_t* __restrict__ label) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    int32_t x = (int32_t)i;
    while (parent[x] != x) x = parent[x];  // stable parents: decreasing ids
    label[i] = x;
}

// Volume of each component, at its root: sum over its triangles of v0 . (v1 x v2) / 6.
__global__ void k_cc_volume(const int32_t* __restrict__ faces, int64_t nf, const float* __restrict__ verts,
                            const int32_t* __restrict__ label, double* __restrict__ vol) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nf) return;
    const float* a = verts + 3 * (int64_t)faces[3 * t];
    const float* b = verts + 3 * (int64_t)faces[3 * t + 1];
    const float* c = verts + 3 * (int64_t)faces[3 * t + 2];
    const double ax = a[0], ay = a[1], az = a[2], bx = b[0], by = b[1], bz = b[2], cx = c[0], cy = c[1], cz = c[2];
    const double term = ax * (by * cz - bz * cy) + ay * (bz * cx - bx * cz) + az * (bx * cy - by * cx);
    atomicAdd(vol + label[faces[3 * t]], term / 6.0);
}

}  // namespace

extern "C" {

// Connected components of a triangle mesh (faces: 3 int32 vertex ids each, < n_verts): d_label[v]
// = the smallest vertex id of v's component (n_verts int32), d_count[0] = number of components
// (isolated vertices count as components), d_comp_volume[r] = signed volume of the component with
// root r (n_verts float64; other entries 0; summed with atomics, so the last bits may depend on
// the order of the additions), d_err[0] = unions that gave up (0).  d_parent: n_verts int32 scratch.
int fb_mesh_components_device(const int32_t* d_faces, int64_t n_faces, const float* d_verts, int64_t n_verts,
                              int32_t* d_parent, int32_t* d_label, double* d_comp_volume, int32_t* d_count,
                              int32_t* d_err, void* stream) noexcept {
    if (n_faces < 0 || n_verts < 0 || n_verts > INT32_MAX || !d_count || !d_err ||
        (n_faces > 0 && (!d_faces || !d_verts)) || (n_verts > 0 && (!d_parent || !d_label || !d_comp_volume)))
        return FB_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    FB_CUDA(cudaMemsetAsync(d_count, 0, 4, st));
    FB_CUDA(cudaMemsetAsync(d_err, 0, 4, st));
    if (n_verts == 0) return FB_OK;
    k_cc_init<<<fb_div_up(n_verts, 256), 256, 0, st>>>(d_parent, d_comp_volume, n_verts);
    FB_LAUNCH();
    if (n_faces > 0) {
        k_cc_union<<<fb_div_up(n_faces, 256), 256, 0, st>>>(d_faces, n_faces, d_parent, d_err);
        FB_LAUNCH();
    }
    k_cc_label<<<fb_div_up(n_verts, 256), 256, 0, st>>>(d_parent, n_verts, d_count);
    FB_LAUNCH();
    k_cc_flatten<<<fb_div_up(n_verts, 256), 256, 0, st>>>(d_parent, n_verts, d_label);
    FB_LAUNCH();
    if (n_faces > 0) {
        k_cc_volume<<<fb_div_up(n_faces, 256), 256, 0, st>>>(d_faces, n_faces, d_verts, d_label, d_comp_volume);
        FB_LAUNCH();
    }
    return FB_OK;
}

// Bit words per active block of the edge map (3 B^3 + 3 B^2 slots).
int64_t fb_mc_words(int32_t block) { return block >= 1 && block <= kMcMaxBlock ? mc_words(block) : -1; }

// Scratch int32 words the count pass's scans need for n_active blocks.
int64_t fb_mc_scan_words(int64_t n_active) { return n_active < 0 ? -1 : scan_scratch_words(n_active + 1) + 1; }

// Pass 1 of the export mesh (faltkarna_v1.py:302-350 + marching cubes): the slot map (d_slot,
// n_blocks int32), each active block's edge bits and word prefixes (d_bits, d_wpre: n_active x
// fb_mc_words), and in d_vcount / d_tcount (n_active + 1 int32 each) the exclusive offsets of the
// blocks' vertices and triangles, their totals in the last entry, and the same totals in 64 bits in
// d_totals[0..1] (the int32 offsets are valid while both stay below 2^31; the caller checks them).
// Stream-ordered; block <= 32.  Status 1 for invalid arguments.
int fb_mc_count_device(const int32_t* d_kind, const int32_t* d_active, int64_t n_active, const float* d_tiles,
                       int64_t nx, int64_t ny, int64_t nz, int32_t block, double ox, double oy, double oz,
                       double pitch, double level, float big, int32_t* d_slot, uint32_t* d_bits, int32_t* d_wpre,
                       int32_t* d_vcount, int32_t* d_tcount, int64_t* d_totals, int32_t* d_scan,
                       int64_t scan_words, void* stream) noexcept {
    McField F;
    if (int rc = mc_field(F, d_kind, d_tiles, nx, ny, nz, block, ox, oy, oz, pitch, level, big, d_slot)) return rc;
    if (n_active < 0 || !d_vcount || !d_tcount || !d_scan || !d_totals ||
        (n_active > 0 && (!d_active || !d_tiles || !d_bits || !d_wpre)))
        return FB_INVALID;
    if (scan_words < scan_scratch_words(n_active + 1) + 1) return FB_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t nblocks = ((nx + block - 1) / block) * F.nby * F.nbz;
    FB_CUDA(cudaMemsetAsync(d_slot, 0xff, nblocks * 4, st));
    if (n_active > 0) {
        k_mc_slot_map<<<fb_div_up(n_active, 256), 256, 0, st>>>(d_active, n_active, d_slot);
        FB_LAUNCH();
    }
    FB_CUDA(cudaMemsetAsync(d_vcount + n_active, 0, 4, st));
    FB_CUDA(cudaMemsetAsync(d_tcount + n_active, 0, 4, st));
    FB_CUDA(cudaMemsetAsync(d_totals, 0, 16, st));
    if (int rc = mc_launch<false>(F, d_active, n_active, d_bits, d_wpre, d_vcount, d_tcount, nullptr, nullptr,
                                  nullptr, nullptr, nullptr, reinterpret_cast<unsigned long long*>(d_totals), st))
        return rc;
    if (int rc = scan_exclusive(d_vcount, n_active + 1, d_scan, d_scan + 1, scan_words - 1, st)) return rc;
    if (int rc = scan_exclusive(d_tcount, n_active + 1, d_scan, d_scan + 1, scan_words - 1, st)) return rc;
    return FB_OK;
}

// Pass 2: vertices (float32 x, y, z world coordinates, d_vcount[n_active] of them; d_vkey, if not
// null, the vertex's edge as (linear index of its lower end) * 3 + axis), triangles
// (int32 vertex ids, d_tcount[n_active] of them, outward normals) and the enclosed volume
// sum(v0 . (v1 x v2)) / 6 in float64 (d_volume[0]; d_vol_part: n_active float64 scratch), summed in a
// fixed order.  The arguments of pass 1 unchanged.  d_err[0] counts triangle corners without a
// vertex and blocks with another number of triangles than pass 1 counted (0 unless the field changed in
// between; such corners are -1, and nothing is written beyond the counted totals).
int fb_mc_emit_device(const int32_t* d_kind, const int32_t* d_active, int64_t n_active, const float* d_tiles,
                      int64_t nx, int64_t ny, int64_t nz, int32_t block, double ox, double oy, double oz, double pitch,
                      double level, float big, const int32_t* d_slot, const uint32_t* d_bits, const int32_t* d_wpre,
                      const int32_t* d_vcount, const int32_t* d_tcount, float* d_verts, int64_t* d_vkey,
                      int32_t* d_faces, double* d_vol_part, double* d_volume, int32_t* d_err, void* stream) noexcept {
    McField F;
    if (int rc = mc_field(F, d_kind, d_tiles, nx, ny, nz, block, ox, oy, oz, pitch, level, big, d_slot)) return rc;
    if (n_active < 0 || !d_vcount || !d_tcount || !d_volume || !d_err ||
        (n_active > 0 && (!d_active || !d_tiles || !d_bits || !d_wpre || !d_vol_part)))
        return FB_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    FB_CUDA(cudaMemsetAsync(d_err, 0, 4, st));
    if (int rc = mc_launch<true>(F, d_active, n_active, const_cast<uint32_t*>(d_bits), const_cast<int32_t*>(d_wpre),
                                 const_cast<int32_t*>(d_vcount), const_cast<int32_t*>(d_tcount), d_verts, d_vkey,
                                 d_faces, d_vol_part, d_err, nullptr, st))
        return rc;
    k_mc_volume<<<1, kMcThreads, 0, st>>>(d_vol_part, n_active, d_volume);
    FB_LAUNCH();
    return FB_OK;
}

}  // extern "C"
