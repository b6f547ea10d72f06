// mcwords.cuh — the word machinery of every marching-cubes variant.
//
// A grid's points are grouped in row-aligned 32-point words of sign bits.  Words
// are numbered in raster order, so vertex and triangle numbers are prefix sums
// over words.  A variant supplies a policy (its grid geometry, tilings and vertex
// arithmetic); this file counts, numbers and emits:
//
//   k_words   edge-crossing masks of every word and the counts that follow from
//             signs alone; marks the voxels whose exact values will be read.  A
//             warp takes 32 words (a sub-tile) and turns their mixed cubes into
//             one dense list (a cube per lane), so that neither an empty word nor a
//             full one costs its neighbours time; warps never wait for one another.
//   k_amb     the face and interior tests of the ambiguous cubes, which need values
//             (so with the exact smoothing on demand they come after the repair): a
//             block lists the words of 32 sub-tiles that hold any, then takes them a
//             cube per lane.
//   k_sum     sums of the sub-tiles, scanned per tile of 256 in the block; the last
//             block to finish scans the tiles.
//   k_finish  the active words (those that own output) as one list in word order
//             with their absolute triangle and c-vertex offsets; the words'
//             vertex offsets become absolute.
//   k_emit    a warp takes G active words, numbers their vertices and cubes
//             densely and emits them with all lanes busy; triangles pass through
//             a small queue because cubes make different numbers of them.
//
// A word's record is one uint4 {x, y, z crossing masks, vertex offset}: a
// triangle corner finds its vertex id with one 16-byte load.  Inactive words have
// no record: nothing refers to them.
//
// Measured on a 512^3 CT volume (7.6 M triangles, 4.5 M words, cold caches): masks,
// marks, counts, scan and active list 290 -> 150 us (k_words 85: a block scan per 256
// words had cost 120, waiting for the block's fullest warp); emit 474 -> 207 us
// against one lane per word listing its cubes for the warp, with separate mask and
// offset arrays and the ambiguous tests repeated.  Two emit kernels (vertices,
// triangles) took 255, two vertices per lane in flight 250.  On the brain volume
// (0.2 M triangles, 1.7 k groups of 32 words for 5 k resident warps) the emit went
// from 157 to 23 us with smaller groups.
#pragma once
#include <algorithm>
#include <atomic>

#include "n2m_internal.cuh"

namespace mcw {
constexpr unsigned FULL = 0xffffffffu;
constexpr int SUB = 32;           // words per sub-tile
constexpr int TILE = 256;         // sub-tiles per tile

// bits [lo, hi) of a word, clipped to it
__device__ __forceinline__ unsigned bit_range(int lo, int hi) {
    if (hi <= 0 || lo >= 32 || hi <= lo) return 0u;
    const unsigned h = hi >= 32 ? FULL : (1u << hi) - 1u, l = lo <= 0 ? 0u : (1u << lo) - 1u;
    return h & ~l;
}
// position of the r-th (from 0) set bit of m, which has more than r
__device__ __forceinline__ int nth_bit(unsigned m, int r) {
    int p = 0;
#pragma unroll
    for (int s = 16; s; s >>= 1) {
        const int c = __popc(m & ((1u << s) - 1u));
        if (r >= c) {
            r -= c;
            m >>= s;
            p += s;
        }
    }
    return p;
}
// the lane whose items hold number k, given every lane's first item number
__device__ __forceinline__ int find_lane(const unsigned *pre, unsigned k) {
    int l = 0;
#pragma unroll
    for (int s = 16; s; s >>= 1)
        if (pre[l + s] <= k) l += s;
    return l;
}
__device__ __forceinline__ unsigned warp_excl(unsigned v, int lane, unsigned &total) {
    unsigned i = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(FULL, i, o);
        if (lane >= o) i += t;
    }
    total = __shfl_sync(FULL, i, 31);
    return i - v;
}

// one word of a grid
struct Geo {
    int x0, y, z;         // grid point of bit 0 (x0 may be negative: bits before the grid)
    unsigned WX, slice;   // words per row and slice of its grid
    unsigned inm, hxm;    // bits of grid points; of those with a +x neighbour
    bool hy, hz, nx;      // a row, a slice, a word of the row follows
    int tag;              // the policy's own (box number, interior flag)
};

// sign words of a word's cubes: a = (y, z), b = (y+1, z), c = (y, z+1), d = (y+1, z+1), and bit 0 of the word after
// each (nxt bits 0..3)
struct Corners {
    unsigned a, b, c, d, nxt;
};
__device__ __forceinline__ Corners load_corners(const unsigned *__restrict__ signs, unsigned w, const Geo &g) {
    Corners q{__ldg(signs + w), 0u, 0u, 0u, 0u};
    if (g.nx) q.nxt = __ldg(signs + w + 1) & 1u;
    if (g.hy) {
        q.b = __ldg(signs + w + g.WX);
        if (g.nx) q.nxt |= (__ldg(signs + w + g.WX + 1) & 1u) << 1;
    }
    if (g.hz) {
        q.c = __ldg(signs + w + g.slice);
        if (g.nx) q.nxt |= (__ldg(signs + w + g.slice + 1) & 1u) << 2;
    }
    if (g.hy && g.hz) {
        q.d = __ldg(signs + w + g.slice + g.WX);
        if (g.nx) q.nxt |= (__ldg(signs + w + g.slice + g.WX + 1) & 1u) << 3;
    }
    return q;
}
__device__ __forceinline__ unsigned plus_x(unsigned w, unsigned next) { return w >> 1 | next << 31; }
// cubes whose corner signs differ
__device__ __forceinline__ unsigned mixed_cubes(const Corners &q, const Geo &g) {
    if (!(g.hy && g.hz)) return 0u;
    const unsigned a1 = plus_x(q.a, q.nxt), b1 = plus_x(q.b, q.nxt >> 1), c1 = plus_x(q.c, q.nxt >> 2), d1 = plus_x(q.d, q.nxt >> 3);
    return (q.a | a1 | q.b | b1 | q.c | c1 | q.d | d1) & ~(q.a & a1 & q.b & b1 & q.c & c1 & q.d & d1) & g.hxm;
}
// the tables' corner order (x,y,z) (x+1,y,z) (x+1,y+1,z) (x,y+1,z) and the same at z+1
__device__ __forceinline__ int cube_index(unsigned a, unsigned b, unsigned c, unsigned d, unsigned nxt, int i) {
    const unsigned pa = __funnelshift_r(a, nxt & 1u, i) & 3u, pb = __funnelshift_r(b, nxt >> 1 & 1u, i) & 3u,
                   pc = __funnelshift_r(c, nxt >> 2 & 1u, i) & 3u, pd = __funnelshift_r(d, nxt >> 3 & 1u, i) & 3u;
    return (int)(pa | (pb >> 1 | (pb & 1u) << 1) << 2 | pc << 4 | (pd >> 1 | (pd & 1u) << 1) << 6);
}

// The tiling of one cube: offset of its edge codes, triangles, whether it has a c-vertex
struct CubeTiling {
    int off, n;
    bool cv;
};
constexpr unsigned TESTS = 0xffu;   // quick(): the tiling depends on corner values

// what the count pass leaves behind (see McWork)
struct Out {
    uint4 *words;      // per active word (its vertex offset within the sub-tile until k_finish)
    unsigned *cnt;     // per active word, triangles | c-vertices << 16
    unsigned *amb;     // per active word, its ambiguous cubes
    unsigned *ambat;   // per word with any, its first entry in tilings
    unsigned *tilings; // of the ambiguous cubes: code offset | triangles << 22 | c-vertex << 26; nwords entries
    uint4 *sub;        // per sub-tile {vertices, its active words, its words with ambiguous cubes, -}
    uint4 *pre;        // per sub-tile, what precedes it in its tile {vertices, triangles, c-vertices, active words}
    uint4 *part;       // per tile, what precedes it, likewise
    uint4 *total;
    unsigned *ctr;     // tiles finished, group counter of the emit, tilings
    unsigned nwords, nsub;
};

__device__ __forceinline__ uint4 add4(uint4 a, uint4 b) { return make_uint4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// marks voxels of a volume in a bitmap of row-aligned words (bit x & 31 of word (z*ny + y)*W + x/32): word wx of row
// (y, z), of which y may be one row and z one slice past the volume, and bit nx of a row its padding column (they wrap
// into the next row or slice as the padded grid reads them, src/MarchingCubes.c:1097-1115)
struct Marks {
    unsigned *need;         // null: none wanted
    int nx, ny, nz;
    unsigned W;
    __device__ __forceinline__ void put(int wx, int y, int z, unsigned bits) const {
        if (!bits) return;
        if (y >= ny) {
            y -= ny;
            z++;
        }
        if (z >= nz) return;
        const int p = nx - 32 * wx;   // bit of the padding column
        const unsigned in = bits & bit_range(0, p);
        if (in) atomicOr(need + ((size_t)z * ny + y) * W + wx, in);
        if (p >= 0 && p < 32 && (bits >> p & 1u)) {
            if (++y >= ny) {
                y -= ny;
                z++;
            }
            if (z < nz) atomicOr(need + ((size_t)z * ny + y) * W, 1u);
        }
    }
};

template <class P>
__global__ void __launch_bounds__(256) k_words(P pol, const unsigned *__restrict__ signs, Out o, Marks marks) {
    grid_wait();
    __shared__ unsigned qt[256], pre[8][32], cor[8][6][32], cnt[8][32], amb[8][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    qt[threadIdx.x] = pol.quick(threadIdx.x);
    __syncthreads();
    for (unsigned sub = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; sub < o.nsub; sub += (gridDim.x * blockDim.x) >> 5) {
        const unsigned w = sub * SUB + (unsigned)lane;
        unsigned xm = 0, ym = 0, zm = 0, mix = 0;
        Geo g;
        if (w < o.nwords && pol.geo(w, g)) {
            const Corners q = load_corners(signs, w, g);
            xm = (q.a ^ plus_x(q.a, q.nxt)) & g.hxm;
            ym = g.hy ? (q.a ^ q.b) & g.inm : 0u;
            zm = g.hz ? (q.a ^ q.c) & g.inm : 0u;
            mix = mixed_cubes(q, g);
            if (mix) {
                cor[wid][0][lane] = q.a;
                cor[wid][1][lane] = q.b;
                cor[wid][2][lane] = q.c;
                cor[wid][3][lane] = q.d;
                cor[wid][4][lane] = q.nxt;
                cor[wid][5][lane] = mix;
            }
        }
        const unsigned nv = __popc(xm) + __popc(ym) + __popc(zm);
        const bool act = (nv | mix) != 0u;
        const unsigned acts = __ballot_sync(FULL, act);
        if (!acts) {
            if (lane == 0) o.sub[sub] = make_uint4(0u, 0u, 0u, 0u);
            continue;
        }
        cnt[wid][lane] = 0u;
        amb[wid][lane] = 0u;
        unsigned both;   // vertices | cubes << 16
        const unsigned ex = warp_excl(nv | __popc(mix) << 16, lane, both);
        const unsigned ncube = both >> 16;
        pre[wid][lane] = ex >> 16;
        __syncwarp();
        for (unsigned k = lane; k < ncube; k += 32) {
            const int l = find_lane(pre[wid], k);
            const int i = nth_bit(cor[wid][5][l], (int)(k - pre[wid][l]));
            const int lut = cube_index(cor[wid][0][l], cor[wid][1][l], cor[wid][2][l], cor[wid][3][l], cor[wid][4][l], i);
            const unsigned n = qt[lut] & 0xffu;
            if (n == TESTS) atomicOr(&amb[wid][l], 1u << i);
            else atomicAdd(&cnt[wid][l], n);
        }
        __syncwarp();
        const unsigned am = amb[wid][lane], ambs = __ballot_sync(FULL, am != 0u);
        if (lane == 0) o.sub[sub] = make_uint4(both & 0xffffu, acts, ambs, 0u);
        if (act) {
            o.words[w] = make_uint4(xm, ym, zm, ex & 0xffffu);
            o.cnt[w] = cnt[wid][lane];
            if (P::CVERTS) o.amb[w] = am;
            if (marks.need) {   // both ends of every crossing edge; every corner of the ambiguous cubes
                int wx, vy, vz;
                pol.voxel_word(g, wx, vy, vz);
                const unsigned am2 = am | am << 1;
                marks.put(wx, vy, vz, xm | xm << 1 | ym | zm | am2);
                if ((xm | am) >> 31) marks.put(wx + 1, vy, vz, 1u);
                marks.put(wx, vy + 1, vz, ym | am2);
                marks.put(wx, vy, vz + 1, zm | am2);
                if (am) {
                    marks.put(wx, vy + 1, vz + 1, am2);
                    if (am >> 31) {
                        marks.put(wx + 1, vy + 1, vz, 1u);
                        marks.put(wx + 1, vy, vz + 1, 1u);
                        marks.put(wx + 1, vy + 1, vz + 1, 1u);
                    }
                }
            }
        }
        __syncwarp();   // the shared lists are reused
    }
}

constexpr unsigned NO_TILING = 0xffffffffu;
constexpr int AMB_T = 128, AMB_S = 32, AMB_W = 8;   // threads of k_amb, sub-tiles of a block, words of a warp at a time
template <class P>
__global__ void __launch_bounds__(AMB_T) k_amb(P pol, const unsigned *__restrict__ signs, Out o) {
    grid_wait();
    __shared__ unsigned short list[AMB_S * SUB];
    __shared__ unsigned nlist, pre[4][32], cor[4][6][32], words[4][32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) nlist = 0u;
    __syncthreads();
    const unsigned sub = blockIdx.x * AMB_S + (unsigned)tid, w0 = blockIdx.x * AMB_S * SUB;
    unsigned m = tid < AMB_S && sub < o.nsub ? o.sub[sub].z : 0u;
    if (m) {
        unsigned at = atomicAdd(&nlist, (unsigned)__popc(m));
        for (; m; m &= m - 1) list[at++] = (unsigned short)(tid * SUB + __ffs(m) - 1);
    }
    __syncthreads();
    const unsigned n = nlist;
    for (unsigned a0 = (unsigned)wid * AMB_W; a0 < n; a0 += AMB_W * AMB_T / 32) {
        unsigned am = 0;
        if (lane < AMB_W && a0 + (unsigned)lane < n) {
            const unsigned w = w0 + list[a0 + lane];
            Geo g;
            pol.geo(w, g);
            const Corners q = load_corners(signs, w, g);
            am = o.amb[w];
            words[wid][lane] = w;
            cor[wid][0][lane] = q.a;
            cor[wid][1][lane] = q.b;
            cor[wid][2][lane] = q.c;
            cor[wid][3][lane] = q.d;
            cor[wid][4][lane] = q.nxt;
            cor[wid][5][lane] = am;
        }
        unsigned ncube, at = 0;
        pre[wid][lane] = warp_excl(__popc(am), lane, ncube);
        if (lane == 0) at = atomicAdd(o.ctr + 2, ncube);
        at = __shfl_sync(FULL, at, 0);
        const bool room = at + ncube <= o.nwords;          // else the emit repeats the tests
        if (am) o.ambat[words[wid][lane]] = room ? at + pre[wid][lane] : NO_TILING;
        __syncwarp();
        for (unsigned k = lane; k < ncube; k += 32) {
            const int l = find_lane(pre[wid], k);
            const int i = nth_bit(cor[wid][5][l], (int)(k - pre[wid][l]));
            const int lut = cube_index(cor[wid][0][l], cor[wid][1][l], cor[wid][2][l], cor[wid][3][l], cor[wid][4][l], i);
            Geo g;
            pol.geo(words[wid][l], g);
            const CubeTiling T = pol.tests(g, g.x0 + i, g.y, g.z, lut);
            atomicAdd(o.cnt + words[wid][l], (unsigned)T.n | (T.cv ? 1u << 16 : 0u));
            if (room) o.tilings[at + k] = (unsigned)T.off | (unsigned)T.n << 22 | (T.cv ? 1u << 26 : 0u);
        }
        __syncwarp();
    }
}

__device__ __forceinline__ uint4 warp_incl4(uint4 v, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        uint4 t;
        t.x = __shfl_up_sync(FULL, v.x, d); t.y = __shfl_up_sync(FULL, v.y, d);
        t.z = __shfl_up_sync(FULL, v.z, d); t.w = __shfl_up_sync(FULL, v.w, d);
        if (lane >= d) v = add4(v, t);
    }
    return v;
}
// exclusive scan over a block of 256, *all: its total
__device__ __forceinline__ uint4 block_excl4(uint4 v, uint4 *wsum, int lane, int wid, uint4 *all) {
    const uint4 in = warp_incl4(v, lane);
    if (lane == 31) wsum[wid] = in;
    __syncthreads();
    uint4 before = make_uint4(in.x - v.x, in.y - v.y, in.z - v.z, in.w - v.w), t = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        if (k < wid) before = add4(before, wsum[k]);
        t = add4(t, wsum[k]);
    }
    *all = t;
    return before;
}

// (a template only so that each unit has its own)
template <class P>
__global__ void __launch_bounds__(TILE) k_sum(Out o) {
    grid_wait();
    __shared__ uint4 wsum[8];
    __shared__ bool last;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const unsigned s = blockIdx.x * TILE + (unsigned)tid;
    const uint4 rec = s < o.nsub ? o.sub[s] : make_uint4(0u, 0u, 0u, 0u);
    unsigned mine = 0;   // this lane's sub-tile: triangles (at most 12288) | c-vertices << 16
    if (rec.y) {         // its 32 counts at once (only those of active words are set)
        const uint4 *c4 = (const uint4 *)(o.cnt + (size_t)s * SUB);
        uint4 c[SUB / 4];
#pragma unroll
        for (int q = 0; q < SUB / 4; q++) c[q] = __ldg(c4 + q);
#pragma unroll
        for (int q = 0; q < SUB / 4; q++) {
            const unsigned m = rec.y >> (4 * q);
            mine += (m & 1u ? c[q].x : 0u) + (m & 2u ? c[q].y : 0u) + (m & 4u ? c[q].z : 0u) + (m & 8u ? c[q].w : 0u);
        }
    }
    uint4 all;
    const uint4 before = block_excl4(make_uint4(rec.x, mine & 0xffffu, mine >> 16, (unsigned)__popc(rec.y)), wsum, lane, wid, &all);
    if (s < o.nsub) o.pre[s] = before;
    if (tid == 0) {
        o.part[blockIdx.x] = all;
        __threadfence();
        last = atomicAdd(o.ctr, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const unsigned n = gridDim.x, each = (n + TILE - 1) / TILE, p0 = min(n, (unsigned)tid * each), p1 = min(n, p0 + each);
    uint4 sum = make_uint4(0u, 0u, 0u, 0u);
    for (unsigned k = p0; k < p1; k++) sum = add4(sum, __ldcg(o.part + k));
    uint4 at = block_excl4(sum, wsum, lane, wid, &all);
    for (unsigned k = p0; k < p1; k++) {
        const uint4 v = __ldcg(o.part + k);
        o.part[k] = at;
        at = add4(at, v);
    }
    if (tid == 0) *o.total = all;
}

// what precedes sub-tile s: vertices, triangles, c-vertices, active words
__device__ __forceinline__ uint4 sub_offset(const Out &o, unsigned s) { return add4(o.pre[s], o.part[s / TILE]); }

// a warp takes FIN sub-tiles at once, a lane per word
constexpr int FIN = 4;
template <class P>
__global__ void __launch_bounds__(256) k_finish(P pol, Out o, uint4 *act) {
    grid_wait();
    const int lane = threadIdx.x & 31;
    const uint4 total = *o.total;
    for (unsigned s0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * FIN; s0 < o.nsub; s0 += ((gridDim.x * blockDim.x) >> 5) * FIN) {
        unsigned m[FIN], c[FIN];
        uint4 b[FIN];
#pragma unroll
        for (int u = 0; u < FIN; u++) m[u] = s0 + u < o.nsub ? o.sub[s0 + u].y : 0u;
#pragma unroll
        for (int u = 0; u < FIN; u++) {
            const unsigned w = (s0 + u) * SUB + (unsigned)lane;
            c[u] = m[u] >> lane & 1u ? __ldg(o.cnt + w) : 0u;
            b[u] = make_uint4(0u, 0u, 0u, 0u);
            if (m[u]) {
                b[u] = sub_offset(o, s0 + u);
                unsigned eshift, cshift;   // added to edge-vertex and c-vertex numbers
                pol.shifts(o, s0 + u, total, eshift, cshift);
                b[u].x += eshift;
                b[u].z += cshift;
            }
        }
#pragma unroll
        for (int u = 0; u < FIN; u++) {
            if (!m[u]) continue;
            unsigned t;
            const unsigned w = (s0 + u) * SUB + (unsigned)lane, e = warp_excl(c[u], lane, t);
            if (m[u] >> lane & 1u) {
                o.words[w].w += b[u].x;
                act[b[u].w + __popc(m[u] & ((1u << lane) - 1u))] = make_uint4(w, b[u].y + (e & 0xffffu), b[u].z + (e >> 16), 0u);
            }
        }
    }
}

// id of the vertex on the `axis` edge of the point at bit l of word w
__device__ __forceinline__ int vertex_id(const uint4 *__restrict__ words, unsigned w, unsigned l, int axis) {
    const uint4 m = __ldg(words + w);
    const unsigned lt = (1u << l) - 1u;
    unsigned id = m.w + __popc(m.x & lt) + __popc(m.y & lt) + __popc(m.z & lt);
    if (axis >= 1) id += (m.x >> l) & 1u;
    if (axis == 2) id += (m.y >> l) & 1u;
    return (int)id;
}
// tiling edge code 0..11 -> owner offset (bit 0: +x, 1: +y, 2: +z) and axis (bits 3-4)
__device__ __forceinline__ unsigned edge_code(int code) {
    constexpr unsigned long long k = (0x00ull << 0) | (0x09ull << 5) | (0x02ull << 10) | (0x08ull << 15) | (0x04ull << 20) |
                                     (0x0dull << 25) | (0x06ull << 30) | (0x0cull << 35) | (0x10ull << 40) |
                                     (0x11ull << 45) | (0x13ull << 50) | (0x12ull << 55);
    return (unsigned)(k >> (5 * code)) & 31u;
}

constexpr int EW = 4;              // warps per CTA of k_emit
constexpr int TQ = 32 + 32 * 12;   // queued triangles: fewer than 32 left over, 32 cubes of at most 12

// next: a zeroed group counter (groups are handed out one at a time: their work varies); G active words per group
__device__ __forceinline__ unsigned next_group(unsigned *next, int lane) {
    unsigned grp = 0;
    if (lane == 0) grp = atomicAdd(next, 1u);
    return __shfl_sync(FULL, grp, 0);
}

struct EmitShared {
    unsigned prev[32], pre[32];    // first vertex / cube of each lane's word
    unsigned cor[6][32];
    unsigned first_c[32], amb[32]; // c-vertices of the group before each word's; ambiguous cubes
    __align__(8) unsigned tri[TQ]; // lane << 27 | bit << 22 | code offset; before that, 32 vertices on their way out
    int cvert[TQ];                 // the cube's c-vertex
    int out[96];                   // 32 triangles on their way out
};

template <class P>
__global__ void __launch_bounds__(EW * 32, P::CTAS) k_emit(P pol, const unsigned *__restrict__ signs, Out o, const uint4 *__restrict__ act,
                                                           unsigned warps, MeshRoom room, vec3i *tris) {
    grid_wait();
    const uint4 tot = *o.total;
    if (!room.fits(tot)) return;   // emitted again into larger buffers
    // Words per group: more fill the lanes better and share the group's start, fewer leave no SM
    // waiting for a last group.  32 only from eight rounds of groups per resident warp on (1.25 M
    // active words), 8 (a word has about 7 vertices) below one round of 16.  The emit stage with
    // the other choice: 512^3 CT without pre-smoothing (19 M triangles) 513 us with 32, 581 with 16;
    // pre-smoothed (0.6 M active words, four rounds of 32) 249 with 32, 240 with 16; brain (14 k
    // words) 157 with 32, 23 with 8.
    const unsigned nact = tot.w, G = nact >= 256u * warps ? 32u : (nact >= 16u * warps ? 16u : 8u);
    const uint4 *__restrict__ words = o.words;
    __shared__ EmitShared shared[EW];
    __shared__ unsigned qt[256];
    for (int i = threadIdx.x; i < 256; i += EW * 32) qt[i] = pol.quick(i);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    EmitShared &S = shared[threadIdx.x >> 5];
    const unsigned ngroups = (nact + G - 1) / G;
    for (unsigned grp; (grp = next_group(o.ctr + 1, lane)) < ngroups;) {
        const unsigned a = grp * G + (unsigned)lane;
        const bool live = (unsigned)lane < G && a < nact;
        const uint4 e = live ? __ldg(act + a) : make_uint4(0u, 0u, 0u, 0u);
        Geo g{0, 0, 0, 0u, 0u, 0u, 0u, false, false, false, 0};
        uint4 m = make_uint4(0u, 0u, 0u, 0u);
        unsigned mix = 0;
        if (live) {
            m = __ldg(words + e.x);
            if (P::CVERTS) S.amb[lane] = __ldg(o.amb + e.x);
            pol.geo(e.x, g);
            const Corners q = load_corners(signs, e.x, g);
            mix = mixed_cubes(q, g);
            S.cor[0][lane] = q.a;
            S.cor[1][lane] = q.b;
            S.cor[2][lane] = q.c;
            S.cor[3][lane] = q.d;
            S.cor[4][lane] = q.nxt;
        }
        S.cor[5][lane] = mix;
        unsigned both;
        const unsigned ex = warp_excl((__popc(m.x) + __popc(m.y) + __popc(m.z)) | __popc(mix) << 16, lane, both);
        S.prev[lane] = ex & 0xffffu;
        S.pre[lane] = ex >> 16;
        const unsigned nv = both & 0xffffu, nc = both >> 16;
        unsigned tbase = __shfl_sync(FULL, e.y, 0);
        if (!P::MULTI) {   // lanes without a word take part in the queue too
            g.WX = __shfl_sync(FULL, g.WX, 0);
            g.slice = __shfl_sync(FULL, g.slice, 0);
        }
        __syncwarp();
        // ---- vertices, EV per lane with their values in flight together
        constexpr int EV = P::EV;
        for (unsigned k0 = 0; k0 < nv; k0 += 32 * EV) {
            int x[EV], y[EV], z[EV], ax[EV], id[EV];
            typename P::Edge v[EV];
#pragma unroll
            for (int u = 0; u < EV; u++) {
                const unsigned k = min(k0 + 32 * u + (unsigned)lane, nv - 1);
                const int l = find_lane(S.prev, k);
                const int r = (int)(k - S.prev[l]);
                const unsigned mx = __shfl_sync(FULL, m.x, l), my = __shfl_sync(FULL, m.y, l), mz = __shfl_sync(FULL, m.z, l),
                               v0 = __shfl_sync(FULL, m.w, l);
                x[u] = __shfl_sync(FULL, g.x0, l);
                y[u] = __shfl_sync(FULL, g.y, l);
                z[u] = __shfl_sync(FULL, g.z, l);
                const int tag = P::MULTI ? __shfl_sync(FULL, g.tag, l) : 0;
                int p = 0, cb = 0;   // the point holding the word's r-th vertex, vertices before it
#pragma unroll
                for (int s = 16; s; s >>= 1) {
                    const unsigned lt = (1u << (p + s)) - 1u;
                    const int c = __popc(mx & lt) + __popc(my & lt) + __popc(mz & lt);
                    if (c <= r) {
                        p += s;
                        cb = c;
                    }
                }
                const bool bx = mx >> p & 1u, by = my >> p & 1u;
                const int j = r - cb;
                ax[u] = j == 0 ? (bx ? 0 : (by ? 1 : 2)) : (j == 1 && bx && by ? 1 : 2);
                x[u] += p;
                id[u] = (int)(v0 + (unsigned)r);
                v[u] = pol.edge(x[u], y[u], z[u], ax[u], tag);
            }
#pragma unroll
            for (int u = 0; u < EV; u++) {
                const unsigned n = min(32u, nv - min(nv, k0 + 32 * u));
                vec3d q = {0., 0., 0.};
                if ((unsigned)lane < n) q = pol.vertex(v[u], x[u], y[u], z[u], ax[u], id[u]);
                const int id0 = __shfl_sync(FULL, id[u], 0);
                if (__all_sync(FULL, (unsigned)lane >= n || id[u] == id0 + lane)) {   // consecutive: whole sectors
                    double *st = (double *)S.tri, *out = (double *)(pol.pts + id0);
                    __syncwarp();
                    st[3 * lane] = q.x;
                    st[3 * lane + 1] = q.y;
                    st[3 * lane + 2] = q.z;
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < 3; c++)
                        if ((unsigned)(32 * c + lane) < 3 * n) out[32 * c + lane] = st[32 * c + lane];
                } else if ((unsigned)lane < n) {
                    pol.pts[id[u]] = q;
                }
            }
        }
        __syncwarp();   // the queue takes over the stage
        // ---- cubes, one per lane; their triangles go through the queue
        unsigned fill = 0, ccount = 0;
        auto emit = [&](unsigned k, unsigned n) {   // queue entries k .. k + n - 1, n <= 32
            const bool ok = (unsigned)lane < n;
            const unsigned t = ok ? S.tri[k + lane] : 0u;
            const int l = (int)(t >> 27);
            const unsigned w = __shfl_sync(FULL, e.x, l);
            const unsigned WX = P::MULTI ? __shfl_sync(FULL, g.WX, l) : g.WX, slice = P::MULTI ? __shfl_sync(FULL, g.slice, l) : g.slice;
            if (ok) {
                const unsigned b = t >> 22 & 31u;
                const int off = (int)(t & 0x3fffffu);
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const int code = pol.code(off + c);
                    int v;
                    if (P::CVERTS && code == 12) {
                        v = S.cvert[k + lane];
                    } else {
                        const unsigned ec = edge_code(code), bb = b + (ec & 1u);
                        v = vertex_id(words, w + (bb >> 5) + (ec & 2u ? WX : 0u) + (ec & 4u ? slice : 0u), bb & 31u, (int)(ec >> 3));
                    }
                    S.out[3 * lane + (P::REVERSE ? 2 - c : c)] = v;
                }
            }
            __syncwarp();
            int *out = (int *)(tris + tbase + k);   // whole sectors
#pragma unroll
            for (int c = 0; c < 3; c++)
                if ((unsigned)(32 * c + lane) < 3 * n) out[32 * c + lane] = S.out[32 * c + lane];
            __syncwarp();
        };
        for (unsigned k0 = 0; k0 < nc; k0 += 32) {
            const bool ok = k0 + (unsigned)lane < nc;
            const unsigned k = min(k0 + (unsigned)lane, nc - 1);
            const int l = find_lane(S.pre, k);
            const int r = (int)(k - S.pre[l]);
            const int i = nth_bit(S.cor[5][l], r);
            const int lut = cube_index(S.cor[0][l], S.cor[1][l], S.cor[2][l], S.cor[3][l], S.cor[4][l], i);
            const unsigned q = qt[lut];
            CubeTiling T{(int)(q >> 8), ok ? (int)(q & 0xffu) : 0, false};
            int v12 = -1;
            if (P::CVERTS) {
                if (__any_sync(FULL, ok && T.n == (int)TESTS)) {
                    const int x0 = __shfl_sync(FULL, g.x0, l), y = __shfl_sync(FULL, g.y, l), z = __shfl_sync(FULL, g.z, l),
                              tag = __shfl_sync(FULL, g.tag, l);
                    const unsigned c0 = __shfl_sync(FULL, e.z, l), w = __shfl_sync(FULL, e.x, l);
                    const Geo gl{x0, y, z, 0u, 0u, 0u, 0u, false, false, false, tag};
                    if (ok && T.n == (int)TESTS) {   // decided by k_amb
                        const unsigned at = __ldg(o.ambat + w);
                        if (at != NO_TILING) {
                            const unsigned t = __ldg(o.tilings + at + __popc(S.amb[l] & ((1u << i) - 1u)));
                            T = CubeTiling{(int)(t & 0x3fffffu), (int)(t >> 22 & 15u), (t >> 26 & 1u) != 0u};
                        } else {
                            T = pol.tests(gl, x0 + i, y, z, lut);
                        }
                    }
                    // number the c-vertices within their words
                    const unsigned cvb = __ballot_sync(FULL, ok && T.cv), cex = ccount + __popc(cvb & ((1u << lane) - 1u));
                    if (ok && r == 0) S.first_c[l] = cex;
                    __syncwarp();
                    if (ok && T.cv) {
                        v12 = (int)(c0 + cex - S.first_c[l]);
                        pol.cvertex(gl, x0 + i, y, z, v12);
                    }
                    ccount += __popc(cvb);
                } else if (ok && r == 0) {
                    S.first_c[l] = ccount;
                }
            }
            unsigned made;
            const unsigned at = fill + warp_excl((unsigned)T.n, lane, made);
            for (int j = 0; j < T.n; j++) {
                S.tri[at + j] = (unsigned)l << 27 | (unsigned)i << 22 | (unsigned)(T.off + 3 * j);
                if (P::CVERTS) S.cvert[at + j] = v12;
            }
            fill += made;
            __syncwarp();
            unsigned head = 0;
            for (; fill - head >= 32; head += 32) emit(head, 32u);
            if (head) {   // the rest to the front
                __syncwarp();
                const unsigned rest = fill - head;
                const unsigned t = (unsigned)lane < rest ? S.tri[head + lane] : 0u;
                const int cv = P::CVERTS && (unsigned)lane < rest ? S.cvert[head + lane] : -1;
                __syncwarp();
                S.tri[lane] = t;
                if (P::CVERTS) S.cvert[lane] = cv;
                fill = rest;
                tbase += head;
                __syncwarp();
            }
        }
        if (fill) emit(0u, fill);
        __syncwarp();   // the lists are reused by the next group
    }
}

// ---- host side ----------------------------------------------------------------------
// buffers of a grid of nwords sign words
inline n2m_status prepare(McWork &w, size_t nwords, uint4 *d_total, Out &o) {
    const size_t nsub = (nwords + SUB - 1) / SUB, tiles = (nsub + TILE - 1) / TILE;
    o.nwords = (unsigned)nwords;
    o.nsub = (unsigned)nsub;
    CKS(w.words.ensure(nwords * sizeof(uint4)));
    CKS(w.act.ensure(nwords * sizeof(uint4)));
    CKS(w.cnt.ensure(4 * nwords * sizeof(unsigned)));
    CKS(w.sub.ensure((2 * nsub + tiles) * sizeof(uint4) + 4 * sizeof(unsigned)));
    o.words = w.words.as<uint4>();
    o.cnt = w.cnt.as<unsigned>();
    o.amb = o.cnt + nwords;
    o.ambat = o.amb + nwords;
    o.tilings = o.ambat + nwords;
    o.sub = w.sub.as<uint4>();
    o.pre = o.sub + nsub;
    o.part = o.pre + nsub;
    o.ctr = (unsigned *)(o.part + tiles);
    o.total = d_total;
    return N2M_OK;
}

// what follows from signs alone (and the marks, if wanted); the counters are cleared here
template <class P>
n2m_status count_signs(const P &pol, const unsigned *signs, const Out &o, const Marks &marks, cudaStream_t s) {
    CK(cudaMemsetAsync(o.ctr, 0, 4 * sizeof(unsigned), s));
    n2m_launch(k_words<P>, std::max(1u, std::min((o.nsub + 7) / 8, 152u * 32u)), 256, 0, s, pol, signs, o, marks);
    CKL();
    return N2M_OK;
}
// the rest: values are final
template <class P>
n2m_status count_values(const P &pol, const unsigned *signs, McWork &w, const Out &o, bool tests, cudaStream_t s) {
    if (tests) n2m_launch(k_amb<P>, (o.nsub + AMB_S - 1) / AMB_S, AMB_T, 0, s, pol, signs, o);
    n2m_launch(k_sum<P>, (o.nsub + TILE - 1) / TILE, TILE, 0, s, o);
    n2m_launch(k_finish<P>, std::max(1u, std::min((o.nsub + 8 * FIN - 1) / (8 * FIN), 152u * 16u)), 256, 0, s, pol, o,
               w.act.as<uint4>());
    CKL();
    return N2M_OK;
}

// CTAs of a kernel that fit the GPU at once, kept per device ordinal
inline n2m_status resident_ctas(const void *fn, std::atomic<int> (&of)[64], int &n) {
    int dev = 0;
    CK(cudaGetDevice(&dev));
    n = dev < 64 ? of[dev].load(std::memory_order_relaxed) : 0;
    if (!n) {
        int sms = 0, per_sm = 0;
        CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, EW * 32, 0));
        n = sms * std::max(per_sm, 1);
        if (dev < 64) of[dev].store(n, std::memory_order_relaxed);
    }
    return N2M_OK;
}

// the counts are taken on the device (the grid is what fits the GPU at once); a mesh beyond `room` is not emitted
template <class P>
n2m_status emit(const P &pol, const unsigned *signs, McWork &w, const Out &o, const MeshRoom &room, vec3i *d_tris, cudaStream_t s) {
    static std::atomic<int> resident[64];   // work comes from an atomic counter, so any grid is correct
    int n = 0;
    CKS(resident_ctas((const void *)k_emit<P>, resident, n));
    n2m_launch(k_emit<P>, (unsigned)n, EW * 32, 0, s, pol, signs, o, w.act.as<uint4>(), (unsigned)n * EW, room, d_tris);
    CKL();
    return N2M_OK;
}
}  // namespace mcw
