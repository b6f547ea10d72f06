// mcwords.cuh — the word machinery of every marching-cubes variant.
//
// A grid's points are grouped in row-aligned 32-point words of sign bits.  Words
// are numbered in raster order, so vertex and triangle numbers are prefix sums
// over words.  A variant supplies a policy (its grid geometry, tilings and vertex
// arithmetic); this file counts, numbers and emits:
//
//   k_words   edge-crossing masks of every word and the counts that follow from
//             signs alone; marks the voxels whose exact values will be read; lists
//             the words holding ambiguous cubes.  A warp turns the mixed cubes of its
//             32 words into one dense list (a cube per lane), so that neither an empty
//             word nor a full one costs its neighbours time.  Sub-tiles of 256 words
//             are scanned in the block; the last block to finish scans the tiles.
//   k_amb     the face and interior tests of the listed words' ambiguous cubes, which
//             need values (so with the exact smoothing on demand they come after the
//             repair), again a cube per lane: their loads no longer hold up k_words.
//   k_sum     triangle and c-vertex sums, over active words only.
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
// Measured on the 512^3 CT volume (7.1 M triangles, cold caches): emit 474 -> 218 us
// against one lane per word listing its cubes for the warp and separate mask and
// offset arrays; masks, marks, counts, scan and active list 290 -> 178 us.  On the brain volume
// (0.2 M triangles, 1.7 k groups of 32 words for 5 k resident warps) the emit went
// from 157 to 23 us.
#pragma once
#include <algorithm>
#include <atomic>

#include "n2m_internal.cuh"

namespace mcw {
constexpr unsigned FULL = 0xffffffffu;
constexpr int SUB = 256;          // words per sub-tile

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
    uint4 *words;           // per active word
    unsigned *cnt;          // per active word, triangles | c-vertices << 16
    unsigned *amb;          // per active word, its ambiguous cubes
    unsigned *amblist;      // words with any
    unsigned char *staged;  // per sub-tile, its active words in order (number within the sub-tile)
    uint2 *sub;             // per sub-tile, what precedes it in its tile {vertices, active words | own active words << 20}
    uint2 *subt;            // the same {triangles, c-vertices}
    uint2 *part, *partt;    // per tile, what precedes it, likewise
    uint4 *total;           // {vertices, triangles, c-vertices, active words}
    unsigned *ctr;          // tiles finished (two passes), words in amblist, group counter of the emit
    unsigned nwords, nsub, per;   // per: sub-tiles per tile (tile = block)
};

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

// turns n per-tile sums into what precedes each, by one block; the total goes to *all
__device__ __forceinline__ void scan_parts(uint2 *part, unsigned n, uint2 *psum, int tid, uint2 &all) {
    const int lane = tid & 31, wid = tid >> 5;
    const unsigned each = (n + SUB - 1) / SUB, p0 = min(n, (unsigned)tid * each), p1 = min(n, p0 + each);
    uint2 s = make_uint2(0u, 0u);
    for (unsigned k = p0; k < p1; k++) {
        const uint2 v = __ldcg(part + k);
        s.x += v.x;
        s.y += v.y;
    }
    unsigned tx, ty;
    uint2 before;
    before.x = warp_excl(s.x, lane, tx);
    before.y = warp_excl(s.y, lane, ty);
    if (lane == 0) psum[wid] = make_uint2(tx, ty);
    __syncthreads();
    all = make_uint2(0u, 0u);
    for (int k = 0; k < SUB / 32; k++) {
        if (k < wid) {
            before.x += psum[k].x;
            before.y += psum[k].y;
        }
        all.x += psum[k].x;
        all.y += psum[k].y;
    }
    for (unsigned k = p0; k < p1; k++) {
        const uint2 v = __ldcg(part + k);
        part[k] = before;
        before.x += v.x;
        before.y += v.y;
    }
}
// whether this block is the last to hand in its tile's sums (all threads call it)
__device__ __forceinline__ bool last_tile(uint2 *part, uint2 sums, unsigned *done, bool &flag) {
    if (threadIdx.x == 0) {
        part[blockIdx.x] = sums;
        __threadfence();
        flag = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (flag) __threadfence();
    return flag;
}

template <class P>
__global__ void __launch_bounds__(SUB) k_words(P pol, const unsigned *__restrict__ signs, Out o, Marks marks) {
    __shared__ unsigned qt[256], pre[8][32], cor[8][6][32], cnt[SUB], amb[SUB], abase;
    __shared__ uint2 wsum[8];
    __shared__ bool last;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    qt[tid] = pol.quick(tid);
    __syncthreads();
    uint2 run = make_uint2(0u, 0u);   // vertices, active words of the tile so far
    const unsigned s1 = min(o.nsub, (blockIdx.x + 1) * o.per);
    for (unsigned sub = blockIdx.x * o.per; sub < s1; sub++) {
        const unsigned w = sub * SUB + (unsigned)tid;
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
        cnt[tid] = 0u;
        amb[tid] = 0u;
        unsigned ncube;
        pre[wid][lane] = warp_excl(__popc(mix), lane, ncube);
        __syncwarp();
        for (unsigned k = lane; k < ncube; k += 32) {
            const int l = find_lane(pre[wid], k);
            const int i = nth_bit(cor[wid][5][l], (int)(k - pre[wid][l]));
            const int lut = cube_index(cor[wid][0][l], cor[wid][1][l], cor[wid][2][l], cor[wid][3][l], cor[wid][4][l], i);
            const unsigned n = qt[lut] & 0xffu;
            if (n == TESTS) atomicOr(&amb[wid * 32 + l], 1u << i);
            else atomicAdd(&cnt[wid * 32 + l], n);
        }
        __syncwarp();
        // a sub-tile has at most 24576 vertices and 256 active words (256 with ambiguous cubes)
        const unsigned nv = __popc(xm) + __popc(ym) + __popc(zm), am = amb[tid];
        const bool act = (nv | mix) != 0u;
        unsigned ta, tb, ea = warp_excl(nv | (act ? 1u << 16 : 0u), lane, ta);
        const unsigned ab = __ballot_sync(FULL, am != 0u);
        tb = __popc(ab);
        if (lane == 0) wsum[wid] = make_uint2(ta, tb);
        __syncthreads();
        uint2 all = make_uint2(0u, 0u);
        unsigned eb = __popc(ab & ((1u << lane) - 1u));
#pragma unroll
        for (int k = 0; k < SUB / 32; k++) {
            const uint2 t = wsum[k];
            if (k < wid) {
                ea += t.x;
                eb += t.y;
            }
            all.x += t.x;
            all.y += t.y;
        }
        if (tid == 0 && all.y) abase = atomicAdd(o.ctr + 2, all.y);
        if (act) {
            o.words[w] = make_uint4(xm, ym, zm, ea & 0xffffu);
            o.staged[(size_t)sub * SUB + (ea >> 16)] = (unsigned char)tid;
            o.cnt[w] = cnt[tid];
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
        if (tid == 0) o.sub[sub] = make_uint2(run.x, run.y | (all.x >> 16) << 20);
        run.x += all.x & 0xffffu;
        run.y += all.x >> 16;
        __syncthreads();   // abase; wsum is reused
        if (am) o.amblist[abase + eb] = w;
    }
    if (!last_tile(o.part, run, o.ctr, last)) return;
    uint2 all;
    scan_parts(o.part, gridDim.x, wsum, tid, all);
    if (tid == 0) {
        o.total->x = all.x;
        o.total->w = all.y;
    }
}

// the ambiguous cubes of the listed words, a warp per 32 words
template <class P>
__global__ void __launch_bounds__(128) k_amb(P pol, const unsigned *__restrict__ signs, Out o) {
    __shared__ unsigned pre[4][32], cor[4][6][32], words[4][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned n = o.ctr[2];
    for (unsigned a0 = (blockIdx.x * 4 + (unsigned)wid) * 32; a0 < n; a0 += gridDim.x * 128) {
        unsigned am = 0;
        if (a0 + (unsigned)lane < n) {
            const unsigned w = o.amblist[a0 + lane];
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
        unsigned ncube;
        pre[wid][lane] = warp_excl(__popc(am), lane, ncube);
        __syncwarp();
        for (unsigned k = lane; k < ncube; k += 32) {
            const int l = find_lane(pre[wid], k);
            const int i = nth_bit(cor[wid][5][l], (int)(k - pre[wid][l]));
            const int lut = cube_index(cor[wid][0][l], cor[wid][1][l], cor[wid][2][l], cor[wid][3][l], cor[wid][4][l], i);
            Geo g;
            pol.geo(words[wid][l], g);
            const CubeTiling T = pol.tests(g, g.x0 + i, g.y, g.z, lut);
            atomicAdd(o.cnt + words[wid][l], (unsigned)T.n | (T.cv ? 1u << 16 : 0u));
        }
        __syncwarp();
    }
}

// triangle and c-vertex sums of the sub-tiles, a warp each, in rounds of 8 (a template only to be emitted once per unit)
template <class P>
__global__ void __launch_bounds__(SUB) k_sum(Out o) {
    __shared__ uint2 wsum[8];
    __shared__ bool last;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    uint2 run = make_uint2(0u, 0u);
    const unsigned s0 = blockIdx.x * o.per, s1 = min(o.nsub, s0 + o.per);
    for (unsigned r = s0; r < s1; r += 8) {
        const unsigned sub = r + (unsigned)wid;
        uint2 t = make_uint2(0u, 0u);
        if (sub < s1) {
            const unsigned n = o.sub[sub].y >> 20;
            for (unsigned k = (unsigned)lane; k < n; k += 32) {
                const unsigned c = o.cnt[sub * SUB + o.staged[(size_t)sub * SUB + k]];
                t.x += c & 0xffffu;
                t.y += c >> 16;
            }
        }
        t.x = __reduce_add_sync(FULL, t.x);
        t.y = __reduce_add_sync(FULL, t.y);
        if (lane == 0) wsum[wid] = t;
        __syncthreads();
        uint2 before = run;
        for (int k = 0; k < 8; k++) {
            if (k < wid) {
                before.x += wsum[k].x;
                before.y += wsum[k].y;
            }
            run.x += wsum[k].x;
            run.y += wsum[k].y;
        }
        if (lane == 0 && sub < s1) o.subt[sub] = before;
        __syncthreads();
    }
    if (!last_tile(o.partt, run, o.ctr + 1, last)) return;
    uint2 all;
    scan_parts(o.partt, gridDim.x, wsum, tid, all);
    if (tid == 0) {
        o.total->y = all.x;
        o.total->z = all.y;
    }
}

// what precedes sub-tile s: vertices, triangles, c-vertices, active words
__device__ __forceinline__ uint4 sub_offset(const Out &o, unsigned s) {
    const uint2 a = o.sub[s], b = o.subt[s], pa = o.part[s / o.per], pb = o.partt[s / o.per];
    return make_uint4(a.x + pa.x, b.x + pb.x, b.y + pb.y, (a.y & 0xfffffu) + pa.y);
}

// a warp per sub-tile
template <class P>
__global__ void __launch_bounds__(256) k_finish(P pol, Out o, uint4 *act) {
    const int lane = threadIdx.x & 31;
    const uint4 total = *o.total;
    for (unsigned s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < o.nsub; s += (gridDim.x * blockDim.x) >> 5) {
        const unsigned n = o.sub[s].y >> 20;
        if (!n) continue;
        uint4 b = sub_offset(o, s);
        unsigned eshift, cshift;   // added to edge-vertex and c-vertex numbers
        pol.shifts(o, s, total, eshift, cshift);
        for (unsigned k0 = 0; k0 < n; k0 += 32) {
            const unsigned k = k0 + (unsigned)lane;
            const unsigned w = s * SUB + (k < n ? o.staged[(size_t)s * SUB + k] : 0u);
            const unsigned c = k < n ? o.cnt[w] : 0u;
            unsigned tt, tc;
            const unsigned et = warp_excl(c & 0xffffu, lane, tt), ec = warp_excl(c >> 16, lane, tc);
            if (k < n) {
                o.words[w].w += b.x + eshift;
                act[b.w + k] = make_uint4(w, b.y + et, b.z + ec + cshift, 0u);
            }
            b.y += tt;
            b.z += tc;
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

struct EmitShared {
    unsigned prev[32], prec[32];   // first vertex / cube of each lane's word
    unsigned cor[6][32];
    unsigned first_c[32];          // c-vertices of the group before each word's
    unsigned tri[TQ];              // lane << 27 | bit << 22 | code offset
    int cvert[TQ];                 // the cube's c-vertex
};

// next: a zeroed group counter (groups are handed out one at a time: their work varies); G active words per group
template <class P>
__global__ void __launch_bounds__(EW * 32) k_emit(P pol, const unsigned *__restrict__ signs, const uint4 *__restrict__ words,
                                                  const uint4 *__restrict__ act, unsigned nact, unsigned G, vec3i *tris,
                                                  unsigned *next) {
    __shared__ EmitShared shared[EW];
    __shared__ unsigned qt[256];
    for (int i = threadIdx.x; i < 256; i += EW * 32) qt[i] = pol.quick(i);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    EmitShared &S = shared[threadIdx.x >> 5];
    const unsigned ngroups = (nact + G - 1) / G;
    for (;;) {
        unsigned grp = 0;
        if (lane == 0) grp = atomicAdd(next, 1u);
        grp = __shfl_sync(FULL, grp, 0);
        if (grp >= ngroups) break;
        const unsigned a = grp * G + (unsigned)lane;
        const bool live = (unsigned)lane < G && a < nact;
        const uint4 e = live ? __ldg(act + a) : make_uint4(0u, 0u, 0u, 0u);
        Geo g{0, 0, 0, 0u, 0u, 0u, 0u, false, false, false, 0};
        uint4 m = make_uint4(0u, 0u, 0u, 0u);
        unsigned mix = 0;
        if (live) {
            pol.geo(e.x, g);
            m = __ldg(words + e.x);
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
        S.prec[lane] = ex >> 16;
        const unsigned nv = both & 0xffffu, nc = both >> 16;
        unsigned tbase = __shfl_sync(FULL, e.y, 0);
        __syncwarp();
        // ---- vertices, one per lane
        for (unsigned k0 = 0; k0 < nv; k0 += 32) {
            const unsigned k = k0 + (unsigned)lane;
            const int l = find_lane(S.prev, min(k, nv - 1));
            const int r = (int)(min(k, nv - 1) - S.prev[l]);
            const unsigned mx = __shfl_sync(FULL, m.x, l), my = __shfl_sync(FULL, m.y, l), mz = __shfl_sync(FULL, m.z, l),
                           v0 = __shfl_sync(FULL, m.w, l);
            const int x0 = __shfl_sync(FULL, g.x0, l), y = __shfl_sync(FULL, g.y, l), z = __shfl_sync(FULL, g.z, l),
                      tag = __shfl_sync(FULL, g.tag, l);
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
            const int j = r - cb, ax = j == 0 ? (bx ? 0 : (by ? 1 : 2)) : (j == 1 && bx && by ? 1 : 2);
            if (k < nv) pol.vertex(x0 + p, y, z, ax, tag, (int)(v0 + (unsigned)r));
        }
        // ---- cubes, one per lane; their triangles go through the queue
        unsigned fill = 0, ccount = 0;
        auto emit = [&](unsigned k, bool ok) {
            const unsigned t = ok ? S.tri[k] : 0u;
            const int l = (int)(t >> 27);
            const unsigned w = __shfl_sync(FULL, e.x, l);
            const unsigned WX = P::MULTI ? __shfl_sync(FULL, g.WX, l) : g.WX, slice = P::MULTI ? __shfl_sync(FULL, g.slice, l) : g.slice;
            if (!ok) return;
            const unsigned b = t >> 22 & 31u;
            const int off = (int)(t & 0x3fffffu);
            int tv[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const int code = pol.code(off + c);
                if (code == 12) {
                    tv[c] = S.cvert[k];
                } else {
                    const unsigned ec = edge_code(code), bb = b + (ec & 1u);
                    tv[c] = vertex_id(words, w + (bb >> 5) + (ec & 2u ? WX : 0u) + (ec & 4u ? slice : 0u), bb & 31u, (int)(ec >> 3));
                }
            }
            tris[tbase + k] = P::REVERSE ? vec3i{tv[2], tv[1], tv[0]} : vec3i{tv[0], tv[1], tv[2]};
        };
        if (!P::MULTI) {   // lanes without a word take part in the queue too
            g.WX = __shfl_sync(FULL, g.WX, 0);
            g.slice = __shfl_sync(FULL, g.slice, 0);
        }
        for (unsigned k0 = 0; k0 < nc; k0 += 32) {
            const unsigned k = k0 + (unsigned)lane;
            const bool ok = k < nc;
            const int l = find_lane(S.prec, min(k, nc - 1));
            const int r = (int)(min(k, nc - 1) - S.prec[l]);
            const int i = nth_bit(S.cor[5][l], r);
            const int lut = cube_index(S.cor[0][l], S.cor[1][l], S.cor[2][l], S.cor[3][l], S.cor[4][l], i);
            const unsigned q = qt[lut];
            CubeTiling T{(int)(q >> 8), ok ? (int)(q & 0xffu) : 0, false};
            if (__any_sync(FULL, ok && T.n == (int)TESTS)) {
                const int x0 = __shfl_sync(FULL, g.x0, l), y = __shfl_sync(FULL, g.y, l), z = __shfl_sync(FULL, g.z, l),
                          tag = __shfl_sync(FULL, g.tag, l);
                Geo gl{x0, y, z, 0u, 0u, 0u, 0u, false, false, false, tag};
                if (ok && T.n == (int)TESTS) T = pol.tests(gl, x0 + i, y, z, lut);
            }
            int v12 = -1;
            const unsigned cvb = __ballot_sync(FULL, ok && T.cv);
            if (P::CVERTS) {   // number the c-vertices within their words
                const unsigned cex = ccount + __popc(cvb & ((1u << lane) - 1u));
                if (ok && r == 0) S.first_c[l] = cex;
                __syncwarp();
                const unsigned c0 = __shfl_sync(FULL, e.z, l);
                const int x0 = __shfl_sync(FULL, g.x0, l), y = __shfl_sync(FULL, g.y, l), z = __shfl_sync(FULL, g.z, l),
                          tag = __shfl_sync(FULL, g.tag, l);
                if (ok && T.cv) {
                    v12 = (int)(c0 + cex - S.first_c[l]);
                    Geo gl{x0, y, z, 0u, 0u, 0u, 0u, false, false, false, tag};
                    pol.cvertex(gl, x0 + i, y, z, v12);
                }
                ccount += __popc(cvb);
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
            for (; fill - head >= 32; head += 32) emit(head + (unsigned)lane, true);
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
        if (fill) emit((unsigned)lane, (unsigned)lane < fill);
        __syncwarp();   // the lists are reused by the next group
    }
}

// ---- host side ----------------------------------------------------------------------
// Sub-tiles per tile: about 16 tiles per SM, so that the last block's scan stays short.
inline unsigned subs_per_tile(size_t nsub) { return (unsigned)std::max<size_t>(1, (nsub + 152 * 16 - 1) / (152 * 16)); }

// buffers of a grid of nwords sign words
inline n2m_status prepare(McWork &w, size_t nwords, uint4 *d_total, Out &o) {
    const size_t nsub = (nwords + SUB - 1) / SUB;
    o.nwords = (unsigned)nwords;
    o.nsub = (unsigned)nsub;
    o.per = subs_per_tile(nsub);
    const size_t tiles = (nsub + o.per - 1) / o.per;
    CKS(w.words.ensure(nwords * sizeof(uint4)));
    CKS(w.act.ensure(nwords * sizeof(uint4)));
    CKS(w.cnt.ensure(3 * nwords * sizeof(unsigned)));
    CKS(w.staged.ensure(nsub * SUB));
    CKS(w.sub.ensure(2 * (nsub + tiles) * sizeof(uint2) + 4 * sizeof(unsigned)));
    o.words = w.words.as<uint4>();
    o.cnt = w.cnt.as<unsigned>();
    o.amb = o.cnt + nwords;
    o.amblist = o.amb + nwords;
    o.staged = w.staged.as<unsigned char>();
    o.sub = w.sub.as<uint2>();
    o.subt = o.sub + nsub;
    o.part = o.subt + nsub;
    o.partt = o.part + tiles;
    o.ctr = (unsigned *)(o.partt + tiles);
    o.total = d_total;
    return N2M_OK;
}

// what follows from signs alone (and the marks, if wanted); the counters are cleared here
template <class P>
n2m_status count_signs(const P &pol, const unsigned *signs, const Out &o, const Marks &marks, cudaStream_t s) {
    CK(cudaMemsetAsync(o.ctr, 0, 4 * sizeof(unsigned), s));
    { k_words<P><<<(o.nsub + o.per - 1) / o.per, SUB, 0, s>>>(pol, signs, o, marks); N2M_COUNT(); }
    CKL();
    return N2M_OK;
}
// the rest: values are final
template <class P>
n2m_status count_values(const P &pol, const unsigned *signs, McWork &w, const Out &o, bool tests, cudaStream_t s) {
    if (tests) {
        const unsigned b = std::max(1u, std::min((o.nwords / 32 + 127) / 128, 152u * 8u));   // 1 word in 32 fills it
        k_amb<P><<<b, 128, 0, s>>>(pol, signs, o);
        N2M_COUNT();
    }
    { k_sum<P><<<(o.nsub + o.per - 1) / o.per, SUB, 0, s>>>(o); N2M_COUNT(); }
    { k_finish<P><<<std::max(1u, std::min((o.nsub + 7) / 8, 152u * 8u)), 256, 0, s>>>(pol, o, w.act.as<uint4>()); N2M_COUNT(); }
    CKL();
    return N2M_OK;
}

template <class P>
n2m_status emit(const P &pol, const unsigned *signs, McWork &w, const Out &o, unsigned nact, vec3i *d_tris, cudaStream_t s) {
    // CTAs that fit the GPU at once, per device ordinal (work comes from an atomic counter, so any grid is correct)
    static std::atomic<int> resident_of[64];
    int dev = 0;
    CK(cudaGetDevice(&dev));
    int resident = dev < 64 ? resident_of[dev].load(std::memory_order_relaxed) : 0;
    if (!resident) {
        int sms = 0, per_sm = 0;
        CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_emit<P>, EW * 32, 0));
        resident = sms * std::max(per_sm, 1);
        if (dev < 64) resident_of[dev].store(resident, std::memory_order_relaxed);
    }
    // 32 words per group keep the per-group work small; below two groups per resident warp smaller groups
    // spread the mesh over the GPU instead (8 words still fill the lanes: a word has about 7 vertices)
    const unsigned warps = (unsigned)resident * EW;
    const unsigned G = nact >= 64u * warps ? 32u : (nact >= 16u * warps ? 16u : 8u);
    const unsigned groups = (nact + G - 1) / G;
    const unsigned blocks = std::min<unsigned>((groups + EW - 1) / EW, (unsigned)resident);
    { k_emit<P><<<blocks, EW * 32, 0, s>>>(pol, signs, o.words, w.act.as<uint4>(), nact, G, d_tris, o.ctr + 3); N2M_COUNT(); }
    CKL();
    return N2M_OK;
}
}  // namespace mcw
