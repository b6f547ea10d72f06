// mc.cu — Lewiner MC33 marching cubes (src/MarchingCubes.c:116-1143) as two
// passes over the padded bounding-box grid, plus the classic case table of
// the same framework (-o 1).
//
// Numbering is the reference's: the edge vertices of grid point p (its +x,
// +y, +z edges, in that order) come after those of every point before p in
// raster order; c-vertices follow all edge vertices in cube raster order;
// triangles are in cube raster order, tiling order within a cube.  So the
// mesh is the reference's mesh before its weld, vertex for vertex.
//
// The sign bit of every grid point, packed in 32-point words (k_signs), then the
// word machinery of mcwords.cuh: counts, offsets, and an emit in which every
// edge vertex is made exactly once (this replaces the reference's vertex weld
// for shared edges).  Words are aligned with the volume's 32-voxel groups (the
// grid's first point is bit lo0 & 31), so a word of signs is a word of any
// bitmap of the volume.
// Vertices whose final coordinates sit within 1.5e-5 of a grid point (edge
// vertices) or of a grid plane (c-vertices) are recorded as weld candidates:
// only such vertices can lie within the weld tolerance (1e-5) of another.
#include <float.h>

#include <algorithm>

#include "mc33.cuh"
#include "mcwords.cuh"

namespace {
using namespace mc33;
struct GV {  // device view of the padded grid
    const float *vol;
    int dx, dy, dz;
    long long nvox, dxy;
    int lo0, lo1, lo2, NX, NY, NZ;
    unsigned WX;   // words per row
    int xoff;      // bit of grid point x = 0 in a row's first word
    float iso, edge_max, pad;
};

// value of grid point (x,y,z) minus isolevel, as marchingCubes() builds it
// (src/MarchingCubes.c:1097-1115, incl. the row wrap past x = dim0-1), with
// meshify's edge darkening (src/meshify.c:348-369) applied on the fly and
// run()'s FLT_EPSILON clamp (src/MarchingCubes.c:131-132).
__device__ __forceinline__ float gval(const GV &g, int x, int y, int z) {
    const long long j = (long long)(g.lo0 + x) + (long long)(y + g.lo1) * g.dx + (long long)(z + g.lo2) * g.dxy;
    float v;
    if (j < g.nvox) {
        v = __ldg(g.vol + j);
        // the voxel j really is: the grid ends at dim, so a coordinate is past the volume by at most
        // one (the padding column / row), which wraps into the next row / slice
        int vx = g.lo0 + x, vy = y + g.lo1, vz = z + g.lo2;
        if (vx >= g.dx) {
            vx -= g.dx;
            vy++;
        }
        if (vy >= g.dy) {
            vy -= g.dy;
            vz++;
        }
        if (vx == 0 || vy == 0 || vz == 0 || vx == g.dx - 1 || vy == g.dy - 1 || vz == g.dz - 1)
            v = fminf(g.edge_max, v);
        v = __fsub_rn(v, g.iso);
    } else {
        v = g.pad;
    }
    if (fabsf(v) < N2M_FLT_EPS) v = N2M_FLT_EPS;
    return v;
}

// ---- signs --------------------------------------------------------------------
// The sign (grid value > 0) of every grid point as one bit: bit b of word
// (z*NY + y)*WX + xw is grid point x = 32*xw - xoff + b, i.e. voxel column
// 32*(lo0/32 + xw) + b; bits outside the grid are 0.  The FLT_EPSILON clamp maps
// (-eps, eps) to +eps, so positive <=> value - iso > -eps.

// bits of word xw that are grid points
__device__ __forceinline__ unsigned grid_bits(const GV &g, int xw) {
    return mcw::bit_range(g.xoff - 32 * xw, g.xoff + g.NX - 32 * xw);
}

// Signs from a volume, a warp per row, SW words at a time with all their loads in
// flight.  Words strictly inside the volume and the grid read the volume directly;
// border words (a row's first and last, every word of a row on a face) apply gval's
// cases lane by lane on the linear voxel index j = row start + x: the padding column
// (x one past the volume) is the next row's first voxel, which is on a face; a row on
// a face of the volume (or the padding row, which wraps to y = 0 of the next slice)
// has every point darkened; j past the volume is the padding value.
constexpr int SW = 16;

__device__ __forceinline__ unsigned border_word(const GV &g, long long rb, bool rface, int xw, int lane) {
    const int x = xw * 32 + lane - g.xoff, vx = g.lo0 + x;
    const bool in = x >= 0 && x < g.NX;
    float d = g.pad;
    if (in && rb + x < g.nvox) {
        const float v = __ldg(g.vol + rb + x);
        d = __fsub_rn((rface || vx == 0 || vx >= g.dx - 1) ? fminf(g.edge_max, v) : v, g.iso);
    }
    return __ballot_sync(0xffffffffu, in && d > -N2M_FLT_EPS);
}

__global__ void __launch_bounds__(256) k_signs(GV g, unsigned nrows, unsigned *signs) {
    grid_wait();
    const int lane = threadIdx.x & 31, WX = (int)g.WX;
    const int vb0 = g.lo0 - g.xoff;   // voxel column of a row's first bit
    // words whose 32 points lie strictly inside the volume in x and inside the grid
    const int xs0 = vb0 == 0 || g.xoff ? 1 : 0;
    const int lim = min(g.dx - 1, g.lo0 + g.NX);   // columns below this
    const int xs1 = lim - vb0 >= 32 ? (lim - vb0) / 32 : 0;
    for (unsigned row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < nrows; row += (gridDim.x * blockDim.x) >> 5) {
        const int y = (int)(row % (unsigned)g.NY), z = (int)(row / (unsigned)g.NY);
        const int vy = g.lo1 + y, vz = g.lo2 + z;
        const bool rface = !(vy >= 1 && vy <= g.dy - 2 && vz >= 1 && vz <= g.dz - 2);
        const long long rb = (long long)g.lo0 + (long long)vy * g.dx + (long long)vz * g.dxy;   // j of grid x = 0
        const float *rp = g.vol + (rb - g.xoff) + lane;
        unsigned *out = signs + (size_t)row * g.WX;
        const int f0 = rface ? WX : min(xs0, WX), f1 = rface ? WX : max(f0, min(xs1, WX));   // direct words [f0, f1)
        for (int xw = 0; xw < f0; xw++) {
            const unsigned m = border_word(g, rb, rface, xw, lane);
            if (lane == 0) out[xw] = m;
        }
        for (int xw0 = f0; xw0 < f1; xw0 += SW) {
            float raw[SW];
#pragma unroll
            for (int k = 0; k < SW; k++) raw[k] = xw0 + k < f1 ? __ldg(rp + (xw0 + k) * 32) : 0.f;
            unsigned mine = 0;
#pragma unroll
            for (int k = 0; k < SW; k++) {
                const unsigned m = __ballot_sync(0xffffffffu, __fsub_rn(raw[k], g.iso) > -N2M_FLT_EPS);
                if (lane == k) mine = m;
            }
            if (lane < SW && xw0 + lane < f1) out[xw0 + lane] = mine;
        }
        for (int xw = f1; xw < WX; xw++) {
            const unsigned m = border_word(g, rb, rface, xw, lane);
            if (lane == 0) out[xw] = m;
        }
    }
}

// A sign bitmap of the volume: OdWork::vsign (nys groups of 8 rows per slice), or plain row words (nys 0)
struct SignMap {
    const unsigned *bits;
    unsigned wv, nys;   // words per row
    int ny;
    __device__ __forceinline__ unsigned word(int x, int y, int z) const {
        return __ldg(bits + (nys ? od_vsign_word((unsigned)x, (unsigned)y, (unsigned)z, wv, nys)
                                 : ((size_t)z * ny + y) * wv + ((unsigned)x >> 5)));
    }
};

// Signs from the volume's sign bitmap, one thread per word and no values read:
// darkening is min(edge_max, v), whose sign is the voxel's bit and edge_max's own, and
// the padding's sign is the same for every padding point.  512^3 (cold caches): 98 us
// when the border words (two per row of 16) still read their voxels, 25 us now.
__global__ void __launch_bounds__(256) k_signs_bits(GV g, unsigned nwords, unsigned *signs, SignMap map) {
    grid_wait();
    const bool dark = __fsub_rn(g.edge_max, g.iso) > -N2M_FLT_EPS, padp = g.pad > -N2M_FLT_EPS;
    auto voxel = [&](int x, int y, int z) {   // sign of a voxel of a y or z row past the volume too; x = 0
        if (y >= g.dy) {
            y -= g.dy;
            z++;
        }
        return z < g.dz ? dark && (map.word(x, y, z) & 1u) : padp;
    };
    for (unsigned w = blockIdx.x * blockDim.x + threadIdx.x; w < nwords; w += gridDim.x * blockDim.x) {
        const unsigned xw = w % g.WX, row = w / g.WX;
        int vy = g.lo1 + (int)(row % (unsigned)g.NY), vz = g.lo2 + (int)(row / (unsigned)g.NY);
        const unsigned in = grid_bits(g, (int)xw);
        if (vy >= g.dy) {   // the padding row is row 0 of the next slice
            vy -= g.dy;
            vz++;
        }
        unsigned m = 0;
        if (vz >= g.dz) {
            m = padp ? in : 0u;
        } else {
            const int vb = g.lo0 - g.xoff + 32 * (int)xw;
            if (vb < g.dx) m = map.word(vb, vy, vz);
            m &= mcw::bit_range(0, g.dx - vb);
            if (!dark) {
                if (vy == 0 || vz == 0 || vy == g.dy - 1 || vz == g.dz - 1) m = 0u;
                else m &= mcw::bit_range(vb == 0 ? 1 : 0, g.dx - 1 - vb);
            }
            if (g.dx - vb >= 0 && g.dx - vb < 32 && (in >> (g.dx - vb) & 1u) && voxel(0, vy + 1, vz)) m |= 1u << (g.dx - vb);
            m &= in;
        }
        signs[w] = m;
    }
}

// ---- emit pass -------------------------------------------------------------------
// grid value at p (strictly inside the volume: no darkening, wrap or padding)
__device__ __forceinline__ float ival(const GV &g, const float *p) {
    const float v = __fsub_rn(__ldg(p), g.iso);
    return fabsf(v) < N2M_FLT_EPS ? N2M_FLT_EPS : v;
}

// corner values of cube (x, y, z), by gval's rules
__device__ __noinline__ void cube_values(const GV &g, int x, int y, int z, float *c) {
    const int vx = g.lo0 + x, vy = g.lo1 + y, vz = g.lo2 + z;
    if (vx >= 1 && vx + 1 <= g.dx - 2 && vy >= 1 && vy + 1 <= g.dy - 2 && vz >= 1 && vz + 1 <= g.dz - 2) {   // strictly inside
        const float *p = g.vol + ((long long)vx + (long long)vy * g.dx + (long long)vz * g.dxy);
        const long long sy = g.dx, sz = g.dxy;
        c[0] = ival(g, p); c[1] = ival(g, p + 1); c[2] = ival(g, p + 1 + sy); c[3] = ival(g, p + sy);
        c[4] = ival(g, p + sz); c[5] = ival(g, p + 1 + sz); c[6] = ival(g, p + 1 + sy + sz); c[7] = ival(g, p + sy + sz);
    } else {
        c[0] = gval(g, x, y, z); c[1] = gval(g, x + 1, y, z); c[2] = gval(g, x + 1, y + 1, z); c[3] = gval(g, x, y + 1, z);
        c[4] = gval(g, x, y, z + 1); c[5] = gval(g, x + 1, y, z + 1); c[6] = gval(g, x + 1, y + 1, z + 1);
        c[7] = gval(g, x, y + 1, z + 1);
    }
}
__device__ __noinline__ mcw::CubeTiling tested_tiling(const GV &g, int x, int y, int z, int lut, bool classic) {
    float c[8];
    cube_values(g, x, y, z, c);
    const Tiling T = select_tiling(c, lut, classic);
    return mcw::CubeTiling{T.off, T.n, T.cv};
}

// mcwords.cuh's policy for the padded Lewiner grid
struct Policy {
    static constexpr bool MULTI = false, REVERSE = true, CVERTS = true;
    static constexpr int CTAS = 8, EV = 1;   // of k_emit: CTAs per SM, vertices per lane in flight
    GV g;
    bool classic;
    vec3d *pts;
    int *cand, *ccand;
    unsigned *ncand, *nccand;
    int cap;
    unsigned *near;   // marks of vertices close to a grid point, or null
    __device__ __forceinline__ unsigned quick(int lut) const {
        Tiling T = {0, 0, false};
        return quick_tiling(lut, classic, T) ? (unsigned)T.off << 8 | (unsigned)T.n : mcw::TESTS;
    }
    __device__ __forceinline__ int code(int off) const { return d_lut[off]; }
    __device__ __forceinline__ bool geo(unsigned w, mcw::Geo &q) const {
        const unsigned row = w / g.WX, xw = w - row * g.WX;
        q.z = (int)(row / (unsigned)g.NY);
        q.y = (int)(row - (unsigned)q.z * (unsigned)g.NY);
        q.x0 = 32 * (int)xw - g.xoff;
        q.WX = g.WX;
        q.slice = g.WX * (unsigned)g.NY;
        q.inm = mcw::bit_range(-q.x0, g.NX - q.x0);
        q.hxm = mcw::bit_range(-q.x0, g.NX - 1 - q.x0);
        q.hy = q.y < g.NY - 1;
        q.hz = q.z < g.NZ - 1;
        q.nx = xw + 1 < g.WX;
        q.tag = 0;
        return true;
    }
    __device__ __forceinline__ void voxel_word(const mcw::Geo &q, int &wx, int &vy, int &vz) const {
        wx = (g.lo0 + q.x0) >> 5;
        vy = g.lo1 + q.y;
        vz = g.lo2 + q.z;
    }
    __device__ __forceinline__ void shifts(const mcw::Out &, unsigned, const uint4 &total, unsigned &e, unsigned &c) const {
        e = 0;
        c = total.x;   // c-vertices follow every edge vertex
    }
    __device__ __forceinline__ mcw::CubeTiling tests(const mcw::Geo &, int x, int y, int z, int lut) const {
        return tested_tiling(g, x, y, z, lut, classic);
    }
    __device__ __forceinline__ void cvertex(const mcw::Geo &, int x, int y, int z, int id) const {
        float c[8];
        cube_values(g, x, y, z, c);
        emit_cvertex(c, x, y, z, (float)g.lo0, (float)g.lo1, (float)g.lo2, id, pts, ccand, nccand, cap);
        mark_near(near, id);
    }
    struct Edge {
        float c0, c1;
    };
    __device__ __forceinline__ Edge edge(int x, int y, int z, int ax, int) const {
        const int vx = g.lo0 + x, vy = g.lo1 + y, vz = g.lo2 + z;
        if (vx >= 1 && vx + 1 <= g.dx - 2 && vy >= 1 && vy + 1 <= g.dy - 2 && vz >= 1 && vz + 1 <= g.dz - 2) {
            const float *q = g.vol + ((long long)vx + (long long)vy * g.dx + (long long)vz * g.dxy);
            return Edge{ival(g, q), ival(g, q + (ax == 0 ? 1ll : (ax == 1 ? (long long)g.dx : g.dxy)))};
        }
        return Edge{gval(g, x, y, z), gval(g, x + (ax == 0), y + (ax == 1), z + (ax == 2))};
    }
    __device__ __forceinline__ vec3d vertex(const Edge &c, int x, int y, int z, int ax, int id) const {
        return edge_vertex(c.c0, c.c1, x, y, z, ax, (float)g.lo0, (float)g.lo1, (float)g.lo2, id, cand, ncand, cap, near);
    }
};

// ---- adjoint of the vertex positions w.r.t. the processed volume -----------------
// Same value fetch as gval, also returning the voxel the value depends on (-1
// for padding, a darkened boundary voxel clamped to edge_max, or a value
// clamped to FLT_EPSILON: those are constant in the forward pass).
__device__ __forceinline__ float gval_src(const GV &g, int x, int y, int z, long long &src) {
    const long long j = (long long)(g.lo0 + x) + (long long)(y + g.lo1) * g.dx + (long long)(z + g.lo2) * g.dxy;
    float v;
    src = -1;
    if (j < g.nvox) {
        v = __ldg(g.vol + j);
        src = j;
        int vx = g.lo0 + x, vy = y + g.lo1, vz = z + g.lo2;   // wrapped as in gval
        if (vx >= g.dx) {
            vx -= g.dx;
            vy++;
        }
        if (vy >= g.dy) {
            vy -= g.dy;
            vz++;
        }
        if ((vx == 0 || vy == 0 || vz == 0 || vx == g.dx - 1 || vy == g.dy - 1 || vz == g.dz - 1) && !(v <= g.edge_max)) {
            v = g.edge_max;
            src = -1;
        }
        v = __fsub_rn(v, g.iso);
    } else {
        v = g.pad;
    }
    if (fabsf(v) < N2M_FLT_EPS) {
        v = N2M_FLT_EPS;
        src = -1;
    }
    return v;
}

// u = c0/(c0-c1): du/dc0 = -c1/(c0-c1)^2, du/dc1 = c0/(c0-c1)^2
__device__ __forceinline__ void edge_adjoint(float gax, float c0, float c1, long long s0, long long s1, float *gs) {
    const float den = c0 - c1;
    if (den == 0.f || gax == 0.f) return;
    const float inv2 = 1.f / (den * den);
    if (s0 >= 0) atomicAdd(gs + s0, -gax * c1 * inv2);
    if (s1 >= 0) atomicAdd(gs + s1, gax * c0 * inv2);
}

__device__ __forceinline__ float comp(const float3 &v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }

// one warp per active word; gv = dL/d(raw vertex position)
__global__ void __launch_bounds__(256) k_mc_backward(GV g, bool classic, const uint4 *__restrict__ words,
                                                     const uint4 *__restrict__ act, unsigned nactive,
                                                     const float3 *__restrict__ gv, float *gs) {
    grid_wait();
    const unsigned lane = threadIdx.x & 31u;
    for (unsigned aw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; aw < nactive; aw += (gridDim.x * blockDim.x) >> 5) {
        const uint4 a = act[aw];
        const unsigned w = a.x, row = w / g.WX, xw = w - row * g.WX;
        const int z = (int)(row / (unsigned)g.NY), y = (int)(row - (unsigned)z * (unsigned)g.NY);
        const int x = (int)(xw * 32u + lane) - g.xoff;
        const uint4 m = words[w];
        const bool in = x >= 0 && x < g.NX;
        const bool hx = in && x < g.NX - 1, hy = in && y < g.NY - 1, hz = in && z < g.NZ - 1;
        const bool cube = hx && hy && hz;
        const bool ex = (m.x >> lane) & 1u, ey = (m.y >> lane) & 1u, ez = (m.z >> lane) & 1u;
        float c[8];
        long long sr[8];
        if (in) {
            c[0] = gval_src(g, x, y, z, sr[0]);
            c[1] = hx ? gval_src(g, x + 1, y, z, sr[1]) : c[0];
            c[3] = hy ? gval_src(g, x, y + 1, z, sr[3]) : c[0];
            c[4] = hz ? gval_src(g, x, y, z + 1, sr[4]) : c[0];
            if (cube) {
                c[2] = gval_src(g, x + 1, y + 1, z, sr[2]);
                c[5] = gval_src(g, x + 1, y, z + 1, sr[5]);
                c[6] = gval_src(g, x + 1, y + 1, z + 1, sr[6]);
                c[7] = gval_src(g, x, y + 1, z + 1, sr[7]);
            }
        }
        if (ex | ey | ez) {
            const unsigned lt = (1u << lane) - 1u;
            int id = (int)(m.w + __popc(m.x & lt) + __popc(m.y & lt) + __popc(m.z & lt));
            if (ex) { edge_adjoint(gv[id].x, c[0], c[1], sr[0], sr[1], gs); id++; }
            if (ey) { edge_adjoint(gv[id].y, c[0], c[3], sr[0], sr[3], gs); id++; }
            if (ez) edge_adjoint(gv[id].z, c[0], c[4], sr[0], sr[4], gs);
        }
        Tiling T = {0, 0, false};
        if (cube) {
            const int lut = cube_lut(c);
            if (lut != 0 && lut != 255) T = select_tiling(c, lut, classic);
        }
        int cb = T.cv;
        for (int d = 1; d < 32; d <<= 1) {
            const int b = __shfl_up_sync(0xffffffffu, cb, d);
            if ((int)lane >= d) cb += b;
        }
        cb -= T.cv;
        if (!T.cv) continue;
        // c-vertex = mean of the cube's crossing edge vertices
        const float3 gc = gv[a.z + cb];
        int n = 0;
        for (int e = 0; e < 12; e++) n += (c[k_edge[e][2]] > 0.f) != (c[k_edge[e][3]] > 0.f);
        if (!n) continue;
        const float inv = 1.f / (float)n;
        for (int e = 0; e < 12; e++) {
            const int ax = k_edge[e][1], ca = k_edge[e][2], cbn = k_edge[e][3];
            if ((c[ca] > 0.f) == (c[cbn] > 0.f)) continue;
            edge_adjoint(comp(gc, ax) * inv, c[ca], c[cbn], sr[ca], sr[cbn], gs);
        }
    }
}

// vertices within 1.5e-5 of a c-vertex candidate become weld candidates too
__global__ void k_ccand(const vec3d *__restrict__ pts, int np, const int *__restrict__ cc, int ncc, int *cand,
                        unsigned *ncand, int cap) {
    grid_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
        const vec3d a = pts[i];
        for (int k = 0; k < ncc; k++) {
            const int j = cc[k];
            if (j == i) continue;
            const vec3d b = pts[j];
            const double dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
            if (fabs(dx) < 1.5e-5 && fabs(dy) < 1.5e-5 && fabs(dz) < 1.5e-5) {
                unsigned q = atomicAdd(ncand, 1u);
                if (q < (unsigned)cap) cand[q] = i;
                break;
            }
        }
    }
}

GV make_gv(const McGrid &g) {
    GV v;
    v.vol = g.vol;
    v.dx = g.dim[0]; v.dy = g.dim[1]; v.dz = g.dim[2];
    v.dxy = (long long)g.dim[0] * g.dim[1];
    v.nvox = v.dxy * g.dim[2];
    v.lo0 = g.lo[0]; v.lo1 = g.lo[1]; v.lo2 = g.lo[2];
    v.NX = g.n[0]; v.NY = g.n[1]; v.NZ = g.n[2];
    v.xoff = g.lo[0] & 31;
    v.WX = (unsigned)(g.n[0] + v.xoff + 31) / 32u;
    v.iso = g.iso; v.edge_max = g.edge_max; v.pad = g.pad_val;
    return v;
}
}  // namespace

namespace {
n2m_status grid_words(const GV &v, size_t &nwords) {
    nwords = (size_t)v.WX * v.NY * v.NZ;
    if (nwords >= 0xffffffffULL - mcw::SUB) {
        n2m_set_error("grid too large");
        return N2M_ERR_TOO_LARGE;
    }
    return N2M_OK;
}
}  // namespace

n2m_status mc_count(const McGrid &g, int variant, McWork &w, uint4 *d_total, cudaStream_t s, OdWork &od, const OdRepair *repair,
                    const LabelPost *post) {
    const GV v = make_gv(g);
    size_t nwords;
    CKS(grid_words(v, nwords));
    mcw::Out o;
    CKS(mcw::prepare(w, nwords, d_total, o));
    CKS(w.signs.ensure(nwords * sizeof(unsigned)));
    unsigned *signs = w.signs.as<unsigned>();
    const unsigned blocks = (unsigned)std::min<size_t>((nwords + 255) / 256, 152u * 16u), wv = (unsigned)(v.dx + 31) / 32u;
    if (post || repair) {
        const SignMap map{post ? post->S : od.vsign.as<unsigned>(), wv, post ? 0u : (unsigned)(v.dy + 7) / 8u, v.dy};
        n2m_launch(k_signs_bits, blocks, 256, 0, s, v, (unsigned)nwords, signs, map);
    } else {
        const unsigned nrows = (unsigned)g.n[1] * (unsigned)g.n[2];
        n2m_launch(k_signs, std::min<unsigned>((nrows + 7) / 8, 152u * 16u), 256, 0, s, v, nrows, signs);
    }
    const bool classic = variant == N2M_CUBES_CLASSIC_TABLE;
    const Policy pol{v, classic, nullptr, nullptr, nullptr, nullptr, nullptr, 0};
    mcw::Marks marks{nullptr, v.dx, v.dy, v.dz, wv};
    if (post || repair) CKS(od_marks(od, g.dim, &marks.need, s));
    CKS(mcw::count_signs(pol, signs, o, marks, s));
    // final values where anything below reads them
    if (repair) CKS(od_repair(*repair, s));
    else if (post) CKS(lab_apply((float *)g.vol, v.dx, v.dy, v.dz, marks.need, *post, s));
    return mcw::count_values(pol, signs, w, o, !classic, s);
}

n2m_status mc_emit(const McGrid &g, int variant, McWork &w, MarchOut *d_out, const MeshRoom &room, vec3d *d_pts, vec3i *d_tris,
                   int *d_cand, int cand_cap, unsigned *d_near, cudaStream_t s) {
    const GV v = make_gv(g);
    size_t nwords;
    CKS(grid_words(v, nwords));
    mcw::Out o;
    CKS(mcw::prepare(w, nwords, &d_out->tot, o));
    const Policy pol{v, variant == N2M_CUBES_CLASSIC_TABLE, d_pts, d_cand, d_cand + cand_cap, &d_out->ncand, &d_out->nccand,
                     cand_cap, d_near};
    return mcw::emit(pol, w.signs.as<unsigned>(), w, o, room, d_tris, s);
}

n2m_status mc_backward(const McGrid &g, int variant, McWork &w, const McCounts &c, const float3 *d_gv, float *d_gs,
                       cudaStream_t s) {
    const GV v = make_gv(g);
    if (c.nactive == 0) return N2M_OK;
    const unsigned blocks = std::min<unsigned>((c.nactive + 7) / 8, 152u * 16u);
    n2m_launch(k_mc_backward, blocks, 256, 0, s, v, variant == N2M_CUBES_CLASSIC_TABLE, w.words.as<uint4>(), w.act.as<uint4>(),
               c.nactive, d_gv, d_gs);
    CKL();
    return N2M_OK;
}

n2m_status mc_ccand_scan(const vec3d *d_pts, int np, const int *d_ccand, int nccand, int *d_cand,
                         unsigned *d_ncand, int cand_cap, cudaStream_t s) {
    if (nccand <= 0) return N2M_OK;
    const int blocks = (np + 255) / 256 < 4096 ? (np + 255) / 256 : 4096;
    n2m_launch(k_ccand, blocks > 0 ? blocks : 1, 256, 0, s, d_pts, np, d_ccand, nccand, d_cand, d_ncand, cand_cap);
    CKL();
    return N2M_OK;
}
