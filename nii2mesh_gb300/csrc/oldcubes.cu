// oldcubes.cu — Bourke's classic marching cubes as the reference's
// USE_CLASSIC_CUBES build runs it (src/oldcubes.c:22-40, :401-463, :465-522),
// with edge-owned vertices instead of three private vertices per triangle.
//
// Cubes span [lo, hi-2] (absolute voxel coordinates, no padding).  A corner
// bit is set when value < isolevel.  The reference interpolates every copy
// of an edge vertex in double, oriented as the copying cube lists the edge,
// and its weld keeps the position of the LAST copy (src/meshify.c:99-100).
// Each edge here is computed once, in double, in the orientation of the last
// cube (raster order) that uses it, so positions are the reference's
// post-weld positions bit for bit.  The weld candidates (the few vertices near
// a grid point) can merge with vertices of other edges; the reference merges
// copies, so oc_copies / oc_copy_positions list every triangle corner that
// names a candidate (3*triangle + corner, its order in the reference's
// triangle soup) with the position the emitting cube gives that copy, and the
// host weld groups the copies as the reference does.
#include <algorithm>

#include "mc_tables.h"
#include "mcwords.cuh"

namespace {
__device__ const unsigned short d_edge[256] = N2M_CLASSIC_EDGE_INIT;
__device__ const signed char d_tri[256 * 16] = N2M_CLASSIC_TRI_INIT;

struct OV {
    const float *vol;
    int dx, dy, dz;
    long long dxy;
    int lo0, lo1, lo2, hi0, hi1, hi2;   // cube range [lo, hi-2]
    int NX, NY, NZ;                     // grid points: hi - lo
    unsigned WX;            // words per row
    int xoff;               // bit of grid point x = 0 in a row's first word
    float iso, edge_max;
};

// darkened voxel value (src/meshify.c:368-369)
__device__ __forceinline__ float oval(const OV &g, int X, int Y, int Z) {
    float v = __ldg(g.vol + (long long)Z * g.dxy + (long long)Y * g.dx + X);
    if (X == 0 || Y == 0 || Z == 0 || X == g.dx - 1 || Y == g.dy - 1 || Z == g.dz - 1) v = fminf(g.edge_max, v);
    return v;
}

__device__ __forceinline__ int ocube_ntri(int ci) {
    if (!d_edge[ci]) return 0;
    int n = 0;
    while (n < 5 && d_tri[ci * 16 + 3 * n] != -1) n++;
    return n;
}

// ---- signs --------------------------------------------------------------------
// Bit b of word (z*NY + y)*WX + xw is grid point x = 32*xw - xoff + b (voxel column
// 32*(lo0/32 + xw) + b): set when the point is below the isolevel, darkened value
// included; bits outside the grid are 0.

// Signs from a volume: a warp per row, OS_W words at a time with all their loads in flight.
constexpr int OS_W = 16;
__global__ void __launch_bounds__(256) k_oc_signs(OV g, unsigned nrows, unsigned *signs) {
    grid_wait();
    const int lane = threadIdx.x & 31;
    for (unsigned row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < nrows; row += (gridDim.x * blockDim.x) >> 5) {
        const int y = (int)(row % (unsigned)g.NY), z = (int)(row / (unsigned)g.NY);
        const int vy = g.lo1 + y, vz = g.lo2 + z;
        const bool rface = vy == 0 || vz == 0 || vy == g.dy - 1 || vz == g.dz - 1;
        const float *rp = g.vol + (long long)vz * g.dxy + (long long)vy * g.dx + g.lo0;
        unsigned *out = signs + (size_t)row * g.WX;
        for (unsigned xw0 = 0; xw0 < g.WX; xw0 += OS_W) {
            float raw[OS_W];
#pragma unroll
            for (int k = 0; k < OS_W; k++) {
                const int x = (int)(xw0 + k) * 32 + lane - g.xoff;
                raw[k] = xw0 + k < g.WX && x >= 0 && x < g.NX ? __ldg(rp + x) : 0.f;
            }
            unsigned mine = 0;
#pragma unroll
            for (int k = 0; k < OS_W; k++) {
                const int x = (int)(xw0 + k) * 32 + lane - g.xoff, vx = g.lo0 + x;
                const float v = rface || vx == 0 || vx == g.dx - 1 ? fminf(g.edge_max, raw[k]) : raw[k];
                const unsigned m = __ballot_sync(0xffffffffu, x >= 0 && x < g.NX && v < g.iso);
                if (lane == k) mine = m;
            }
            if (lane < OS_W && xw0 + lane < g.WX) out[xw0 + lane] = mine;
        }
    }
}

// Signs from a sign bitmap of the volume with bit = value >= iso (OdWork::vsign, wv words
// per row, nys groups of 8 rows; nys 0: plain row words), one thread per word: the
// complement, and a darkened point is below the isolevel if its voxel or edge_max is.
__global__ void __launch_bounds__(256) k_oc_signs_bits(OV g, unsigned nwords, unsigned *signs,
                                                       const unsigned *__restrict__ vsign, unsigned wv, unsigned nys) {
    grid_wait();
    const bool dark = g.edge_max < g.iso;
    for (unsigned w = blockIdx.x * blockDim.x + threadIdx.x; w < nwords; w += gridDim.x * blockDim.x) {
        const unsigned row = w / g.WX, xw = w - row * g.WX;
        const int vz = g.lo2 + (int)(row / (unsigned)g.NY), vy = g.lo1 + (int)(row % (unsigned)g.NY);
        const int x0 = 32 * (int)xw - g.xoff, vb = g.lo0 + x0;
        unsigned m = ~__ldg(vsign + (nys ? od_vsign_word((unsigned)vb, (unsigned)vy, (unsigned)vz, wv, nys)
                                         : ((size_t)vz * g.dy + vy) * wv + ((unsigned)vb >> 5)));
        if (dark) {
            if (vy == 0 || vz == 0 || vy == g.dy - 1 || vz == g.dz - 1) m = 0xffffffffu;
            else m |= ~mcw::bit_range(vb == 0 ? 1 : 0, g.dx - 1 - vb);
        }
        signs[w] = m & mcw::bit_range(-x0, g.NX - x0);
    }
}

__device__ __forceinline__ void ogeo(const OV &g, unsigned w, mcw::Geo &q) {
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
}

// ---- emit pass -------------------------------------------------------------------
// exact float -> double and int -> double by assembling the bits: conversions issue on the pipe that this part
// shares with FP64, which bounds the interpolation below
__device__ __forceinline__ double f2d(float f) {
    const unsigned u = __float_as_uint(f), e = (u >> 23) & 0xffu;
    if (e - 1u < 0xfeu)   // normal
        return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(u << 29));
    return (double)f;
}
__device__ __forceinline__ double i2d(int v) {   // v >= 0
    if (v == 0) return 0.0;
    const int p = 31 - __clz(v);
    const unsigned long long m = (unsigned long long)(unsigned)v << (52 - p);
    return __longlong_as_double((long long)(((unsigned long long)(p + 1023) << 52) + (m & 0xfffffffffffffull)));
}

// The edge vertex of grid point (x, y, z) along axis ax, interpolated as the
// last cube (raster order) that lists the edge orients it.  VertexInterp
// (src/oldcubes.c:22-40) moves only the coordinate along the edge:
// p = p1 + mu*(p2-p1) with mu = (iso - v1)/(v2 - v1), and p2 - p1 is 1 or -1, so the
// product is mu or -mu.  A vertex near a grid point becomes a weld candidate (a wider
// float test spares the others the double one).
__device__ __forceinline__ vec3d oc_vertex(const OV &g, float v0, float v1, int x, int y, int z, int ax, int id, int *cand,
                                           unsigned *ncand, int cap, unsigned *near) {
    const int X = g.lo0 + x, Y = g.lo1 + y, Z = g.lo2 + z;
    const int c0 = g.lo0, c1 = g.lo1, c2 = g.lo2, e0 = g.hi0 - 2, e1 = g.hi1 - 2, e2 = g.hi2 - 2;
    bool fwd = true;   // z: every user lists the edge bottom to top
    if (ax == 0) {     // last user: (X,Y,Z) fwd > (X,Y-1,Z) rev > (X,Y,Z-1) fwd > (X,Y-1,Z-1) rev
        if (Y <= e1 && Z <= e2) fwd = true;
        else if (Y - 1 >= c1 && Z <= e2) fwd = false;
        else fwd = Y <= e1 && Z - 1 >= c2;
    } else if (ax == 1) {   // (X,Y,Z) rev > (X-1,Y,Z) fwd > (X,Y,Z-1) rev > (X-1,Y,Z-1) fwd
        if (X <= e0 && Z <= e2) fwd = false;
        else if (X - 1 >= c0 && Z <= e2) fwd = true;
        else fwd = !(X <= e0 && Z - 1 >= c2);
    }
    const int i0 = ax == 0 ? X : (ax == 1 ? Y : Z);
    const float va = fwd ? v0 : v1, vb = fwd ? v1 : v0;
    const double iso = f2d(g.iso), da = f2d(va), db = f2d(vb);
    const double mu = __ddiv_rn(__dsub_rn(iso, da), __dsub_rn(db, da));
    const double r = __dadd_rn(i2d(fwd ? i0 : i0 + 1), fwd ? mu : -mu);
    const float mf = __fdividef(__fsub_rn(g.iso, va), __fsub_rn(vb, va));   // within 1e-6 of mu, or 0, Inf or NaN
    if (!(mf > NEAR_CORNER + 1e-5f && mf < 1.f - NEAR_CORNER - 1e-5f)) {
        mark_near(near, id);
        if (!(mf > 2e-5f && mf < 1.f - 2e-5f) && fabs(r - rint(r)) < 1.5e-5) {
            const unsigned k = atomicAdd(ncand, 1u);
            if (k < (unsigned)cap) cand[k] = id;
        }
    }
    return {ax == 0 ? r : i2d(X), ax == 1 ? r : i2d(Y), ax == 2 ? r : i2d(Z)};
}

// mcwords.cuh's policy for the unpadded classic grid
struct Policy {
    static constexpr bool MULTI = false, REVERSE = false, CVERTS = false;
    static constexpr int CTAS = 8, EV = 2;   // of k_emit: CTAs per SM, vertices per lane in flight
    OV g;
    vec3d *pts;
    int *cand;
    unsigned *ncand;
    int cap;
    unsigned *near;
    __device__ __forceinline__ unsigned quick(int lut) const { return (unsigned)(lut * 16) << 8 | (unsigned)ocube_ntri(lut); }
    __device__ __forceinline__ int code(int off) const { return d_tri[off]; }
    __device__ __forceinline__ bool geo(unsigned w, mcw::Geo &q) const {
        ogeo(g, w, q);
        return true;
    }
    __device__ __forceinline__ void voxel_word(const mcw::Geo &q, int &wx, int &vy, int &vz) const {
        wx = (g.lo0 + q.x0) >> 5;
        vy = g.lo1 + q.y;
        vz = g.lo2 + q.z;
    }
    __device__ __forceinline__ void shifts(const mcw::Out &, unsigned, const uint4 &, unsigned &e, unsigned &c) const { e = c = 0; }
    __device__ __forceinline__ mcw::CubeTiling tests(const mcw::Geo &, int, int, int, int) const { return {0, 0, false}; }
    __device__ __forceinline__ void cvertex(const mcw::Geo &, int, int, int, int) const {}
    struct Edge {
        float v0, v1;
    };
    __device__ __forceinline__ Edge edge(int x, int y, int z, int ax, int) const {
        const int X = g.lo0 + x, Y = g.lo1 + y, Z = g.lo2 + z;
        return Edge{oval(g, X, Y, Z), oval(g, X + (ax == 0), Y + (ax == 1), Z + (ax == 2))};
    }
    __device__ __forceinline__ vec3d vertex(const Edge &v, int x, int y, int z, int ax, int id) const {
        return oc_vertex(g, v.v0, v.v1, x, y, z, ax, id, cand, ncand, cap, near);
    }
};

// weld candidates as a bitmap over the vertices
__global__ void k_oc_candbits(const int *__restrict__ cand, unsigned ncand, unsigned *bits) {
    grid_wait();
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < ncand; i += gridDim.x * blockDim.x) {
        const unsigned v = (unsigned)cand[i];
        atomicOr(bits + (v >> 5), 1u << (v & 31u));
    }
}

// every triangle corner (3*t + c) that names a weld candidate (bit set)
__global__ void k_oc_copies(const vec3i *__restrict__ tris, unsigned nt, const unsigned *__restrict__ bits,
                            unsigned *out, unsigned *count, unsigned cap) {
    grid_wait();
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += gridDim.x * blockDim.x) {
        const vec3i T = tris[t];
        const int v[3] = {T.x, T.y, T.z};
#pragma unroll
        for (int c = 0; c < 3; c++)
            if ((__ldg(bits + ((unsigned)v[c] >> 5)) >> ((unsigned)v[c] & 31u)) & 1u) {
                const unsigned k = atomicAdd(count, 1u);
                if (k < cap) out[k] = 3u * t + (unsigned)c;
            }
    }
}

// Bourke's corners (bit 0: +x, 1: +y, 2: +z) and each edge's two corners, in
// the order VertexInterp takes them (src/oldcubes.c:418-441)
__constant__ unsigned char c_corner[8] = {0, 1, 3, 2, 4, 5, 7, 6};
__constant__ unsigned char c_edge_ab[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6},
                                               {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};

// The copy of a vertex that corner q = 3t + c holds in the reference's
// triangle soup: the cube that emitted triangle t (the word whose triangle
// range holds t, then the cube within it) and the position that cube's
// VertexInterp gives, in the edge's orientation within that cube.
__global__ void k_oc_copy_pos(OV g, const unsigned *__restrict__ signs, const uint4 *__restrict__ act, unsigned nact,
                              const vec3i *__restrict__ tris, const unsigned *__restrict__ qs, unsigned n, int *vid,
                              vec3d *pos) {
    grid_wait();
    const double iso = (double)g.iso;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned q = qs[i], t = q / 3u, c = q - 3u * t;
        unsigned lo = 0, hi = nact - 1;   // the last active word whose first triangle is <= t
        while (lo < hi) {
            const unsigned mid = lo + (hi - lo + 1) / 2;
            if (act[mid].y <= t) lo = mid;
            else hi = mid - 1;
        }
        const uint4 A = act[lo];
        mcw::Geo G;
        ogeo(g, A.x, G);
        const mcw::Corners K = mcw::load_corners(signs, A.x, G);
        unsigned k = t - A.y;
        int p = 0, ci = 0;
        for (unsigned mix = mcw::mixed_cubes(K, G); mix; mix &= mix - 1) {
            p = __ffs(mix) - 1;
            ci = mcw::cube_index(K.a, K.b, K.c, K.d, K.nxt, p);
            const unsigned nc = (unsigned)ocube_ntri(ci);
            if (k < nc) break;
            k -= nc;
        }
        const int e = d_tri[ci * 16 + 3 * (int)k + (int)c];
        const unsigned ca = c_corner[c_edge_ab[e][0]], cb = c_corner[c_edge_ab[e][1]];
        const int X = g.lo0 + G.x0 + p, Y = g.lo1 + G.y, Z = g.lo2 + G.z;
        const int ax = X + (int)(ca & 1u), ay = Y + (int)((ca >> 1) & 1u), az = Z + (int)(ca >> 2);
        const int bx = X + (int)(cb & 1u), by = Y + (int)((cb >> 1) & 1u), bz = Z + (int)(cb >> 2);
        const double va = oval(g, ax, ay, az), vb = oval(g, bx, by, bz);
        const double mu = __ddiv_rn(__dsub_rn(iso, va), __dsub_rn(vb, va));
        vec3d P = {(double)ax, (double)ay, (double)az};
        if (ax != bx) P.x = __dadd_rn(P.x, __dmul_rn(mu, (double)(bx - ax)));
        if (ay != by) P.y = __dadd_rn(P.y, __dmul_rn(mu, (double)(by - ay)));
        if (az != bz) P.z = __dadd_rn(P.z, __dmul_rn(mu, (double)(bz - az)));
        const vec3i T = tris[t];
        vid[i] = c == 0 ? T.x : (c == 1 ? T.y : T.z);
        pos[i] = P;
    }
}

OV make_ov(const float *vol, const int dim[3], const int lo[3], const int hi[3], float iso, float edge_max) {
    OV g;
    g.vol = vol;
    g.dx = dim[0]; g.dy = dim[1]; g.dz = dim[2];
    g.dxy = (long long)dim[0] * dim[1];
    g.lo0 = lo[0]; g.lo1 = lo[1]; g.lo2 = lo[2];
    g.hi0 = hi[0]; g.hi1 = hi[1]; g.hi2 = hi[2];
    g.NX = hi[0] - lo[0]; g.NY = hi[1] - lo[1]; g.NZ = hi[2] - lo[2];
    g.xoff = lo[0] & 31;
    g.WX = (unsigned)(g.NX + g.xoff + 31) / 32u;
    g.iso = iso;
    g.edge_max = edge_max;
    return g;
}
}  // namespace

n2m_status oc_count(const float *vol, const int dim[3], const int lo[3], const int hi[3], float iso, float edge_max,
                    McWork &w, uint4 *d_total, cudaStream_t s, OdWork &od, const OdRepair *repair, const LabelPost *post) {
    const OV g = make_ov(vol, dim, lo, hi, iso, edge_max);
    if (g.NX < 2 || g.NY < 2 || g.NZ < 2) {
        CK(cudaMemsetAsync(d_total, 0, sizeof(uint4), s));
        return N2M_OK;
    }
    const size_t nwords = (size_t)g.WX * g.NY * g.NZ;
    if (nwords >= 0xffffffffULL - mcw::SUB) {
        n2m_set_error("grid too large");
        return N2M_ERR_TOO_LARGE;
    }
    mcw::Out o;
    CKS(mcw::prepare(w, nwords, d_total, o));
    CKS(w.signs.ensure(nwords * sizeof(unsigned)));
    unsigned *signs = w.signs.as<unsigned>();
    const unsigned wblocks = (unsigned)std::min<size_t>((nwords + 255) / 256, 152u * 16u);
    const unsigned wv = (unsigned)(g.dx + 31) / 32u;
    if (post || repair) {
        n2m_launch(k_oc_signs_bits, wblocks, 256, 0, s, g, (unsigned)nwords, signs, post ? post->S : od.vsign.as<unsigned>(),
                   wv, post ? 0u : (unsigned)(g.dy + 7) / 8u);
    } else {
        const unsigned nrows = (unsigned)g.NY * (unsigned)g.NZ;
        n2m_launch(k_oc_signs, std::min<unsigned>((nrows + 7) / 8, 152u * 16u), 256, 0, s, g, nrows, signs);
    }
    const Policy pol{g, nullptr, nullptr, nullptr, 0};
    mcw::Marks marks{nullptr, g.dx, g.dy, g.dz, wv};
    if (post || repair) CKS(od_marks(od, dim, &marks.need, s));
    CKS(mcw::count_signs(pol, signs, o, marks, s));
    // final values where the emit reads them
    if (repair) CKS(od_repair(*repair, s));
    else if (post) CKS(lab_apply((float *)vol, g.dx, g.dy, g.dz, marks.need, *post, s));
    return mcw::count_values(pol, signs, w, o, false, s);
}

n2m_status oc_emit(const float *vol, const int dim[3], const int lo[3], const int hi[3], float iso, float edge_max,
                   McWork &w, MarchOut *d_out, const MeshRoom &room, vec3d *d_pts, vec3i *d_tris, int *d_cand,
                   int cand_cap, unsigned *d_near, cudaStream_t s) {
    const OV g = make_ov(vol, dim, lo, hi, iso, edge_max);
    if (g.NX < 2 || g.NY < 2 || g.NZ < 2) return N2M_OK;   // no cube: oc_count left zero counts and no words
    mcw::Out o;
    CKS(mcw::prepare(w, (size_t)g.WX * g.NY * g.NZ, &d_out->tot, o));
    return mcw::emit(Policy{g, d_pts, d_cand, &d_out->ncand, cand_cap, d_near}, w.signs.as<unsigned>(), w, o, room, d_tris, s);
}

n2m_status oc_copies(const vec3i *d_tris, int nt, int nv, const int *d_cand, int ncand, unsigned *d_bits,
                     unsigned *d_out, unsigned *d_count, unsigned cap, cudaStream_t s) {
    CK(cudaMemsetAsync(d_bits, 0, (size_t)(nv + 31) / 32 * sizeof(unsigned), s));
    CK(cudaMemsetAsync(d_count, 0, sizeof(unsigned), s));
    n2m_launch(k_oc_candbits, (unsigned)std::max(1, std::min((ncand + 255) / 256, 1024)), 256, 0, s, d_cand, (unsigned)ncand,
               d_bits);
    n2m_launch(k_oc_copies, (unsigned)std::max(1, std::min((nt + 255) / 256, 152 * 16)), 256, 0, s, d_tris, (unsigned)nt,
               d_bits, d_out, d_count, cap);
    CKL();
    return N2M_OK;
}

n2m_status oc_copy_positions(const float *vol, const int dim[3], const int lo[3], const int hi[3], float iso,
                             float edge_max, const McWork &w, unsigned nactive, const vec3i *d_tris, const unsigned *d_q,
                             int n, int *d_vid, vec3d *d_pos, cudaStream_t s) {
    const OV g = make_ov(vol, dim, lo, hi, iso, edge_max);
    if (n <= 0 || nactive == 0) return N2M_OK;
    n2m_launch(k_oc_copy_pos, (unsigned)std::min((n + 127) / 128, 1024), 128, 0, s, g, w.signs.as<unsigned>(),
               w.act.as<uint4>(), nactive, d_tris, d_q, (unsigned)n, d_vid, d_pos);
    CKL();
    return N2M_OK;
}
