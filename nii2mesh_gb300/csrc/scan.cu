// scan.cu — device-wide exclusive prefix sum, in place.  Reduce-then-scan: per-tile
// sums, a single-CTA scan of the tile sums (looping for any count), then a per-tile scan
// that adds its offset.
#include "n2m_internal.cuh"

namespace {
constexpr int SB = 256;          // threads per CTA
constexpr int SI = 8;            // items per thread
constexpr int TILE = SB * SI;    // items per tile

__device__ unsigned block_exscan_u32(unsigned &v) {
    __shared__ unsigned wsum[SB / 32];
    __shared__ unsigned tot;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        const unsigned s = lane < SB / 32 ? wsum[lane] : 0u;
        unsigned si = s;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(0xffffffffu, si, o);
            if (lane >= o) si += t;
        }
        if (lane < SB / 32) wsum[lane] = si - s;
    }
    __syncthreads();
    const unsigned woff = wsum[wid];
    if (threadIdx.x == SB - 1) tot = woff + incl;
    v = woff + incl - v;
    __syncthreads();
    const unsigned total = tot;
    __syncthreads();
    return total;
}

__global__ void __launch_bounds__(SB) k_tile_sums_u32(const unsigned *__restrict__ d, size_t n, unsigned *part) {
    grid_wait();
    const size_t base = (size_t)blockIdx.x * TILE;
    unsigned s = 0;
    for (int i = 0; i < SI; i++) {
        const size_t k = base + (size_t)i * SB + threadIdx.x;
        if (k < n) s += d[k];
    }
    const unsigned t = block_exscan_u32(s);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

__global__ void __launch_bounds__(SB) k_scan_parts_u32(unsigned *part, size_t np, unsigned *total) {
    grid_wait();
    unsigned carry = 0;
    for (size_t base = 0; base < np; base += SB) {
        const size_t k = base + threadIdx.x;
        unsigned v = k < np ? part[k] : 0u;
        const unsigned t = block_exscan_u32(v);
        if (k < np) part[k] = v + carry;
        carry += t;
    }
    if (threadIdx.x == 0) *total = carry;
}

__global__ void __launch_bounds__(SB) k_tile_scan_u32(unsigned *d, size_t n, const unsigned *part) {
    grid_wait();
    const size_t base = (size_t)blockIdx.x * TILE + (size_t)threadIdx.x * SI;
    unsigned it[SI], s = 0;
    for (int i = 0; i < SI; i++) {
        it[i] = base + i < n ? d[base + i] : 0u;
        s += it[i];
    }
    block_exscan_u32(s);
    unsigned run = s + part[blockIdx.x];
    for (int i = 0; i < SI; i++) {
        if (base + i < n) d[base + i] = run;
        run += it[i];
    }
}
}  // namespace

n2m_status scan_u32(unsigned *d, size_t n, unsigned *d_total, ScanWork &w, cudaStream_t s) {
    if (n == 0) {
        CK(cudaMemsetAsync(d_total, 0, sizeof(unsigned), s));
        return N2M_OK;
    }
    const size_t tiles = (n + TILE - 1) / TILE;
    CKS(w.part.ensure(tiles * sizeof(unsigned)));
    n2m_launch(k_tile_sums_u32, (unsigned)tiles, SB, 0, s, d, n, w.part.as<unsigned>());
    n2m_launch(k_scan_parts_u32, 1, SB, 0, s, w.part.as<unsigned>(), tiles, d_total);
    n2m_launch(k_tile_scan_u32, (unsigned)tiles, SB, 0, s, d, n, w.part.as<unsigned>());
    CKL();
    return N2M_OK;
}
