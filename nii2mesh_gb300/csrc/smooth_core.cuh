// smooth_core.cuh — the running range, bounding box and non-finite count of the
// values that a kernel produces.
#pragma once
#include <float.h>
#include <limits.h>

#include "exact.cuh"
#include "n2m_internal.cuh"

namespace smooth {
// running range / bbox / non-finite count of the values a thread produced
struct Acc {
    float mn, mx;
    int lo0, lo1, lo2, hi0, hi1, hi2;
    unsigned nf;
    __device__ void init() {
        mn = FLT_MAX; mx = -FLT_MAX;
        lo0 = lo1 = lo2 = INT_MAX;
        hi0 = hi1 = hi2 = INT_MIN;
        nf = 0;
    }
    __device__ __forceinline__ void add(float v, int x, int y, int z, float iso) {
        if (!isfinite(v)) { nf++; return; }
        mn = fminf(mn, v);
        mx = fmaxf(mx, v);
        if (v >= iso) {
            lo0 = min(lo0, x); lo1 = min(lo1, y); lo2 = min(lo2, z);
            hi0 = max(hi0, x); hi1 = max(hi1, y); hi2 = max(hi2, z);
        }
    }
    // the K values of one lane's run along z (x, y fixed; z = z0 + k), those
    // whose bit is set in `take`: min/max per value, the bbox once per run
    template <int K>
    __device__ __forceinline__ void add_run(const float (&r)[K], unsigned take, int x, int y, int z0, float iso) {
        unsigned ge = 0;
#pragma unroll
        for (int k = 0; k < K; k++) {
            if (!(take >> k & 1u)) continue;
            const float v = r[k];
            if (!isfinite(v)) { nf++; continue; }
            mn = fminf(mn, v);
            mx = fmaxf(mx, v);
            ge |= (unsigned)(v >= iso) << k;
        }
        if (ge) {
            lo0 = min(lo0, x); lo1 = min(lo1, y); lo2 = min(lo2, z0 + __ffs(ge) - 1);
            hi0 = max(hi0, x); hi1 = max(hi1, y); hi2 = max(hi2, z0 + 31 - __clz(ge));
        }
    }
    // block-wide reduction, one set of atomics per CTA
    __device__ void flush(VolStats *st, bool minmax) {
        const unsigned full = 0xffffffffu;
        for (int o = 16; o; o >>= 1) {
            mn = fminf(mn, __shfl_xor_sync(full, mn, o));
            mx = fmaxf(mx, __shfl_xor_sync(full, mx, o));
            lo0 = min(lo0, __shfl_xor_sync(full, lo0, o)); lo1 = min(lo1, __shfl_xor_sync(full, lo1, o));
            lo2 = min(lo2, __shfl_xor_sync(full, lo2, o)); hi0 = max(hi0, __shfl_xor_sync(full, hi0, o));
            hi1 = max(hi1, __shfl_xor_sync(full, hi1, o)); hi2 = max(hi2, __shfl_xor_sync(full, hi2, o));
            nf += __shfl_xor_sync(full, nf, o);
        }
        __shared__ Acc part[32];
        const int nthr = blockDim.x * blockDim.y;
        const int tid = threadIdx.y * blockDim.x + threadIdx.x;
        if ((tid & 31) == 0) part[tid >> 5] = *this;
        __syncthreads();
        if (tid == 0) {
            Acc a = part[0];
            for (int w = 1; w < (nthr + 31) / 32; w++) {
                const Acc &b = part[w];
                a.mn = fminf(a.mn, b.mn); a.mx = fmaxf(a.mx, b.mx);
                a.lo0 = min(a.lo0, b.lo0); a.lo1 = min(a.lo1, b.lo1); a.lo2 = min(a.lo2, b.lo2);
                a.hi0 = max(a.hi0, b.hi0); a.hi1 = max(a.hi1, b.hi1); a.hi2 = max(a.hi2, b.hi2);
                a.nf += b.nf;
            }
            // hundreds of blocks at one cache line: only what still changes something
            auto low = [](int *p, int v) { if (v < *(volatile int *)p) atomicMin(p, v); };
            auto high = [](int *p, int v) { if (v > *(volatile int *)p) atomicMax(p, v); };
            if (minmax && a.mn <= a.mx) {
                low(&st->vmin, f2ord(a.mn));
                high(&st->vmax, f2ord(a.mx));
            }
            if (a.lo0 != INT_MAX) {
                low(&st->lo[0], a.lo0); low(&st->lo[1], a.lo1); low(&st->lo[2], a.lo2);
                high(&st->hi[0], a.hi0); high(&st->hi[1], a.hi1); high(&st->hi[2], a.hi2);
            }
            if (a.nf) atomicAdd(&st->nonfinite, a.nf);
        }
    }
};
}  // namespace smooth
