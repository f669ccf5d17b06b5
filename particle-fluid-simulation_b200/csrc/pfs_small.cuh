// pfs_small.cuh — the density pass of a small world, one warp per slot, shared by
// the FP32 form (Dens32, pfs_neighbors.cu) and the FP16-cell form (Dens16,
// pfs_fp16.cu).
//
// Up to SMALL_SLOTS slots the flat walk is latency: 16 thread blocks for 2,047
// particles, each thread of which looks up 27 ranges and walks them alone (34 us),
// after two launches for a spatial order that only serves caches.  Here lanes
// 0 .. 26 look a slot's ranges up together, the lanes hold 32 candidates at a time
// and evaluate the in-range terms together, and only the sums run in order: 10 us
// for 2,047 slots, 16 for 16,384, and the slots are their own processing order.
// Candidates, terms, order, lists and queue are the flat walk's.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "pfs_common.cuh"
#include "pfs_step.cuh"

namespace pfs {
namespace {

constexpr int SMALL_THREADS = 128;

template <class F>
__global__ void __launch_bounds__(SMALL_THREADS)
k_density_small(DevParams P, F form, const float4* __restrict__ xp, const int2* __restrict__ table,
                uint32_t* __restrict__ order, float2* __restrict__ rr, float4* __restrict__ fr,
                int32_t* __restrict__ nlist,
                int32_t* __restrict__ ncount, uint32_t* __restrict__ scanq, uint32_t* __restrict__ scanq_n,
                uint32_t* __restrict__ err) {
    const uint32_t full = 0xffffffffu, n = P.n;
    const uint32_t i = (blockIdx.x * SMALL_THREADS + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    if (i >= n) return;
    const float4 sp = xp[i];
    const float h = P.h;
    // lane d < 27: sample point d (z outer, x inner), its cell and its table range
    const int dz = lane / 9, dy = (lane / 3) % 3, dx = lane % 3;
    auto off = [&](int d) { return d == 0 ? PFS_MUL(h, -1.0f) : (d == 1 ? PFS_MUL(h, 0.0f) : h); };
    const float sx = PFS_ADD(sp.x, off(dx)), sy = PFS_ADD(sp.y, off(dy)), sz = PFS_ADD(sp.z, off(dz));
    const bool vx = !(sx < P.minx) && !(sx > P.maxx), vy = !(sy < P.miny) && !(sy > P.maxy),
               vz = !(sz < P.minz) && !(sz > P.maxz);
    int32_t cx = cell_coord(sx, P.minx, h), cy = cell_coord(sy, P.miny, h), cz = cell_coord(sz, P.minz, h);
    const bool dens = vx && vy && vz && lane < 27;
    // the sample-point cells are the cells around the particle's own (lane 13): its
    // in-range candidates are its force-pass list
    const int32_t ox = __shfl_sync(full, cx, 13) + dx - 1, oy = __shfl_sync(full, cy, 13) + dy - 1,
                  oz = __shfl_sync(full, cz, 13) + dz - 1;
    const bool around = (!vx || cx == ox) && (!vy || cy == oy) && (!vz || cz == oz);
    const bool listing = __all_sync(full, lane >= 27 || around) && __shfl_sync(full, (int)dens, 13) != 0;
    if (listing) {
        cx = ox;
        cy = oy;
        cz = oz;
    }
    int2 se = make_int2(-1, -1);
    bool bad = false;
    if (dens || (listing && lane < 27)) {
        se = __ldg(table + slot_of(P, cell_hash((uint32_t)cx, (uint32_t)cy, (uint32_t)cz)));
        if (se.x != -1 && (se.x < 0 || se.y > (int32_t)n || se.x > se.y)) {
            atomicOr(err, ERR_TABLE_RANGE);
            bad = true;
            se.x = -1;
        }
    }
    const bool list_ok = listing && !__any_sync(full, bad);
    const uint32_t in_box = __ballot_sync(full, dens);
    // the ranges one after another: the first position of each, and its slot offset
    const uint32_t len = se.x == -1 ? 0u : (uint32_t)(se.y - se.x);
    uint32_t incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += t;
    }
    const uint32_t total = __shfl_sync(full, incl, 31);
    const uint32_t sub = (uint32_t)se.x - (incl - len);
    const float3 me = form.self(xp, i);
    typename F::Sum sum;
    uint32_t cnt = 0;  // list entries
    for (uint32_t base = 0; base < total; base += 32) {
        const uint32_t q = base + (uint32_t)lane;
        int r = 0;
#pragma unroll
        for (int w = 16; w > 0; w >>= 1)
            if (__shfl_sync(full, incl, r + w - 1) <= q) r += w;
        const uint32_t j = q + __shfl_sync(full, sub, r);
        float dd = 0.0f;
        bool in = false;
        if (q < total) {
            dd = form.dist2(form.stage(j), -me.x, -me.y, -me.z);
            in = form.in_table_reach(dd, P.skip_d2);
        }
        float t, tn;
        form.terms(P, dd, t, tn);
        for (uint32_t m = __ballot_sync(full, in && (in_box >> r & 1u)); m; m &= m - 1u) {
            const int k = __ffs(m) - 1;
            sum.add(true, __shfl_sync(full, t, k), __shfl_sync(full, tn, k));
        }
        const bool put = listing && in && j != i;
        const uint32_t m = __ballot_sync(full, put);
        const uint32_t at = cnt + (uint32_t)__popc(m & lt);
        if (put && at < P.list_cap) nlist[(size_t)at * n + i] = (int32_t)j;
        cnt += (uint32_t)__popc(m);
    }
    if (lane == 0) {
        const bool scan = !(list_ok && cnt <= P.list_cap);
        put_rr(rr, fr, i, sum.finish(P));
        order[i] = i;
        ncount[i] = scan ? -1 : (int32_t)cnt;
        if (scan) {
            const uint32_t k = atomicAdd(scanq_n + CTR_SCANQ, 1u);
            if (k < n) scanq[k] = i;
        }
    }
}

template <class F>
cudaError_t launch_density_small(const DevParams& P, const StepBuffers& b, const F& form, cudaStream_t s) {
    const unsigned g = (P.n + SMALL_THREADS / 32 - 1) / (SMALL_THREADS / 32);
    k_density_small<F><<<g, SMALL_THREADS, 0, s>>>(P, form, b.xp, b.table, b.order, b.rr, b.records(), b.nlist, b.ncount, b.scanq,
                                                   b.scanq_n, b.err);
    return cudaGetLastError();
}

}  // namespace
}  // namespace pfs
