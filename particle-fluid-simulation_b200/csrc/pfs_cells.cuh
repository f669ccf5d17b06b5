// pfs_cells.cuh — the cell-grouped density pass of the grid search, shared by the
// FP32 form (k_density_cells<Dens32>, pfs_neighbors.cu) and the FP16-cell form
// (k_density_cells<Dens16>, pfs_fp16.cu).  The candidates of a particle and
// their order are calculateDensities.comp:114-131's: the 27 sample cells (z
// outer, x inner), each cell's table run in slot order; only the in-range ones
// are ever looked at (pfs_geo.cuh gives the argument).
//
// The one-warp-per-particle form of this pass (k_density_geo) gathers, sorts and
// sums each particle's neighbours by itself: 5,000 to 16,000 warp instructions
// per particle, most of them the same for all particles of a cell.  Here the
// work is grouped by cell (300,000 dense particles on 4,096 slots: 6.25 ms before,
// 1.5 here and 0.13 for the particles left; instruction issue binds it, 0.7 of the
// slots at 94 registers and five blocks on an SM):
//   1. the spatial order keeps the particles of a block of 2^bsx x 2^bsy x 2^bsz
//      cells consecutive, cell by cell, about 104 in all where the fluid is as
//      dense as it was created; a thread block takes one such block at a time;
//   2. the particles of the block's cells and of the layer of cells around them
//      (three to seven times the block's own) are read once.  Each belongs to
//      the table slot of its key; those whose slot is one of the slots of these
//      cells are collected by slot (a small hash table) and ranked by slot
//      number within it, which is the order of the table run.  They are staged in
//      shared memory, as many z layers of the neighbourhood at a time as fit;
//   3. a warp takes up to 32 of the particles, cell by cell: each lane holds two
//      candidates of the cell's 27 runs, and each of the cell's particles is
//      tested against all 64 at once, two per packed instruction; the two
//      ballots are all that is kept of the test;
//   4. when the ballots' space is full, and after each stage, the lanes become
//      the particles: each walks the set bits of its own ballots in order, sums
//      the terms and writes its list entries.
// The sums see the reference's terms in the reference's order, so the results
// are the table walk's, bit for bit.
//
// Left to the one-warp-per-particle pass: particles whose 27 sample cells are not
// the cells around their own or that lie within rounding of a cell face (edge),
// blocks for which that pass is faster (cells_rule, pfs_world.cu: they are never
// listed), and blocks whose neighbourhood does not fit even layer by layer.
#pragma once

#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "pfs_common.cuh"
#include "pfs_step.cuh"

namespace pfs {
namespace {

constexpr int CELLS_THREADS = 128;
constexpr int CELLS_WARPS = CELLS_THREADS / 32;
constexpr int CELLS_RUNS = 216;   // a block of 4 x 4 x 4 cells and the layer around it
constexpr int CELLS_HASH = 512;   // slots of those runs, by open addressing
constexpr uint32_t CELLS_ALL = (1u << 27) - 1u;  // every sample point in the box
constexpr uint32_t CELLS_SLOW = 1u << 31;        // meta: left to the one-particle pass

struct CellsShared {
    uint16_t run[CELLS_RUNS];         // hash entry of the staged run
    uint32_t off[CELLS_HASH + 4];     // staged candidates before a hash entry
    float4 nxy[CELLS_THREADS];        // the tile's particles: (-x, -x, -y, -y)
    float2 nz[CELLS_THREADS];         // (-z, -z)
    uint32_t slot[CELLS_THREADS];
    uint32_t meta[CELLS_THREADS];     // sample points in the box, one bit per cell
    uint32_t cell[CELLS_THREADS];     // cell in the block
    uint32_t start[68];               // the block's particles before cell c
    uint32_t warp_sum[CELLS_WARPS];
    uint32_t work, seg, found;
    DevParams P;
};

// What only the building of a stage needs.
struct CellsBuild {
    uint32_t first[CELLS_RUNS];      // cells of the neighbourhood: first position
    uint32_t chunk[CELLS_RUNS + 4];  // read chunks before cell r
    uint32_t end[CELLS_RUNS];        // end position
    uint32_t key[CELLS_HASH];        // table slot of a hash entry
    uint32_t cnt[CELLS_HASH];        // candidates still to place
};

// Dynamic shared memory: `entries` staged candidates (position, slot), then per
// warp `words` pairs of ballots and, for each of `slots` groups of 64 candidates,
// their entry numbers (11 bits) and cells (5 bits).  While a stage is built the
// warps' part holds CellsBuild and the candidates (slot number, hash entry) as
// found and by slot.
struct CellsLayout {
    uint32_t entries, words, slots;
};
__host__ __device__ __forceinline__ uint32_t cells_warp_bytes(const CellsLayout& y) {
    return y.words * 8u + y.slots * 128u;
}
__host__ __device__ __forceinline__ size_t cells_dyn_bytes(const CellsLayout& y) {
    const size_t test = CELLS_WARPS * (size_t)cells_warp_bytes(y), build = sizeof(CellsBuild) + 12 * (size_t)y.entries;
    return (size_t)y.entries * 16 + (test > build ? test : build);
}
static_assert(CELLS_STAGE_MAX <= 2048, "entry numbers have 11 bits");

// Two floats in one register pair, operated on by one instruction; each half is
// an IEEE round-to-nearest operation.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Exclusive scan of v[0, R) in place, R <= 4 * CELLS_THREADS; v[R] and the return
// value: the total.
__device__ __forceinline__ uint32_t cells_scan(uint32_t* warp_sum, uint32_t* v, uint32_t R) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t k = 4u * tid;
    uint32_t x[4], own = 0;
#pragma unroll
    for (int u = 0; u < 4; u++) {
        x[u] = k + u < R ? v[k + u] : 0u;
        own += x[u];
    }
    uint32_t incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    uint32_t base = incl - own, total = 0;
#pragma unroll
    for (int w = 0; w < CELLS_WARPS; w++) {
        base += w < warp ? warp_sum[w] : 0u;
        total += warp_sum[w];
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
        if (k + u < R) v[k + u] = base;
        base += x[u];
    }
    if (tid == 0) v[R] = total;
    __syncthreads();
    return total;
}

__device__ __forceinline__ uint32_t cells_hash(uint32_t slot) { return slot * 2654435761u >> 23; }

// Stage the runs of the neighbourhood layers [z0, z0 + zs) (layer 0 lies below
// the box) of the box of cells [b, b + dim): candidates by hash entry, in slot
// order, in ent, S.off.  Returns false, for the whole block, when they do not fit.
template <class F>
__device__ __forceinline__ bool cells_build(const DevParams& P, const F& form, CellsShared& S,
                                            const CellsLayout& lay, float4* ent, uint32_t* work, const int3 b,
                                            const int3 dim, int z0, int zs, const uint32_t* __restrict__ order,
                                            const uint32_t* __restrict__ skeys,
                                            const uint32_t* __restrict__ bcount,
                                            const uint32_t* __restrict__ boffset, uint32_t* __restrict__ err) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t full = 0xffffffffu, lt = (1u << lane) - 1u;
    const uint32_t n = P.n;
    const int nx = dim.x + 2, ny = dim.y + 2;
    const uint32_t R = (uint32_t)(nx * ny * (dim.z + 2));
    CellsBuild& B = *reinterpret_cast<CellsBuild*>(work);
    const uint32_t E = lay.entries;  // (a multiple of 64)
    uint32_t* sj = work + sizeof(CellsBuild) / 4;  // by slot
    uint32_t* zj = sj + E;                         // as found
    uint16_t* sb = reinterpret_cast<uint16_t*>(zj + E);
    uint16_t* zb = sb + E;
    __syncthreads();  // the previous stage is no longer read
    for (int k = tid; k < CELLS_HASH; k += CELLS_THREADS) {
        B.key[k] = 0xffffffffu;
        B.cnt[k] = 0u;
    }
    if (tid == 0) S.found = 0u;
    __syncthreads();
    // chunks of 8 candidates where cells hold a few, else of 32
    const int gs = S.start[64] >= 12u << (P.bsx + P.bsy + P.bsz) ? 5 : 3;
    // r / nx and r / (nx ny) by reciprocals: exact for r < 216
    const uint32_t ix = 65535u / (uint32_t)nx + 1u, iy = 65535u / (uint32_t)ny + 1u;
    for (uint32_t r = tid; r < R; r += CELLS_THREADS) {
        const uint32_t qy = r * ix >> 16, qz = qy * iy >> 16;
        const int rx = (int)(r - qy * nx), ry = (int)(qy - qz * ny), rz = (int)qz;
        const int ex = b.x - 1 + rx, ey = b.y - 1 + ry, ez = b.z - 1 + rz;
        uint32_t c = 0, o = 0;
        if (ex >= 0 && ey >= 0 && ez >= 0 && ex < (int)P.ngx && ey < (int)P.ngy && ez < (int)P.ngz) {
            const uint32_t id = spatial_id(P, (uint32_t)ex, (uint32_t)ey, (uint32_t)ez);
            c = __ldg(bcount + id);
            if (c) {
                o = __ldg(boffset + id);
                if (o > n || c > n - o) {
                    atomicOr(err, ERR_SORT_COUNT);
                    c = 0;
                }
            }
        }
        B.first[r] = o;
        B.end[r] = o + c;
        B.chunk[r] = (c + (1u << gs) - 1u) >> gs;
        if (rz >= z0 && rz < z0 + zs) {  // a run of this stage
            const uint32_t slot = slot_of(P, cell_hash((uint32_t)ex, (uint32_t)ey, (uint32_t)ez));
            uint32_t hk = cells_hash(slot);
            for (;;) {  // the table is never full: 216 runs, 512 entries
                const uint32_t was = atomicCAS(&B.key[hk], 0xffffffffu, slot);
                if (was == 0xffffffffu || was == slot) break;
                hk = (hk + 1u) & (CELLS_HASH - 1u);
            }
            S.run[r] = (uint16_t)hk;
        }
    }
    __syncthreads();
    const uint32_t C = cells_scan(S.warp_sum, B.chunk, R);
    // a pile: the neighbourhood has at most six layers, so far more candidates
    // than eight stages hold do not fit; they are not worth reading
    if (C << gs > 8u * E + (R << gs)) return false;
    // read the neighbourhood: a warp takes 256 candidates' worth of chunks a
    // round (each lane looks one chunk's cell up), eight loads in flight
    const int per = 32 >> gs;  // chunks per load
    for (uint32_t cb = 8u * per * warp; cb < C; cb += 8u * per * CELLS_WARPS) {
        uint32_t j0 = 0, j1 = 0;
        if (lane < 8 * per && cb + lane < C) {
            uint32_t lo = 0, hi = R;  // last cell whose first chunk is <= cb + lane
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (B.chunk[mid] <= cb + lane) lo = mid; else hi = mid;
            }
            j0 = B.first[lo] + ((cb + lane - B.chunk[lo]) << gs);
            j1 = B.end[lo];
        }
        uint32_t j[8], key[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int from = u * per + (lane >> gs);  // chunk of this lane
            const uint32_t q = __shfl_sync(full, j0, from) + (lane & ((1 << gs) - 1));
            j[u] = q < __shfl_sync(full, j1, from) ? __ldcg(order + q) : 0xffffffffu;
        }
#pragma unroll
        for (int u = 0; u < 8; u++) key[u] = j[u] < n ? __ldg(skeys + j[u]) : 0xfffffffeu;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            if (!__any_sync(full, j[u] < n)) continue;
            uint32_t hk = cells_hash(key[u]), was = B.key[hk];
            while (was != key[u] && was != 0xffffffffu) {
                hk = (hk + 1u) & (CELLS_HASH - 1u);
                was = B.key[hk];
            }
            const bool in = was == key[u];
            const uint32_t m = __ballot_sync(full, in);
            uint32_t z = 0;
            if (lane == 0 && m) z = atomicAdd(&S.found, (uint32_t)__popc(m));
            z = __shfl_sync(full, z, 0) + __popc(m & lt);
            if (in) {
                atomicAdd(&B.cnt[hk], 1u);
                if (z < E) {
                    zj[z] = j[u];
                    zb[z] = (uint16_t)hk;
                }
            }
        }
    }
    __syncthreads();
    const uint32_t total = S.found;
    if (total > E) return false;
    for (int k = tid; k < CELLS_HASH; k += CELLS_THREADS) S.off[k] = B.cnt[k];
    __syncthreads();
    cells_scan(S.warp_sum, S.off, CELLS_HASH);
    for (uint32_t k = tid; k < total; k += CELLS_THREADS) {
        const uint32_t hk = zb[k], p = S.off[hk] + atomicSub(&B.cnt[hk], 1u) - 1u;
        sj[p] = zj[k];
        sb[p] = (uint16_t)hk;
    }
    __syncthreads();
    // place of each candidate in its run: the candidates of the run in lower slots
    for (uint32_t p = tid; p < total; p += CELLS_THREADS) {
        const uint32_t me = sj[p], hk = sb[p], lo = S.off[hk], hi = S.off[hk + 1];
        const float4 c = form.stage(me);
        uint32_t rank = lo;
#pragma unroll 8
        for (uint32_t q = lo; q < hi; q++) rank += sj[q] < me ? 1u : 0u;
        ent[rank] = c;
    }
    __syncthreads();
    return true;
}

// Density pass over the blocks listed in clist.  F: the form (Dens32, Dens16):
// staging a candidate, the packed distance and reach test, the terms and sums.
template <class F, bool BATCH>
__global__ void __launch_bounds__(CELLS_THREADS, 5)
k_density_cells(DevParams P0, SceneRef sr, F form, const float4* __restrict__ xp,
                const uint32_t* __restrict__ skeys, const uint32_t* __restrict__ order,
                const uint32_t* __restrict__ clist, const CellsRule* __restrict__ crules,
                const uint32_t* __restrict__ bcount, const uint32_t* __restrict__ boffset, CellsLayout lay,
                float2* __restrict__ rr, float4* __restrict__ fr, int32_t* __restrict__ nlist,
                int32_t* __restrict__ ncount, uint32_t* __restrict__ scanq, uint32_t* __restrict__ scanq_n,
                uint32_t* __restrict__ slowq, uint32_t* __restrict__ err) {
    extern __shared__ float4 s_dyn[];
    __shared__ CellsShared S;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t full = 0xffffffffu;
    const uint32_t n = P0.n;
    float4* ent = s_dyn;
    uint32_t* work = reinterpret_cast<uint32_t*>(s_dyn + lay.entries);
    uint32_t* zone = work + warp * (cells_warp_bytes(lay) / 4);
    uint2* ballots = reinterpret_cast<uint2*>(zone);                      // [words]
    uint16_t* at = reinterpret_cast<uint16_t*>(zone + 2u * lay.words);     // [slots][64]
    const DevParams& P = BATCH ? S.P : P0;
    const uint32_t nblk = min(scanq_n[CTR_BLOCKS], n);
    for (;;) {
        __syncthreads();
        if (tid == 0) S.work = atomicAdd(scanq_n + CTR_CELLS, 1u);
        __syncthreads();
        if (S.work >= nblk) return;
        const uint32_t id0 = clist[S.work];
        // the block's cells: particles before each, and its segment of the order
        const uint32_t cells = 1u << (BATCH ? (uint32_t)crules[id0 >> 8].shift : (uint32_t)(P0.bsx + P0.bsy + P0.bsz));
        if (warp == 0) {
            const uint32_t c0 = (uint32_t)lane < cells ? bcount[id0 + lane] : 0u;
            const uint32_t c1 = (uint32_t)lane + 32u < cells ? bcount[id0 + 32 + lane] : 0u;
            uint32_t i0 = c0, i1 = c1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t a = __shfl_up_sync(full, i0, o), e = __shfl_up_sync(full, i1, o);
                if (lane >= o) {
                    i0 += a;
                    i1 += e;
                }
            }
            i1 += __shfl_sync(full, i0, 31);
            S.start[lane] = i0 - c0;
            S.start[32 + lane] = i1 - c1;
            if (lane == 31) S.start[64] = i1;
            if (c0) S.seg = boffset[id0 + lane] - (i0 - c0);  // the same from every cell
            if (c1) S.seg = boffset[id0 + 32 + lane] - (i1 - c1);
        }
        __syncthreads();
        const uint32_t seg = S.seg, members = S.start[64];
        if (members == 0u) continue;
        if (seg > n || members > n - seg) {
            if (tid == 0) atomicOr(err, ERR_SORT_COUNT);
            continue;
        }
        if constexpr (BATCH) {
            const uint32_t i0 = order[seg];
            if (i0 >= n) {
                if (tid == 0) atomicOr(err, ERR_PERM_RANGE);
                continue;
            }
            const uint32_t* from = reinterpret_cast<const uint32_t*>(sr.scenes + sr.sid[i0]);
            for (uint32_t k = tid; k < sizeof(DevParams) / 4; k += CELLS_THREADS)
                reinterpret_cast<uint32_t*>(&S.P)[k] = from[k];
            __syncthreads();
        }
        const uint32_t lb = (id0 - P.block_base) >> (P.bsx + P.bsy + P.bsz);
        const int3 dim = make_int3(1 << P.bsx, 1 << P.bsy, 1 << P.bsz);
        const int3 b = make_int3((int)(lb % P.nbx) << P.bsx, (int)(lb / P.nbx % P.nby) << P.bsy,
                                 (int)(lb / (P.nbx * P.nby)) << P.bsz);
        const float h = P.h, skip = P.skip_d2;
        // as many layers at a time as the block's own density fills seven eighths of
        // the stage with; where that does not fit, one at a time
        const int layers = dim.z + 2;
        const float runs = (float)((dim.x + 2) * (dim.y + 2)), density = (float)members / (float)cells;
        for (int zs = cells_layers(runs, layers, density, (float)(1u << __popc(P.mask)), (float)lay.entries);; zs = 1) {
            bool fits = true, staged = false;
            for (uint32_t t0 = 0; t0 < members; t0 += CELLS_THREADS) {
                // ---- the tile's particles
                __syncthreads();
                const uint32_t tile = min(members - t0, (uint32_t)CELLS_THREADS);
                const uint32_t t = seg + t0 + tid;
                const bool have = (uint32_t)tid < tile;
                bool slow = false;
                if (have) {
                    uint32_t i = order[t];
                    if (i >= n) {
                        atomicOr(err, ERR_PERM_RANGE);
                        i = 0;
                    }
                    const float4 sp = xp[i];
                    const float off[3] = {PFS_MUL(h, -1.0f), PFS_MUL(h, 0.0f), h};
                    bool vx[3], vy[3], vz[3];
                    int32_t cx[3], cy[3], cz[3];
#pragma unroll
                    for (int a = 0; a < 3; a++) {
                        const float sx = PFS_ADD(sp.x, off[a]), sy = PFS_ADD(sp.y, off[a]),
                                    sz = PFS_ADD(sp.z, off[a]);
                        vx[a] = !(sx < P.minx) && !(sx > P.maxx);
                        vy[a] = !(sy < P.miny) && !(sy > P.maxy);
                        vz[a] = !(sz < P.minz) && !(sz > P.maxz);
                        cx[a] = cell_coord(sx, P.minx, h);
                        cy[a] = cell_coord(sy, P.miny, h);
                        cz[a] = cell_coord(sz, P.minz, h);
                    }
                    // the sample-point cells are the cells around the particle's own
                    const bool listing = vx[1] && vy[1] && vz[1] && (!vx[0] || cx[0] == cx[1] - 1) &&
                                         (!vx[2] || cx[2] == cx[1] + 1) && (!vy[0] || cy[0] == cy[1] - 1) &&
                                         (!vy[2] || cy[2] == cy[1] + 1) && (!vz[0] || cz[0] == cz[1] - 1) &&
                                         (!vz[2] || cz[2] == cz[1] + 1);
                    // and no face is within rounding of it
                    auto near_face = [&](float v, float mn, int32_t c) {
                        const float f = PFS_DIV(PFS_SUB(v, mn), h) - (float)c;
                        return !(f > P.edge && f < 1.0f - P.edge);
                    };
                    const uint32_t lx = (uint32_t)(cx[1] - b.x), ly = (uint32_t)(cy[1] - b.y),
                                   lz = (uint32_t)(cz[1] - b.z);
                    slow = !listing || lx >= (uint32_t)dim.x || ly >= (uint32_t)dim.y || lz >= (uint32_t)dim.z ||
                           near_face(sp.x, P.minx, cx[1]) || near_face(sp.y, P.miny, cy[1]) ||
                           near_face(sp.z, P.minz, cz[1]);
                    const uint32_t mx = (vx[0] ? 1u : 0u) | (vx[1] ? 2u : 0u) | (vx[2] ? 4u : 0u);
                    const uint32_t my = (vy[0] ? mx : 0u) | (vy[1] ? mx << 3 : 0u) | (vy[2] ? mx << 6 : 0u);
                    const uint32_t meta = (vz[0] ? my : 0u) | (vz[1] ? my << 9 : 0u) | (vz[2] ? my << 18 : 0u);
                    const float3 q = form.self(xp, i);
                    S.nxy[tid] = make_float4(-q.x, -q.x, -q.y, -q.y);
                    S.nz[tid] = make_float2(-q.z, -q.z);
                    S.slot[tid] = i;
                    S.meta[tid] = slow ? CELLS_SLOW : meta;
                    // its cell in the block, by the segment it is in
                    uint32_t c = 0;
#pragma unroll
                    for (uint32_t s = 32; s > 0; s >>= 1)
                        if (c + s < 64u && S.start[c + s] <= t0 + tid) c += s;
                    S.cell[tid] = c;
                }
                // left to the one-particle pass
                auto leave = [&](bool which) {
                    if (!which) return;
                    const uint32_t q = atomicAdd(scanq_n + CTR_SLOW, 1u);
                    if (q < n) slowq[q] = t;
                };
                __syncthreads();
                // ---- this warp's share of the tile: an even one, since a warp without
                // particles would only wait at the next barrier (full warps instead:
                // batch of 32 scenes 8.5 against 7.9 ms)
                const uint32_t share = (tile + CELLS_WARPS - 1u) / CELLS_WARPS;
                const uint32_t w0 = min(warp * share, tile), w1 = min(w0 + share, tile);
                const bool mine = w0 + lane < w1;
                const uint32_t ms = mine ? w0 + lane : 0u;
                const float nx0 = S.nxy[ms].x, ny0 = S.nxy[ms].z, nz0 = S.nz[ms].x;
                const uint32_t self = S.slot[ms], mycell = S.cell[ms], mymeta = S.meta[ms];
                const bool done = mine && !(mymeta & CELLS_SLOW);  // this pass writes its result
                const uint32_t tm = seg + t0 + ms;
                uint32_t lcnt = 0;  // list entries
                const uint32_t lcap = done ? P.list_cap : 0u;
                int32_t* const row = nlist + tm;
                typename F::Sum sum;
                const int nx = dim.x + 2, ny = dim.y + 2;
                for (int z0 = 0; z0 < layers && fits; z0 += zs) {
                    if (!staged || zs < layers)
                        fits = cells_build(P, form, S, lay, ent, work, b, dim, z0, min(zs, layers - z0), order,
                                           skeys, bcount, boffset, err);
                    if (!fits) break;
                    staged = true;
                    if (w0 >= w1) continue;
                    const int z1 = min(z0 + zs, layers);
                    // this lane's ballots: nk words (two per group of 64), the first
                    // pair at wb, the next ones gm pairs apart; entry numbers from ab
                    uint32_t nk = 0, wb = 0, gm = 0, ab = 0;
                    uint32_t used_w = 0, used_s = 0;
                    auto drain = [&]() {
                        __syncwarp();
                        const bool walls = __any_sync(full, nk && mymeta != CELLS_ALL);
                        const uint32_t* bw = reinterpret_cast<const uint32_t*>(ballots);
                        auto word = [&](uint32_t k) { return k < nk ? bw[2u * (wb + (k >> 1) * gm) + (k & 1u)] : 0u; };
                        uint32_t k = 0, w = word(0), wn = word(1);
                        const uint16_t* an = at + ab;
                        // the next entry of this lane and its cell (has: there is one)
                        auto next = [&](bool& has, float4& c, uint32_t& d) {
                            const bool adv = w == 0u && k + 1u < nk;
                            k += adv ? 1u : 0u;
                            an += adv ? 32 : 0;
                            w = adv ? wn : w;
                            wn = adv ? word(k + 1u) : wn;
                            has = w != 0u;
                            const uint32_t e = an[(__ffs(w) - 1) & 31];
                            w &= w - 1u;
                            c = ent[e & 2047u];
                            d = e >> 11;
                        };
                        auto list = [&](bool has, uint32_t j) {
                            const bool put = has && j != self;
                            if (put && lcnt < lcap) __stcs(row + (size_t)lcnt * n, (int32_t)j);
                            lcnt += put ? 1u : 0u;
                        };
                        // two entries a trip: their distances and terms are independent,
                        // only the sums are serial
                        while (__any_sync(full, w != 0u || k + 1u < nk)) {
                            bool h0, h1;
                            float4 e0, e1;
                            uint32_t c0, c1;
                            next(h0, e0, c0);
                            next(h1, e1, c1);
                            float a2, a3, b2, b3;
                            form.terms(P, form.dist2(e0, nx0, ny0, nz0), a2, a3);
                            form.terms(P, form.dist2(e1, nx0, ny0, nz0), b2, b3);
                            // near a wall: the sample point of the entry's cell is in the box
                            sum.add(h0 && (!walls || mymeta >> c0 & 1u), a2, a3);
                            sum.add(h1 && (!walls || mymeta >> c1 & 1u), b2, b3);
                            list(h0, __float_as_uint(e0.w));
                            list(h1, __float_as_uint(e1.w));
                        }
                        nk = used_w = used_s = 0u;
                        __syncwarp();
                    };
                    uint32_t todo = __ballot_sync(full, mine);
                    while (todo) {
                        const int a = __ffs(todo) - 1;
                        const uint32_t c = __shfl_sync(full, mycell, a);
                        const bool member = mine && mycell == c;
                        const uint32_t grp = __ballot_sync(full, member);
                        todo &= ~grp;
                        const uint32_t g = __popc(grp);
                        // the cell's 27 runs, those of these layers
                        const int lx = (int)c & (dim.x - 1), ly = (int)c >> P.bsx & (dim.y - 1),
                                  lz = (int)c >> (P.bsx + P.bsy);
                        uint32_t st = 0, ln = 0;
                        {
                            const int dz = lane * 57 >> 9, dr = lane - 9 * dz, dy = dr * 11 >> 5, dx = dr - 3 * dy;
                            if (lane < 27 && lz + dz >= z0 && lz + dz < z1) {
                                const uint32_t hk = S.run[lx + dx + nx * (ly + dy + ny * (lz + dz))];
                                st = S.off[hk];
                                ln = S.off[hk + 1] - st;
                            }
                        }
                        uint32_t incl = ln;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const uint32_t v = __shfl_up_sync(full, incl, o);
                            if (lane >= o) incl += v;
                        }
                        const uint32_t L = __shfl_sync(full, incl, 31);
                        const uint32_t sub = st - (incl - ln);  // entry = q + sub of its run
                        // entry of position q of the concatenated runs, and its cell
                        auto locate = [&](uint32_t q) -> uint32_t {
                            int r = 0;
#pragma unroll
                            for (int w = 16; w > 0; w >>= 1)
                                if (__shfl_sync(full, incl, r + w - 1) <= q) r += w;
                            return ((q + __shfl_sync(full, sub, r)) & 2047u) | (uint32_t)r << 11;
                        };
                        const float4 none = make_float4(INFINITY, INFINITY, INFINITY, 0.0f);
                        for (uint32_t q0 = 0; q0 < L; q0 += 64) {
                            if (used_s == lay.slots || used_w + g > lay.words) drain();
                            if (member && nk == 0u) {
                                wb = used_w + (uint32_t)(lane - a);
                                gm = g;
                                ab = used_s * 64u;
                            }
                            const uint32_t at0 = locate(q0 + lane), at1 = locate(q0 + 32 + lane);
                            const float4 c0 = q0 + lane < L ? ent[at0 & 2047u] : none;
                            const float4 c1 = q0 + 32 + lane < L ? ent[at1 & 2047u] : none;
                            at[used_s * 64u + lane] = q0 + lane < L ? (uint16_t)at0 : (uint16_t)0;
                            at[used_s * 64u + 32u + lane] = q0 + 32 + lane < L ? (uint16_t)at1 : (uint16_t)0;
                            const f32x2 x2 = pack2(c0.x, c1.x), y2 = pack2(c0.y, c1.y), z2 = pack2(c0.z, c1.z);
                            const float4* pxy = S.nxy + w0 + a;
                            const float2* pz = S.nz + w0 + a;
                            uint2* out = ballots + used_w;
#pragma unroll 4
                            for (uint32_t m = 0; m < g; m++) {
                                const float4 mxy = pxy[m];
                                const float2 mz = pz[m];
                                float d0, d1;
                                form.dist2_pair(x2, y2, z2, pack2(mxy.x, mxy.y), pack2(mxy.z, mxy.w),
                                                pack2(mz.x, mz.y), d0, d1);
                                const uint32_t b0w = __ballot_sync(full, form.in_reach(d0, skip));
                                const uint32_t b1w = __ballot_sync(full, form.in_reach(d1, skip));
                                out[m] = make_uint2(b0w, b1w);  // every lane stores the same pair
                            }
                            used_w += g;
                            used_s++;
                            if (member) nk += 2u;
                        }
                    }
                    drain();
                }
                if (!fits) {
                    if (zs > 1) break;  // again, one layer at a time
                    leave(have);
                    continue;
                }
                leave(slow);
                const bool scan = done && lcnt > lcap;
                if (done) {
                    put_rr(rr, fr, self, sum.finish(P));
                    ncount[tm] = scan ? -1 : (int32_t)lcnt;
                }
                if (scan) {  // the force pass scans for itself
                    const uint32_t q = atomicAdd(scanq_n + CTR_GEOQ, 1u);
                    if (q < n) scanq[n - 1u - q] = self;
                }
            }
            if (fits || zs == 1) break;
        }
    }
}

// Resident thread blocks of k_density_cells on the current device.
template <class K>
unsigned cells_grid(K kernel, size_t dyn) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, CELLS_THREADS, dyn);
    return (unsigned)std::max(1, per_sm) * (unsigned)std::max(1, sms);
}

// Launch the pass over the table's grid-search particles.  A sparse scene's warp
// spans many cells of one or two groups of 64 candidates each and sums once, at
// the end: 24 groups.  A dense scene's 32 particles of one cell share its groups:
// 16 groups, 352 pairs of ballots, and five thread blocks fit an SM.
inline CellsLayout cells_layout(uint32_t entries) {
    return entries > 1024u ? CellsLayout{entries, 352u, 16u} : CellsLayout{entries, 256u, 24u};
}

template <class F>
cudaError_t launch_cells(const DevParams& P, const StepBuffers& b, const F& form, cudaStream_t s) {
    const CellsLayout lay = cells_layout(b.cells_entries);
    const size_t dyn = cells_dyn_bytes(lay);
    auto k = b.sr.scenes ? k_density_cells<F, true> : k_density_cells<F, false>;
    // The limit belongs to the kernel, not to this table: the largest stage's for
    // every table, so that another thread's world never lowers it between this call
    // and the launch or the graph's instantiation.  The launch asks for its own size.
    const size_t most = std::max(cells_dyn_bytes(cells_layout(CELLS_STAGE_MAX)), cells_dyn_bytes(cells_layout(1024u)));
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e != cudaSuccess) return e;
    const unsigned grid = std::max(1u, std::min(cells_grid(k, dyn), P.n));
    k<<<grid, CELLS_THREADS, dyn, s>>>(P, b.sr, form, b.xp, b.skeys, b.order, b.clist, b.crules, b.bcount, b.boffset,
                                       lay, b.rr, b.records(), b.nlist, b.ncount, b.scanq, b.scanq_n, b.keys_tmp, b.err);
    return cudaGetLastError();
}

}  // namespace
}  // namespace pfs
