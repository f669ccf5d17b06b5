// pfs_density_map.cu — density map of a world's state into a headless float
// grid: the reference's updateDensityMap.comp (:93-147), which fills the 3-D
// image its ray-marching renderers sample.
//
// Per voxel of the image the reference allocates (renderer.c:774-781): the cell
// of the voxel centre ((-1,-1,-1) outside the box), the 27 cells around it in the
// shader's order (z outer, x inner), each skipped when out of bounds by the
// shader's voxel rule, and over the table range of each cell's key the smoothing
// kernel m (h - d)^2 of every position with d^2 < h^2, divided by the volume.
// Every float operation is one IEEE round-to-nearest operation in the shader's
// order, so the map equals the oracle's bit for bit.  The table of the last sort
// is rebuilt from its sorted keys for the call (the step's integrate clears it)
// and cleared again.
//
// Where the table has few slots the work is grouped by cell (k_map_cells; map_route has
// the rule), as in the density pass of the grid search (pfs_cells.cuh).  One thread per voxel walking its own 27 runs waits on
// 27 table look-ups, and reads, where the table has few slots, hundreds of
// distant particles per run: 5.2 ms for the reference's 300,000 particles (4,096
// slots) at 917,504 voxels, 0.6 ms in all now.  Here a thread block takes a block of cells, reads
// their runs once (a 4-byte packed position per entry, CELLS_CODE_STEPS steps per
// cell, decides what is near), stages what is near in run order and slot order,
// tests each cell's voxels against 64 staged positions per warp step, and sums a
// voxel's terms in one lane, in the shader's order.  Voxels outside the box, and
// voxels of cells whose neighbourhood does not fit the stage, walk their runs, a thread
// each (k_density_map), behind it.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#include "pfs_cells.cuh"
#include "pfs_common.cuh"
#include "pfs_flat.cuh"
#include "pfs_step.cuh"

namespace pfs {

namespace {

constexpr int MAP_THREADS = 256;

// outOfBounds (updateDensityMap.comp:93-96): negative, beyond the extent, or
// the far corner itself.
__device__ __forceinline__ bool map_out(int32_t x, int32_t y, int32_t z, int3 m) {
    if (x < 0 || y < 0 || z < 0) return true;
    if (x > m.x || y > m.y || z > m.z) return true;
    return x == m.x && y == m.y && z == m.z;
}

__global__ void __launch_bounds__(MAP_THREADS)
k_table_runs(uint32_t n, const uint32_t* __restrict__ skeys, int2* __restrict__ table, int set) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const uint32_t k = skeys[s];
    if (k >= n) return;
    const bool head = (s == 0) || (skeys[s - 1] != k);
    const bool tail = (s == n - 1) || (skeys[s + 1] != k);
    if (!set) {
        if (head) table[k] = make_int2(-1, -1);
        return;
    }
    if (head) table[k].x = (int32_t)s;
    if (tail) table[k].y = (int32_t)(s + 1);
}

// Packed positions of the state (bits as cells_code; NaN is marked in bit 31).  Each
// position marks its cell (marks: a byte per cell of the grid padded to whole
// blocks of 4 x 4 x 4) and, for rounding, those a sixteenth away: a cell coordinate
// is below CELLS_MAX_GRID and good to 2^-6.
__global__ void __launch_bounds__(MAP_THREADS)
k_map_code(DevParams P, const float4* __restrict__ x, uint32_t* __restrict__ code, uint8_t* __restrict__ marks) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < P.n;
    const float4 p = live ? x[i] : make_float4(NAN, NAN, NAN, 0.0f);
    const float s = (float)CELLS_CODE_STEPS;
    const float u[3] = {PFS_DIV(PFS_SUB(p.x, P.minx), P.h), PFS_DIV(PFS_SUB(p.y, P.miny), P.h),
                        PFS_DIV(PFS_SUB(p.z, P.minz), P.h)};
    const uint32_t g[3] = {(P.ngx & ~3u) + 4, (P.ngy & ~3u) + 4, (P.ngz & ~3u) + 4};
    auto field = [&](float v) { return (uint32_t)__float2int_rd(v * s) & 511u; };
    const bool nan = isnan(p.x) || isnan(p.y) || isnan(p.z);
    if (live) code[i] = field(u[0]) | field(u[1]) << 10 | field(u[2]) << 20 | CELLS_GUARD | (nan ? 0x80000000u : 0u);
    int lo[3], hi[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const bool near = u[a] > -2.0f && u[a] < (float)g[a] + 2.0f;  // elsewhere nothing reaches the box
        lo[a] = near ? max(__float2int_rd(u[a] - 0.0625f), 0) : 0;
        hi[a] = near ? min(__float2int_rd(u[a] + 0.0625f), (int)g[a] - 1) : -1;
        if (near && hi[a] < 0) hi[a] = 0;                             // a cell outside marks the
        if (near && lo[a] >= (int)g[a]) lo[a] = (int)g[a] - 1;        // nearest inside
    }
    // the positions of a table run come from few cells: one lane marks for all that
    // mark the same (every lane for itself: 46 us for 300,000 particles; so: 35)
    const bool marks_any = lo[0] <= hi[0] && lo[1] <= hi[1] && lo[2] <= hi[2];
    const unsigned long long same =
        !marks_any ? ~0ull
                   : (unsigned long long)lo[0] | (unsigned long long)lo[1] << 17 | (unsigned long long)lo[2] << 34 |
                         (unsigned long long)((hi[0] - lo[0]) | (hi[1] - lo[1]) << 1 | (hi[2] - lo[2]) << 2) << 51;
    if ((int)(threadIdx.x & 31) != __ffs(__match_any_sync(0xffffffffu, same)) - 1) return;
    for (int z = lo[2]; z <= hi[2]; z++)
        for (int y = lo[1]; y <= hi[1]; y++)
            for (int q = lo[0]; q <= hi[0]; q++) {
                uint8_t* m = marks + ((size_t)q + (size_t)g[0] * ((size_t)y + (size_t)g[1] * (size_t)z));
                if (__ldcg(m) == 0u) __stcg(m, (uint8_t)1);
            }
}

struct MapArgs {
    float cs;    // voxel size
    int3 img;    // voxels of the image
    int3 bound;  // the shader's own extent
};

__device__ __forceinline__ float map_centre(float mn, int32_t v, float cs) {
    return PFS_ADD(mn, PFS_MUL(PFS_ADD((float)v, 0.5f), cs));
}

__device__ __forceinline__ bool map_inside(const DevParams& P, float x, float y, float z) {
    return !(x < P.minx || y < P.miny || z < P.minz || x > P.maxx || y > P.maxy || z > P.maxz);
}

// A position's term at squared distance s < h^2.
__device__ __forceinline__ float map_term(const DevParams& P, float s) {
    const float dist = PFS_SQRT(s);
    const float a = PFS_SUB(P.h, dist);
    return PFS_MUL(P.m, dist >= P.h ? 0.0f : PFS_MUL(a, a));
}

// One voxel by its own 27-run walk.
__device__ float map_walk(const DevParams& P, const MapArgs& A, float cxp, float cyp, float czp,
                          const float4* __restrict__ x, const int2* __restrict__ table, uint32_t* __restrict__ err) {
    const float h = P.h;
    int32_t c0 = -1, c1 = -1, c2 = -1;
    if (map_inside(P, cxp, cyp, czp)) {
        c0 = cell_coord(cxp, P.minx, h);
        c1 = cell_coord(cyp, P.miny, h);
        c2 = cell_coord(czp, P.minz, h);
    }
    const uint32_t n = P.n;
    float density = 0.0f;
#pragma unroll 1
    for (int q = 0; q < 27; q++) {
        const int32_t kx = c0 + q % 3 - 1, ky = c1 + (q / 3) % 3 - 1, kz = c2 + q / 9 - 1;
        if (map_out(kx, ky, kz, A.bound)) continue;
        const int2 se = __ldg(table + slot_of(P, cell_hash((uint32_t)kx, (uint32_t)ky, (uint32_t)kz)));
        if (se.x == -1) continue;
        if (se.x < 0 || se.y > (int32_t)n || se.x > se.y) {
            atomicOr(err, ERR_TABLE_RANGE);
            continue;
        }
        for (int32_t i = se.x; i < se.y; i++) {
            const float4 p = __ldg(x + i);
            const float d0 = PFS_SUB(cxp, p.x), d1 = PFS_SUB(cyp, p.y), d2 = PFS_SUB(czp, p.z);
            const float dist2 = PFS_ADD(PFS_ADD(PFS_MUL(d0, d0), PFS_MUL(d1, d1)), PFS_MUL(d2, d2));
            if (dist2 < P.r2) density = PFS_ADD(density, map_term(P, dist2));
        }
    }
    return PFS_DIV(PFS_MUL(density, 1.0f), P.volume);
}

// What k_map_cells writes for a voxel it leaves (no result: theirs are numbers or the
// one NaN that arithmetic gives).
constexpr uint32_t MAP_LEFT = 0x7fc5a1e7u;

// A thread per voxel: every voxel (ALL), or, behind the cells' pass, those the shader
// skips (0), the rest of those whose centre lies outside the box, and those left.
template <bool ALL>
__global__ void __launch_bounds__(MAP_THREADS)
k_density_map(DevParams P, MapArgs A, const float4* __restrict__ x, const int2* __restrict__ table,
              float* __restrict__ out, uint32_t* __restrict__ err) {
    const uint64_t nx = (uint64_t)A.img.x, ny = (uint64_t)A.img.y, nz = (uint64_t)A.img.z;
    const uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nx * ny * nz) return;
    const int32_t vx = (int32_t)(idx % nx), vy = (int32_t)((idx / nx) % ny), vz = (int32_t)(idx / (nx * ny));
    if (map_out(vx, vy, vz, A.bound)) {
        out[idx] = 0.0f;
        return;
    }
    const float cx = map_centre(P.minx, vx, A.cs), cy = map_centre(P.miny, vy, A.cs), cz = map_centre(P.minz, vz, A.cs);
    if (ALL || !map_inside(P, cx, cy, cz) || __float_as_uint(out[idx]) == MAP_LEFT)
        out[idx] = map_walk(P, A, cx, cy, cz, x, table, err);
}

// Every voxel, by the flat walk of pfs_flat.cuh (a thread per voxel, the voxels of
// a block sorted by their candidate totals, one loop over the 27 runs together).
// A loop per run ran with 12 of 32 lanes: neighbouring voxels' runs differ in
// length, their totals little.  1,000,000 voxels of a 1,048,576-particle slab:
// 310 -> 250 us (now the L1 binds it: a lane's candidate is a line of its own).
// Voxels with more than FLAT_RCAP run words walk by themselves.
__global__ void __launch_bounds__(FLAT_THREADS, FLAT_BLOCKS)
k_map_flat(DevParams P, MapArgs A, const float4* __restrict__ x, const int2* __restrict__ table,
           float* __restrict__ out, uint32_t* __restrict__ err) {
    __shared__ FlatShared S;
    __shared__ float s_dd[FLAT_CAP][FLAT_THREADS];  // per thread: deferred terms
    const int tid = threadIdx.x;
    const uint32_t n = P.n;
    const uint64_t nx = (uint64_t)A.img.x, ny = (uint64_t)A.img.y, nz = (uint64_t)A.img.z;
    const uint64_t first = (uint64_t)blockIdx.x * FLAT_THREADS;
    __shared__ uint32_t s_first[3];  // the block's first voxel
    if (tid == 0) {
        s_first[0] = (uint32_t)(first % nx);
        s_first[1] = (uint32_t)((first / nx) % ny);
        s_first[2] = (uint32_t)(first / (nx * ny));
    }
    __syncthreads();
    auto voxel = [&](int col, float& cx, float& cy, float& cz) {  // false: none, or one the shader skips
        const uint64_t idx = first + (uint64_t)col;
        const uint32_t ix = s_first[0] + (uint32_t)col, iy = s_first[1] + ix / (uint32_t)nx;
        const int32_t vx = (int32_t)(ix % (uint32_t)nx), vy = (int32_t)(iy % (uint32_t)ny),
                      vz = (int32_t)(s_first[2] + iy / (uint32_t)ny);
        cx = map_centre(P.minx, vx, A.cs);
        cy = map_centre(P.miny, vy, A.cs);
        cz = map_centre(P.minz, vz, A.cs);
        return idx < nx * ny * nz && !map_out(vx, vy, vz, A.bound);
    };
    float cx, cy, cz;
    const bool mine = voxel(tid, cx, cy, cz);
    int nr = 0;
    uint32_t tot = 0;
    if (mine) {
        int32_t c0 = -1, c1 = -1, c2 = -1;
        if (map_inside(P, cx, cy, cz)) {
            c0 = cell_coord(cx, P.minx, P.h);
            c1 = cell_coord(cy, P.miny, P.h);
            c2 = cell_coord(cz, P.minz, P.h);
        }
        // map_out of the 27 cells by axis
        uint32_t hx[3], hy[3];
        bool ox[3], oy[3], ex[3], ey[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const int32_t kx = c0 + a - 1, ky = c1 + a - 1;
            hx[a] = (uint32_t)kx * 73856093u;
            hy[a] = (uint32_t)ky * 19349663u;
            ox[a] = kx < 0 || kx > A.bound.x;
            oy[a] = ky < 0 || ky > A.bound.y;
            ex[a] = kx == A.bound.x;
            ey[a] = ky == A.bound.y;
        }
#pragma unroll 1
        for (int dz = -1; dz <= 1; dz++) {
            const int32_t kz = c2 + dz;
            if (kz < 0 || kz > A.bound.z) continue;
            const uint32_t hz = (uint32_t)kz * 83492791u;
            const bool ez = kz == A.bound.z;
            // a layer's nine table entries are loaded together
            int2 row[9];
#pragma unroll
            for (int q = 0; q < 9; q++)
                row[q] = ox[q % 3] || oy[q / 3] || (ex[q % 3] && ey[q / 3] && ez)
                             ? make_int2(-1, -1)
                             : __ldg(table + slot_of(P, hash_finalize(hx[q % 3] ^ hy[q / 3] ^ hz)));
#pragma unroll
            for (int q = 0; q < 9; q++) {
                const int2 se = row[q];
                if (se.x == -1) continue;
                if (se.x < 0 || se.y > (int32_t)n || se.x > se.y) {
                    atomicOr(err, ERR_TABLE_RANGE);
                    continue;
                }
                uint32_t s0 = (uint32_t)se.x, len = (uint32_t)(se.y - se.x);
                tot += len;
                while (len > 0) {
                    const uint32_t l = min(len, FLAT_LEN_MAX);
                    if (nr < FLAT_RCAP) S.rng[nr][tid] = s0 | (l << 24);
                    nr++;
                    s0 += l;
                    len -= l;
                }
            }
        }
    }
    const bool own = nr > FLAT_RCAP;
    if (nr == 0 || own) S.rng[0][tid] = 0u;  // an empty walk
    S.meta[tid] = (uint8_t)(own ? FLAT_OVER : 0u);
    const uint32_t key = flat_sort(((own ? 0u : tot) << 7) | (uint32_t)tid, reinterpret_cast<uint32_t*>(&s_dd[0][0]), S);
    const int src = (int)(key & 127u);
    const uint32_t meta = S.meta[src];
    flat_move(src, S);
    const bool live = voxel(src, cx, cy, cz);
    float density = 0.0f;
    float* dp = &s_dd[0][tid];
    float* const dfull = &s_dd[FLAT_CAP - 1][tid];
    auto test = [&](const float4 p, int32_t, bool, bool valid) {
        const float d0 = PFS_SUB(cx, p.x), d1 = PFS_SUB(cy, p.y), d2 = PFS_SUB(cz, p.z);
        const float dist2 = PFS_ADD(PFS_ADD(PFS_MUL(d0, d0), PFS_MUL(d1, d1)), PFS_MUL(d2, d2));
        *dp = dist2;
        dp += (valid && dist2 < P.r2) ? FLAT_THREADS : 0;
    };
    auto drain_if_full = [&]() {
        if (__any_sync(0xffffffffu, dp >= dfull)) {
            for (int c = 0; c < FLAT_CAP; c++)
                if (&s_dd[c][tid] < dp) density = PFS_ADD(density, map_term(P, s_dd[c][tid]));
            dp = &s_dd[0][tid];
        }
    };
    flat_walk(S, (int32_t)(key >> 7), 0, true, [&](int32_t j) { return __ldg(x + j); }, test, drain_if_full);
    for (const float* e = &s_dd[0][tid]; e < dp; e += FLAT_THREADS) density = PFS_ADD(density, map_term(P, *e));
    const uint64_t idx = first + (uint64_t)src;
    if (live)
        out[idx] = (meta & FLAT_OVER) ? map_walk(P, A, cx, cy, cz, x, table, err)
                                      : PFS_DIV(PFS_MUL(density, 1.0f), P.volume);
    else if (idx < nx * ny * nz)
        out[idx] = 0.0f;
}

// Voxels per warp up to which it evaluates terms as it tests: about 50 instructions
// per voxel and 64 positions and three per term for all lanes together, against
// 20 and 55.
constexpr uint32_t MAP_DIRECT = 8;
// Positions a block of the map stages at a time (22 KB).
constexpr uint32_t MAP_STAGE = 1408;

struct MapShared {
    uint32_t rs[CELLS_RUNS];         // table runs of the staged layers: first slot
    uint32_t re[CELLS_RUNS];         // and end
    uint32_t chunk[CELLS_RUNS + 4];  // scan chunks before run r
    uint32_t off[CELLS_RUNS + 4];    // staged positions before run r
    float4 nxy[CELLS_THREADS];       // the tile's voxel centres: (-x, -x, -y, -y)
    float2 nz[CELLS_THREADS];        // (-z, -z)
    uint32_t cell[CELLS_THREADS];    // cell in the block
    uint32_t start[65];              // the block's voxels before cell c
    int32_t first[3][8];             // per axis: first voxel of the block's cells 0 .. and past the last
    uint32_t warp_sum[CELLS_WARPS], kept[CELLS_WARPS];
};

// Stage layers [z0, z0 + zs) of the neighbourhood of the cells [b, b + dim):
// positions near them in run order and slot order.  Returns how many there are; fits:
// whether the stage holds them.
__device__ __forceinline__ uint32_t map_build(const DevParams& P, const MapArgs& A, MapShared& S, const CellsLayout& lay,
                                          float4* ent, uint32_t* zone, const int3 b, const int3 dim, int z0, int zs,
                                          const float4* __restrict__ x, const int2* __restrict__ table,
                                          const uint32_t* __restrict__ code, bool& fits, uint32_t* __restrict__ err) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t full = 0xffffffffu, lt = (1u << lane) - 1u;
    const uint32_t n = P.n, zcap = cells_warp_bytes(lay) / 4;
    const int nx = dim.x + 2, ny = dim.y + 2;
    const uint32_t R = (uint32_t)(nx * ny * zs);
    // scan chunks of 8 entries where runs hold a few, else of 32
    const int gs = (P.mask + 1u) >> __popc(P.mask) >= 10u ? 5 : 3;
    __syncthreads();  // the previous stage is no longer read
    const uint32_t ix = 65535u / (uint32_t)nx + 1u, iy = 65535u / (uint32_t)ny + 1u;  // exact for r < 216
    for (uint32_t r = tid; r < R; r += CELLS_THREADS) {
        const uint32_t qy = r * ix >> 16, qz = qy * iy >> 16;
        const int ex = b.x - 1 + (int)(r - qy * nx), ey = b.y - 1 + (int)(qy - qz * ny), ez = b.z - 1 + z0 + (int)qz;
        int2 se = make_int2(-1, -1);
        if (!map_out(ex, ey, ez, A.bound))
            se = __ldg(table + slot_of(P, cell_hash((uint32_t)ex, (uint32_t)ey, (uint32_t)ez)));
        if (se.x != -1 && (se.x < 0 || se.y > (int32_t)n || se.x > se.y)) {
            atomicOr(err, ERR_TABLE_RANGE);
            se.x = -1;
        }
        const uint32_t s0 = se.x == -1 ? 0u : (uint32_t)se.x, s1 = se.x == -1 ? 0u : (uint32_t)se.y;
        S.rs[r] = s0;
        S.re[r] = s1;
        S.chunk[r] = (s1 - s0 + (1u << gs) - 1u) >> gs;
        S.off[r] = 0u;
    }
    __syncthreads();
    const uint32_t C = cells_scan(S.warp_sum, S.chunk, R);
    // near: between one step below the layer under the box and one step past the
    // layer above it (the sum carries into the guard bit from there on)
    const uint32_t lo = ((uint32_t)(CELLS_CODE_STEPS * (b.x - 1) - 1) & 511u) |
                        (((uint32_t)(CELLS_CODE_STEPS * (b.y - 1) - 1) & 511u) << 10) |
                        (((uint32_t)(CELLS_CODE_STEPS * (b.z - 1) - 1) & 511u) << 20);
    const uint32_t add = (uint32_t)(512 - CELLS_CODE_STEPS * (dim.x + 2) - 2) |
                         ((uint32_t)(512 - CELLS_CODE_STEPS * (dim.y + 2) - 2) << 10) |
                         ((uint32_t)(512 - CELLS_CODE_STEPS * (dim.z + 2) - 2) << 20);
    auto keep = [&](uint32_t c) {
        const uint32_t t = ((c - lo) & ~CELLS_GUARD & 0x3fffffffu) + add;
        return ((t & CELLS_GUARD) | (c >> 31)) == 0u;
    };
    // each warp scans a contiguous share of the chunks, 32 chunks a round (each
    // lane looks one chunk's run up), eight loads in flight
    uint32_t zn = 0;
    const uint32_t c_end = (uint32_t)((uint64_t)C * (warp + 1u) / CELLS_WARPS);
    const int per = 32 >> gs;  // chunks per load
    for (uint32_t cb = (uint32_t)((uint64_t)C * warp / CELLS_WARPS); cb < c_end; cb += 32) {
        uint32_t run = 0, j0 = 0, j1 = 0;
        if (cb + lane < c_end) {
            uint32_t l = 0, u = R;  // last run whose first chunk is <= cb + lane
            while (u - l > 1) {
                const uint32_t mid = (l + u) >> 1;
                if (S.chunk[mid] <= cb + lane) l = mid; else u = mid;
            }
            run = l;
            j0 = S.rs[run] + ((cb + lane - S.chunk[run]) << gs);
            j1 = S.re[run];
        }
        const uint32_t left = min(c_end - cb, 32u);
        for (uint32_t u0 = 0; u0 < left; u0 += 8 * per) {
            uint32_t c[8], j[8], rn[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int from = (int)u0 + u * per + (lane >> gs);  // chunk of this lane
                const uint32_t q = __shfl_sync(full, j0, from), e = __shfl_sync(full, j1, from);
                rn[u] = __shfl_sync(full, run, from);
                j[u] = q + (lane & ((1 << gs) - 1));
                const bool in = j[u] < e;
                c[u] = in ? __ldg(code + j[u]) : 0x80000000u;
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const bool in = keep(c[u]);
                const uint32_t m = __ballot_sync(full, in);
                if (m) {
                    if (in) {
                        const uint32_t z = zn + __popc(m & lt);
                        if (z < zcap) zone[z] = j[u];
                        // the chunk's first kept lane counts it for its run
                        const uint32_t gm = gs == 5 ? m : (m >> (lane & 24) & 255u) << (lane & 24);
                        if (!(gm & lt)) atomicAdd(&S.off[rn[u]], (uint32_t)__popc(gm));
                    }
                    zn += __popc(m);
                }
            }
        }
    }
    if (lane == 0) S.kept[warp] = zn;
    __syncthreads();
    uint32_t base = 0, total = 0, most = 0;
#pragma unroll
    for (int w = 0; w < CELLS_WARPS; w++) {
        const uint32_t k = S.kept[w];
        base += w < warp ? k : 0u;
        total += k;
        most = max(most, k);
    }
    fits = most <= zcap && total <= lay.entries;
    if (!fits) return total;
#pragma unroll 4
    for (uint32_t k = lane; k < zn; k += 32) ent[base + k] = __ldg(x + zone[k]);
    cells_scan(S.warp_sum, S.off, R);
    return total;
}

// Per axis, the first voxel of the cells b + 0 .. b + 7 (the voxel of a cell is
// the one whose centre lies in it): from the quotient, then by the cell rule.
__device__ __forceinline__ void map_first(const DevParams& P, const MapArgs& A, const int3 b, int32_t first[3][8]) {
    const int tid = threadIdx.x;
    if (tid >= 24) return;
    const int a = tid >> 3, k = tid & 7;
    const int c = (a == 0 ? b.x : (a == 1 ? b.y : b.z)) + k;
    const float mn = a == 0 ? P.minx : (a == 1 ? P.miny : P.minz);
    const int top = a == 0 ? A.img.x : (a == 1 ? A.img.y : A.img.z);
    int v = min(max((int)floorf((float)c * P.h / A.cs - 0.5f) - 2, 0), top);
    while (v < top && cell_coord(map_centre(mn, v, A.cs), mn, P.h) < c) v++;
    first[a][k] = v;
}

// Most of a box is empty: blocks of 4 x 4 x 4 cells with no marked cell in them or
// next to them are set to 0 here, and only the blocks (nbx x nby x nbz of 2^bs cells)
// of the others are listed for k_map_cells.  (Finding the empty ones by scanning
// the 216 runs around each, which in a table of few slots hold hundreds of distant
// positions, took 133 us of a 300,000-particle scene's map; marking takes 31 and this 11.)
__global__ void __launch_bounds__(CELLS_THREADS)
k_map_coarse(DevParams P, MapArgs A, const uint8_t* __restrict__ marks, float* __restrict__ out,
             uint32_t* __restrict__ list, uint32_t* __restrict__ listed) {
    __shared__ int32_t s_first[3][8];
    const int tid = threadIdx.x;
    const uint32_t gx = (P.ngx >> 2) + 1, gy = (P.ngy >> 2) + 1;
    const uint32_t blk = blockIdx.x;
    const int3 b = make_int3((int)(blk % gx) << 2, (int)(blk / gx % gy) << 2, (int)(blk / (gx * gy)) << 2);
    const int3 g = make_int3((int)gx << 2, (int)gy << 2, (int)((P.ngz >> 2) + 1) << 2);
    bool any = false;
    for (int r = tid; r < 216; r += CELLS_THREADS) {
        const int cx = b.x - 1 + r % 6, cy = b.y - 1 + r / 6 % 6, cz = b.z - 1 + r / 36;
        if (cx >= 0 && cy >= 0 && cz >= 0 && cx < g.x && cy < g.y && cz < g.z)
            any = any || marks[(size_t)cx + (size_t)g.x * ((size_t)cy + (size_t)g.y * (size_t)cz)] != 0;
    }
    if (__syncthreads_or(any)) {
        const uint32_t fx = 4u >> P.bsx, fy = 4u >> P.bsy, fz = 4u >> P.bsz;
        const uint32_t k = tid;
        if (k < fx * fy * fz) {
            const uint32_t qx = ((uint32_t)b.x >> P.bsx) + k % fx, qy = ((uint32_t)b.y >> P.bsy) + k / fx % fy,
                           qz = ((uint32_t)b.z >> P.bsz) + k / (fx * fy);
            if (qx < P.nbx && qy < P.nby && qz < P.nbz)
                list[atomicAdd(listed, 1u)] = qx + P.nbx * (qy + P.nby * qz);
        }
        return;
    }
    map_first(P, A, b, s_first);
    __syncthreads();
    // (a map may have 2^31 voxels, and a block all of them)
    const uint32_t wx = s_first[0][4] - s_first[0][0], wy = s_first[1][4] - s_first[1][0],
                   wz = s_first[2][4] - s_first[2][0];
    for (uint32_t k = tid; k < wx * wy * wz; k += CELLS_THREADS) {
        const int vx = s_first[0][0] + (int)(k % wx), vy = s_first[1][0] + (int)(k / wx % wy),
                  vz = s_first[2][0] + (int)(k / (wx * wy));
        if (map_out(vx, vy, vz, A.bound) ||
            !map_inside(P, map_centre(P.minx, vx, A.cs), map_centre(P.miny, vy, A.cs), map_centre(P.minz, vz, A.cs)))
            continue;  // k_density_map's
        out[((uint64_t)vz * (uint64_t)A.img.y + (uint64_t)vy) * (uint64_t)A.img.x + (uint64_t)vx] =
            PFS_DIV(0.0f, P.volume);
    }
}

__global__ void __launch_bounds__(CELLS_THREADS, 5)
k_map_cells(DevParams P, MapArgs A, CellsLayout lay, const float4* __restrict__ x, const int2* __restrict__ table,
            const uint32_t* __restrict__ code, const uint32_t* __restrict__ list, const uint32_t* __restrict__ listed,
            float* __restrict__ out, uint32_t* __restrict__ err) {
    extern __shared__ float4 s_dyn[];
    __shared__ MapShared S;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t full = 0xffffffffu, lt = (1u << lane) - 1u;
    float4* ent = s_dyn;
    uint32_t* zone = reinterpret_cast<uint32_t*>(s_dyn + lay.entries) + warp * (cells_warp_bytes(lay) / 4);
    uint2* ballots = reinterpret_cast<uint2*>(zone);                      // [words]
    uint16_t* at = reinterpret_cast<uint16_t*>(zone + 2u * lay.words);     // [slots][64]
    const uint32_t nblk = *listed;
    const int3 dim0 = make_int3(1 << P.bsx, 1 << P.bsy, 1 << P.bsz);
    const int cells = dim0.x * dim0.y * dim0.z;
    for (uint32_t at_blk = blockIdx.x; at_blk < nblk; at_blk += gridDim.x) {
        const uint32_t blk = list[at_blk];
        const int3 b0 = make_int3((int)(blk % P.nbx) << P.bsx, (int)(blk / P.nbx % P.nby) << P.bsy,
                                  (int)(blk / (P.nbx * P.nby)) << P.bsz);
        __syncthreads();
        map_first(P, A, b0, S.first);
        __syncthreads();
        if (warp == 0) {  // voxels before each cell
            auto count = [&](int c) -> uint32_t {
                if (c >= cells) return 0u;
                const int lx = c & (dim0.x - 1), ly = c >> P.bsx & (dim0.y - 1), lz = c >> (P.bsx + P.bsy);
                return (uint32_t)((S.first[0][lx + 1] - S.first[0][lx]) * (S.first[1][ly + 1] - S.first[1][ly]) *
                                  (S.first[2][lz + 1] - S.first[2][lz]));
            };
            const uint32_t c0 = count(lane), c1 = count(lane + 32);
            uint32_t i0 = c0, i1 = c1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(full, i0, o), w = __shfl_up_sync(full, i1, o);
                if (lane >= o) {
                    i0 += u;
                    i1 += w;
                }
            }
            i1 += __shfl_sync(full, i0, 31);
            S.start[lane] = i0 - c0;
            S.start[32 + lane] = i1 - c1;
            if (lane == 31) S.start[64] = i1;
        }
        __syncthreads();
        const uint32_t voxels = S.start[64];
        if (voxels == 0u) continue;
        // The whole neighbourhood in one stage (most blocks have little near them);
        // where that does not fit, as many layers as it suggests, and then one.  Then
        // cell by cell, in the same way, where there are blocks for every thread block
        // or a walk takes longer (of a few blocks each one's cells in turn are what the
        // map waits for, 25 us and more a cell: 1,372 voxels 0.6 ms), and what is left walks.
        const float run = (float)P.n / (float)(1u << __popc(P.mask));
        const bool split = cells > 1 && (nblk >= gridDim.x || (float)cells * (25.0f + 0.15f * run) < 4.0f * run);
        int cell = -1, zs = dim0.z + 2;
        bool leave = false;
        for (;;) {
            const bool whole = cell < 0;
            const int3 dim = whole ? dim0 : make_int3(1, 1, 1);
            const int3 b = whole ? b0
                                 : make_int3(b0.x + (cell & (dim0.x - 1)), b0.y + (cell >> P.bsx & (dim0.y - 1)),
                                             b0.z + (cell >> (P.bsx + P.bsy)));
            const uint32_t p_lo = whole ? 0u : S.start[cell], p_hi = whole ? voxels : S.start[cell + 1];
            const int layers = dim.z + 2;
            bool fits = !leave, staged = false;
            uint32_t held = 0;
            for (uint32_t t0 = p_lo; t0 < p_hi && (fits || leave); t0 += CELLS_THREADS) {
                // ---- the tile's voxels
                __syncthreads();
                const uint32_t tile = min(p_hi - t0, (uint32_t)CELLS_THREADS);
                uint64_t idx = 0;
                bool mine_out = false;  // this thread's voxel is this kernel's to write
                if ((uint32_t)tid < tile) {
                    uint32_t c = 0;
#pragma unroll
                    for (uint32_t s = 32; s > 0; s >>= 1)
                        if (c + s < 64u && S.start[c + s] <= t0 + tid) c += s;
                    const int lx = (int)c & (dim0.x - 1), ly = (int)c >> P.bsx & (dim0.y - 1),
                              lz = (int)c >> (P.bsx + P.bsy);
                    const uint32_t k = t0 + tid - S.start[c];
                    const uint32_t wx = (uint32_t)(S.first[0][lx + 1] - S.first[0][lx]),
                                   wy = (uint32_t)(S.first[1][ly + 1] - S.first[1][ly]);
                    const int vx = S.first[0][lx] + (int)(k % wx), vy = S.first[1][ly] + (int)(k / wx % wy),
                              vz = S.first[2][lz] + (int)(k / (wx * wy));
                    const float cx = map_centre(P.minx, vx, A.cs), cy = map_centre(P.miny, vy, A.cs),
                                cz = map_centre(P.minz, vz, A.cs);
                    S.nxy[tid] = make_float4(-cx, -cx, -cy, -cy);
                    S.nz[tid] = make_float2(-cz, -cz);
                    S.cell[tid] = c;
                    idx = ((uint64_t)vz * (uint64_t)A.img.y + (uint64_t)vy) * (uint64_t)A.img.x + (uint64_t)vx;
                    mine_out = !map_out(vx, vy, vz, A.bound) && map_inside(P, cx, cy, cz);
                }
                __syncthreads();
                // ---- this warp's share of the tile: lane l holds the voxel of thread
                // w0 + l while it sums
                const uint32_t share = (tile + CELLS_WARPS - 1u) / CELLS_WARPS;
                const uint32_t w0 = min(warp * share, tile), w1 = min(w0 + share, tile);
                const bool mine = w0 + lane < w1;
                const uint32_t ms = mine ? w0 + lane : 0u;
                const float nx0 = S.nxy[ms].x, ny0 = S.nxy[ms].z, nz0 = S.nz[ms].x;
                const uint32_t mycell = S.cell[ms];
                float density = 0.0f;
                // a warp of few voxels (a dense scene's blocks are small) evaluates the
                // terms as it tests, a lane each, and leaves only the sums to a lane
                const bool direct = share <= MAP_DIRECT;
                const int nx = dim.x + 2, ny = dim.y + 2;
                for (int z0 = 0; z0 < layers && fits; z0 += zs) {
                    if (!staged || zs < layers)
                        held = map_build(P, A, S, lay, ent, zone, b, dim, z0, min(zs, layers - z0), x, table, code, fits,
                                         err);
                    if (!fits) break;
                    staged = true;
                    if (w0 >= w1) continue;
                    const int z1 = min(z0 + zs, layers);
                    // ballots as in the density pass: nk words, the first pair at wb,
                    // the next ones gm pairs apart; entry numbers from ab
                    uint32_t nk = 0, wb = 0, gm = 0, ab = 0;
                    uint32_t used_w = 0, used_s = 0;
                    // direct: this lane's terms wait in its part of the warp's space
                    float* terms = reinterpret_cast<float*>(zone);
                    const uint32_t tcap = cells_warp_bytes(lay) / 4u / max(share, 1u);
                    uint32_t cnt = 0;
                    auto flush = [&]() {
                        __syncwarp();
                        const float* t = terms + lane * tcap;
                        const uint32_t trips = __reduce_max_sync(full, cnt);
#pragma unroll 4
                        for (uint32_t k = 0; k < trips; k++)
                            if (k < cnt) density = PFS_ADD(density, t[k]);
                        cnt = 0;
                        __syncwarp();
                    };
                    auto drain = [&]() {
                        __syncwarp();
                        const uint32_t* bw = reinterpret_cast<const uint32_t*>(ballots);
                        auto word = [&](uint32_t k) { return k < nk ? bw[2u * (wb + (k >> 1) * gm) + (k & 1u)] : 0u; };
                        uint32_t k = 0, w = word(0), wn = word(1);
                        const uint16_t* an = at + ab;
                        auto next = [&](bool& has, float& term) {
                            const bool adv = w == 0u && k + 1u < nk;
                            k += adv ? 1u : 0u;
                            an += adv ? 32 : 0;
                            w = adv ? wn : w;
                            wn = adv ? word(k + 1u) : wn;
                            has = w != 0u;
                            const float4 c = ent[an[(__ffs(w) - 1) & 31]];
                            w &= w - 1u;
                            const float d0 = PFS_ADD(c.x, nx0), d1 = PFS_ADD(c.y, ny0), d2 = PFS_ADD(c.z, nz0);
                            term = map_term(P, PFS_ADD(PFS_ADD(PFS_MUL(d0, d0), PFS_MUL(d1, d1)), PFS_MUL(d2, d2)));
                        };
                        while (__any_sync(full, w != 0u || k + 1u < nk)) {
                            bool h0, h1;
                            float t0v, t1v;
                            next(h0, t0v);
                            next(h1, t1v);
                            // (adding +0 changes nothing: the sum starts at +0)
                            density = PFS_ADD(density, h0 ? t0v : 0.0f);
                            density = PFS_ADD(density, h1 ? t1v : 0.0f);
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
                        // the cell's rows of three runs in these layers
                        const int lx = whole ? (int)c & (dim0.x - 1) : 0, ly = whole ? (int)c >> P.bsx & (dim0.y - 1) : 0,
                                  lz = whole ? (int)c >> (P.bsx + P.bsy) : 0;
                        uint32_t st = 0, ln = 0;
                        {
                            const int dz = lane * 11 >> 5, dy = lane - 3 * dz;
                            if (lane < 9 && lz + dz >= z0 && lz + dz < z1) {
                                const int r0 = lx + nx * (ly + dy + ny * (lz + dz - z0));
                                st = S.off[r0];
                                ln = S.off[r0 + 3] - st;
                            }
                        }
                        uint32_t incl = ln;
#pragma unroll
                        for (int o = 1; o < 16; o <<= 1) {
                            const uint32_t v = __shfl_up_sync(full, incl, o);
                            if (lane >= o) incl += v;
                        }
                        const uint32_t L = __shfl_sync(full, incl, 8);
                        const uint32_t sub = st - (incl - ln);  // entry = q + sub of its row
                        auto locate = [&](uint32_t q) -> uint32_t {
                            int r = 0;
#pragma unroll
                            for (int w = 8; w > 0; w >>= 1)
                                if (__shfl_sync(full, incl, r + w - 1) <= q) r += w;
                            const uint32_t e = q + __shfl_sync(full, sub, min(r, 8));
                            return q < L ? e : 0u;
                        };
                        const float4 none = make_float4(INFINITY, INFINITY, INFINITY, 0.0f);
                        for (uint32_t q0 = 0; q0 < L; q0 += 64) {
                            if (!direct && (used_s == lay.slots || used_w + g > lay.words)) drain();
                            if (member && nk == 0u) {
                                wb = used_w + (uint32_t)(lane - a);
                                gm = g;
                                ab = used_s * 64u;
                            }
                            const uint32_t at0 = locate(q0 + lane), at1 = locate(q0 + 32 + lane);
                            const float4 c0 = q0 + lane < L ? ent[at0] : none;
                            const float4 c1 = q0 + 32 + lane < L ? ent[at1] : none;
                            if (!direct) {
                                at[used_s * 64u + lane] = (uint16_t)at0;
                                at[used_s * 64u + 32u + lane] = (uint16_t)at1;
                            }
                            const f32x2 x2 = pack2(c0.x, c1.x), y2 = pack2(c0.y, c1.y), z2 = pack2(c0.z, c1.z);
                            const float4* pxy = S.nxy + w0 + a;
                            const float2* pz = S.nz + w0 + a;
                            if (direct) {
                                for (uint32_t m = 0; m < g; m++) {
                                    const float4 mxy = pxy[m];
                                    const float mz = pz[m].y;
                                    auto dist2 = [&](const float4 e) {
                                        const float d0 = PFS_ADD(e.x, mxy.x), d1 = PFS_ADD(e.y, mxy.z),
                                                    d2 = PFS_ADD(e.z, mz);
                                        return PFS_ADD(PFS_ADD(PFS_MUL(d0, d0), PFS_MUL(d1, d1)), PFS_MUL(d2, d2));
                                    };
                                    const float s0 = dist2(c0), s1 = dist2(c1);
                                    const bool i0 = s0 < P.r2, i1 = s1 < P.r2;
                                    const uint32_t in0 = __ballot_sync(full, i0), in1 = __ballot_sync(full, i1);
                                    const uint32_t n0 = __popc(in0), add = n0 + __popc(in1);
                                    uint32_t cm = __shfl_sync(full, cnt, a + m);
                                    if (cm + add > tcap) {
                                        flush();
                                        cm = 0;
                                    }
                                    float* to = terms + (a + m) * tcap + cm;
                                    if (i0) to[__popc(in0 & lt)] = map_term(P, s0);
                                    if (i1) to[n0 + __popc(in1 & lt)] = map_term(P, s1);
                                    if (lane == a + (int)m) cnt += add;
                                }
                                continue;
                            }
                            uint2* to = ballots + used_w;
#pragma unroll 4
                            for (uint32_t m = 0; m < g; m++) {
                                const float4 mxy = pxy[m];
                                const float2 mz = pz[m];
                                const f32x2 d0 = add2(x2, pack2(mxy.x, mxy.y)), d1 = add2(y2, pack2(mxy.z, mxy.w)),
                                            d2 = add2(z2, pack2(mz.x, mz.y));
                                // (the sums unpacked: packed ones would be contracted)
                                float ax, ay, az, bx, by, bz;
                                unpack2(mul2(d0, d0), ax, bx);
                                unpack2(mul2(d1, d1), ay, by);
                                unpack2(mul2(d2, d2), az, bz);
                                const uint32_t b0w = __ballot_sync(full, PFS_ADD(PFS_ADD(ax, ay), az) < P.r2);
                                const uint32_t b1w = __ballot_sync(full, PFS_ADD(PFS_ADD(bx, by), bz) < P.r2);
                                to[m] = make_uint2(b0w, b1w);  // every lane stores the same pair
                            }
                            used_w += g;
                            used_s++;
                            if (member) nk += 2u;
                        }
                    }
                    if (direct)
                        flush();
                    else
                        drain();
                }
                // the sums go back to the threads that know the voxels
                __syncthreads();
                if (mine) S.nz[ms].x = density;
                __syncthreads();
                if (mine_out) {
                    if (fits)
                        out[idx] = PFS_DIV(PFS_MUL(S.nz[tid].x, 1.0f), P.volume);
                    else if (leave)
                        out[idx] = __uint_as_float(MAP_LEFT);
                }
            }
            if (!fits && !leave) {
                // (a layer of the middle holds more than the mean)
                const float fit = 0.85f * (float)lay.entries * (float)zs / (float)held;
                if (zs > 1 && fit >= 0.7f) {
                    zs = zs == layers ? min(max((int)fit, 1), layers - 1) : 1;
                } else if (whole && split) {
                    cell = 0;
                    zs = 3;
                } else {
                    leave = true;
                }
                continue;
            }
            if (whole || cell + 1 == cells) break;
            cell++;
            zs = 3;
            leave = false;
        }
    }
}

}  // namespace

// Positions a layer of a block's neighbourhood holds: its cells' own, and in a table of
// few slots those of the whole neighbourhood that share a slot with one of them, once
// for each.
static double map_layer(int sx, int sy, int sz, double per_cell, double slots) {
    const double runs = ((1 << sx) + 2.25) * ((1 << sy) + 2.25);
    return runs * per_cell * (1.0 + runs * ((1 << sz) + 2.25) / slots);
}

// Cells per block: about 64 voxels (half a tile, for small maps' sake), as many
// cells as the stage holds at the fluid's density, and runs that are mostly of
// different slots; at most 4 x 4 x 4.
static void map_blocks(DevParams* P, float cell_size, double per_cell) {
    const double vpc = std::pow((double)P->h / (double)cell_size, 3.0);
    const double slots = (double)(1ull << __builtin_popcount(P->mask));
    P->cshift = 0;
    P->bsx = P->bsy = P->bsz = 0;
    for (int total = 1; total <= 6; total++) {
        const int sx = (total + 2) / 3, sy = (total - sx + 1) / 2, sz = total - sx - sy;
        const double runs = (double)((1 << sx) + 2) * ((1 << sy) + 2) * ((1 << sz) + 2);
        if (map_layer(sx, sy, sz, per_cell, slots) > (double)MAP_STAGE || (double)(1 << (total - 1)) * vpc >= 128.0 ||
            runs > 1.5 * slots)
            break;
        P->bsx = sx;
        P->bsy = sy;
        P->bsz = sz;
    }
    // one cell past the grid: a centre within rounding of the box's far face may
    // round into it
    P->nbx = (P->ngx >> P->bsx) + 1;
    P->nby = (P->ngy >> P->bsy) + 1;
    P->nbz = (P->ngz >> P->bsz) + 1;
}

// Which kernel makes a map: the blocks of cells (M: map_blocks), the flat walk or a thread
// per voxel: the least of what each takes, in us.  Fitted to the three kernels' times of
// 2,650 maps (300 to 260,000 particles, 4 to 16,384 slots, 0.3 to 100 particles a cell,
// 1/37 to 27 voxels a cell, the box 3% to all full; one deviation 40 to 60%); the kernel
// taken was slower than a thread per voxel by more than 5% in 18 of them, and 0.51 of it
// in the mean, where the least of the three is 0.48.  So a map of 666 particles on 32 slots,
// 1,372 voxels, walks (83 us, blocks 610), the reference's 300,000 on 4,096 are grouped
// (0.6 ms, walks 5.2), a full table's runs, which hold a few entries, are walked flat
// (1M-particle slab, 1M voxels: 0.25 ms, blocks 0.38, a thread per voxel 0.31), and runs of
// hundreds a thread per voxel, with twice the flat walk's threads on an SM.
enum MapRoute { MAP_PLAIN, MAP_FLAT, MAP_CELLS };
static MapRoute map_route(const DevParams& P, const DevParams& M, const MapArgs& A, double per_cell) {
    const double n = P.n, slots = (double)(1ull << __builtin_popcount(P.mask));
    // entries of a run of an empty cell, and of one in the fluid
    const double run = n / slots, wet_run = run + per_cell;
    const double thousands = 1e-3 * (double)A.img.x * (double)A.img.y * (double)A.img.z;
    const double voxels_a_cell = std::pow((double)P.h / (double)A.cs, 3.0);
    const double wet = std::min(thousands, 1e-3 * n / per_cell * voxels_a_cell), dry = thousands - wet;
    const double plain = 41.0 + 4.0 * wet_run + dry * (0.12 + 0.0246 * run) + wet * (0.104 + 0.0271 * wet_run);
    const double flat = 27.5 + 2.72 * wet_run + dry * (0.075 + 0.0349 * run) + wet * (0.071 + 0.0349 * wet_run);
    // (from here on some runs are more than the flat walk's words, and walked anyway)
    const MapRoute walk = wet_run <= 32.0 && (run < 4.0 || flat < 0.8 * plain) ? MAP_FLAT : MAP_PLAIN;
    // the list of blocks takes a sort buffer; and a grid of many more cells than voxels
    // has little to group
    const double blocks = (double)M.nbx * M.nby * M.nbz;
    if (run < 4.0 || std::max(P.ngx, std::max(P.ngy, P.ngz)) > CELLS_MAX_GRID || blocks > std::min(1e3 * thousands, n))
        return walk;
    const int layers = (1 << M.bsz) + 2;
    const double R = (double)((1 << M.bsx) + 2) * ((1 << M.bsy) + 2) * layers;
    const double layer = map_layer(M.bsx, M.bsy, M.bsz, per_cell, slots), held = layer * layers;
    if (layer > (double)MAP_STAGE) return walk;  // its voxels would be left
    const double block_voxels = (double)(1 << (M.bsx + M.bsy + M.bsz)) * voxels_a_cell;
    const double tiles = std::max(1.0, std::ceil(block_voxels / 128.0));
    const double scans = 0.9 * held <= 0.95 * MAP_STAGE ? 1.0 : 1.0 + tiles;
    const double block = 6.9 + scans * (2.5 + 0.00178 * R * wet_run) + 0.0134 * held * tiles +
                         block_voxels * (0.0138 + 0.00102 * 27.0 * per_cell * (1.0 + R / slots));
    // blocks that are or lie beside fluid, of 740 resident ones
    const double side = std::cbrt(n / per_cell) + 2.0;
    const double near = std::min(blocks, (side / (1 << M.bsx) + 0.5) * (side / (1 << M.bsy) + 0.5) *
                                             (side / (1 << M.bsz) + 0.5));
    const double grouped = 37.0 + 0.62e-3 * n + 0.028 * thousands + block * std::max(1.0, near / 757.0);
    return grouped < 0.8 * (walk == MAP_FLAT ? flat : plain) ? MAP_CELLS : walk;
}

cudaError_t launch_density_map(const DevParams& P, const StepBuffers& b, float cell_size, double per_cell,
                               const int32_t image[3], const int32_t bound[3], float* out, cudaStream_t s) {
    const uint32_t n = P.n;
    if (n == 0) return cudaSuccess;
    const unsigned g = (n + MAP_THREADS - 1) / MAP_THREADS;
    k_table_runs<<<g, MAP_THREADS, 0, s>>>(n, b.skeys, b.table, 1);
    const MapArgs A = {cell_size, make_int3(image[0], image[1], image[2]), make_int3(bound[0], bound[1], bound[2])};
    const uint64_t voxels = (uint64_t)A.img.x * (uint64_t)A.img.y * (uint64_t)A.img.z;
    if (voxels) {
        const unsigned gv = (unsigned)((voxels + MAP_THREADS - 1) / MAP_THREADS);
        DevParams M = P;
        map_blocks(&M, cell_size, per_cell);
        const MapRoute route = map_route(P, M, A, per_cell);
        if (route == MAP_PLAIN) {
            k_density_map<true><<<gv, MAP_THREADS, 0, s>>>(P, A, b.x, b.table, out, b.err);
        } else if (route == MAP_FLAT) {
            const cudaError_t e = flat_carveout(k_map_flat);
            if (e != cudaSuccess) return e;
            const unsigned gf = (unsigned)((voxels + FLAT_THREADS - 1) / FLAT_THREADS);
            k_map_flat<<<gf, FLAT_THREADS, 0, s>>>(P, A, b.x, b.table, out, b.err);
        } else {
            // the marks take the neighbour lists' buffer (64 bytes for each 4 x 4 x 4 cells,
            // of which there are at most n)
            const uint32_t coarse = ((P.ngx >> 2) + 1) * ((P.ngy >> 2) + 1) * ((P.ngz >> 2) + 1);
            static_assert(NLIST_CAP * 4 >= 64, "marks in the neighbour lists");
            uint8_t* marks = reinterpret_cast<uint8_t*>(b.nlist);
            cudaError_t e = cudaMemsetAsync(marks, 0, (size_t)coarse * 64, s);
            if (e != cudaSuccess) return e;
            k_map_code<<<g, MAP_THREADS, 0, s>>>(P, b.x, b.keys_tmp, marks);
            const CellsLayout lay = {MAP_STAGE, 256u, 20u};
            const size_t dyn = (size_t)lay.entries * 16 + CELLS_WARPS * (size_t)cells_warp_bytes(lay);
            e = cudaFuncSetAttribute(k_map_cells, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
            uint32_t* listed = b.scanq_n + CTR_BLOCKS;
            if (e == cudaSuccess) e = cudaMemsetAsync(listed, 0, 4, s);
            if (e != cudaSuccess) return e;
            k_map_coarse<<<coarse, CELLS_THREADS, 0, s>>>(M, A, marks, out, b.vals_tmp, listed);
            k_map_cells<<<std::min(cells_grid(k_map_cells, dyn), M.nbx * M.nby * M.nbz), CELLS_THREADS, dyn, s>>>(
                M, A, lay, b.x, b.table, b.keys_tmp, b.vals_tmp, listed, out, b.err);
            k_density_map<false><<<gv, MAP_THREADS, 0, s>>>(P, A, b.x, b.table, out, b.err);
        }
    }
    k_table_runs<<<g, MAP_THREADS, 0, s>>>(n, b.skeys, b.table, 0);
    return cudaGetLastError();
}

}  // namespace pfs
