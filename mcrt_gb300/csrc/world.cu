// world.cu — the procedural voxel world on the GPU: a seeded terrain generator
// and the chunked face mesher that turns the voxel grid into the triangle mesh
// the tracer renders.
//
// Voxel grid: one byte per voxel (block id), index (x * ny + y) * nz + z — the
// XZY-major order of the reference's chunks (world/chunk.rs:26-31) extended to
// the whole grid.  Chunks are 16 x ny x 16 columns; chunk (i, k) of the grid has
// chunk coordinates (chunk_x0 + i, chunk_z0 + k) and world origin
// chunk_world_origin (world/chunk.rs:131-137).
//
// Mesher: world/mesher.rs:97-366.  A warp takes two (chunk, face direction,
// layer) slices of an X or Y direction, or one of a Z direction: it stages the
// slice's visible faces in shared memory (a face is visible when its block is
// opaque and the neighbour along the normal is not; outside the grid counts as
// air, as the reference's missing neighbour chunks do) and grows the greedy
// rectangles of a row together.  A count pass, an exclusive scan and an emit
// pass place every quad where the reference's sequential loop would: chunks in
// (x outer, z inner) order, then +X, -X, +Y, -Y, +Z, -Z, layers, then the greedy
// order within the slice.  MCRT_MESH_FACES emits one quad per visible face in
// the same order (the exposed-face mesh).
#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace mcrt {

namespace {

// ------------------------------------------------------------------ noise
// Lattice value noise: a PCG hash of the integer lattice point and the seed
// gives a value in [0, 1); values are blended with the smoothstep fade
// t^2 (3 - 2t).  fBm sums octaves with frequency * lacunarity and
// amplitude * gain per octave, normalised by the amplitude sum.
__device__ __forceinline__ uint32_t lattice_hash(int32_t x, int32_t y, int32_t z, uint32_t seed) {
    uint32_t h = pcg_hash((uint32_t)x * 0x8da6b343u ^ seed);
    h = pcg_hash(h ^ ((uint32_t)y * 0xd8163841u));
    return pcg_hash(h ^ ((uint32_t)z * 0xcb1ab31fu));
}
__device__ __forceinline__ float lattice_value(int32_t x, int32_t y, int32_t z, uint32_t seed) {
    return (float)(lattice_hash(x, y, z, seed) >> 8) * (1.0f / 16777216.0f);
}
__device__ __forceinline__ float fade(float t) { return t * t * (3.0f - 2.0f * t); }
__device__ __forceinline__ float lerpf(float a, float b, float t) { return a + (b - a) * t; }

__device__ float value_noise2(float x, float z, uint32_t seed) {
    float fx0 = floorf(x), fz0 = floorf(z);
    int32_t ix = (int32_t)fx0, iz = (int32_t)fz0;
    float tx = fade(x - fx0), tz = fade(z - fz0);
    float a = lerpf(lattice_value(ix, 0, iz, seed), lattice_value(ix + 1, 0, iz, seed), tx);
    float b = lerpf(lattice_value(ix, 0, iz + 1, seed), lattice_value(ix + 1, 0, iz + 1, seed), tx);
    return lerpf(a, b, tz);
}
__device__ float value_noise3(float x, float y, float z, uint32_t seed) {
    float fx0 = floorf(x), fy0 = floorf(y), fz0 = floorf(z);
    int32_t ix = (int32_t)fx0, iy = (int32_t)fy0, iz = (int32_t)fz0;
    float tx = fade(x - fx0), ty = fade(y - fy0), tz = fade(z - fz0);
    float c[2];
    for (int k = 0; k < 2; ++k) {
        float a = lerpf(lattice_value(ix, iy, iz + k, seed), lattice_value(ix + 1, iy, iz + k, seed), tx);
        float b = lerpf(lattice_value(ix, iy + 1, iz + k, seed), lattice_value(ix + 1, iy + 1, iz + k, seed), tx);
        c[k] = lerpf(a, b, ty);
    }
    return lerpf(c[0], c[1], tz);
}
__device__ float fbm2(float x, float z, uint32_t octaves, float lac, float gain, uint32_t seed) {
    float sum = 0.0f, amp = 1.0f, norm = 0.0f, f = 1.0f;
    for (uint32_t o = 0; o < octaves; ++o) {
        sum += amp * value_noise2(x * f, z * f, seed + o * 0x9e3779b9u);
        norm += amp;
        amp *= gain;
        f *= lac;
    }
    return sum / norm;
}
__device__ float fbm3(float x, float y, float z, uint32_t octaves, float lac, float gain, uint32_t seed) {
    float sum = 0.0f, amp = 1.0f, norm = 0.0f, f = 1.0f;
    for (uint32_t o = 0; o < octaves; ++o) {
        sum += amp * value_noise3(x * f, y * f, z * f, seed + o * 0x9e3779b9u);
        norm += amp;
        amp *= gain;
        f *= lac;
    }
    return sum / norm;
}

// ------------------------------------------------------------------ generator
// Block ids of the reference's registry (world/block.rs:14-24).
constexpr uint8_t kAir = 0, kLimestone = 1, kRedSoil = 2, kGrass = 3, kSand = 4, kWater = 5, kShrub = 8,
                  kGravel = 9, kCaveGlow = 10;

// Column: limestone (gravel patches) below, 3 blocks of red soil (sand near the
// sea), a grass (sand) top, caves carved by 3D fBm above cave_min_y, glowing
// flora on some cave floors, water up to the sea level, shrubs on some grass
// tops.
//
// Bound by integer hashing (up to 40 hashes per voxel below the surface), so
// what counts is how many warps share it: a block takes 32 columns (lane =
// column, z fastest, so a row of one y is 32 contiguous bytes) and its eight
// warps take every eighth y.  With one thread per column the 128^3 grid ran
// 512 warps, less than one per scheduler, in 92 us; it now takes 41 us.
// The second pass decorates from the blocks of the first: whether a block is
// air does not change in it, so the order over y does not matter.
constexpr uint32_t kGenWarps = 8;

__global__ void __launch_bounds__(32 * kGenWarps) k_world_generate(mcrt_world_params P, uint8_t *vox) {
    extern __shared__ uint8_t s_col[];                       // [ny][32]: the blocks of the first pass
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t t = blockIdx.x * 32u + lane;
    const uint32_t ny = P.ny;
    const bool active = t < P.nx * P.nz;
    const uint32_t x = active ? t / P.nz : 0u, z = active ? t - x * P.nz : 0u;
    const int32_t gx = P.chunk_x0 * 16 + (int32_t)x, gz = P.chunk_z0 * 16 + (int32_t)z;
    const float hn = fbm2((float)gx * P.height_freq, (float)gz * P.height_freq, P.height_octaves, P.lacunarity,
                          P.gain, P.seed);
    const float hf = P.height_base + P.height_amp * (2.0f * hn - 1.0f);
    int32_t surface = (int32_t)floorf(hf);
    surface = max(1, min(surface, (int32_t)ny - 2));
    const bool beach = (float)surface <= P.sand_line;
    for (uint32_t y = warp; y < ny; y += kGenWarps) {
        const int32_t yi = (int32_t)y;
        uint8_t b = kAir;
        if (yi <= surface) {
            if (yi == surface) b = beach ? kSand : kGrass;
            else if (yi >= surface - 3) b = beach ? kSand : kRedSoil;
            else {
                b = kLimestone;
                if (value_noise3((float)gx * 0.11f, (float)yi * 0.11f, (float)gz * 0.11f, P.seed ^ 0x5bd1e995u) > 0.72f)
                    b = kGravel;
            }
            if (y >= P.cave_min_y) {
                const float c = fbm3((float)gx * P.cave_freq, (float)yi * P.cave_freq, (float)gz * P.cave_freq,
                                     P.cave_octaves, P.lacunarity, P.gain, P.seed ^ 0x6c62272eu);
                if (0.5f + (c - 0.5f) * P.cave_contrast > P.cave_threshold) b = kAir;
            }
        } else if ((float)yi <= P.sea_level) {
            b = kWater;
        }
        s_col[y * 32u + lane] = b;
    }
    __syncthreads();
    if (!active) return;
    uint8_t *col = vox + (size_t)x * ny * P.nz + z;
    for (uint32_t y = warp; y < ny; y += kGenWarps) {
        const int32_t yi = (int32_t)y;
        uint8_t b = s_col[y * 32u + lane];
        if (y >= 1u && y + 1u < ny && yi < surface) {
            // cave floors: a solid block under a carved voxel below the surface
            if (b != kAir && s_col[(y + 1u) * 32u + lane] == kAir &&
                (lattice_hash(gx, yi, gz, P.seed ^ 0x27d4eb2fu) & 7u) == 0u)
                b = kCaveGlow;
        } else if (yi == surface + 1) {
            // shrubs on some grass tops (nothing decorates the surface block itself); at two layers the
            // surface is the top one, and surface + 1 no layer of the grid
            if (b == kAir && s_col[(uint32_t)surface * 32u + lane] == kGrass &&
                (lattice_hash(gx, 0, gz, P.seed ^ 0x165667b1u) & 15u) == 0u)
                b = kShrub;
        }
        col[(size_t)y * P.nz] = b;
    }
}

// ------------------------------------------------------------------ mesher
// BLOCK_META[id].opaque (world/block.rs:53-125): ids 1..10 occlude, air and
// unassigned ids do not.
__device__ __forceinline__ bool opaque(uint8_t id) { return id >= 1 && id <= 10; }

struct MeshGrid {
    const uint8_t *vox;
    uint32_t nx, ny, nz, ncz;
    int32_t chunk_x0, chunk_z0;
    uint32_t per_chunk;     // slices per chunk: 16 + 16 + ny + ny + 16 + 16
    uint32_t units;         // warps per chunk: slices of the X and Y directions in pairs, of Z one by one
    uint32_t pitch_z;       // cells of a row of a Z slice (v = y), a multiple of 32
};

// What one warp meshes: two neighbouring layers of an X or Y direction (their
// rows are 16 cells of v = z: a half warp each) or one layer of a Z direction
// (rows of ny cells of v = y, 32 at a time).
struct MeshUnit {
    uint32_t cx, cz;        // chunk index in the grid
    int axis, sign, ua, va;
    uint32_t layer, udim, vdim;
    bool pair, second;      // two layers; the second one exists
    uint32_t slice;         // the (first) slice
};

__device__ __forceinline__ MeshUnit unit_of(const MeshGrid &G, uint32_t k) {
    MeshUnit m;
    const uint32_t c = k / G.units;
    uint32_t r = k - c * G.units;
    m.cx = c / G.ncz;
    m.cz = c - m.cx * G.ncz;
    const uint32_t dims[3] = {16u, G.ny, 16u};
    uint32_t first = c * G.per_chunk;
    int dir = 0;
    for (; dir < 6; ++dir) {                       // +X, -X, +Y, -Y, +Z, -Z (mesher.rs:77-84)
        const uint32_t layers = dims[dir >> 1], n = dir < 4 ? (layers + 1u) >> 1 : layers;
        if (r < n) break;
        r -= n;
        first += layers;
    }
    m.axis = dir >> 1;
    m.sign = (dir & 1) ? -1 : 1;
    m.pair = dir < 4;
    m.layer = m.pair ? 2u * r : r;
    m.second = m.pair && m.layer + 1u < dims[m.axis];
    m.slice = first + m.layer;
    m.ua = m.axis == 0 ? 1 : 0;                    // mesher.rs:137-141
    m.va = m.axis == 2 ? 1 : 2;
    m.udim = dims[m.ua];
    m.vdim = dims[m.va];
    return m;
}

struct MeshOut {
    float4 *v;                   // mcrt_gpu_vertex records, 3 float4 each
    uint4 *t;                    // mcrt_gpu_triangle records
    const uint32_t *quad_base;   // per slice
    const uint32_t *mat_of;      // 256 block -> material slot
    float voxel;
};

// emit_quad (mesher.rs:308-366) of n staged quads (quad index, u0 | v0 << 16,
// h | w << 16, block id | second layer << 8), by the whole warp: consecutive
// lanes write consecutive 16-byte words of the vertex records.
__device__ __forceinline__ void emit_quads(const MeshGrid &G, const MeshUnit &m, const MeshOut &O, const uint4 *quads,
                                           uint32_t n, uint32_t lane) {
    const float s = O.voxel;
    const float ox = (float)(G.chunk_x0 + (int32_t)m.cx) * 16.0f * s;
    const float oz = (float)(G.chunk_z0 + (int32_t)m.cz) * 16.0f * s;
    const uint32_t face = m.sign > 0 ? 1u : 0u;
    for (uint32_t i = lane; i < 12u * n; i += 32u) {
        const uint32_t k = i / 12u, part = i - 12u * k, corner = part / 3u, what = part - 3u * corner;
        const uint4 e = quads[k];
        float4 r;
        if (what == 0u) {                                     // corners (u0, v0), (u0+h, v0), (u0+h, v0+w), (u0, v0+w)
            const uint32_t uu = (e.y & 0xffffu) + ((corner == 1u || corner == 2u) ? (e.z & 0xffffu) : 0u);
            const uint32_t vv = (e.y >> 16) + (corner >= 2u ? e.z >> 16 : 0u);
            const float pa = (float)(m.layer + (e.w >> 8) + face) * s, pu = (float)uu * s, pv = (float)vv * s;
            const float px = m.axis == 0 ? pa : pu;           // u is x on the Y and Z axes
            const float py = m.axis == 1 ? pa : (m.axis == 0 ? pu : pv);
            const float pz = m.axis == 2 ? pa : pv;
            r = make_float4(ox + px, 0.0f + py, oz + pz, 1.0f);
        } else if (what == 1u) {
            const float sg = (float)m.sign;
            r = make_float4(m.axis == 0 ? sg : 0.0f, m.axis == 1 ? sg : 0.0f, m.axis == 2 ? sg : 0.0f, 0.0f);
        } else {
            r = make_float4((corner == 1u || corner == 2u) ? 1.0f : 0.0f, corner >= 2u ? 1.0f : 0.0f, 0.0f, 0.0f);
        }
        O.v[(size_t)e.x * 12u + part] = r;
    }
    for (uint32_t i = lane; i < 2u * n; i += 32u) {
        const uint4 e = quads[i >> 1];
        const uint32_t b = 4u * e.x, mat = __ldg(O.mat_of + (e.w & 0xffu));
        uint4 t;
        if (i & 1u) t = m.sign > 0 ? make_uint4(b, b + 2, b + 3, mat) : make_uint4(b, b + 3, b + 2, mat);
        else t = m.sign > 0 ? make_uint4(b, b + 1, b + 2, mat) : make_uint4(b, b + 2, b + 1, mat);
        O.t[(size_t)e.x * 2u + (i & 1u)] = t;
    }
}

// Meshing of one unit by one warp (mesher.rs:185-243); EMIT = false counts the
// quads of each slice.
//
// The reference grows rectangles cell by cell: at the first free cell of a row
// a run of equal blocks along v, then rows along u while the whole run
// repeats.  Runs of one row do not touch each other (a rectangle only takes
// cells of its own columns in later rows), so the warp grows all rectangles
// that start in a row at once: lane = column, a run lives on while the ballot
// of its columns is full, and taken cells are cleared in the staged slice.
// Every lane reads and writes its own columns only.  Rows longer than 32 cells
// (Z directions of grids above 32 blocks) agree through a flag per run in
// shared memory instead of a ballot.
//
// Bound by the grid reads (bytes, L1/L2) and the stores of the quads (224 B
// each).  One thread per slice re-read the grid for every comparison and wrote
// its quads alone: 2350 us to count and 2680 us to emit the greedy mesh of a
// 128^3 world, 127 and 134 us this way.
constexpr uint32_t kMeshStage = 64;      // staged quads per warp: written out at 32 or more

__host__ __device__ __forceinline__ size_t mesh_cell_bytes(uint32_t ny, uint32_t pitch_z) {
    const uint32_t x = 32u * ny, z = 16u * pitch_z;
    return (size_t)(x > z ? x : z) > 512u ? (x > z ? x : z) : 512u;
}
__host__ __device__ __forceinline__ size_t mesh_warp_bytes(uint32_t ny, uint32_t pitch_z) {
    return kMeshStage * 16u + ((mesh_cell_bytes(ny, pitch_z) + 7u * pitch_z + 15u) & ~(size_t)15u);
}

template <bool EMIT>
__global__ void __launch_bounds__(128) k_world_mesh(MeshGrid G, uint32_t n_units, int greedy, uint32_t *counts,
                                                    MeshOut O) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t k = blockIdx.x * (blockDim.x >> 5) + warp;
    if (k >= n_units) return;                                // whole warps
    uint8_t *mem = smem + warp * mesh_warp_bytes(G.ny, G.pitch_z);
    uint4 *stage = reinterpret_cast<uint4 *>(mem);
    uint8_t *cells = mem + kMeshStage * 16u;
    const uint32_t P = G.pitch_z;
    uint16_t *run_start = reinterpret_cast<uint16_t *>(cells + mesh_cell_bytes(G.ny, P));   // wide rows: per column
    uint16_t *run_end = run_start + P, *run_h = run_end + P;                                // per run, at its start
    uint8_t *run_fail = reinterpret_cast<uint8_t *>(run_h + P);
    const MeshUnit m = unit_of(G, k);
    const uint32_t half = m.pair ? lane >> 4 : 0u;
    const uint32_t chunks = m.pair ? 1u : P >> 5, pitch = m.pair ? 32u : P;
    const unsigned lt = (1u << lane) - 1u;
    const unsigned group = m.pair ? 0xffffu << (16u * half) : 0xffffffffu;    // lanes of this lane's slice
    // ---- the faces of the slice(s): a block id where the block is opaque and the neighbour along the normal is
    //      not (outside the grid: air, mesher.rs:261-300), else 0
    {
        const size_t stride[3] = {(size_t)G.ny * G.nz, G.nz, 1};
        const uint32_t layer = m.layer + half;
        const uint32_t org[3] = {m.cx * 16u, 0u, m.cz * 16u}, dims[3] = {G.nx, G.ny, G.nz};
        const int64_t q = (int64_t)org[m.axis] + layer + m.sign;
        const bool inside = q >= 0 && q < (int64_t)dims[m.axis];
        const int64_t step = m.sign * (int64_t)stride[m.axis];
        const bool exists = half == 0u || m.second;
        for (uint32_t c = 0; c < chunks; ++c) {
            const uint32_t v = m.pair ? lane & 15u : 32u * c + lane;
            const bool in = exists && v < m.vdim;
            const uint8_t *p = G.vox + (org[0] * stride[0] + org[2]) + layer * stride[m.axis] + v * stride[m.va];
            const size_t su = stride[m.ua];
            uint8_t *out = cells + 32u * c + lane;
#pragma unroll 8
            for (uint32_t u = 0; u < m.udim; ++u) {
                const uint8_t id = in ? __ldg(p + u * su) : (uint8_t)0;
                const uint8_t nb = in && inside ? __ldg(p + u * su + step) : (uint8_t)0;
                out[u * pitch] = opaque(id) && !opaque(nb) ? id : (uint8_t)0;
            }
        }
    }
    __syncwarp();
    uint32_t quads = 0;                                      // of this lane's slice
    uint32_t qbase = 0;
    if (EMIT && (half == 0u || m.second)) qbase = O.quad_base[m.slice + half];
    uint32_t staged = 0;
    auto push = [&](bool p, uint32_t u0, uint32_t v0, uint32_t h, uint32_t w, uint32_t id) {
        const unsigned mask = __ballot_sync(0xffffffffu, p);
        if (EMIT) {
            if (p)
                stage[staged + __popc(mask & lt)] = make_uint4(qbase + quads + __popc(mask & group & lt),
                                                               u0 | (v0 << 16), h | (w << 16), id | (half << 8));
            staged += __popc(mask);
            if (staged >= kMeshStage - 32u) {
                __syncwarp();
                emit_quads(G, m, O, stage, staged, lane);
                __syncwarp();
                staged = 0;
            }
        }
        quads += __popc(mask & group);
    };
    if (!greedy) {
        for (uint32_t u = 0; u < m.udim; ++u)
            for (uint32_t c = 0; c < chunks; ++c) {
                const uint32_t id = cells[u * pitch + 32u * c + lane];
                if (__any_sync(0xffffffffu, id != 0u)) push(id != 0u, u, m.pair ? lane & 15u : 32u * c + lane, 1u, 1u, id);
            }
    } else if (chunks == 1u) {
        const bool first = m.pair ? (lane & 15u) == 0u : lane == 0u;
        const bool last = m.pair ? (lane & 15u) == 15u : lane == 31u;
        for (uint32_t u0 = 0; u0 < m.udim; ++u0) {
            const uint32_t id = cells[u0 * 32u + lane];
            if (!__any_sync(0xffffffffu, id != 0u)) continue;
            const uint32_t before = __shfl_up_sync(0xffffffffu, id, 1), after = __shfl_down_sync(0xffffffffu, id, 1);
            const bool start = id && (first || id != before), end = id && (last || id != after);
            const unsigned starts = __ballot_sync(0xffffffffu, start), ends = __ballot_sync(0xffffffffu, end);
            const uint32_t s = 31u - __clz((starts & (lt | (1u << lane))) | 1u);
            const uint32_t e = (uint32_t)__ffs((ends & ~lt) | 0x80000000u) - 1u;
            const unsigned run = (e == 31u ? 0xffffffffu : (2u << e) - 1u) & ~((1u << s) - 1u);   // where id != 0
            bool alive = id != 0u;
            uint32_t h = 1;
            for (uint32_t u = u0 + 1; u < m.udim; ++u) {
                const unsigned same = __ballot_sync(0xffffffffu, alive && cells[u * 32u + lane] == id);
                alive = alive && (same & run) == run;
                if (!__any_sync(0xffffffffu, alive)) break;
                if (alive) {
                    cells[u * 32u + lane] = 0;
                    ++h;
                }
            }
            push(start, u0, m.pair ? lane & 15u : lane, h, e - s + 1u, id);
        }
    } else {
        for (uint32_t u0 = 0; u0 < m.udim; ++u0) {
            __syncwarp();                                    // the cells cleared from the rows above
            const uint8_t *row = cells + u0 * pitch;
            uint32_t alive = 0, last_start = 0;              // bit c: this lane's column of chunk c
            for (uint32_t c = 0; c < chunks; ++c) {
                const uint32_t v = 32u * c + lane, id = row[v];
                const bool start = id && (v == 0u || row[v - 1u] != id);
                const unsigned starts = __ballot_sync(0xffffffffu, start);
                const unsigned mine = starts & (lt | (1u << lane));
                run_start[v] = (uint16_t)(mine ? 32u * c + 31u - __clz(mine) : last_start);
                if (starts) last_start = 32u * c + 31u - __clz(starts);
                if (id) alive |= 1u << c;
                run_fail[v] = 0;
                run_h[v] = 1;
            }
            if (!__any_sync(0xffffffffu, alive != 0u)) continue;
            const uint32_t own = alive;
            for (uint32_t c = 0; c < chunks; ++c) {          // the end of a run, noted at its start
                const uint32_t v = 32u * c + lane;
                if ((own >> c) & 1u)
                    if (v + 1u == m.vdim || row[v + 1u] != row[v]) run_end[run_start[v]] = (uint16_t)(v + 1u);
            }
            __syncwarp();
            for (uint32_t u = u0 + 1; u < m.udim; ++u) {
                uint8_t *next = cells + u * pitch;
                for (uint32_t c = 0; c < chunks; ++c) {
                    const uint32_t v = 32u * c + lane;
                    if (((alive >> c) & 1u) && next[v] != row[v]) run_fail[run_start[v]] = 1;
                }
                __syncwarp();
                for (uint32_t c = 0; c < chunks; ++c) {
                    const uint32_t v = 32u * c + lane;
                    if (!((alive >> c) & 1u)) continue;
                    if (run_fail[run_start[v]]) {
                        alive &= ~(1u << c);
                    } else {
                        next[v] = 0;
                        if (run_start[v] == v) run_h[v] = (uint16_t)(u + 1u - u0);
                    }
                }
                __syncwarp();
                if (!__any_sync(0xffffffffu, alive != 0u)) break;
            }
            __syncwarp();
            for (uint32_t c = 0; c < chunks; ++c) {
                const uint32_t v = 32u * c + lane;
                const bool start = ((own >> c) & 1u) && run_start[v] == v;
                if (__any_sync(0xffffffffu, start))
                    push(start, u0, v, start ? run_h[v] : 0u, start ? run_end[v] - v : 0u, row[v]);
            }
        }
    }
    if (EMIT) {
        __syncwarp();
        emit_quads(G, m, O, stage, staged, lane);
    } else {
        if (lane == 0u) counts[m.slice] = quads;
        if (lane == 16u && m.second) counts[m.slice + 1u] = quads;
    }
}

}  // namespace

void launch_world_generate(const mcrt_world_params &P, uint8_t *vox, cudaStream_t st) {
    const uint32_t n = P.nx * P.nz;
    k_world_generate<<<(n + 31) / 32, 32 * kGenWarps, 32 * P.ny, st>>>(P, vox);
    ::mcrt::note_launch();
}

cudaError_t world_mesh(const uint8_t *d_vox, uint32_t nx, uint32_t ny, uint32_t nz, int32_t chunk_x0, int32_t chunk_z0,
                       bool greedy, const uint32_t *d_mat_of, float voxel, WorldMeshBuffers &M, cudaStream_t st) {
    MeshGrid G;
    G.vox = d_vox;
    G.nx = nx; G.ny = ny; G.nz = nz;
    G.ncz = nz / 16;
    G.chunk_x0 = chunk_x0;
    G.chunk_z0 = chunk_z0;
    G.per_chunk = 64 + 2 * ny;
    const uint32_t n_chunks = (nx / 16) * (nz / 16), n_slices = n_chunks * G.per_chunk;
    G.units = 48 + 2 * ((ny + 1) / 2);
    G.pitch_z = (ny + 31) / 32 * 32;
    const uint32_t n_units = n_chunks * G.units;
    // warps per block: four, or as many as fit 48 KB (one at ny = 1024: 41 KB)
    const size_t warp_bytes = mesh_warp_bytes(ny, G.pitch_z);
    const int warps = (int)std::max<size_t>(1, std::min<size_t>(4, (48 * 1024) / warp_bytes));
    const size_t smem = warps * warp_bytes;
    if (smem > 48 * 1024) return cudaErrorInvalidValue;
    const size_t scan_words = scan_tmp_words(n_slices + 1);
    cudaError_t e;
    if ((e = M.counts.ensure((size_t)(n_slices + 1) * 4 * 2 + scan_words * 4)) != cudaSuccess) return e;
    uint32_t *counts = M.counts.as<uint32_t>();
    uint32_t *base = counts + n_slices + 1;
    uint32_t *tmp = base + n_slices + 1;
    if ((e = cudaMemsetAsync(counts + n_slices, 0, 4, st)) != cudaSuccess) return e;
    const int blocks = (int)((n_units + warps - 1) / warps);
    MeshOut O{};
    k_world_mesh<false><<<blocks, 32 * warps, smem, st>>>(G, n_units, greedy ? 1 : 0, counts, O);
    ::mcrt::note_launch();
    exclusive_scan_u32(counts, base, n_slices + 1, tmp, st);
    uint32_t total = 0;
    if ((e = cudaMemcpyAsync(&total, base + n_slices, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
    if ((uint64_t)total * 2 >= (1ull << 27) - 1) return cudaErrorInvalidValue;   // triangle-id bound of the tracer
    if ((e = M.vertices.ensure((size_t)std::max(total, 1u) * 4 * sizeof(mcrt_gpu_vertex))) != cudaSuccess) return e;
    if ((e = M.triangles.ensure((size_t)std::max(total, 1u) * 2 * sizeof(mcrt_gpu_triangle))) != cudaSuccess) return e;
    O.v = M.vertices.as<float4>();
    O.t = M.triangles.as<uint4>();
    O.quad_base = base;
    O.mat_of = d_mat_of;
    O.voxel = voxel;
    k_world_mesh<true><<<blocks, 32 * warps, smem, st>>>(G, n_units, greedy ? 1 : 0, counts, O);
    ::mcrt::note_launch();
    M.n_quads = total;
    return cudaGetLastError();
}

}  // namespace mcrt
