// tension3.cu -- surface tension for the 3D step (Tension3.java): the colour, its blurs, the capillary stress and
// the grid update with the stress's force; node (k*ny + j)*nx + i. The passes run over tiles of nodes, and in a step
// that sorts only over the tiles the fluid can reach.
//
// Every operation is the reference's, in its order, rounded once (the _rn intrinsics keep the compiler from
// fusing a multiply into an add), so the passes give the same bits as the float restatement on the CPU. Reads of
// a neighbour are held to the wall ring [1, n-2] on every axis, as Tension3.at does (Tension3.java:215-221).
#include <algorithm>

#include "mpm3_kernels.cuh"

namespace vf {

namespace {

constexpr float MIN_COLOUR = 0.3f;    // Tension.MIN_COLOUR (Tension.java:74)
constexpr float MASS_FLOOR = 0.3f;    // Tension.MASS_FLOOR (Tension.java:77)
constexpr float EPS2 = (float)(1e-4 * 1e-4);   // Tension3.EPS squared, formed in double (Tension3.java:57, 145)
constexpr int WALL3 = 1;              // Flip3.WALL

__device__ __forceinline__ int held(int c, int size) { return min(max(c, WALL3), size - 1 - WALL3); }

__device__ __forceinline__ int64_t index3(const Dims3& d, int i, int j, int k) {
    return ((int64_t)k * d.ny + j) * d.nx + i;
}

// The passes work on tiles of TT_X x TT_Y x TT_Z nodes, a CTA of 256 threads a tile at a time. A tile's nodes and a
// one-node halo, each read at its held coordinates, are staged in shared memory (34 x 10 x 10 floats in rows of 36, so
// a thread's float2 reads stay aligned), a warp a row at a time; every neighbour read of the reference is then a
// shared-memory read.
constexpr int TT_X = TENSION3_TX, TT_Y = TENSION3_TY, TT_Z = TENSION3_TZ;
constexpr int TH_Y = TT_Y + 2, TH_Z = TT_Z + 2, TROW = 36;
constexpr int TENSION_THREADS = 256;
using TensionTile = float[TH_Z][TH_Y][TROW];

// The a-th tile of a pass: of the list of live tiles, or of all tiles when there is none.
__device__ __forceinline__ int tile_count(const TensionTiles& t) { return t.list ? *t.count : t.tnx * t.tny * t.tnz; }

__device__ __forceinline__ void tile_origin(const TensionTiles& t, int a, int& x0, int& y0, int& z0) {
    const int tile = t.list ? t.list[a] : a;
    x0 = tile % t.tnx * TT_X;
    y0 = tile / t.tnx % t.tny * TT_Y;
    z0 = tile / (t.tnx * t.tny) * TT_Z;
}

// Stages the tile at (x0, y0, z0) and its halo. For SCALED (the first blur: src is the grid, float4 {m, ...}) a staged
// value is the node's mass over a full node's, no more than one; a full node on the wall ring holds half a rest mass
// for each wall through it. That depends on the node read alone, so it is formed once per staged node.
template <bool SCALED>
__device__ __forceinline__ void stage_tile(TensionTile& tile, const void* src, float rho0, const Dims3& d, int x0, int y0,
                                           int z0) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cx[2] = {held(x0 + lane - 1, d.nx), held(x0 + 31 + lane, d.nx)};   // columns lane, and 32 + lane (2 lanes)
    auto colour = [&](float mass, int x, int y, int z) {
        const int c[3] = {x, y, z}, size[3] = {d.nx, d.ny, d.nz};
        float full = rho0;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            if (c[a] == WALL3) full = __fmul_rn(0.5f, full);
            if (c[a] == size[a] - 1 - WALL3) full = __fmul_rn(0.5f, full);
        }
        return fminf(__fdiv_rn(mass, full), 1.0f);
    };
    constexpr int ROWS = TH_Y * TH_Z, PER = (ROWS + 7) / 8;
    float v[PER], w[PER];
#pragma unroll
    for (int r = 0; r < PER; r++) {   // every row's loads in flight together
        const int row = warp + 8 * r;
        v[r] = w[r] = 0.0f;
        if (row < ROWS) {
            const int64_t n = index3(d, 0, held(y0 + row % TH_Y - 1, d.ny), held(z0 + row / TH_Y - 1, d.nz));
            if (SCALED) {
                const float4* g = static_cast<const float4*>(src);
                v[r] = g[n + cx[0]].x;
                if (lane < 2) w[r] = g[n + cx[1]].x;
            } else {
                const float* g = static_cast<const float*>(src);
                v[r] = g[n + cx[0]];
                if (lane < 2) w[r] = g[n + cx[1]];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < PER; r++) {
        const int row = warp + 8 * r;
        if (row >= ROWS) continue;
        const int ly = row % TH_Y, lz = row / TH_Y;
        if (SCALED) {
            const int y = held(y0 + ly - 1, d.ny), z = held(z0 + lz - 1, d.nz);
            v[r] = colour(v[r], cx[0], y, z);
            if (lane < 2) w[r] = colour(w[r], cx[1], y, z);
        }
        tile[lz][ly][lane] = v[r];
        if (lane < 2) tile[lz][ly][32 + lane] = w[r];
    }
    __syncthreads();
}

}  // namespace

// The live tiles of this step: those the cell scan marked (mark, zeroed again here) listed in any order; and a tile that
// was live before and no longer is has both colour planes cleared, so that outside the live tiles the planes hold the
// zeros that a pass over every tile would write there. A warp takes 32 tiles.
__global__ void __launch_bounds__(256) k_tension3_tiles(TensionTiles t, float* c0, float* c1, Dims3 d) {
    const int lane = threadIdx.x & 31, n = t.tnx * t.tny * t.tnz;
    for (int base = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 32; base < n; base += gridDim.x * 256) {
        const int tile = base + lane;
        const bool live = tile < n && t.mark[tile] != 0, was = tile < n && t.prev[tile] != 0;
        if (live) t.mark[tile] = 0;
        if (live != was) t.prev[tile] = live ? 1 : 0;
        const unsigned m = __ballot_sync(0xffffffffu, live);
        int at = 0;
        if (lane == 0 && m) at = atomicAdd(t.count, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (live) t.list[at + __popc(m & ((1u << lane) - 1))] = tile;
        for (unsigned left = __ballot_sync(0xffffffffu, was && !live); left; left &= left - 1) {
            const int q = base + __ffs(left) - 1;
            const int x = q % t.tnx * TT_X + lane, y0 = q / t.tnx % t.tny * TT_Y, z0 = q / (t.tnx * t.tny) * TT_Z;
            for (int r = 0; r < TT_Y * TT_Z; r++) {
                const int y = y0 + r % TT_Y, z = z0 + r / TT_Y;
                if (x < d.nx && y < d.ny && z < d.nz) c0[index3(d, x, y, z)] = c1[index3(d, x, y, z)] = 0.0f;
            }
        }
    }
}

// Tension3.blur (Tension3.java:73-107): the [1 2 1]^3/64 blur of the node mass taken to a colour (SCALED) or of the last
// colour, dk outermost and di innermost, each read held to the wall ring. The weights are powers of two, so a product
// is exact and adding it is one fused operation with the same bits as the reference's multiply and add (but for
// products below the normal range, far under anything the later passes can see).
//
// A thread blurs two neighbours along x over half the tile's z-layers: a row's four values are two 8-byte reads, kept
// for the three layers that use them, so a node costs 27 adds and 1.5 shared reads.
template <bool SCALED>
__global__ void __launch_bounds__(TENSION_THREADS) k_tension3_blur(const void* src, float* dst, const Params3* params,
                                                                   Dims3 d, TensionTiles t) {
    __shared__ __align__(16) TensionTile tile;
    const float rho0 = SCALED ? params->rho0 : 0.0f;
    const int px = threadIdx.x & 15, ty = (threadIdx.x >> 4) & 7, zh = threadIdx.x >> 7;
    const int n = tile_count(t);
    for (int a = blockIdx.x; a < n; a += gridDim.x) {
        int x0, y0, z0;
        tile_origin(t, a, x0, y0, z0);
        stage_tile<SCALED>(tile, src, rho0, d, x0, y0, z0);
        const int i = x0 + 2 * px, j = y0 + ty, kz = zh * (TT_Z / 2);
        float win[3][3][4];   // [layer][row][x - 1 .. x + 2], sliding one layer per output node
        auto layer = [&](int p, int lz) {
#pragma unroll
            for (int r = 0; r < 3; r++) {
                const float2 lo = *reinterpret_cast<const float2*>(&tile[lz][ty + r][2 * px]);
                const float2 hi = *reinterpret_cast<const float2*>(&tile[lz][ty + r][2 * px + 2]);
                win[p][r][0] = lo.x;
                win[p][r][1] = lo.y;
                win[p][r][2] = hi.x;
                win[p][r][3] = hi.y;
            }
        };
        layer(1, kz);
        layer(2, kz + 1);
#pragma unroll
        for (int tz = 0; tz < TT_Z / 2; tz++) {
#pragma unroll
            for (int r = 0; r < 3; r++)
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    win[0][r][q] = win[1][r][q];
                    win[1][r][q] = win[2][r][q];
                }
            layer(2, kz + tz + 2);
            float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
            for (int dk = 0; dk < 3; dk++)
#pragma unroll
                for (int dj = 0; dj < 3; dj++)
#pragma unroll
                    for (int di = 0; di < 3; di++) {
                        const float weight = (float)((2 - abs(di - 1)) * (2 - abs(dj - 1)) * (2 - abs(dk - 1))) / 64.0f;
                        s0 = __fmaf_rn(weight, win[dk][dj][di], s0);
                        s1 = __fmaf_rn(weight, win[dk][dj][di + 1], s1);
                    }
            const int k = z0 + kz + tz;
            if (i < d.nx && j < d.ny && k < d.nz) {
                float* o = dst + index3(d, i, j, k);
                if ((d.nx & 1) == 0) {
                    *reinterpret_cast<float2*>(o) = make_float2(s0, s1);
                } else {
                    o[0] = s0;
                    if (i + 1 < d.nx) o[1] = s1;
                }
            }
        }
        __syncthreads();   // the tile is free for the next
    }
}

// Tension3.stress (Tension3.java:128-154): the stress over sigma from the colour's central differences g,
// diagonal (|g|^2 - g_a^2)/|g| and off the diagonal -g_a g_b/|g|, |g| kept off zero by EPS. Only nodes holding
// MIN_COLOUR are ever read (k_grid3_tension's open faces join two of them), so only those are written.
__global__ void __launch_bounds__(TENSION_THREADS) k_tension3_stress(const float* colour, float* stress, Dims3 d,
                                                                     TensionTiles t) {
    __shared__ __align__(16) TensionTile tile;
    const int64_t n = (int64_t)d.nx * d.ny * d.nz;
    const int tx = (threadIdx.x & 31) + 1, ty = (threadIdx.x >> 5) + 1;
    const int tiles = tile_count(t);
    for (int a = blockIdx.x; a < tiles; a += gridDim.x) {
        int x0, y0, z0;
        tile_origin(t, a, x0, y0, z0);
        stage_tile<false>(tile, colour, 0.0f, d, x0, y0, z0);
        const int i = x0 + tx - 1, j = y0 + ty - 1;
        for (int tz = 1; tz <= TT_Z; tz++) {
            const int k = z0 + tz - 1;
            if (i >= d.nx || j >= d.ny || k >= d.nz || !(tile[tz][ty][tx] > MIN_COLOUR)) continue;
            float g[3];
            g[0] = __fmul_rn(0.5f, __fsub_rn(tile[tz][ty][tx + 1], tile[tz][ty][tx - 1]));
            g[1] = __fmul_rn(0.5f, __fsub_rn(tile[tz][ty + 1][tx], tile[tz][ty - 1][tx]));
            g[2] = __fmul_rn(0.5f, __fsub_rn(tile[tz + 1][ty][tx], tile[tz - 1][ty][tx]));
            const float xx = __fmul_rn(g[0], g[0]), yy = __fmul_rn(g[1], g[1]), zz = __fmul_rn(g[2], g[2]);
            const float length = __fsqrt_rn(__fadd_rn(__fadd_rn(xx, __fadd_rn(yy, zz)), EPS2));
            const int64_t node = index3(d, i, j, k);
            stress[0 * n + node] = __fdiv_rn(__fadd_rn(yy, zz), length);
            stress[1 * n + node] = __fdiv_rn(__fadd_rn(xx, zz), length);
            stress[2 * n + node] = __fdiv_rn(__fadd_rn(xx, yy), length);
            stress[3 * n + node] = -__fdiv_rn(__fmul_rn(g[0], g[1]), length);
            stress[4 * n + node] = -__fdiv_rn(__fmul_rn(g[0], g[2]), length);
            stress[5 * n + node] = -__fdiv_rn(__fmul_rn(g[1], g[2]), length);
        }
        __syncthreads();   // the tile is free for the next
    }
}

// Flip3.gridWithTension (Flip3.java:267-310) with Tension3.force (Tension3.java:162-200): the force over sigma on
// a node is the flux of the stress across its six faces, the mean of T_ab at the two nodes a face joins, over
// the faces whose nodes both hold MIN_COLOUR, on nodes of the wall ring or inside it; across a face in the wall
// only the normal stress crosses.
__device__ __forceinline__ void tension_node(const Step3& s, const float* colour, const float* stress, const Params3& p,
                                             int i, int j, int k) {
    const Dims3 d = s.d;
    const int64_t node = index3(d, i, j, k);
    const float4 g4 = s.grid[node];
    float v[3];
    grid_velocity_free(g4, p, v);
    const float mass = g4.x;
    if (mass > EMPTY3) {
        const int64_t n = (int64_t)d.nx * d.ny * d.nz;
        const int at[3] = {i, j, k};
        const int size[3] = {d.nx, d.ny, d.nz};
        // the stress planes a face along axis a carries, component c: T_ac (txx tyy tzz txy txz tyz)
        const int tensor[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
        bool ring = colour[node] > MIN_COLOUR;
#pragma unroll
        for (int a = 0; a < 3; a++) ring = ring && !(at[a] < WALL3) && !(at[a] > size[a] - 1 - WALL3);
        float force[3] = {0.0f, 0.0f, 0.0f};
        if (ring) {
#pragma unroll
            for (int a = 0; a < 3; a++) {
#pragma unroll
                for (int sign = -1; sign <= 1; sign += 2) {
                    int c3[3] = {held(i, d.nx), held(j, d.ny), held(k, d.nz)};
                    c3[a] = held(at[a] + sign, size[a]);
                    const int64_t there = index3(d, c3[0], c3[1], c3[2]);
                    if (!(colour[there] > MIN_COLOUR)) continue;
                    const bool wall = sign < 0 ? !(at[a] > WALL3) : !(at[a] < size[a] - 1 - WALL3);
                    const float shear = wall ? 0.0f : 1.0f;
                    const float half = 0.5f * (float)sign;
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const float* t = stress + (int64_t)tensor[a][c] * n;
                        const float flux = __fmul_rn(half, __fadd_rn(t[node], t[there]));
                        force[c] = __fadd_rn(force[c], c == a ? flux : __fmul_rn(shear, flux));
                    }
                }
            }
        }
        const float push = __fdiv_rn(__fmul_rn(p.dt, p.sigma), fmaxf(mass, __fmul_rn(MASS_FLOOR, p.rho0)));
#pragma unroll
        for (int a = 0; a < 3; a++) v[a] = __fadd_rn(v[a], __fmul_rn(push, force[a]));
    }
    const float3 w = grid_walls(v, i, j, k, d, p);
    s.vel[node] = make_float4(w.x, w.y, w.z, 0.0f);
}

__global__ void __launch_bounds__(TENSION_THREADS) k_grid3_tension(Step3 s, const float* colour, const float* stress,
                                                                   TensionTiles t) {
    const Params3 p = *s.params;
    const int tiles = tile_count(t);
    for (int a = blockIdx.x; a < tiles * TT_Z; a += gridDim.x) {   // a tile's layer at a time, a node a thread
        int x0, y0, z0;
        tile_origin(t, a / TT_Z, x0, y0, z0);
        const int i = x0 + (threadIdx.x & 31), j = y0 + (threadIdx.x >> 5), k = z0 + a % TT_Z;
        if (i < s.d.nx && j < s.d.ny && k < s.d.nz) tension_node(s, colour, stress, p, i, j, k);
    }
}

cudaError_t launch_tension3_tiles(const TensionTiles& t, float* c0, float* c1, const Dims3& d, cudaStream_t stream) {
    const int n = t.tnx * t.tny * t.tnz;
    k_tension3_tiles<<<std::min((n + 255) / 256, sm_count()), 256, 0, stream>>>(t, c0, c1, d);
    return cudaGetLastError();
}

// A pass's CTAs: one a tile where they all fit the GPU at once (eight CTAs of 256 threads an SM), else that many, each
// taking the tiles of its stride.
static int tension_blocks(const TensionTiles& t) { return std::min(t.tnx * t.tny * t.tnz, 8 * sm_count()); }

cudaError_t launch_tension3_blur(bool scaled, const void* src, float* dst, const Params3* params, const Dims3& d,
                                 const TensionTiles& t, cudaStream_t stream) {
    if (scaled)
        k_tension3_blur<true><<<tension_blocks(t), TENSION_THREADS, 0, stream>>>(src, dst, params, d, t);
    else
        k_tension3_blur<false><<<tension_blocks(t), TENSION_THREADS, 0, stream>>>(src, dst, params, d, t);
    return cudaGetLastError();
}

cudaError_t launch_tension3_stress(const float* colour, float* stress, const Dims3& d, const TensionTiles& t,
                                   cudaStream_t stream) {
    k_tension3_stress<<<tension_blocks(t), TENSION_THREADS, 0, stream>>>(colour, stress, d, t);
    return cudaGetLastError();
}

cudaError_t launch_grid3_tension(const Step3& s, const float* colour, const float* stress, const TensionTiles& t,
                                 cudaStream_t stream) {
    k_grid3_tension<<<std::min(TT_Z * t.tnx * t.tny * t.tnz, 8 * sm_count()), TENSION_THREADS, 0, stream>>>(s, colour, stress,
                                                                                                         t);
    return cudaGetLastError();
}

}  // namespace vf
