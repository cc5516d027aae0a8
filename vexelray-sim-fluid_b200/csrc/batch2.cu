// batch2.cu -- many independent 2D scenes (each a FlipStep: sort by cell, scatter, grid, advect;
// FlipStep.java:81-193, Flip.java) stepped by ONE cooperative persistent kernel launch per step,
// the launches replayed from a CUDA graph. No counterpart in the reference, which steps one scene
// per ParticleSimulation; the per-node arithmetic, the stencils and the particles' moves are the single-scene
// step's (mpm2_device.cuh); the stencil sums are in paired fp32 with fused multiply-adds.
//
// Layout in HBM (scenes side by side, no per-scene allocation):
//   particles   two sets (ping-pong by step parity) of 10 f32 a slot: float4 {x y m j}, float4 {c00 c01 c10 c11},
//               float2 {u v}. The scatter reads one cell's particles a lane; of ten arrays each such read fetched
//               a 32-byte sector for 4 bytes. scene s owns slots [p0, p0 + np) of every field, and keeps them: the sort is by
//               (scene, tile, cell), so a scene's particles never leave its range
//   grid        two buffers (by step parity) of float4 {m, mu, mv, 0} per node; scene s's nodes at
//               g0 + j*nx + i
//   tiles       a scene's (nx-2) x (ny-2) stencil cells are cut into tiles of tx x ty cells, ntx x nty
//               of them; the tile entries of all scenes, each scene's followed by a sentinel, hold the
//               per-step counts and the run starts (by parity)
//   cells       cell keys tile-major: key = c0 + tile * tx*ty + (ly * tx + lx), one count and one cursor
//               per key
//
// One step = five phases separated by a grid-wide barrier (the launch is cooperative, so every CTA is
// resident; the barrier's wait is bounded and sets a status bit rather than hang):
//   1  tile scan     per scene: tile counts -> run starts (parity buffer), counts zeroed; each tile's run cut
//                    into chunks, counted per scene
//   2  cell scan     a warp per non-empty tile: cell counts -> cursors (cell starts), counts zeroed; CTA 0 lays
//                    the scenes' chunks out one after another. The tiles are dealt to the warps one by one: 32
//                    neighbouring tiles a warp left the full ones with few warps (136 -> 21 us a step of 256 scenes).
//   3  permute       per slot: perm[cursor[key]++] = slot, one cursor bump per run of equal keys of a warp. Within a
//                    cell the order is the atomics' (unspecified, as in the reference's CountingSort,
//                    SortTest.java:121-134); what the scatter needs is each cell's particles contiguous. The
//                    chunks enter the item list, and the other parity's grid is cleared over the windows of
//                    the tiles the previous step scattered into.
//   4  scatter       a warp per chunk, the first dealt and the rest drawn: the tile's cells clipped to the chunk (the cursors hold
//                    each run's end) are ordered by count, largest first, and taken in rounds of 32, a lane a cell
//                    (several lanes a cell where a round has few); a lane sums Flip.scatter's 27 amounts over its
//                    particles in registers, two at a time, their fields copied to shared memory a pair ahead, and
//                    when the round's fullest cell is done all its lanes add their sums into the warp's private node
//                    window (a round's lanes hold distinct cells, so distinct nodes at each stencil offset: plain
//                    read-modify-write); then one 16-byte red.global.add.v4.f32 per touched window node
//   5  gather        a group of threads per chunk, chunks dealt in turn: the tile window's node velocities (Flip.grid,
//                    fused) in shared memory, then per particle Flip.advectBody; the particle is written to its sorted slot
//                    of the other set, and its next cell tallied in shared memory for the next step's sort.
// Chunks bound a work item, so a dense tile (tens of thousands of particles in the 64^2 scenes) spreads over
// many warps instead of one.
//
// What bounds it and what it measured, 256 scenes of 64^2 to 512^2 nodes with 16.7M particles, a step (us):
//   scatter 583 -> 299  a warp's lanes read 32 cells' particles: with ten arrays of floats that was 320 sectors of 32
//                       bytes a step of a warp; with three of records it is 96. Tried: a CTA a chunk with the chunk
//                       staged in shared memory in slot order, a thread a cell, 390 (instructions and barriers); 24
//                       warps an SM in 80 registers, 460.
//   gather  539 -> 240  an item's reads hang one on another (item, sources, particles, window), each a trip to memory:
//                       now the next items' are in flight during this one's arithmetic, in paired fp32; floor 155
//   permute 198 -> 164, cell scan 136 -> 21, tile scan 8
#include <algorithm>
#include <cmath>
#include <map>
#include <string>
#include <vector>

#include "mpm2_device.cuh"
#include "sort.cuh"

using namespace vf;

namespace {

struct Scene2 {
    int nx, ny, np;
    int tx, ty, ntx, nty, tc;   // tile shape in cells (powers of two), tiles per axis, cells per tile
    int lgx, lgy;               // log2 of tx, ty
    int wmul;                   // 65536 / (tx + 2) rounded up: window node j is in row (j * wmul) >> 16
    int p0;                     // first particle slot
    int t0;                     // first tile entry: ntx*nty tiles, then a sentinel
    int c0;                     // first cell key
    int64_t g0;                 // first grid node
    Params2 prm;
};

// A work item: a chunk of a tile's particles, with what the scatter and gather read of its scene ahead of it.
struct __align__(16) Item2 {
    int c0, c1, t, s;        // slots [c0, c1), tile entry, scene
    long long g0;            // the grid node of the tile's first cell
    int nx, ny;              // the scene's grid
    int x0, y0, cb, lg;      // the tile's first cell, its first cell key, log2 of its sides: x | y << 8
};

// The batch's device state, passed by value to the step kernel.
struct Batch2 {
    const Scene2* scene;
    int nscenes;
    const int* tile_scene;     // tile entry -> scene, -1 for a sentinel
    int nentries;              // tile entries (every scene's tiles and its sentinel)
    float* part[2];            // a set: float4 {x y m j} per slot, then float4 {c00 c01 c10 c11}, then float2 {u v}
    int64_t stride;            // slots of a set
    int np;                    // all scenes' particles
    int ncells;                // all scenes' cell keys
    int* key;                  // per slot of the current set: the cell key for this step's sort
    int* perm;                 // sorted slot -> slot of the current set
    int* cell_count;
    int* cursor;               // per cell: its run's start after the cell scan, its end after the permute
    int* tile_count;
    int* tile_start[2];        // per tile entry, by step parity: run start; the sentinel holds the scene's end
    int* chunk_start;          // per tile entry: its first chunk within its scene; the sentinel the scene's chunks
    int* scene_chunks;         // per scene: its chunks
    int* scene_chunk_start;    // per scene (and one past): its first chunk in the item list
    Item2* item;               // per chunk, written by the permute phase
    int item_cap;              // item's length
    float4* grid[2];
    unsigned* work;            // the scatter's count of chunks drawn
    unsigned* step;            // device step counter (its parity picks the buffers)
    GridBarrier* bar;
    int wmax, tcmax, ring;     // window nodes and cells of the largest tile, pairs in flight (shared memory)
    int gmin;                  // the fewest threads of a group of the gather (shared memory)
    unsigned* done;            // CTAs finished with the launch (the last one closes the phase clock)
    unsigned long long* phase_ns;   // device time per phase summed over launches, the launch count, a stamp
    uint32_t* status;
};

constexpr int NPHASE = 5;         // tile scan, cell scan, permute, scatter, gather
// Particles of a work item per thread of a CTA: a tile's run in chunks of equal length. Five: the 1,024 of a 16 x 16 tile
// with four a cell, and the tiles a little over it, are one chunk of a 256-thread CTA (at four, half of them were two).
constexpr int PER_THREAD = 5;

// Shared memory of one warp in the scatter: its node window (m, mu, mv arrays of the largest tile's window), the cell
// queue: per cell of the largest tile its particles' range within the chunk, the non-empty cells by descending count,
// count buckets, the queue's head; and the particles on their way.
constexpr int QBUCKETS = 32;               // count buckets (31 particles and more share the last)
constexpr int PAIR_WORDS = 2 * 32 * 10;    // two particles a lane on their way to shared memory in the scatter
__host__ __device__ constexpr int window_words(int wmax) { return (3 * wmax + 3) & ~3; }   // 16-byte aligned
__host__ __device__ constexpr int warp_smem_floats(int wmax, int tcmax, int ring) {   // tcmax a multiple of 64
    return window_words(wmax) + tcmax + tcmax / 2 + QBUCKETS + 4 + ring * PAIR_WORDS;
}

// Shared memory of a group of the gather: two windows of grid nodes, one of node velocities and the next step's tallies.
__host__ __device__ constexpr int group_smem_floats(int wmax, int tcmax) { return ((4 * 2 + 2) * wmax + tcmax + 3) & ~3; }

// Shared memory of a CTA: its warps' in the scatter, or its groups' in the gather, at least one.
__host__ __device__ constexpr int batch_smem_floats(int threads, int wmax, int tcmax, int ring) {
    const int scatter = threads / 32 * warp_smem_floats(wmax, tcmax, ring), gather = group_smem_floats(wmax, tcmax);
    return scatter > gather ? scatter : gather;
}

// One particle's fields as the scatter reads them.
struct Part2 {
    float4 a, c;
    float2 v;
};

// A set's three arrays.
struct Set2 {
    float4* a;   // x y m j
    float4* c;   // c00 c01 c10 c11
    float2* v;   // u v
};

__host__ __device__ __forceinline__ Set2 set_of(float* part, int64_t st) {
    return Set2{reinterpret_cast<float4*>(part), reinterpret_cast<float4*>(part + 4 * st),
                reinterpret_cast<float2*>(part + 8 * st)};
}

// One particle on its way to a lane's place in shared memory; zeros where there is none.
__device__ __forceinline__ void copy_part2(const Set2& to, const Set2& in, int src, bool some) {
    const int n = some ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to.a)),
                 "l"(in.a + src), "r"(n) : "memory");
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to.c)),
                 "l"(in.c + src), "r"(n) : "memory");
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to.v)),
                 "l"(in.v + src), "r"(n >> 1) : "memory");
}

__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }

// bspline_weights with every weight in both halves of a pair: the pairs that paired multiply-adds take.
__device__ __forceinline__ void pair_weights(float f, float2 w[3]) {
    const float2 ff = both(f), half = both(0.5f);
    const float2 a = __ffma2_rn(ff, both(-1.0f), both(1.5f)), c = __fadd2_rn(ff, both(-1.0f)), e = __fadd2_rn(ff, both(-0.5f));
    w[0] = __fmul2_rn(half, __fmul2_rn(a, a));
    w[1] = __ffma2_rn(make_float2(-c.x, -c.y), c, both(0.75f));
    w[2] = __fmul2_rn(half, __fmul2_rn(e, e));
}

// A particle's amounts (Flip.scatter, Flip.java:269-303) added to a cell's sums: m[k] the mass of stencil node k,
// v[k] its momentum pair. With d1 = 1 - f the offset of the stencil's middle node and G the affine matrix times the
// mass with the impulse on its diagonal, a node's momentum over its weight is m v + G d1 + (i - 1) G.x + (j - 1) G.y.
__device__ __forceinline__ void scatter_pairs2(float fx, float fy, const Part2& q, float sp, float (&m)[9],
                                               float2 (&v)[9]) {
    float2 wx[3], wy[3];
    pair_weights(fx, wx);
    pair_weights(fy, wy);
    const float mass = q.a.z;
    const float2 gx = make_float2(fmaf(mass, q.c.x, sp), mass * q.c.z);
    const float2 gy = make_float2(mass * q.c.y, fmaf(mass, q.c.w, sp));
    float2 mid = __fmul2_rn(both(mass), q.v);
    mid = __ffma2_rn(gx, both(1.0f - fx), mid);
    mid = __ffma2_rn(gy, both(1.0f - fy), mid);
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const float2 at = j == 0 ? __ffma2_rn(gy, both(-1.0f), mid) : j == 1 ? mid : __fadd2_rn(mid, gy);
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const float2 val = i == 0 ? __ffma2_rn(gx, both(-1.0f), at) : i == 1 ? at : __fadd2_rn(at, gx);
            const float2 w = __fmul2_rn(wx[i], wy[j]);
            m[3 * j + i] = fmaf(w.x, mass, m[3 * j + i]);
            v[3 * j + i] = __ffma2_rn(val, w, v[3 * j + i]);
        }
    }
}

// The sums of Flip.advectBody (Flip.java:494-545) over a particle's stencil, by rows: sum w g, sum w dx g and
// sum w dy g of the node velocities g, as (u, v) pairs.
template <class Vel>
__device__ __forceinline__ Gathered2 gather_pairs2(float fx, float fy, Vel vel) {
    float2 wx[3], wy[3], wdx[3];
    pair_weights(fx, wx);
    pair_weights(fy, wy);
    const float2 d1x = both(1.0f - fx), d1y = both(1.0f - fy);
    wdx[0] = __fmul2_rn(wx[0], both(-fx));
    wdx[1] = __fmul2_rn(wx[1], d1x);
    wdx[2] = __fmul2_rn(wx[2], both(2.0f - fx));
    float2 mean, bx, by;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const float2 g0 = vel(3 * j), g1 = vel(3 * j + 1), g2 = vel(3 * j + 2);
        const float2 row = __ffma2_rn(g2, wx[2], __ffma2_rn(g1, wx[1], __fmul2_rn(g0, wx[0])));
        const float2 rowx = __ffma2_rn(g2, wdx[2], __ffma2_rn(g1, wdx[1], __fmul2_rn(g0, wdx[0])));
        const float2 wdy = __fmul2_rn(wy[j], j == 0 ? both(-fy) : j == 1 ? d1y : both(2.0f - fy));
        mean = j == 0 ? __fmul2_rn(row, wy[0]) : __ffma2_rn(row, wy[j], mean);
        bx = j == 0 ? __fmul2_rn(rowx, wy[0]) : __ffma2_rn(rowx, wy[j], bx);
        by = j == 0 ? __fmul2_rn(row, wdy) : __ffma2_rn(row, wdy, by);
    }
    return Gathered2{mean.x, mean.y, bx.x, by.x, bx.y, by.y, 0.0f};
}

// impulse_factor with the quotients from reciprocals: 1 / J by one Newton step from the approximate reciprocal (J is
// clamped to [1/10, 10]), m / rho0 corrected by its remainder (Markstein) where `vol`, the reciprocal of rho0, is
// given (0: divided). Both are the quotients that a division rounds: on this GPU the same bits for every float J in
// [1/10, 10], and for 9.7e9 pairs of masses from 2^-60 to 2^60 and densities from 2^-40 to 2^40.
__device__ __forceinline__ float impulse2(const Params2& q, float vol, float m, float j) {
    float jp;
    if (q.tait) {
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(j));
        r = fmaf(r, fmaf(-j, r, 1.0f), r);
        const float r2 = r * r;
        jp = q.bulk * ((r2 * r2) * r2 - j);
    } else {
        jp = q.bulk * (1.0f - j);
    }
    float v = m * vol;
    v = fmaf(fmaf(-v, q.rho0, m), vol, v);
    if (vol == 0.0f) v = __fdiv_rn(m, q.rho0);
    return (4.0f * (q.dt * v)) * jp;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// The next-step cell key and tile entry of a particle at (x, y) in scene sc.
__device__ __forceinline__ void batch_key(const Scene2& sc, float x, float y, int& key, int& tile) {
    int col, row;
    stencil_cell2(x, y, sc.nx, sc.ny, col, row);
    const int local = (row >> sc.lgy) * sc.ntx + (col >> sc.lgx);
    tile = sc.t0 + local;
    key = sc.c0 + local * sc.tc + ((row & (sc.ty - 1)) << sc.lgx) + (col & (sc.tx - 1));
}

// The gather of a step's items by groups of G threads, a chunk each, in parts of PER_THREAD particles a thread.
template <int THREADS, int G>
__device__ __forceinline__ void gather_items(const Batch2& B, int items, const Set2& in, const Set2& out, const float4* g_cur,
                                             float* dyn, Item2 (*rings)[4]) {
    const int gid = threadIdx.x / G, tid = threadIdx.x & (G - 1), lane = threadIdx.x & 31;
    constexpr int groups = THREADS / G;
    auto sync = [&] {
        if constexpr (G == 32) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(gid + 1), "r"(G) : "memory");
    };
    // The items are dealt to the groups like cards. A group takes one at a time, with the next particles, the sources of
    // the ones after and the third item on their way: an item's reads hang one on another (item, sources, particles),
    // each a trip to memory as long as the work on an item.
    Item2* ring = rings[gid];   // the items in hand and the one after
    const int first = blockIdx.x * groups + gid, deal = gridDim.x * groups;
    auto fetch_item = [&](int i) {   // the group's i-th; an empty one past the last. Part of the next group of copies.
        const int64_t k = first + (int64_t)i * deal;
        if (tid < 3)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(&ring[i & 3]) + 16 * tid),
                         "l"(reinterpret_cast<const char*>(B.item + (k < items ? k : 0)) + 16 * tid), "r"(k < items ? 16 : 0)
                         : "memory");
    };
    const int my_items = items > first ? (items - 1 - first) / deal + 1 : 0;
    float4* raw = reinterpret_cast<float4*>(dyn + gid * group_smem_floats(B.wmax, B.tcmax));   // two windows as the scatter left them
    float2* vw = reinterpret_cast<float2*>(raw + 2 * B.wmax);
    int* tally = reinterpret_cast<int*>(vw + B.wmax);          // the next step's cells of the tile
    // a window's nodes, each to be read by the thread that copies it (zeros outside the grid)
    auto window = [&](const Item2& it, int b) {
        const int wx = (1 << (it.lg & 255)) + 2, wn = wx * ((1 << (it.lg >> 8)) + 2), wmul = (65536 + wx - 1) / wx;
        if (it.c0 >= it.c1) return;
#pragma unroll 4
        for (int j = tid; j < wn; j += G) {
            const int row = (j * wmul) >> 16, col = j - row * wx;
            const bool ok = it.x0 + col < it.nx && it.y0 + row < it.ny;
            const float4* from = g_cur + it.g0 + (ok ? (int64_t)row * it.nx + col : 0);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(raw + b * B.wmax + j)), "l"(from), "r"(ok ? 16 : 0)
                         : "memory");
        }
    };
    int bad = 0;
    // a part of an item: PER_THREAD particles a thread, from slot `at` on
    auto sources = [&](const Item2& it, int at, int (&src)[PER_THREAD]) {
#pragma unroll
        for (int i = 0; i < PER_THREAD; i++) {
            const int slot = at + tid + i * G;
            src[i] = slot < it.c1 ? B.perm[slot] : -1;
        }
    };
    auto fetch = [&](const Item2& it, int at, const int (&src)[PER_THREAD], float4 (&q)[PER_THREAD]) {
#pragma unroll
        for (int i = 0; i < PER_THREAD; i++) {
            const int slot = at + tid + i * G;
            if (slot >= it.c1) continue;
            const bool ok = (unsigned)src[i] < (unsigned)B.np;
            bad |= !ok;
            q[i] = __ldg(in.a + (ok ? src[i] : slot));
        }
    };
    // the part after the one at (n, at): of the same item, or the next one's first
    auto step_on = [&](int& n, int& at) {
        at += PER_THREAD * G;
        if (at >= ring[n & 3].c1) at = ring[++n & 3].c0;
    };
    int src[PER_THREAD];
    float4 q[PER_THREAD], qn[PER_THREAD];
#pragma unroll
    for (int i = 0; i < PER_THREAD; i++) q[i] = qn[i] = make_float4(1, 1, 0, 1);
    __syncthreads();
    for (int i = 0; i < 3; i++) fetch_item(i);
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    int n1 = 0, at1 = ring[0].c0;   // the part after the one in hand
    window(ring[0], 0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    sources(ring[0], at1, src);
    fetch(ring[0], at1, src, q);
    step_on(n1, at1);
    sources(ring[n1 & 3], at1, src);
    for (int j = tid; j < B.tcmax; j += G) tally[j] = 0;
    for (int n = 0; n < my_items; n++) {
        const int b = n & 1;
        const Item2 cur = ring[n & 3];
        const int lgx = cur.lg & 255, lgy = cur.lg >> 8, tx = 1 << lgx, ty = 1 << lgy, wx = tx + 2, wn = wx * (ty + 2);
        const int x0 = cur.x0, y0 = cur.y0, nx = cur.nx, ny = cur.ny;
        const Scene2& sc = B.scene[cur.s];
        const Params2 prm = sc.prm;
        const float hi_x = (float)nx - 1.5f, hi_y = (float)ny - 1.5f;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (cur.c0 < cur.c1) {
            for (int j = tid; j < wn; j += G) {
                const float4 gv = raw[b * B.wmax + j];
                const int row = (j * sc.wmul) >> 16;
                vw[j] = grid_velocity2(gv.x, gv.y, gv.z, x0 + j - row * wx, y0 + row, nx, ny, prm);
            }
        }
        sync();
        fetch_item(n + 3);
        window(ring[(n + 1) & 3], b ^ 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        int stayed = 0;
        int at = cur.c0;
        do {   // once for an empty item too, as step_on counts
            // the next part's particles, and the sources of the one after
            fetch(ring[n1 & 3], at1, src, qn);
            step_on(n1, at1);
            sources(ring[n1 & 3], at1, src);
#pragma unroll
            for (int i0 = 0; i0 < PER_THREAD; i0 += 2) {   // two particles' arithmetic together, then their writes
                Advected2 a[2];
                bool in_tile[2];
#pragma unroll
                for (int w = 0; w < 2; w++) {
                    if (i0 + w >= PER_THREAD) break;
                    const float4 p = q[min(i0 + w, PER_THREAD - 1)];
                    int col, row;
                    stencil_cell2(p.x, p.y, nx, ny, col, row);
                    const int lx = col - x0, ly = row - y0;
                    const float fx = __fsub_rn(clampf(p.x, 0.5f, hi_x), (float)col);
                    const float fy = __fsub_rn(clampf(p.y, 0.5f, hi_y), (float)row);
                    in_tile[w] = (unsigned)lx < (unsigned)tx && (unsigned)ly < (unsigned)ty;
                    const float2* from = vw + (in_tile[w] ? ly * wx + lx : 0);
                    a[w] = advect_gathered2(gather_pairs2(fx, fy, [&](int o) { return from[(o / 3) * wx + o % 3]; }), p.x,
                                            p.y, p.w, nx, ny, prm);
                }
#pragma unroll
                for (int w = 0; w < 2; w++) {
                    const int i = i0 + w, slot = at + tid + i * G;
                    if (i >= PER_THREAD || slot >= cur.c1) break;
                    if (!in_tile[w]) {   // left as it is
                        bad = 1;
                        const int from = (unsigned)B.perm[slot] < (unsigned)B.np ? B.perm[slot] : slot;
                        const float2 v = in.v[from];
                        const float4 c = in.c[from];
                        a[w] = Advected2{q[i].x, q[i].y, v.x, v.y, c.x, c.y, c.z, c.w, q[i].w};
                    }
                    out.a[slot] = make_float4(a[w].x, a[w].y, q[i].z, a[w].j);
                    out.c[slot] = make_float4(a[w].c00, a[w].c01, a[w].c10, a[w].c11);
                    out.v[slot] = make_float2(a[w].u, a[w].w);
                    int col, row;
                    stencil_cell2(a[w].x, a[w].y, nx, ny, col, row);
                    const int cx = col - x0, cy = row - y0;
                    if ((unsigned)cx < (unsigned)tx && (unsigned)cy < (unsigned)ty) {
                        const int local = (cy << lgx) + cx;
                        B.key[slot] = cur.cb + local;
                        atomicAdd(&tally[local], 1);
                        stayed++;
                    } else {   // into another tile
                        int key, tile;
                        batch_key(sc, a[w].x, a[w].y, key, tile);
                        B.key[slot] = key;
                        if (key >= 0 && key < B.ncells && tile >= 0 && tile < B.nentries) {
                            atomicAdd(&B.cell_count[key], 1);
                            atomicAdd(&B.tile_count[tile], 1);
                        } else {
                            bad = 1;
                        }
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < PER_THREAD; i++) q[i] = qn[i];
        } while ((at += PER_THREAD * G) < cur.c1);
        stayed = __reduce_add_sync(0xffffffffu, stayed);
        if (lane == 0 && stayed) atomicAdd(&B.tile_count[cur.t], stayed);
        sync();
        for (int j = tid; j < tx * ty; j += G) {
            const int c = tally[j];
            if (c) {
                atomicAdd(&B.cell_count[cur.cb + j], c);
                tally[j] = 0;
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");   // the empty items past the last
    if (bad) set_status(B.status, ST_OOB);
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) k_batch2_step(Batch2 B) {
    extern __shared__ __align__(16) float dyn[];
    __shared__ int scan_smem[33];
    // a step after one whose grid barrier gave up does nothing: the barrier's count is no longer consistent
    __shared__ int dead;
    if (threadIdx.x == 0) dead = (*(volatile uint32_t*)B.status & ST_TIMEOUT) != 0;
    __syncthreads();
    if (dead) return;
    const unsigned par = *B.step & 1u;   // read before the first barrier; CTA 0 advances it after
    const Set2 in = set_of(B.part[par], B.stride), out = set_of(B.part[par ^ 1u], B.stride);
    int* ts_cur = B.tile_start[par];
    const int* ts_prev = B.tile_start[par ^ 1u];
    float4* g_cur = B.grid[par];
    float4* g_next = B.grid[par ^ 1u];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int gwarp = blockIdx.x * nwarps + warp, nwarps_all = gridDim.x * nwarps;
    constexpr int CHUNK = PER_THREAD * THREADS;
    // the phase clock: CTA 0 stamps the start and every barrier, the last CTA to finish the end
    __shared__ unsigned long long stamp;
    if (blockIdx.x == 0 && threadIdx.x == 0) stamp = global_ns();
    auto phase_done = [&](int k) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            const unsigned long long now = global_ns();
            atomicAdd(&B.phase_ns[k], now - stamp);
            stamp = now;
            if (k == NPHASE - 2) B.phase_ns[NPHASE + 1] = now;   // the last phase's start
        }
    };

    // ---- 1. tile scan, per scene: tile counts -> run starts, and the tiles' chunks of <= CHUNK particles
    for (int s = blockIdx.x; s < B.nscenes; s += gridDim.x) {
        const Scene2 sc = B.scene[s];
        const int nt = sc.ntx * sc.nty;
        int carry = 0, ccarry = 0;
        for (int base = 0; base < nt; base += blockDim.x) {
            const int i = base + threadIdx.x;
            const int c = i < nt ? B.tile_count[sc.t0 + i] : 0;
            int total, ctotal;
            const int ex = block_exclusive(c, scan_smem, &total);
            const int cex = block_exclusive((c + CHUNK - 1) / CHUNK, scan_smem, &ctotal);
            if (i < nt) {
                ts_cur[sc.t0 + i] = sc.p0 + carry + ex;
                B.chunk_start[sc.t0 + i] = ccarry + cex;
                B.tile_count[sc.t0 + i] = 0;
            }
            carry += total;
            ccarry += ctotal;
        }
        if (threadIdx.x == 0) {
            ts_cur[sc.t0 + nt] = sc.p0 + carry;
            B.chunk_start[sc.t0 + nt] = ccarry;
            B.scene_chunks[s] = ccarry;
            if (carry != sc.np) set_status(B.status, ST_RANK);
        }
    }
    if (!grid_barrier(B.bar, B.status)) return;
    phase_done(0);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(B.step, 1u);

    // ---- 2. cell scan, a warp per non-empty tile: the tile's cell counts -> cursors (cell starts); CTA 0 first
    // lays out the scenes' chunks one scene after another
    if (blockIdx.x == 0) {
        int carry = 0;
        for (int base = 0; base < B.nscenes; base += blockDim.x) {
            const int i = base + threadIdx.x;
            int total;
            const int ex = block_exclusive(i < B.nscenes ? B.scene_chunks[i] : 0, scan_smem, &total);
            if (i < B.nscenes) B.scene_chunk_start[i] = carry + ex;
            carry += total;
        }
        if (threadIdx.x == 0) B.scene_chunk_start[B.nscenes] = carry;
    }
    // The tiles dealt to the warps like cards (a scene's full tiles lie together, its empty ones too), 32 at a time:
    // a lane reads one tile's run and scene (the reads of the warp's 32 tiles in flight together); then the warp
    // scans the non-empty ones one at a time, every lane on the tile's cells.
    for (int64_t t0 = gwarp; t0 < B.nentries; t0 += 32ll * nwarps_all) {
        const int tl = (int)min(t0 + (int64_t)lane * nwarps_all, (int64_t)B.nentries);
        const int sl = tl < B.nentries ? B.tile_scene[tl] : -1;
        int tsl = 0, tel = 0, tcl = 0, cbl = 0;
        bool live = false;
        if (sl >= 0) {
            tsl = ts_cur[tl];
            tel = ts_cur[tl + 1];
            const Scene2& sc = B.scene[sl];
            if (tel > tsl) {
                if (tsl < sc.p0 || tel > sc.p0 + sc.np) {   // counts that do not add up
                    set_status(B.status, ST_RANK);
                } else {
                    live = true;
                    tcl = sc.tc;                           // 64 .. 512 cells: 2 .. 16 per lane
                    cbl = sc.c0 + (tl - sc.t0) * sc.tc;
                }
            }
        }
        unsigned todo = __ballot_sync(0xffffffffu, live);
        while (todo) {
            const int l = __ffs(todo) - 1;
            todo &= todo - 1;
            const int ts = __shfl_sync(0xffffffffu, tsl, l), te = __shfl_sync(0xffffffffu, tel, l);
            const int tc = __shfl_sync(0xffffffffu, tcl, l);
            const int per = tc >> 5;
            const int cb = __shfl_sync(0xffffffffu, cbl, l) + lane * per;
            int2* count = reinterpret_cast<int2*>(B.cell_count + cb);   // cb is even: keys start at multiples of 64
            int2* cursor = reinterpret_cast<int2*>(B.cursor + cb);
            int2 c[8];
            int sum = 0;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                c[k] = 2 * k < per ? count[k] : make_int2(0, 0);
                sum += c[k].x + c[k].y;
            }
            int run = ts + warp_inclusive(sum) - sum;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                if (2 * k < per) {
                    cursor[k] = make_int2(run, run + c[k].x);
                    count[k] = make_int2(0, 0);
                    run += c[k].x + c[k].y;
                }
            }
            if (lane == 31 && run != te) set_status(B.status, ST_RANK);
        }
    }
    if (!grid_barrier(B.bar, B.status)) return;
    phase_done(1);

    // ---- 3. permute: perm[cursor[key]++] = slot, sixteen slots per thread, one cursor bump per run of equal keys of
    // a warp (the order within a cell is the atomics' order: unspecified, as in the reference's CountingSort); the
    // tiles' chunks entered in the item list; and the other parity's grid cleared over the windows of the tiles
    // the previous step scattered into
    {
        // PK slots a thread (a warp's slots consecutive), the next iteration's keys read while this one's atomics
        // are in flight
        constexpr int PK = 16;
        const int n32 = (B.np + 31) & ~31;
        const int stride = gridDim.x * blockDim.x;
        auto key_at = [&](int i) {
            int v = i < B.np ? B.key[i] : -1;
            if (i < B.np && (v < 0 || v >= B.ncells)) {
                set_status(B.status, ST_OOB);
                v = -1;
            }
            return v;
        };
        int kn[PK];
        const int first = blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll
        for (int u = 0; u < PK; u++) kn[u] = key_at(first + u * stride);
        for (int i0 = first; i0 < n32; i0 += PK * stride) {
            int k[PK];
#pragma unroll
            for (int u = 0; u < PK; u++) {
                k[u] = kn[u];
                kn[u] = key_at(i0 + (PK + u) * stride);
            }
            // the slots of a warp are consecutive, and in the last step's sorted order their keys come in runs:
            // one cursor bump per run of equal keys (a key in two runs of the warp takes two, with distinct ranks)
            int base[PK], rank[PK], leader[PK];
#pragma unroll
            for (int u = 0; u < PK; u++) {   // the atomics of the slots in flight together
                const int prev = __shfl_up_sync(0xffffffffu, k[u], 1);
                const unsigned starts = __ballot_sync(0xffffffffu, lane == 0 || prev != k[u]);
                leader[u] = 31 - __clz(starts & (0xffffffffu >> (31 - lane)));
                const unsigned above = starts & ~(0xffffffffu >> (31 - lane));
                const int end = above ? __ffs(above) - 1 : 32;
                rank[u] = lane - leader[u];
                base[u] = (lane == leader[u] && k[u] >= 0) ? atomicAdd(&B.cursor[k[u]], end - leader[u]) : 0;
            }
#pragma unroll
            for (int u = 0; u < PK; u++) {
                const int d = __shfl_sync(0xffffffffu, base[u], leader[u]) + rank[u];
                if (k[u] >= 0) {
                    if (d >= 0 && d < B.np) B.perm[d] = i0 + u * stride;
                    else set_status(B.status, ST_RANK);
                }
            }
        }
    }
    // The tiles as above, a lane a tile: each lane reads its tile's runs and scene (the reads of a warp's
    // tiles in flight together) and enters the tile's chunks in the item list; then the warp clears, one tile at a
    // time with every lane on it, the windows of the tiles the previous step scattered into, from the lanes' values.
    for (int64_t t0 = gwarp; t0 < B.nentries; t0 += 32ll * nwarps_all) {
        const int t = (int)min(t0 + (int64_t)lane * nwarps_all, (int64_t)B.nentries);
        const int s = t < B.nentries ? B.tile_scene[t] : -1;
        int ts = 0, te = 0;
        bool clear = false;
        if (t < B.nentries) {
            ts = ts_cur[t];
            te = ts_cur[t + 1];
            clear = ts_prev[t + 1] > ts_prev[t];
        }
        int x0 = 0, y0 = 0, wx = 0, wn = 0, nxs = 0, nys = 0, wmul = 0;
        int64_t g0 = 0;
        if (s >= 0) {
            const Scene2& sc = B.scene[s];
            if (te > ts && ts >= sc.p0 && te <= sc.p0 + sc.np) {   // the tile's chunks into the item list
                const int item0 = B.scene_chunk_start[s] + B.chunk_start[t];
                const int nch = (te - ts + CHUNK - 1) / CHUNK;
                const int lt = t - sc.t0, ix = (lt % sc.ntx) * sc.tx, iy = (lt / sc.ntx) * sc.ty;
                Item2 it = {0, 0, t, s, sc.g0 + (int64_t)iy * sc.nx + ix, sc.nx, sc.ny, ix, iy, sc.c0 + lt * sc.tc,
                            sc.lgx | sc.lgy << 8};
                const int per = (te - ts + nch - 1) / nch;
                for (int q = 0; q < nch; q++) {
                    it.c0 = min(te, ts + q * per);
                    it.c1 = min(te, it.c0 + per);
                    if (item0 + q >= 0 && item0 + q < B.item_cap) B.item[item0 + q] = it;
                    else set_status(B.status, ST_OOB);
                }
            }
            const int lt = t - sc.t0;
            x0 = (lt % sc.ntx) * sc.tx;
            y0 = (lt / sc.ntx) * sc.ty;
            wx = sc.tx + 2;
            wn = wx * (sc.ty + 2);
            nxs = sc.nx;
            nys = sc.ny;
            wmul = sc.wmul;
            g0 = sc.g0;
        } else {
            clear = false;
        }
        unsigned todo = __ballot_sync(0xffffffffu, clear);
        while (todo) {
            const int l = __ffs(todo) - 1;
            todo &= todo - 1;
            const int cx0 = __shfl_sync(0xffffffffu, x0, l), cy0 = __shfl_sync(0xffffffffu, y0, l);
            const int cwx = __shfl_sync(0xffffffffu, wx, l), cwn = __shfl_sync(0xffffffffu, wn, l);
            const int cnx = __shfl_sync(0xffffffffu, nxs, l), cny = __shfl_sync(0xffffffffu, nys, l);
            const int cwm = __shfl_sync(0xffffffffu, wmul, l);
            const int64_t cg0 = __shfl_sync(0xffffffffu, g0, l);
            for (int j = lane; j < cwn; j += 32) {
                const int row = (j * cwm) >> 16, gi = cx0 + j - row * cwx, gj = cy0 + row;
                if (gi < cnx && gj < cny) g_next[cg0 + (int64_t)gj * cnx + gi] = make_float4(0, 0, 0, 0);
            }
        }
    }
    if (!grid_barrier(B.bar, B.status)) return;
    phase_done(2);
    const int items = min(B.scene_chunk_start[B.nscenes], B.item_cap);

    // ---- 4. scatter: each warp takes a chunk, scatters it alone through its own node window, and draws the next
    float* ww = dyn + warp * warp_smem_floats(B.wmax, B.tcmax, B.ring);
    // The first chunks are dealt one a CTA, then a second and so on: where there are fewer chunks than warps every SM works
    // on as many. Drawn by the warps as they arrive they went to the SMs whose warps came first, 16 to an SM: a step of 134k
    // particles in 8 scenes scattered in 36 to 40 us and takes 27, of 1.2M in 81 in 59 to 69 and takes 40.
    // A warp's next chunk is drawn while it works on the one before: a chunk is short enough for the counter's and
    // the item's round trips to show.
    auto draw = [&] {
        int k = 0;
        if (lane == 0) k = nwarps_all + (int)atomicAdd(B.work, 1u);
        return k;   // lane 0's
    };
    auto item_of = [&](int k) { return *reinterpret_cast<const int4*>(B.item + min(k, items - 1)); };   // with an item at all
    int knext = warp * (int)gridDim.x + (int)blockIdx.x;
    int4 itnext = items > 0 ? item_of(knext) : make_int4(-1, 0, 0, 0);
    while (knext < items) {
        const int4 it = itnext;   // the chunk: its tile entry, scene and slots
        const int drawn = draw();
        auto turn = [&] {
            knext = __shfl_sync(0xffffffffu, drawn, 0);
            itnext = item_of(knext);
        };
        const int t = it.z, s = it.w, c0 = it.x, c1 = it.y;
        if (t < 0 || t >= B.nentries || s < 0 || s >= B.nscenes) {
            if (lane == 0) set_status(B.status, ST_OOB);
            turn();
            continue;
        }
        const Scene2& sc = B.scene[s];
        const int p0 = sc.p0, p1 = sc.p0 + sc.np;
        if (c0 >= c1 || c0 < p0 || c1 > p1) {
            if (lane == 0) set_status(B.status, ST_OOB);
            turn();
            continue;
        }
        const int lt = t - sc.t0;
        const int tx = sc.tx, ty = sc.ty, nx = sc.nx, ny = sc.ny, tc = sc.tc, lgx = sc.lgx, wmul = sc.wmul;
        const int x0 = (lt % sc.ntx) * tx, y0 = (lt / sc.ntx) * ty;   // the tile's first cell = first node
        const int wx = tx + 2, wn = wx * (ty + 2);
        const Params2 prm = sc.prm;
        ushort2* crange = reinterpret_cast<ushort2*>(ww + window_words(B.wmax));   // per cell: its particles from c0
        unsigned short* order = reinterpret_cast<unsigned short*>(crange + B.tcmax);
        int* bucket = reinterpret_cast<int*>(order + B.tcmax);
        int* head = bucket + QBUCKETS;
        float* ring = reinterpret_cast<float*>(head + 4);
        for (int j = lane; j < 3 * wn; j += 32) ww[j] = 0.0f;
        bucket[lane] = 0;
        __syncwarp();
        // the tile's cells (keys cb + j, j = ly * tx + lx; after the permute cursor[key] is the run's end) clipped
        // to the chunk, and counted into the buckets
        const int cb = sc.c0 + lt * tc;
        if (tc > B.tcmax) {
            if (lane == 0) set_status(B.status, ST_OOB);
            turn();
            continue;
        }
        constexpr int CW = 8;   // cells a lane reads together
        int start = c0;         // of the next 32 cells: cell 0 starts at the tile's run start, <= c0
        for (int j0 = lane; j0 < tc; j0 += 32 * CW) {   // tc a multiple of 64
            int e[CW];
#pragma unroll
            for (int u = 0; u < CW; u++) e[u] = j0 + 32 * u < tc ? B.cursor[cb + j0 + 32 * u] : c1;
#pragma unroll
            for (int u = 0; u < CW; u++) {
                const int below = __shfl_up_sync(0xffffffffu, e[u], 1), b0 = lane ? below : start;
                start = __shfl_sync(0xffffffffu, e[u], 31);
                if (j0 + 32 * u < tc) {
                    const int lo = min(max(b0, c0), c1), hi = min(max(e[u], lo), c1);
                    crange[j0 + 32 * u] = make_ushort2((unsigned short)(lo - c0), (unsigned short)(hi - c0));
                    if (hi > lo) atomicAdd(&bucket[QBUCKETS - 1 - min(hi - lo, QBUCKETS - 1)], 1);
                }
            }
        }
        turn();
        __syncwarp();
        {
            const int v = bucket[lane];
            int x = v;   // exclusive scan over the buckets, largest counts first
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            bucket[lane] = x - v;
            if (lane == 31) *head = x;
        }
        __syncwarp();
        const int ncq = *head;   // non-empty cells
        for (int j = lane; j < tc; j += 32) {
            const ushort2 r = crange[j];
            if (r.y > r.x) order[atomicAdd(&bucket[QBUCKETS - 1 - min((int)r.y - (int)r.x, QBUCKETS - 1)], 1)] = (unsigned short)j;
        }
        __syncwarp();
        // the non-empty cells in synchronous rounds of 32, fullest first: a lane sums its cell's 27 amounts
        // (Flip.scatter, Flip.java:269-303) over the cell's particles in registers; when the round's fullest cell is
        // done, all its lanes add their sums into the window at once. A round's cells have like counts, so few lanes
        // wait, and its lanes hold distinct cells, so at one stencil offset they write distinct nodes. (Dealing
        // cells from a queue, a lane taking the next cell when its own was done, left the window adds at scattered
        // times, divergent in nearly every iteration.)
        // A step takes two particles a lane (their arithmetic is two independent chains). The pairs of all rounds are
        // one stream: a pair is copied to shared memory while the one before is summed, and the sources of the next
        // are read. (A round is a few particles long, so reads that began with it would leave it waiting for them;
        // and a register that a load is on its way to cannot be handed on without waiting for it.)
        int fr = -32, fpairs = 0;   // the stream's place: its round, and the pairs left of it
        int fevery = 1;             // lanes a cell in that round
        int fi = 0, fleft = 0;      // the lane's next slot, and its particles left in the round
        int src0 = 0, src1 = 0, have = 0;
        // lanes a cell in the round from rank r0 on, a power of two: the last round's cells may be few
        auto lg_lanes = [&](int r0) { return r0 < ncq && ncq - r0 < 32 ? 31 - __clz(32 / (ncq - r0)) : 0; };
        auto sources_of_pair = [&] {
            if (fpairs == 0) {
                fr += 32;
                fleft = 0;
                const int lg = lg_lanes(fr), at = fr + (lane >> lg), part = lane & ((1 << lg) - 1);
                fevery = 1 << lg;
                if (at < ncq) {
                    const ushort2 r = crange[order[at]];
                    fi = c0 + r.x + part;
                    fleft = ((int)r.y - (int)r.x - part + fevery - 1) >> lg;
                }
                fpairs = max(1, ((int)__reduce_max_sync(0xffffffffu, (unsigned)fleft) + 1) / 2);
            }
            have = fleft;
            if (fleft > 0) src0 = B.perm[fi];
            if (fleft > 1) src1 = B.perm[fi + fevery];
            fi += 2 * fevery;
            fleft -= 2;
            fpairs--;
        };
        unsigned filled = 0, used = 0;   // pairs, so far
        auto at = [&](unsigned pair, int u) {
            float* q = ring + ((pair & (B.ring - 1)) * 2 + u) * (PAIR_WORDS / 2);
            return Set2{reinterpret_cast<float4*>(q) + lane, reinterpret_cast<float4*>(q + 128) + lane,
                        reinterpret_cast<float2*>(q + 256) + lane};
        };
        bool bad = false;   // a source that is not the scene's, or a particle that is not in its cell
        auto copy = [&] {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int src = u ? src1 : src0;
                const bool some = have > u, ok = some && (unsigned)(src - p0) < (unsigned)(p1 - p0);
                bad |= some && !ok;
                copy_part2(at(filled, u), in, ok ? src : p0, ok);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            filled++;
        };
        sources_of_pair();
        if (B.ring > 1) {
            copy();
            sources_of_pair();
        }
        const float vol = prm.rho0 > 1e-30f && prm.rho0 < 1e30f ? __frcp_rn(prm.rho0) : 0.0f;
        const float hi_x = (float)nx - 1.5f, hi_y = (float)ny - 1.5f;
        float am[9];
        float2 av[9];
        for (int r0 = 0; r0 < ncq; r0 += 32) {
#pragma unroll
            for (int a = 0; a < 9; a++) am[a] = av[a].x = av[a].y = 0.0f;
            const int lg = lg_lanes(r0), part = lane & ((1 << lg) - 1);
            const int cell = r0 + (lane >> lg) < ncq ? order[r0 + (lane >> lg)] : -1;
            const int mine = cell >= 0 ? ((int)crange[cell].y - (int)crange[cell].x - part + (1 << lg) - 1) >> lg : 0;
            const float col = (float)(x0 + (cell & (tx - 1))), row = (float)(y0 + (cell >> lgx));
            const int steps = ((int)__reduce_max_sync(0xffffffffu, (unsigned)mine) + 1) / 2;
            for (int n = 0; n < steps; n++) {
                copy();
                sources_of_pair();
                if (B.ring > 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
                else asm volatile("cp.async.wait_group 0;" ::: "memory");
                Part2 q[2];
                float fx[2], fy[2], sp[2];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const Set2 from = at(used, u);
                    q[u] = Part2{*from.a, *from.c, *from.v};
                    // the offsets from the cell that the sort put the particle in, as stencil2 forms them
                    fx[u] = __fsub_rn(clampf(q[u].a.x, 0.5f, hi_x), col);
                    fy[u] = __fsub_rn(clampf(q[u].a.y, 0.5f, hi_y), row);
                    const bool in_cell = fminf(fx[u], fy[u]) >= 0.5f && fmaxf(fx[u], fy[u]) <= 1.5f;
                    const float m = q[u].a.z;
                    if (in_cell ? !(m > 0.0f) : m != 0.0f) {   // nothing to scatter, whatever its other fields
                        bad |= m > 0.0f;
                        q[u] = Part2{make_float4(0, 0, 0, 1), make_float4(0, 0, 0, 0), make_float2(0, 0)};
                    }
                    sp[u] = q[u].a.z > 0.0f ? impulse2(prm, vol, q[u].a.z, q[u].a.w) : 0.0f;
                }
                used++;
                scatter_pairs2(fx[0], fy[0], q[0], sp[0], am, av);
                scatter_pairs2(fx[1], fy[1], q[1], sp[1], am, av);
            }
            for (int o = 1; o < 1 << lg; o <<= 1) {   // a cell's lanes' sums
#pragma unroll
                for (int a = 0; a < 9; a++) {
                    am[a] += __shfl_xor_sync(0xffffffffu, am[a], o);
                    av[a].x += __shfl_xor_sync(0xffffffffu, av[a].x, o);
                    av[a].y += __shfl_xor_sync(0xffffffffu, av[a].y, o);
                }
            }
            const unsigned fm = __ballot_sync(0xffffffffu, cell >= 0 && part == 0);
            if (cell >= 0 && part == 0) {
                const int wb = (cell >> lgx) * wx + (cell & (tx - 1));
#pragma unroll
                for (int o = 0; o < 9; o++) {
                    const int wi = wb + (o / 3) * wx + o % 3;
                    ww[wi] += am[o];
                    ww[wn + wi] += av[o].x;
                    ww[2 * wn + wi] += av[o].y;
                    __syncwarp(fm);
                }
            }
            __syncwarp();   // this round's window writes before the next round's
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (bad) set_status(B.status, ST_OOB);
        __syncwarp();
        for (int j = lane; j < wn; j += 32) {
            const float a = ww[j], bu = ww[wn + j], bv = ww[2 * wn + j];
            if (a == 0.0f && bu == 0.0f && bv == 0.0f) continue;
            const int row = (j * wmul) >> 16, gi = x0 + j - row * wx, gj = y0 + row;
            if (gi >= nx || gj >= ny) {
                set_status(B.status, ST_OOB);
                continue;
            }
            red_add_v4(&g_cur[sc.g0 + (int64_t)gj * nx + gi], a, bu, bv, 0.0f);
        }
        __syncwarp();   // the window is free for the next chunk
    }
    if (!grid_barrier(B.bar, B.status)) return;
    phase_done(3);
    if (blockIdx.x == 0 && threadIdx.x == 0) *B.work = 0;

    // ---- 5. gather: the tile window's node velocities (the grid update) into shared memory, then the chunk's particles
    // advected, PER_THREAD a thread at a time.
    // The CTA's threads work in groups, a chunk each: the fewest of 32, 64 or 128 that take a chunk of the mean length
    // PER_THREAD a thread, and as many more as leave a group for every chunk, up to the CTA's. A whole CTA a chunk left most
    // of its threads idle where tiles hold few particles: at 58 a tile of 8 x 8 cells, 3.8M particles took 367 us in CTAs of
    // 128 threads, 681 of 256 and 1,394 of 512, and take 157; at some 1,000 a tile of 16 x 16 cells, 16.7M particles took
    // 288 us in CTAs of 256, and take 240. Groups with nothing to do: 134k particles, 10.2 us by the mean length alone, 7.1.
    __shared__ Item2 rings[THREADS / 32][4];
    const int mean = items > 0 ? (B.np + items - 1) / items : 0;
    int G = max(B.gmin, mean <= 32 * PER_THREAD ? 32 : mean <= 64 * PER_THREAD ? 64 : 128);
    while (G < 128 && items <= (int)gridDim.x * (THREADS / (2 * G))) G *= 2;
    if (items <= (int)gridDim.x) G = THREADS;
    if (G == 32) gather_items<THREADS, 32>(B, items, in, out, g_cur, dyn, rings);
    else if (G == 64) gather_items<THREADS, 64>(B, items, in, out, g_cur, dyn, rings);
    else if (THREADS == 128 || G == 128) gather_items<THREADS, 128>(B, items, in, out, g_cur, dyn, rings);
    else gather_items<THREADS, THREADS>(B, items, in, out, g_cur, dyn, rings);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(B.done, 1u) == gridDim.x - 1) {   // the last CTA: the launch's end
            atomicExch(B.done, 0u);
            const unsigned long long start = *(volatile unsigned long long*)&B.phase_ns[NPHASE + 1];
            atomicAdd(&B.phase_ns[NPHASE - 1], global_ns() - start);
            atomicAdd(&B.phase_ns[NPHASE], 1ull);
        }
    }
}

// After a load: the uploaded fields (x, y, u, v, m, one after another in the other set's memory) into the first
// set, J 1 and the affine matrix zero, and every particle's first cell key, tallied (the step's first phase expects
// the counts).
__global__ void __launch_bounds__(256) k_batch2_tally(Batch2 B) {
    const int n32 = (B.np + 31) & ~31;
    const Set2 out = set_of(B.part[0], B.stride);
    const float* in = B.part[1];
    const int64_t st = B.stride;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n32; i += gridDim.x * blockDim.x) {
        int key = -1, tile = -1;
        if (i < B.np) {
            int lo = 0, hi = B.nscenes - 1;   // the scene owning slot i: the last with p0 <= i
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (B.scene[mid].p0 <= i) lo = mid;
                else hi = mid - 1;
            }
            const Scene2 sc = B.scene[lo];
            const float x = in[i], y = in[st + i];
            out.a[i] = make_float4(x, y, in[4 * st + i], 1.0f);
            out.c[i] = make_float4(0, 0, 0, 0);
            out.v[i] = make_float2(in[2 * st + i], in[3 * st + i]);
            batch_key(sc, x, y, key, tile);
            B.key[i] = key;
        }
        warp_tally(B.cell_count, key, key >= 0, B.ncells, B.status);
        warp_tally(B.tile_count, tile, tile >= 0, B.nentries, B.status);
    }
}

// Particle readback: one field of `n` particles from slot p0 on.
__global__ void __launch_bounds__(256) k_batch2_field(Set2 set, float* out, int p0, int n, int field) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* a = reinterpret_cast<const float*>(set.a + p0 + i);
    const float* c = reinterpret_cast<const float*>(set.c + p0 + i);
    const float* v = reinterpret_cast<const float*>(set.v + p0 + i);
    out[i] = field <= PY ? a[field] : field <= PV ? v[field - PU] : field <= PJ ? a[field - PM + 2] : c[field - PC00];
}

// Grid readback: one float of every node of one scene.
__global__ void k_batch2_unpack(const float4* grid, float* out, int64_t nodes, int comp) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nodes) return;
    const float4 g = grid[i];
    out[i] = comp == 0 ? g.x : comp == 1 ? g.y : g.z;
}

const int TILES[][2] = VF_BATCH_TILES;
const int BLOCKS[] = VF_BATCH_BLOCKS;
constexpr int GRAPH_STEPS = 16;   // launches per graph replay

const void* step_kernel(int block) {   // block: one of VF_BATCH_BLOCKS
    return block == 128 ? (const void*)k_batch2_step<128> : block == 256 ? (const void*)k_batch2_step<256>
                                                                         : (const void*)k_batch2_step<512>;
}

// The most dynamic shared memory that the kernel may have. The limit belongs to the kernel, which every batch of its CTA size
// launches, so it is never one batch's own: that of a batch of smaller tiles would stop the launches of one made before it.
int32_t allow_shared(const void* kernel, size_t* most) {
    cudaFuncAttributes a;
    int dev = 0, optin = 0;
    VF_TRY_CUDA(cudaFuncGetAttributes(&a, kernel));
    VF_TRY_CUDA(cudaGetDevice(&dev));
    VF_TRY_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    *most = (size_t)optin - a.sharedSizeBytes;
    VF_TRY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*most));
    return VF_OK;
}

bool tile_ok(int tx, int ty) {
    for (auto& t : TILES)
        if (t[0] == tx && t[1] == ty) return true;
    return false;
}

bool block_ok(int b) {
    for (int x : BLOCKS)
        if (x == b) return true;
    return false;
}

}  // namespace

// ------------------------------------------------------------------ the handle

struct vf_mpm2_batch {
    std::vector<Scene2> scenes;
    uint32_t flags = 0;
    int block = 256, ctas = 0;
    size_t smem = 0;
    int64_t np = 0, stride = 0;
    int ncells = 0, nentries = 0;
    cudaStream_t stream = nullptr;
    DeviceBuffer scene_d, tile_scene, part[2], key, perm, cell_count, cursor, tile_count, tile_start[2], grid[2];
    DeviceBuffer chunk_start, scene_chunks, scene_chunk_start, item;
    DeviceBuffer ctl;      // step counter, two work counters, the done count, the barrier, the phase clock
    DeviceBuffer status;
    DeviceBuffer scratch;  // one scene's readout
    HostWords words;
    int64_t nodes = 0;
    int wmax = 0, tcmax = 0, ring = 1, gmin = 32;
    int64_t steps = 0, launches = 0;
    bool loaded = false;
    bool timed_out = false;   // a grid barrier gave up: no step runs again until the next load
    cudaGraphExec_t graph = nullptr;
};

namespace {

Batch2 view(vf_mpm2_batch* h) {
    Batch2 b;
    b.scene = h->scene_d.as<Scene2>();
    b.nscenes = (int)h->scenes.size();
    b.tile_scene = h->tile_scene.as<int>();
    b.nentries = h->nentries;
    b.part[0] = h->part[0].as<float>();
    b.part[1] = h->part[1].as<float>();
    b.stride = h->stride;
    b.np = (int)h->np;
    b.ncells = h->ncells;
    b.key = h->key.as<int>();
    b.perm = h->perm.as<int>();
    b.cell_count = h->cell_count.as<int>();
    b.cursor = h->cursor.as<int>();
    b.tile_count = h->tile_count.as<int>();
    b.tile_start[0] = h->tile_start[0].as<int>();
    b.tile_start[1] = h->tile_start[1].as<int>();
    b.chunk_start = h->chunk_start.as<int>();
    b.scene_chunks = h->scene_chunks.as<int>();
    b.scene_chunk_start = h->scene_chunk_start.as<int>();
    b.item = h->item.as<Item2>();
    b.item_cap = (int)(h->item.bytes / sizeof(Item2));
    b.grid[0] = h->grid[0].as<float4>();
    b.grid[1] = h->grid[1].as<float4>();
    unsigned* ctl = h->ctl.as<unsigned>();
    b.step = ctl;
    b.work = ctl + 1;
    b.wmax = h->wmax;
    b.ring = h->ring;
    b.gmin = h->gmin;
    b.tcmax = h->tcmax;
    b.done = ctl + 3;
    b.bar = reinterpret_cast<GridBarrier*>(ctl + 4);
    b.phase_ns = reinterpret_cast<unsigned long long*>(ctl + 8);
    b.status = h->status.as<uint32_t>();
    return b;
}

int32_t launch_step(vf_mpm2_batch* h) {
    Batch2 b = view(h);
    void* args[] = {&b};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(h->ctas);
    cfg.blockDim = dim3(h->block);
    cfg.dynamicSmemBytes = h->smem;
    cfg.stream = h->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    VF_TRY_CUDA(cudaLaunchKernelExC(&cfg, step_kernel(h->block), args));
    h->launches++;
    return VF_OK;
}

int32_t batch_status(vf_mpm2_batch* h) {
    VF_TRY_CUDA(cudaMemcpyAsync(h->words.p, h->status.ptr, 4, cudaMemcpyDeviceToHost, h->stream));
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    const uint32_t st = h->words.p[0];
    if (st) {
        VF_TRY_CUDA(cudaMemsetAsync(h->status.ptr, 0, 4, h->stream));
        if (st & ST_TIMEOUT) h->timed_out = true;
        set_error("a batch kernel flagged device status 0x%x%s", st,
                  (st & ST_TIMEOUT) ? " (a grid barrier timed out; load the batch again before stepping it)" : "");
        return (st & ST_TIMEOUT) ? VF_ETIMEOUT : VF_EDEVICE;
    }
    return VF_OK;
}

// The readouts' buffer: the largest scene's particles or nodes, from the first readout on.
int32_t read_scratch(vf_mpm2_batch* h) {
    if (h->scratch.ptr) return VF_OK;
    int64_t most = 0;
    for (const Scene2& q : h->scenes) most = std::max(most, std::max((int64_t)q.nx * q.ny, (int64_t)q.np));
    return h->scratch.alloc((size_t)most * 4);
}

// Captures GRAPH_STEPS step launches into one graph.
int32_t build_graph(vf_mpm2_batch* h) {
    if (h->graph) return VF_OK;
    cudaGraph_t g = nullptr;
    VF_TRY_CUDA(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    int32_t rc = VF_OK;
    for (int k = 0; k < GRAPH_STEPS && rc == VF_OK; k++) rc = launch_step(h);
    h->launches -= GRAPH_STEPS;   // captured, not run
    cudaError_t e = cudaStreamEndCapture(h->stream, &g);
    if (rc) {
        if (g) cudaGraphDestroy(g);
        return rc;
    }
    if (e != cudaSuccess) {
        set_error("capturing the batch step failed: %s", cudaGetErrorString(e));
        return VF_ECUDA;
    }
    e = cudaGraphInstantiate(&h->graph, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) {
        h->graph = nullptr;
        set_error("instantiating the batch step graph failed: %s", cudaGetErrorString(e));
        return VF_ECUDA;
    }
    return VF_OK;
}

int32_t params_of(const vf_scene2& s, uint32_t flags, Params2* p) {
    float w[5];
    for (int k = 0; k < 5; k++) w[k] = bits_to_float(s.params[k]);
    VF_REQUIRE(w[0] > 0 && w[3] >= 0 && w[4] > 0, VF_EINVAL,   // Flip.java:204-207
               "dt > 0, bulk >= 0 and rho0 > 0, got dt %g, bulk %g, rho0 %g", w[0], w[3], w[4]);
    *p = Params2{w[0], w[1], w[2], w[3], w[4], (flags & VF_EOS_TAIT) ? 1 : 0,
                 (int)((flags & VF_WALL_STICKY_MASK) >> VF_WALL_STICKY_SHIFT)};
    return VF_OK;
}

}  // namespace

extern "C" {

int32_t vf_mpm2_batch_create(const vf_scene2* scenes, int32_t nscenes, uint32_t flags, int32_t block,
                             vf_mpm2_batch** out) {
    VF_REQUIRE(out, VF_EINVAL, "out is null");
    *out = nullptr;
    VF_REQUIRE(scenes && nscenes >= 1, VF_EINVAL, "a batch needs scenes, got %d", nscenes);
    VF_REQUIRE(!(flags & (VF_RELAX | VF_TENSION)), VF_EINVAL, "a batch steps plain scenes: no relaxation or tension");
    if (block == 0) block = 256;
    VF_REQUIRE(block_ok(block), VF_EINVAL, "block %d is not one of VF_BATCH_BLOCKS", block);
    std::vector<Scene2> sc((size_t)nscenes);
    int64_t np = 0, cells = 0, nodes = 0, entries = 0;
    int wmax = 0, tcmax = 0;
    for (int s = 0; s < nscenes; s++) {
        const vf_scene2& d = scenes[s];
        VF_REQUIRE(d.nx >= 3 && d.ny >= 3, VF_EINVAL, "scene %d: a grid needs at least three nodes each way, got %d x %d",
                   s, d.nx, d.ny);
        VF_REQUIRE(d.particles >= 1, VF_EINVAL, "scene %d: a step needs particles, got %d", s, d.particles);
        int tx = d.tile_x, ty = d.tile_y;
        if (tx == 0 && ty == 0) tx = ty = 16;
        VF_REQUIRE(tile_ok(tx, ty), VF_EINVAL, "scene %d: tile %d x %d is not one of VF_BATCH_TILES", s, tx, ty);
        Scene2& c = sc[s];
        int32_t rc = params_of(d, flags, &c.prm);
        if (rc) {
            set_error("scene %d: %s", s, last_error());
            return rc;
        }
        c.nx = d.nx;
        c.ny = d.ny;
        c.np = d.particles;
        c.tx = tx;
        c.ty = ty;
        c.ntx = (d.nx - 2 + tx - 1) / tx;
        c.nty = (d.ny - 2 + ty - 1) / ty;
        c.tc = tx * ty;
        c.p0 = (int)np;
        c.g0 = nodes;
        np += d.particles;
        nodes += (int64_t)d.nx * d.ny;
        cells += (int64_t)c.ntx * c.nty * c.tc;
        entries += (int64_t)c.ntx * c.nty + 1;
        while (1 << c.lgx < tx) c.lgx++;
        while (1 << c.lgy < ty) c.lgy++;
        c.wmul = (65536 + tx + 1) / (tx + 2);
        wmax = std::max(wmax, (tx + 2) * (ty + 2));
        tcmax = std::max(tcmax, c.tc);
    }
    VF_REQUIRE(np < (1ll << 31) - 64 && cells < (1ll << 31) && entries < (1ll << 30), VF_EINVAL,
               "a batch holds fewer than 2^31 particles and cell keys, got %lld and %lld", (long long)np,
               (long long)cells);
    // tile entries and cell keys laid out densest scene first, so the work-stealing phases take the
    // heaviest tiles first
    std::vector<int> order((size_t)nscenes);
    for (int s = 0; s < nscenes; s++) order[s] = s;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return (double)sc[a].np / ((double)sc[a].nx * sc[a].ny) > (double)sc[b].np / ((double)sc[b].nx * sc[b].ny);
    });
    std::vector<int> tile_scene((size_t)entries, -1);
    int t0 = 0, c0 = 0;
    for (int s : order) {
        Scene2& c = sc[s];
        c.t0 = t0;
        c.c0 = c0;
        const int nt = c.ntx * c.nty;
        for (int i = 0; i < nt; i++) tile_scene[(size_t)t0 + i] = s;
        t0 += nt + 1;
        c0 += nt * c.tc;
    }
    int32_t rc = require_device();
    if (rc) return rc;
    vf_mpm2_batch* h = new vf_mpm2_batch();
    h->scenes = sc;
    h->flags = flags;
    h->block = block;
    h->np = np;
    h->stride = (np + 63) / 64 * 64;
    h->ncells = (int)cells;
    h->nentries = (int)entries;
    h->nodes = nodes;
    h->wmax = wmax;
    h->tcmax = tcmax;
    auto fail = [&](int32_t code) {
        vf_mpm2_batch_destroy(h);
        return code;
    };
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess) {
        set_error("cudaStreamCreate failed");
        return fail(VF_ECUDA);
    }
    // two pairs of the scatter's particles in flight a lane, unless their memory takes a CTA from the SM
    size_t most = 0;
    if ((rc = allow_shared(step_kernel(block), &most))) return fail(rc);
    int per_sm = 0;
    for (int ring = 1; ring <= 2; ring++) {
        const size_t smem = (size_t)batch_smem_floats(block, wmax, tcmax, ring) * sizeof(float);
        int fit = 0;
        if (smem > most ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, step_kernel(block), block, smem) != cudaSuccess) {
            cudaGetLastError();
            fit = 0;
        }
        if (fit < 1 || fit < per_sm) break;
        per_sm = fit;
        h->ring = ring;
        h->smem = smem;
    }
    if (per_sm < 1) {
        set_error("the batch step does not fit on an SM with %d threads and %zu bytes of shared memory", block,
                  (size_t)batch_smem_floats(block, wmax, tcmax, 1) * sizeof(float));
        return fail(VF_ECUDA);
    }
    h->ctas = per_sm * sm_count();
    while ((size_t)(block / h->gmin) * group_smem_floats(wmax, tcmax) * sizeof(float) > h->smem) h->gmin *= 2;
    const size_t pb = (size_t)h->stride * NF2 * 4;
    if ((rc = h->scene_d.alloc(sc.size() * sizeof(Scene2))) || (rc = h->tile_scene.alloc((size_t)entries * 4)) ||
        (rc = h->part[0].alloc(pb)) || (rc = h->part[1].alloc(pb)) || (rc = h->key.alloc((size_t)np * 4)) ||
        (rc = h->perm.alloc((size_t)np * 4)) || (rc = h->cell_count.alloc((size_t)cells * 4)) ||
        (rc = h->cursor.alloc((size_t)cells * 4)) || (rc = h->tile_count.alloc((size_t)entries * 4)) ||
        (rc = h->tile_start[0].alloc((size_t)entries * 4)) || (rc = h->tile_start[1].alloc((size_t)entries * 4)) ||
        (rc = h->grid[0].alloc((size_t)nodes * 16)) || (rc = h->grid[1].alloc((size_t)nodes * 16)) ||
        (rc = h->chunk_start.alloc((size_t)entries * 4)) || (rc = h->scene_chunks.alloc((size_t)nscenes * 4)) ||
        (rc = h->scene_chunk_start.alloc((size_t)(nscenes + 1) * 4)) ||
        (rc = h->item.alloc((size_t)(np / (PER_THREAD * block) + entries + 1) * sizeof(Item2))) ||
        (rc = h->ctl.alloc(128)) || (rc = h->status.alloc(16)) || (rc = h->words.alloc()))
        return fail(rc);
    if (cudaMemcpyAsync(h->scene_d.ptr, sc.data(), sc.size() * sizeof(Scene2), cudaMemcpyHostToDevice, h->stream) !=
            cudaSuccess ||
        cudaMemcpyAsync(h->tile_scene.ptr, tile_scene.data(), (size_t)entries * 4, cudaMemcpyHostToDevice, h->stream) !=
            cudaSuccess ||
        cudaMemsetAsync(h->status.ptr, 0, h->status.bytes, h->stream) != cudaSuccess ||
        cudaStreamSynchronize(h->stream) != cudaSuccess) {
        set_error("uploading the scene table failed");
        return fail(VF_ECUDA);
    }
    *out = h;
    return VF_OK;
}

int32_t vf_mpm2_batch_load(vf_mpm2_batch* h, const float* x, const float* y, const float* u, const float* v,
                           const float* m) {
    VF_REQUIRE(h && x && y && u && v && m, VF_EINVAL, "null argument");
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    float* base = h->part[1].as<float>();   // on the way to the first set
    const float* src[5] = {x, y, u, v, m};
    for (int f = 0; f < 5; f++)
        VF_TRY_CUDA(cudaMemcpyAsync(base + f * h->stride, src[f], (size_t)h->np * 4, cudaMemcpyHostToDevice, h->stream));
    for (DeviceBuffer* b : {&h->cell_count, &h->tile_count, &h->tile_start[0], &h->tile_start[1], &h->grid[0],
                            &h->grid[1], &h->item, &h->ctl, &h->status})
        VF_TRY_CUDA(cudaMemsetAsync(b->ptr, 0, b->bytes, h->stream));
    Batch2 b = view(h);
    k_batch2_tally<<<std::max(1, std::min(div_up(h->np, 256), sm_count() * 8)), 256, 0, h->stream>>>(b);
    VF_CHECK_LAUNCH();
    h->launches++;
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    h->steps = 0;
    h->loaded = true;
    h->timed_out = false;
    return batch_status(h);
}

int32_t vf_mpm2_batch_advance(vf_mpm2_batch* h, int32_t count) {
    VF_REQUIRE(h, VF_EINVAL, "null handle");
    VF_REQUIRE(count >= 0, VF_EINVAL, "count >= 0, got %d", count);
    VF_REQUIRE(h->loaded, VF_ESTATE, "load the batch before stepping it");
    VF_REQUIRE(!h->timed_out, VF_ESTATE, "a grid barrier of this batch timed out; load it again before stepping it");
    int32_t rc;
    int left = count;
    if (left >= GRAPH_STEPS) {
        if ((rc = build_graph(h))) return rc;
        for (; left >= GRAPH_STEPS; left -= GRAPH_STEPS) {
            VF_TRY_CUDA(cudaGraphLaunch(h->graph, h->stream));
            h->launches += GRAPH_STEPS;
        }
    }
    for (; left > 0; left--)
        if ((rc = launch_step(h))) return rc;
    h->steps += count;
    return VF_OK;
}

int32_t vf_mpm2_batch_set_wait_limit(vf_mpm2_batch* h, int32_t polls) {
    VF_REQUIRE(h, VF_EINVAL, "null handle");
    VF_REQUIRE(polls >= 0, VF_EINVAL, "polls >= 0, got %d", polls);
    const unsigned v = (unsigned)polls;
    unsigned* limit = &reinterpret_cast<GridBarrier*>(h->ctl.as<unsigned>() + 4)->limit;
    VF_TRY_CUDA(cudaMemcpyAsync(limit, &v, 4, cudaMemcpyHostToDevice, h->stream));
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    return VF_OK;
}

int32_t vf_mpm2_batch_finish(vf_mpm2_batch* h) {
    VF_REQUIRE(h, VF_EINVAL, "null handle");
    return batch_status(h);
}

int32_t vf_mpm2_batch_read(vf_mpm2_batch* h, int32_t scene, int32_t field, float* out, int64_t n) {
    VF_REQUIRE(h && out, VF_EINVAL, "null argument");
    VF_REQUIRE(scene >= 0 && scene < (int)h->scenes.size(), VF_EINVAL, "no scene %d", scene);
    VF_REQUIRE(h->loaded, VF_ESTATE, "the batch holds no particles yet");
    const Scene2& sc = h->scenes[scene];
    int32_t rc;
    if (field >= VF2_X && field <= VF2_C11) {
        VF_REQUIRE(n == sc.np, VF_EINVAL, "scene %d holds %d particles, got %lld", scene, sc.np, (long long)n);
        if ((rc = read_scratch(h))) return rc;
        k_batch2_field<<<div_up(n, 256), 256, 0, h->stream>>>(set_of(h->part[h->steps & 1].as<float>(), h->stride),
                                                              h->scratch.as<float>(), sc.p0, (int)n, field);
        VF_CHECK_LAUNCH();
        VF_TRY_CUDA(cudaMemcpyAsync(out, h->scratch.ptr, (size_t)n * 4, cudaMemcpyDeviceToHost, h->stream));
    } else if (field >= VF2_GM && field <= VF2_GMV) {
        const int64_t nodes = (int64_t)sc.nx * sc.ny;
        VF_REQUIRE(n == nodes, VF_EINVAL, "scene %d has %lld nodes, got %lld", scene, (long long)nodes, (long long)n);
        VF_REQUIRE(h->steps > 0, VF_ESTATE, "no step has run");
        if ((rc = read_scratch(h))) return rc;
        const float4* g = h->grid[(h->steps - 1) & 1].as<float4>() + sc.g0;
        k_batch2_unpack<<<div_up(nodes, 256), 256, 0, h->stream>>>(g, h->scratch.as<float>(), nodes, field - VF2_GM);
        VF_CHECK_LAUNCH();
        VF_TRY_CUDA(cudaMemcpyAsync(out, h->scratch.ptr, (size_t)nodes * 4, cudaMemcpyDeviceToHost, h->stream));
    } else {
        set_error("no field %d", field);
        return VF_EINVAL;
    }
    return batch_status(h);
}

int32_t vf_mpm2_batch_config(const vf_mpm2_batch* h, int32_t scene, int32_t* tile_x, int32_t* tile_y, int32_t* block,
                             int32_t* ctas) {
    VF_REQUIRE(h, VF_EINVAL, "null handle");
    VF_REQUIRE(scene >= 0 && scene < (int)h->scenes.size(), VF_EINVAL, "no scene %d", scene);
    if (tile_x) *tile_x = h->scenes[scene].tx;
    if (tile_y) *tile_y = h->scenes[scene].ty;
    if (block) *block = h->block;
    if (ctas) *ctas = h->ctas;
    return VF_OK;
}

int32_t vf_mpm2_batch_phases(vf_mpm2_batch* h, double ms[5], int64_t* launches) {
    VF_REQUIRE(h && ms, VF_EINVAL, "null argument");
    unsigned long long ns[NPHASE + 1];
    unsigned long long* dev = reinterpret_cast<unsigned long long*>(h->ctl.as<unsigned>() + 8);
    VF_TRY_CUDA(cudaMemcpyAsync(ns, dev, sizeof ns, cudaMemcpyDeviceToHost, h->stream));
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    for (int k = 0; k < NPHASE; k++) ms[k] = (double)ns[k] / 1e6;
    if (launches) *launches = (int64_t)ns[NPHASE];
    VF_TRY_CUDA(cudaMemsetAsync(dev, 0, sizeof ns, h->stream));
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    return VF_OK;
}

int64_t vf_mpm2_batch_particles(const vf_mpm2_batch* h) { return h ? h->np : 0; }
int64_t vf_mpm2_batch_steps(const vf_mpm2_batch* h) { return h ? h->steps : 0; }
int64_t vf_mpm2_batch_launches(const vf_mpm2_batch* h) { return h ? h->launches : 0; }
void* vf_mpm2_batch_stream(vf_mpm2_batch* h) { return h ? (void*)h->stream : nullptr; }

void vf_mpm2_batch_destroy(vf_mpm2_batch* h) {
    if (!h) return;
    if (h->stream) cudaStreamSynchronize(h->stream);
    if (h->graph) cudaGraphExecDestroy(h->graph);
    for (DeviceBuffer* b : {&h->scene_d, &h->tile_scene, &h->part[0], &h->part[1], &h->key, &h->perm, &h->cell_count,
                            &h->cursor, &h->tile_count, &h->tile_start[0], &h->tile_start[1], &h->grid[0], &h->grid[1],
                            &h->chunk_start, &h->scene_chunks, &h->scene_chunk_start, &h->item, &h->ctl,
                            &h->status, &h->scratch})
        b->release();
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
}

}  // extern "C"
