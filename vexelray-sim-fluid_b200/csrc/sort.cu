// sort.cu -- kernels of the stable counting sort by cell (see sort.cuh).
#include "sort.cuh"

namespace vf {

// ------------------------------------------------------------------ scans

// Four consecutive counts from i on, zeros past n (the arrays start on 16 bytes and i is a multiple of 4).
__device__ __forceinline__ int4 load4(const int* __restrict__ a, int64_t i, int64_t n) {
    if (i + 4 <= n) return *reinterpret_cast<const int4*>(a + i);
    return make_int4(i < n ? a[i] : 0, i + 1 < n ? a[i + 1] : 0, i + 2 < n ? a[i + 2] : 0, 0);
}

__device__ __forceinline__ void store4(int* __restrict__ a, int64_t i, int64_t n, int4 v) {
    if (i + 4 <= n) {
        *reinterpret_cast<int4*>(a + i) = v;
        return;
    }
    if (i < n) a[i] = v.x;
    if (i + 1 < n) a[i + 1] = v.y;
    if (i + 2 < n) a[i + 2] = v.z;
}

__global__ void __launch_bounds__(1024) k_scan_sums(const int* __restrict__ counts, int64_t n, int64_t range,
                                                    int* __restrict__ sums) {
    __shared__ int smem[33];
    griddep_wait();
    const int64_t lo = blockIdx.x * range, hi = min(lo + range, n);
    int sum = 0;
    for (int64_t i = lo + threadIdx.x * 4; i < hi; i += SCAN_TILE) {
        const int4 c = load4(counts, i, n);
        sum += c.x + c.y + c.z + c.w;
    }
    int total;
    block_exclusive(sum, smem, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) k_scan_apply(int* __restrict__ counts, int* __restrict__ starts, int64_t n,
                                                     int64_t range, const int* __restrict__ sums) {
    __shared__ int smem[33];
    griddep_wait();
    int carry = 0;
    if (gridDim.x > 1) block_exclusive(threadIdx.x < blockIdx.x ? sums[threadIdx.x] : 0, smem, &carry);
    const int64_t lo = blockIdx.x * range, hi = min(lo + range, n);
    for (int64_t base = lo; base < hi; base += SCAN_TILE) {
        const int64_t i = base + threadIdx.x * 4;
        const int4 c = load4(counts, i, n);
        int total;
        const int ex = carry + block_exclusive(c.x + c.y + c.z + c.w, smem, &total);
        store4(starts, i, n, make_int4(ex, ex + c.x, ex + c.x + c.y, ex + c.x + c.y + c.z));
        store4(counts, i, n, make_int4(0, 0, 0, 0));
        carry += total;
    }
    if (hi == n && threadIdx.x == 0) starts[n] = carry;
}

cudaError_t launch_scan(int* counts, int* starts, int64_t n, int* sums, cudaStream_t stream) {
    const int64_t tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    const int64_t range = (tiles + SCAN_BLOCKS - 1) / SCAN_BLOCKS * SCAN_TILE;
    const int blocks = (int)((n + range - 1) / range);
    if (blocks > 1) {
        const cudaError_t e = launch_dependent(k_scan_sums, blocks, 1024, 0, stream, counts, n, range, sums);
        if (e != cudaSuccess) return e;
    }
    return launch_dependent(k_scan_apply, blocks, 1024, 0, stream, counts, starts, n, range, sums);
}

// One block of 32 warps; warp w owns the contiguous segment [w*seg, (w+1)*seg) of the bricks and walks
// it 32 bricks at a time, so every load and store of a warp is one coalesced 128-byte line. Pass 1 sums
// each segment; a block scan gives each warp its offsets; pass 2 scans each 32-brick chunk with
// shuffles, writes the starts, appends the non-empty bricks in order and zeroes the counts.
__global__ void __launch_bounds__(1024) k_brick_scan(int* __restrict__ brick_count, int* __restrict__ brick_start,
                                                     int* __restrict__ active, int* __restrict__ n_active, int nb) {
    griddep_wait();
    __shared__ int smem[33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int seg = (nb + 31) / 32;
    const int lo = warp * seg, hi = min(lo + seg, nb);
    int sum = 0, live = 0;
    for (int base = lo; base < hi; base += 32) {
        const int i = base + lane;
        const int c = i < hi ? brick_count[i] : 0;
        sum += c;
        live += c > 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        live += __shfl_xor_sync(0xffffffffu, live, o);
    }
    // one value per warp into the block scan (lane 0 carries it, the rest add nothing)
    int total, total_live;
    int run = block_exclusive(lane == 0 ? sum : 0, smem, &total);
    int slot = block_exclusive(lane == 0 ? live : 0, smem, &total_live);
    run = __shfl_sync(0xffffffffu, run, 0);
    slot = __shfl_sync(0xffffffffu, slot, 0);
    for (int base = lo; base < hi; base += 32) {
        const int i = base + lane;
        const int c = i < hi ? brick_count[i] : 0;
        const int inc = warp_inclusive(c);
        const unsigned nz = __ballot_sync(0xffffffffu, c > 0);
        if (i < hi) {
            brick_start[i] = run + inc - c;
            if (c > 0) active[slot + __popc(nz & ((1u << lane) - 1u))] = i;
            brick_count[i] = 0;
        }
        run += __shfl_sync(0xffffffffu, inc, 31);
        slot += __popc(nz);
    }
    if (threadIdx.x == 0) {
        brick_start[nb] = total;
        n_active[0] = total_live;
        n_active[2] = 0;   // the tiled gather's item counter for this list
    }
}

__global__ void __launch_bounds__(512) k_cell_scan(int* __restrict__ cell_count, int* __restrict__ cell_start,
                                                   int* __restrict__ cursor, const int* __restrict__ brick_start,
                                                   const int* __restrict__ active,
                                                   const int* __restrict__ n_active, BrickMarks marks) {
    griddep_wait();
    __shared__ int smem[33];
    const int na = *n_active;
    if (marks.mark && blockIdx.x == 0 && threadIdx.x == 0) *marks.count = 0;
    for (int a = blockIdx.x; a < na; a += gridDim.x) {
        const int b = active[a];
        if (marks.mark) {
            // the brick's nodes are 8b .. 8b + 9 an axis
            const int n0[3] = {b % marks.nbx * 8 - marks.reach, b / marks.nbx % marks.nby * 8 - marks.reach,
                               b / (marks.nbx * marks.nby) * 8 - marks.reach};
            const int span = 9 + 2 * marks.reach;
            const int x0 = max(n0[0], 0) / marks.tx, x1 = min((n0[0] + span) / marks.tx, marks.tnx - 1);
            const int y0 = max(n0[1], 0) / marks.ty, y1 = min((n0[1] + span) / marks.ty, marks.tny - 1);
            const int z0 = max(n0[2], 0) / marks.tz, z1 = min((n0[2] + span) / marks.tz, marks.tnz - 1);
            const int wx = x1 - x0 + 1, wy = y1 - y0 + 1, n = wx * wy * (z1 - z0 + 1);
            for (int k = threadIdx.x; k < n; k += blockDim.x)
                marks.mark[((z0 + k / (wx * wy)) * marks.tny + y0 + k / wx % wy) * marks.tnx + x0 + k % wx] = 1;
        }
        const int64_t key = (int64_t)b * 512 + threadIdx.x;
        int c = cell_count[key];
        int total;
        int ex = block_exclusive(c, smem, &total);
        cell_start[key] = brick_start[b] + ex;
        if (cursor) cursor[key] = brick_start[b] + ex;
        cell_count[key] = 0;
    }
}

__global__ void k_permute(const int* __restrict__ key, const int* __restrict__ rank, const int* __restrict__ starts,
                          int* __restrict__ perm, int n, int64_t cells, uint32_t* status) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    griddep_wait();
    if (i >= n) return;
    const int k = key[i];
    if (k < 0 || (int64_t)k >= cells) {
        set_status(status, ST_OOB);
        return;
    }
    int d = starts[k] + rank[i];
    if (d < 0 || d >= n) {
        set_status(status, ST_RANK);
        return;
    }
    perm[d] = i;
}

__global__ void __launch_bounds__(256) k_permute_cursor(const int* __restrict__ key, int* __restrict__ cursor,
                                                       int* __restrict__ perm, int n, int64_t nkeys, uint32_t* status) {
    griddep_wait();
    // PERMUTE_PER slots a thread, PERMUTE_PER x 256 a block; a warp's slots for one u are consecutive, so in the
    // last step's sorted order their keys come in runs: one cursor atomic per run, all of a thread's in flight
    // together before their ranks are read
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int base = blockIdx.x * (256 * PERMUTE_PER) + threadIdx.x;
    int k[PERMUTE_PER], leader[PERMUTE_PER], rank[PERMUTE_PER], got[PERMUTE_PER];
#pragma unroll
    for (int u = 0; u < PERMUTE_PER; u++) {
        const int i = base + u * 256;
        k[u] = i < n ? key[i] : -1;
        if (i < n && (k[u] < 0 || (int64_t)k[u] >= nkeys)) {
            set_status(status, ST_OOB);
            k[u] = -1;
        }
    }
#pragma unroll
    for (int u = 0; u < PERMUTE_PER; u++) {
        const int prev = __shfl_up_sync(all, k[u], 1);
        const unsigned starts = __ballot_sync(all, lane == 0 || prev != k[u]);
        leader[u] = 31 - __clz(starts & (0xffffffffu >> (31 - lane)));   // the run's first lane
        const unsigned above = starts & ~(0xffffffffu >> (31 - lane));    // run starts after this lane
        const int end = above ? __ffs(above) - 1 : 32;
        rank[u] = lane - leader[u];
        got[u] = (lane == leader[u] && k[u] >= 0) ? atomicAdd(&cursor[k[u]], end - leader[u]) : 0;
    }
#pragma unroll
    for (int u = 0; u < PERMUTE_PER; u++) {
        const int d = __shfl_sync(all, got[u], leader[u]) + rank[u];
        const int i = base + u * 256;
        if (k[u] < 0) continue;
        if (d < 0 || d >= n) {
            set_status(status, ST_RANK);
            continue;
        }
        perm[d] = i;
    }
}

// Insertion sort of a short run, ascending.
__device__ __forceinline__ void insertion_sort(int* a, int n) {
    for (int i = 1; i < n; i++) {
        int v = a[i];
        int j = i - 1;
        while (j >= 0 && a[j] > v) {
            a[j + 1] = a[j];
            j--;
        }
        a[j + 1] = v;
    }
}

__global__ void k_fixup_cells(int* __restrict__ perm, const int* __restrict__ starts, int64_t cells) {
    int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cells) return;
    int s0 = starts[c], s1 = starts[c + 1];
    if (s1 - s0 > 1) insertion_sort(perm + s0, s1 - s0);
}

// Runs up to this many particles per brick are fixed up in shared memory.
constexpr int FIXUP_CAP = 12288;

__global__ void __launch_bounds__(512) k_fixup_bricks(int* __restrict__ perm, const int* __restrict__ cell_start,
                                                      const int* __restrict__ brick_start,
                                                      const int* __restrict__ active,
                                                      const int* __restrict__ n_active) {
    extern __shared__ int run[];
    const int na = *n_active;
    for (int a = blockIdx.x; a < na; a += gridDim.x) {
        const int b = active[a];
        const int bs = brick_start[b], be = brick_start[b + 1];
        const int n = be - bs;
        const int64_t key = (int64_t)b * 512 + threadIdx.x;
        int s0 = cell_start[key];
        int s1 = threadIdx.x < 511 ? cell_start[key + 1] : be;
        s0 = max(s0, bs);   // a run always lies inside its brick's; clip anything else
        s1 = min(max(s1, s0), be);
        if (n <= FIXUP_CAP) {
            for (int i = threadIdx.x; i < n; i += blockDim.x) run[i] = perm[bs + i];
            __syncthreads();
            if (s1 - s0 > 1) insertion_sort(run + (s0 - bs), s1 - s0);
            __syncthreads();
            for (int i = threadIdx.x; i < n; i += blockDim.x) perm[bs + i] = run[i];
            __syncthreads();
        } else {
            if (s1 - s0 > 1) insertion_sort(perm + s0, s1 - s0);
        }
    }
}

__global__ void k_dense_starts3(const int* __restrict__ cell_start, const int* __restrict__ brick_start,
                                int* __restrict__ out, int64_t nkeys, int np) {
    int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k > nkeys) return;
    if (k == nkeys) {
        out[k] = np;
        return;
    }
    int64_t b = k >> 9;
    bool live = brick_start[b + 1] > brick_start[b];
    out[k] = live ? cell_start[k] : brick_start[b];
}

__global__ void __launch_bounds__(256) k_gather_stable(const float* __restrict__ in, float* __restrict__ out,
                                                       const int* __restrict__ perm, const int* __restrict__ key,
                                                       const int* __restrict__ starts, int n, int64_t stride, int nf) {
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    griddep_wait();
    if (d >= n) return;
    const int src = perm[d];
    const int k = key[src], s0 = starts[k], s1 = starts[k + 1];
    int to = s0;
    for (int e = s0; e < s1; e++) to += perm[e] < src;
    for (int f = 0; f < nf; f++) out[f * stride + to] = in[f * stride + src];
}

__global__ void k_gather_fields(const float* __restrict__ in, float* __restrict__ out, const int* __restrict__ perm,
                                int n, int64_t stride, int nf) {
    int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= n) return;
    int s = perm[d];
    for (int f = 0; f < nf; f++) out[f * stride + d] = in[f * stride + s];
}

}  // namespace vf

