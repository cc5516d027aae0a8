// cnn_wgrad.cu -- the network's weight and bias gradients on tcgen05, for sm_100a.
//
// dW[co][ky][kx][ci] = sum over pixels of dy[y][x][co] * in[y + ky - 2][x + kx - 2][ci]: a contraction over pixels, so K
// is the pixels of a row and both operands are read MN-major, straight from the channels-innermost rows that TMA lays
// into shared memory. A tap is then only an offset: a column tap shifts an operand's start by a pixel, a row tap pairs
// two staged rows, and several taps are one MMA whose M or N blocks lie a pixel or a row apart.
//
// Work: tiles of 4 rows x 128 pixels, a contiguous range a CTA, down 128-pixel strips. Operand A is the tile's 4 rows of
// one tensor, operand B the 8 rows (two above, two below) of the other; rows and pixels outside the image are TMA's
// zeros, so every pair of rows is summed once. The gradients stay in tensor memory over all of a CTA's tiles; at the end
// each is added to the fp32 gradient once.
//   layer 2 (32 -> 32 channels): A the layer's input, B dy. Per row r of A and 16 pixels one MMA of M = 4 column taps x 32
//     input channels (blocks one pixel apart) and N = 5 rows of dy x 32 output channels (160 columns): 20 taps. The fifth
//     column tap: per 16 pixels one MMA of M = 4 rows of A x 32 and N = 8 rows of dy x 32 (256 columns), of whose 32
//     row pairs the 20 within two rows of each other are taps.
//   layers 1 and 3 (8 channels on one side): A the 32-channel tensor with the columns' halo, B the 8-channel one; per
//     column tap and 16 pixels one MMA of M = 4 rows x 32 and N = 8 rows x 8 (64 columns), 5 x 64 columns in all. B's
//     pixels are 16 bytes, so a row is taken as a flat run of numbers: four boxes of 32 pixels x 8 rows a tile, where
//     boxes a pixel wide, 1,056 of them, held layer 1 to 148 us.
// Measured at 1024^2 x 4 samples (event-timed): layers 1, 2, 3 took 412, 1182 and 939 us on mma.sync and take 107,
// 166 and 105 here; reading the two tensors once takes 51, 82 and 51 at the measured copy rate. The MMAs bound all three:
// layer 2 keeps the tensor pipe half busy with N = 160 and 256, the thin layers' N = 64 is under what A's 4 KB from
// shared memory cost an MMA.
//
//   warp 0 (one thread): TMA into a ring of stages; warp 1 (one thread): the MMAs; warps 2-5: clear the tensor memory, sum
//   dy over the tile's own rows for the bias gradient while the stage is up, and write the gradients at the end.
// Every wait is bounded, as in the convolutions (cnn_tc.cu).
#include "cnn.cuh"
#include "tc.cuh"

namespace vf {

namespace {

constexpr int WG_THREADS = 192;
constexpr int WG_M = 128;         // pixels of a tile's row
constexpr int WG_R = 4;           // rows of A
constexpr int WG_RB = 8;          // rows of B

// The staged geometry of a layer (its number). A: rows of 64-byte pixels, 64-byte swizzle; 132 pixels from x0 - 2 on. B:
// layer 2, rows of 128 64-byte pixels; else four segments of 8 rows x 32 16-byte pixels.
template <int LAYER>
struct WgLayout {
    static constexpr bool THIN = LAYER != 2;
    static constexpr int PIX = WG_M + 4;
    static constexpr int A_ROW = (PIX * 64 + 511) / 512 * 512;
    static constexpr int B_ROW = THIN ? 512 : WG_M * 64;
    static constexpr int B_SEG = WG_RB * 512;
    static constexpr int A_BYTES = WG_R * A_ROW, B_BYTES = WG_RB * WG_M * (THIN ? 16 : 64);
    static constexpr int STAGE = A_BYTES + B_BYTES;                   // a multiple of 1024
    static constexpr int STAGES = THIN ? 4 : 2;
    static constexpr uint32_t TX = WG_R * PIX * 64 + B_BYTES;
    static constexpr int SMEM = STAGES * STAGE + (2 * STAGES + 1) * 8 + 16 + 1024;
    static constexpr int COLS = THIN ? 5 * 64 : 160 + 256;
};

__device__ __forceinline__ void tma_row(uint32_t dst, const CUtensorMap* map, int px, int row, int b, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
            dst),
        "l"(map), "r"(0), "r"(px), "r"(row), "r"(b), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void tma_seg(uint32_t dst, const CUtensorMap* map, int at, int row, int b, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
        "l"(map), "r"(at), "r"(row), "r"(b), "r"(bar)
        : "memory");
}

// Eight consecutive channels' bf16 values added to sums.
__device__ __forceinline__ void add8(float (&sum)[8], uint4 v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        sum[2 * k] += __uint_as_float(w[k] << 16);
        sum[2 * k + 1] += __uint_as_float(w[k] & 0xffff0000u);
    }
}

}  // namespace

template <int LAYER>
__global__ void __launch_bounds__(WG_THREADS, 1) k_wgrad_tc(WgradArgs a, const __grid_constant__ CUtensorMap map_a,
                                                            const __grid_constant__ CUtensorMap map_b, uint32_t* status) {
    using L = WgLayout<LAYER>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024 - (su32(smem_raw) & 1023)) & 1023);
    const uint32_t ring = su32(smem), bars = ring + L::STAGES * L::STAGE;
    const uint32_t full = bars, empty = bars + 8 * L::STAGES, done = bars + 16 * L::STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::STAGES * L::STAGE + (2 * L::STAGES + 1) * 8);
    __shared__ volatile int abort_cta;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int q = 0; q < L::STAGES; q++) {
            mbar_init(full + 8 * q, 1);
            mbar_init(empty + 8 * q, 1 + 4);   // the MMAs' commit and the four bias warps
        }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        abort_cta = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tmem_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    if (warp >= 2) {
        for (int c = 0; c < L::COLS; c += 16) tmem_zero_cols<16>(tmem + ((uint32_t)((warp & 3) * 32) << 16) + c);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    const int xs_n = (a.W + WG_M - 1) / WG_M, qy_n = (a.H + WG_R - 1) / WG_R;
    const int total = a.B * xs_n * qy_n;
    const int t0 = (int)((int64_t)blockIdx.x * total / gridDim.x);
    const int t1 = (int)((int64_t)(blockIdx.x + 1) * total / gridDim.x);
    int issued = 0;                       // producer: stages whose copies were issued
    if (warp == 0 && lane == 0) {
        for (int t = t0, n = 0; t < t1 && !abort_cta; t++, n++) {
            const int slot = n % L::STAGES;
            if (n >= L::STAGES && !mbar_wait(empty + 8 * slot, (uint32_t)((n / L::STAGES - 1) & 1), &abort_cta, status)) break;
            const int y0 = t % qy_n * WG_R, x0 = t / qy_n % xs_n * WG_M, b = t / (qy_n * xs_n);
            const uint32_t fb = full + 8 * slot, base = ring + slot * L::STAGE;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb), "r"(L::TX) : "memory");
            for (int r = 0; r < WG_R; r++) tma_row(base + r * L::A_ROW, &map_a, x0 - 2, y0 + r, b, fb);
            if constexpr (L::THIN) {
                for (int k = 0; k < WG_M / 32; k++)
                    tma_seg(base + L::A_BYTES + k * L::B_SEG, &map_b, (x0 + 32 * k) * 8, y0 - 2, b, fb);
            } else {
                for (int r = 0; r < WG_RB; r++) tma_row(base + L::A_BYTES + r * L::B_ROW, &map_b, x0, y0 - 2 + r, b, fb);
            }
            issued = n + 1;
        }
    } else if (warp == 1 && lane == 0) {
        for (int t = t0, n = 0; t < t1 && !abort_cta; t++, n++) {
            const int slot = n % L::STAGES;
            if (!mbar_wait(full + 8 * slot, (uint32_t)((n / L::STAGES) & 1), &abort_cta, status)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t A = ring + slot * L::STAGE, B = A + L::A_BYTES;
#pragma unroll
            for (int ks = 0; ks < WG_M / 16; ks++) {
                if constexpr (LAYER == 2) {
#pragma unroll
                    for (int r = 0; r < WG_R; r++)
                        umma_acc(tmem, desc_mn64(A + r * L::A_ROW + ks * 1024, 64), desc_mn64(B + r * L::B_ROW + ks * 1024, L::B_ROW),
                                 idesc_mn(128, 160));
                    umma_acc(tmem + 160, desc_mn64(A + ks * 1024 + 4 * 64, L::A_ROW), desc_mn64(B + ks * 1024, L::B_ROW),
                             idesc_mn(128, 256));
                } else {
#pragma unroll
                    for (int kx = 0; kx < 5; kx++)
                        // layer 3: A is the input, kx - 2 pixels on from B's; layer 1: A is dy, as many back
                        umma_acc(tmem + kx * 64, desc_mn64(A + ks * 1024 + (LAYER == 3 ? kx : 4 - kx) * 64, L::A_ROW),
                                 desc_mn16(B + ks / 2 * L::B_SEG + ks % 2 * 256, L::B_ROW), idesc_mn(128, 64));
                }
            }
            umma_commit(empty + 8 * slot);
        }
        umma_commit(done);   // arrives when every MMA this thread issued has completed
    } else if (warp >= 2) {
        // the bias gradient: warp w sums row w - 2 of the tile's own rows of dy
        float sum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        constexpr bool THIN = LAYER == 3;                 // dy has 8 channels
        const int chunk = THIN ? 0 : lane & 3;            // the lane's 8 channels
        for (int t = t0, n = 0; t < t1 && !abort_cta; t++, n++) {
            const int slot = n % L::STAGES;
            if (!mbar_wait(full + 8 * slot, (uint32_t)((n / L::STAGES) & 1), &abort_cta, status)) break;
            const unsigned char* stage = smem + slot * L::STAGE;
            if constexpr (THIN) {
                const unsigned char* row = stage + L::A_BYTES + warp * L::B_ROW;   // row w - 2, after two rows of halo
#pragma unroll
                for (int k = 0; k < WG_M / 32; k++) add8(sum, *reinterpret_cast<const uint4*>(row + k * L::B_SEG + lane * 16));
            } else {
                const unsigned char* row = LAYER == 1 ? stage + (warp - 2) * L::A_ROW : stage + L::A_BYTES + warp * L::B_ROW;
#pragma unroll
                for (int k = 0; k < WG_M / 8; k++) {
                    const int px = (lane >> 2) + 8 * k + (LAYER == 1 ? 2 : 0);
                    add8(sum, *reinterpret_cast<const uint4*>(row + px * 64 + ((chunk ^ ((px >> 1) & 3)) << 4)));
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + 8 * slot);
        }
#pragma unroll
        for (int k = 0; k < 8; k++)
#pragma unroll
            for (int o = 16; o >= (THIN ? 1 : 4); o >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
        if (lane < (THIN ? 1 : 4)) {
#pragma unroll
            for (int k = 0; k < 8; k++)
                if (chunk * 8 + k < a.cout_real && sum[k] != 0.0f) atomicAdd(&a.db[chunk * 8 + k], sum[k]);
        }
        // the gradients: this warp's 32 lanes of tensor memory, one block of 32 rows of M
        const bool ok = mbar_wait(done, 0, &abort_cta, status);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int q = warp & 3;
        const uint32_t at = tmem + ((uint32_t)(q * 32) << 16);
        // summed over the CTA in shared memory first (the ring is free once `done` has arrived, for the MMAs, and the four
        // warps have met, for their sums of dy), in the parameters' order:
        // the four warps hold parts of the same gradients, and what reaches L2 is then one coalesced reduction a CTA
        // (each warp reducing straight into the gradient cost layer 1 65 us a launch, 592 adds to each of 2,400 numbers)
        float* acc = reinterpret_cast<float*>(smem);
        const int n = a.cout_real * CNN_TAPS * a.cin_real, tid4 = tid - 64;
        auto sync4 = [] { asm volatile("bar.sync 1, 128;" ::: "memory"); };
        sync4();
        for (int k = tid4; k < n; k += 128) acc[k] = 0.0f;
        sync4();
        auto add = [&](int co, int ky, int kx, int ci, uint32_t g) {
            if (co < a.cout_real && ci < a.cin_real) acc[(co * CNN_TAPS + ky * 5 + kx) * a.cin_real + ci] += __uint_as_float(g);
        };
        if constexpr (LAYER == 2) {
            for (int c = 0; c < 160; c += 16) {   // M block q: column tap q; N block c / 32: row tap 4 - c / 32
                uint32_t v[16];
                tmem_ld_nowait<16>(at + c, v);
                tmem_wait_ld();
#pragma unroll
                for (int k = 0; k < 16; k++) add(c % 32 + k, 4 - c / 32, q, lane, v[k]);
            }
        }
        // the parts of one gradient lie in four blocks of M: A's row q with B's rows q .. q + 4. In each of five rounds the
        // four warps are at different row taps, so no two add to one gradient.
        for (int round = 0; round < 5; round++) {
            const int d = (round + q) % 5, r = q + d;
            if constexpr (LAYER == 2) {
                for (int c = r * 32; c < r * 32 + 32; c += 16) {   // column tap 4
                    uint32_t v[16];
                    tmem_ld_nowait<16>(at + 160 + c, v);
                    tmem_wait_ld();
#pragma unroll
                    for (int k = 0; k < 16; k++) add(c % 32 + k, 4 - d, 4, lane, v[k]);
                }
            } else {
                uint32_t u[5][8];
#pragma unroll
                for (int kx = 0; kx < 5; kx++) tmem_ld_nowait<8>(at + kx * 64 + r * 8, u[kx]);
                tmem_wait_ld();
#pragma unroll
                for (int kx = 0; kx < 5; kx++)
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        if (LAYER == 3) add(k, 4 - d, kx, lane, u[kx][k]);
                        else add(lane, d, kx, k, u[kx][k]);
                    }
            }
            sync4();
        }
        if (__all_sync(0xffffffffu, ok && !abort_cta)) {
            for (int k = tid4; k < n; k += 128)
                if (acc[k] != 0.0f) atomicAdd(&a.dw[k], acc[k]);
        }
    }

    // ---- teardown: nothing in flight may outlive the CTA's shared and tensor memory
    __syncwarp();
    if (warp == 0 && lane == 0 && abort_cta) {
        for (int n = max(0, issued - L::STAGES); n < issued; n++)
            for (int spin = 0; spin < TC_SPINS && !mbar_try(full + 8 * (n % L::STAGES), (uint32_t)((n / L::STAGES) & 1)); spin++) {
            }
    }
    if (warp == 1 && lane == 0) {
        for (int spin = 0; spin < TC_SPINS && !mbar_try(done, 0u); spin++) {
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

namespace {

// The layer's number by its channels.
int wgrad_layer(int cin, int cout) { return cin == 8 && cout == 32 ? 1 : cin == 32 && cout == 32 ? 2 : cin == 32 && cout == 8 ? 3 : 0; }

}  // namespace

const void* wgrad_tc_kernel(int cin, int cout) {
    switch (wgrad_layer(cin, cout)) {
        case 1: return (const void*)k_wgrad_tc<1>;
        case 2: return (const void*)k_wgrad_tc<2>;
        case 3: return (const void*)k_wgrad_tc<3>;
        default: return nullptr;
    }
}

size_t wgrad_tc_smem(int cin, int cout) {
    switch (wgrad_layer(cin, cout)) {
        case 1: return WgLayout<1>::SMEM;
        case 2: return WgLayout<2>::SMEM;
        case 3: return WgLayout<3>::SMEM;
        default: return 0;
    }
}

cudaError_t launch_wgrad_tc(int cin, int cout, const WgradArgs& a, uint32_t* status, cudaStream_t s) {
    const int layer = wgrad_layer(cin, cout);
    EncodeTiled enc = tensor_map_encoder();
    if (!layer || !enc) return cudaErrorInvalidValue;
    // a tensor [B][H][W][32] by rows of `pix` pixels in the 64-byte swizzle; one of 8 channels as [B][H][W * 8] by boxes
    // of 8 rows x 256 numbers
    auto wide = [&](CUtensorMap* map, const __nv_bfloat16* p, int pix) {
        const cuuint64_t dims[4] = {32, (cuuint64_t)a.W, (cuuint64_t)a.H, (cuuint64_t)a.B};
        const cuuint64_t strides[3] = {64, (cuuint64_t)a.W * 64, (cuuint64_t)a.H * a.W * 64};
        const cuuint32_t box[4] = {32, (cuuint32_t)pix, 1, 1}, estr[4] = {1, 1, 1, 1};
        return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void*)p, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    auto thin = [&](CUtensorMap* map, const __nv_bfloat16* p) {
        const cuuint64_t dims[3] = {(cuuint64_t)a.W * 8, (cuuint64_t)a.H, (cuuint64_t)a.B};
        const cuuint64_t strides[2] = {(cuuint64_t)a.W * 16, (cuuint64_t)a.H * a.W * 16};
        const cuuint32_t box[3] = {256, WG_RB, 1}, estr[3] = {1, 1, 1};
        return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void*)p, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    CUtensorMap ma, mb;
    const bool ok = layer == 1   ? wide(&ma, a.dy, WG_M + 4) && thin(&mb, a.in)
                    : layer == 2 ? wide(&ma, a.in, WG_M + 4) && wide(&mb, a.dy, WG_M)
                                 : wide(&ma, a.in, WG_M + 4) && thin(&mb, a.dy);
    if (!ok) return cudaErrorInvalidValue;
    const int total = a.B * ((a.W + WG_M - 1) / WG_M) * ((a.H + WG_R - 1) / WG_R);
    void* args[] = {const_cast<WgradArgs*>(&a), &ma, &mb, &status};
    return cudaLaunchKernel(wgrad_tc_kernel(cin, cout), dim3(total < sm_count() ? total : sm_count()), dim3(WG_THREADS), args,
                            wgrad_tc_smem(cin, cout), s);
}

}  // namespace vf
