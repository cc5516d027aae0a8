// cnn_tc.cu -- the network's 32-input-channel 5x5 convolutions on the fifth-generation tensor cores, with
// warp-specialised roles: TMA into a ring of input rows, one thread issuing tcgen05.mma into tensor memory, and
// eight epilogue warps. For sm_100a.
//
// Work: output tiles of 4 rows x 128 pixels. A CTA takes a contiguous range of tiles down 128-pixel strips, so
// consecutive tiles share 4 of their 8 input rows: the ring holds blocks of 4 input rows (4 blocks for 32 input
// channels, 6 for 8), and a tile that continues its predecessor's strip loads one new block.
//   warp 0 (one thread): per block, one TMA tile load per input row (box: the row's channels x 132 or 136 pixels,
//     zero fill outside the image) into a free ring slot, ahead of the MMAs by up to the ring's depth; they
//     complete on the slot's `full` barrier.
//   warp 1: allocates the tensor memory (2 accumulator sets x 4 rows x C columns, C = output channels); one
//     thread waits for the tile's two blocks and a free accumulator set and issues 80 MMAs (M = 128 pixels,
//     K = 16: one tap's 16 channels): per (input row, tap column, channel half), ONE MMA for all the tile's output
//     rows that read that slice, N = their number x C (the weights staged ky-fastest make their B blocks
//     consecutive rows; the accumulators in reverse row order make their D blocks consecutive columns). It
//     commits to the set's `tfull` barrier and to the `empty` barrier of each block no later tile reads.
//   warps 2-9: wait on `tfull`; warp w reads tensor-memory lanes 32 (w % 4) .. + 31 (its pixels) and half of the
//     columns (channels), or with 8 output channels half of the rows, with one wait, clears them (the MMAs only accumulate), writes bias
//     + ReLU to bf16, or fp32, or the gradient times the ReLU mask, and arrives on the set's `tempty` barrier.
// Every wait is bounded: on expiry the CTA sets ST_TIMEOUT and every role leaves its loop; the CTA then waits
// (bounded) for its copies and MMAs in flight before it frees the tensor memory.
//
// Operand layouts (K-major, 32-byte swizzle): an input row is two planes (channels 0-15, 16-31) of 132 pixels x
// 32 bytes; the A operand of output row r, tap (ky, kx) and channel half kc starts at input row r + ky, plane kc,
// pixel kx. The weights: per k step (tap, half), N rows of 32 bytes.
#include "cnn.cuh"
#include "tc.cuh"

namespace vf {

namespace {

constexpr int TC_THREADS = 320;          // warp 0 TMA, warp 1 MMA, warps 2-9 epilogue
constexpr int TC_M = 128;                  // pixels per MMA
constexpr int TC_TR = 4;                   // output rows per tile

// The staged geometry by input channels. 32: an input row is two planes (channels 0-15, 16-31) of 132 pixels x
// 32 bytes in the 32-byte swizzle; a k step is (tap, channel half). 8: one unswizzled plane of 136 pixels x 16
// bytes; a k step is the taps (ky, 2p) and (ky, 2p + 1), p = 0..2 (the sixth tap, kx = 5, has zero weights and
// reads pixel 130 + 127 at most).
#ifndef TC_WIDE
#define TC_WIDE 1   // 32 input channels: A in 64-byte rows (64-byte swizzle), B in 128-byte rows (128-byte swizzle)
#endif

template <int CIN, int NMMA>
struct TcLayout {
    static constexpr bool SWZ = CIN == 32;
    static constexpr bool WIDE = SWZ && TC_WIDE;
    static constexpr int PIX = SWZ ? TC_M + 4 : TC_M + 8;
    static constexpr int PLANES = SWZ && !WIDE ? 2 : 1;
    static constexpr int CH = WIDE ? 32 : SWZ ? 16 : 8;                        // channels per TMA box
    static constexpr int PLANE = WIDE  ? (PIX * 64 + 511) / 512 * 512
                                 : SWZ ? (PIX * 32 + 255) / 256 * 256
                                       : (PIX * 16 + 127) / 128 * 128;
    static constexpr int ROWB = PLANES * PLANE;
    static constexpr int BLOCKB = TC_TR * ROWB;
    static constexpr uint32_t BOX_BYTES = CH * PIX * 2;
    static constexpr int KSTEPS = SWZ ? CNN_TAPS * 2 : 5 * 3;
    static constexpr int B_BYTES = WIDE ? 3 * 5 * NMMA * 128 : KSTEPS * NMMA * 32;   // WIDE: 3 tap pairs
    static constexpr int RING = SWZ ? 4 : 6;           // ring blocks of TC_TR input rows (as many as fit)
    static constexpr int NBAR = 2 * RING + 4 + 1;      // full[RING], empty[RING], tfull[2], tempty[2], done
    static constexpr int SMEM = RING * BLOCKB + B_BYTES + NBAR * 8 + 16 + 1024;
    static constexpr int TCOLS = 2 * TC_TR * NMMA <= 128 ? 128 : 256;   // two accumulator sets
};

// The tile sequence of a CTA: tiles [t0, t1) of (sample, 128-pixel strip, 4-row quad), quads fastest.
struct TileSeq {
    int xs_n, qy_n;
    __device__ void at(int t, int& b, int& x0, int& y0) const {
        const int qy = t % qy_n, r = t / qy_n;
        y0 = qy * TC_TR;
        x0 = (r % xs_n) * TC_M;
        b = r / xs_n;
    }
    // whether tile t continues tile t - 1's strip (so shares its last input block)
    __device__ bool continues(int t, int t0) const { return t > t0 && t % qy_n != 0; }
};

}  // namespace

template <int CIN, int NMMA, int COUT, int MODE>
__global__ void __launch_bounds__(TC_THREADS, 1) k_conv_tc(ConvArgs a, const __grid_constant__ CUtensorMap tmap,
                                                            uint32_t* status) {
    using L = TcLayout<CIN, NMMA>;
    constexpr int K = conv_k(CIN);
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024 - (su32(smem_raw) & 1023)) & 1023);
    constexpr int TC_RING = L::RING;
    const uint32_t ring = su32(smem);                    // TC_RING blocks
    const uint32_t wts = ring + TC_RING * L::BLOCKB;     // the weights (layout below)
    const uint32_t bars = wts + L::B_BYTES;              // mbarriers
    const uint32_t full = bars, empty = bars + 8 * TC_RING, tfull = bars + 16 * TC_RING, tempty = tfull + 16,
                   done = tempty + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + TC_RING * L::BLOCKB + L::B_BYTES + L::NBAR * 8);
    __shared__ volatile int abort_cta;
    __shared__ float bias_s[32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // the weights once (cp.async), ky fastest so that consecutive taps' blocks are consecutive rows; 32 input
    // channels: per (kx, half kc, ky) NMMA swizzled rows of 32 bytes; 8: per (pair p, half h, ky) NMMA rows of
    // 16 bytes (tap ky * 5 + 2p + h, the zero tap 25 where 2p + h = 5); then barriers and tensor memory
    if constexpr (L::WIDE) {
        // per tap pair P = kx / 2: NMMA x 5 rows (ky fastest) of 128 bytes = [tap (ky, 2P) | tap (ky, 2P + 1)],
        // 16-byte chunk q of row r at chunk q ^ (r % 8) (the 128-byte swizzle; pair blocks 1024-byte aligned)
        for (int i = tid; i < NMMA * (K / 8); i += TC_THREADS) {
            const int co = i / (K / 8), c = i % (K / 8), tap = c / 4, g = c % 4, ky = tap / 5, kx = tap % 5;
            const int r = ky * NMMA + co, q = (kx & 1) * 4 + g;
            cp16(wts + (kx / 2) * 5 * NMMA * 128 + r * 128 + ((q ^ (r & 7)) << 4),
                 co < COUT ? a.w + (int64_t)co * K + c * 8 : a.w, co < COUT ? 16u : 0u);
        }
    } else if constexpr (L::SWZ) {
        for (int i = tid; i < NMMA * (K / 8); i += TC_THREADS) {
            const int co = i / (K / 8), c = i % (K / 8), step = c / 2, half = c % 2;
            const int tap = step / 2, kc = step % 2, ky = tap / 5, kx = tap % 5;
            const int blk = (kx * 2 + kc) * 5 + ky;
            cp16(wts + blk * NMMA * 32 + sw32(co, half), co < COUT ? a.w + (int64_t)co * K + c * 8 : a.w,
                 co < COUT ? 16u : 0u);
        }
    } else {
        for (int i = tid; i < 3 * 2 * 5 * NMMA; i += TC_THREADS) {
            const int co = i % NMMA, ky = (i / NMMA) % 5, h = (i / (5 * NMMA)) % 2, pr = i / (10 * NMMA);
            const int kx = 2 * pr + h, tap = kx <= 4 ? ky * 5 + kx : CNN_TAPS;
            cp16(wts + i * 16, co < COUT ? a.w + (int64_t)co * K + tap * 8 : a.w, co < COUT ? 16u : 0u);
        }
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (tid < 32) bias_s[tid] = (MODE != CONV_GRAD_MASK && a.bias && tid < a.bias_n) ? a.bias[tid] : 0.0f;
    if (tid == 0) {
        for (int q = 0; q < TC_RING; q++) {
            mbar_init(full + 8 * q, 1);
            mbar_init(empty + 8 * q, 1);
        }
        for (int q = 0; q < 2; q++) {
            mbar_init(tfull + 8 * q, 1);
            mbar_init(tempty + 8 * q, 8);
        }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        abort_cta = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tmem_slot)),
                     "r"(L::TCOLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    constexpr int CW = NMMA / 2;   // accumulator columns per epilogue warp: warps 2-5 the first half, 6-9 the second
    if (warp >= 2) {   // both accumulator sets start at zero (the MMAs only accumulate)
        const uint32_t base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + ((warp - 2) >> 2) * CW;
        for (int c = 0; c < 2 * TC_TR; c++) tmem_zero_cols<CW>(base + c * NMMA);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    const int H = a.H, W = a.W;
    const TileSeq seq{(W + TC_M - 1) / TC_M, (H + TC_TR - 1) / TC_TR};
    const int total = a.B * seq.xs_n * seq.qy_n;
    const int t0 = (int)((int64_t)blockIdx.x * total / gridDim.x);
    const int t1 = (int)((int64_t)(blockIdx.x + 1) * total / gridDim.x);
    int issued_blocks = 0;   // producer: blocks whose copies were issued

    if (warp == 0 && lane == 0) {
        // ---- producer
        int n = 0;
        for (int t = t0; t < t1 && !abort_cta; t++) {
            int b, x0, y0;
            seq.at(t, b, x0, y0);
            const bool cont = seq.continues(t, t0);
            for (int k = cont ? 1 : 0; k < 2; k++, n++) {
                const int slot = n % TC_RING;
                if (n >= TC_RING && !mbar_wait(empty + 8 * slot, (uint32_t)((n / TC_RING - 1) & 1), &abort_cta, status))
                    break;
                const uint32_t fb = full + 8 * slot;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb),
                             "r"((uint32_t)(TC_TR * L::PLANES) * L::BOX_BYTES)
                             : "memory");
                const int row0 = y0 - 2 + 4 * k;
                for (int r = 0; r < TC_TR; r++)
                    for (int pl = 0; pl < L::PLANES; pl++) {
                        const uint32_t dst = ring + slot * L::BLOCKB + r * L::ROWB + pl * L::PLANE;
                        asm volatile(
                            "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
                            "%3, %4, %5}], [%6];" ::"r"(dst),
                            "l"(&tmap), "r"(pl * L::CH), "r"(x0 - 2), "r"(row0 + r), "r"(b), "r"(fb)
                            : "memory");
                    }
                issued_blocks = n + 1;
            }
        }
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issue
        int fb = 0, i = 0;
        for (int t = t0; t < t1 && !abort_cta; t++, i++) {
            const bool cont = seq.continues(t, t0);
            fb = i == 0 ? 0 : cont ? fb + 1 : fb + 2;
            if (!cont && !mbar_wait(full + 8 * (fb % TC_RING), (uint32_t)((fb / TC_RING) & 1), &abort_cta, status)) break;
            if (!mbar_wait(full + 8 * ((fb + 1) % TC_RING), (uint32_t)(((fb + 1) / TC_RING) & 1), &abort_cta, status))
                break;
            const int set = i & 1;
            if (i >= 2 && !mbar_wait(tempty + 8 * set, (uint32_t)((i / 2 - 1) & 1), &abort_cta, status)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t r0 = ring + (fb % TC_RING) * L::BLOCKB, r1 = ring + ((fb + 1) % TC_RING) * L::BLOCKB;
            const uint32_t acc = tmem + set * TC_TR * NMMA;
            // input row ir and one k-step slice: ONE MMA for every output row orow = ir - ky of the tile that reads
            // the slice: the weights are staged ky-fastest, so the n taps' B blocks are n * NMMA consecutive rows,
            // and the accumulators lie in reverse row order, so the rows' D blocks are consecutive: N = n * NMMA.
            // Descriptors are linear in the start address (16-byte units in the low bits, no carry below 256 KB),
            // so each is a base plus a compile-time offset.
#ifndef TC_ORDER
#define TC_ORDER 1   // 1: consecutive MMAs alternate between the tile's first and last input rows
#endif
            // one MMA of input row ir and k slice (kx or pair p, channel half kc)
            auto mma = [&](int ir, int kx, int kc) {
                constexpr int last = TC_TR - 1;
                const int ky0 = ir - last > 0 ? ir - last : 0, ky1 = ir < 4 ? ir : 4;
                const int n = ky1 - ky0 + 1;
                const uint32_t id = idesc(TC_M, n * NMMA);
                const uint32_t d = acc + (last - (ir - ky0)) * NMMA;
                const uint32_t row = (ir < 4 ? r0 : r1) + (ir & 3) * L::ROWB;
                if constexpr (L::WIDE) {
                    // A: pixel rows of 64 bytes, channel half kc at +32; B: the pair block of kx, its half at
                    // +64 (kx odd), channel half at +32
                    umma_acc(d, desc_sw64(row) + (uint64_t)((kx * 64 + kc * 32) >> 4),
                             desc_sw128(wts) + (uint64_t)(((kx / 2) * 5 * NMMA * 128 + ky0 * NMMA * 128 + (kx & 1) * 64 +
                                                           kc * 32) >> 4),
                             id);
                } else if constexpr (L::SWZ) {
                    umma_acc(d, desc_sw32(row) + (uint64_t)((kc * L::PLANE + kx * 32) >> 4),
                             desc_sw32(wts) + (uint64_t)((((kx * 2 + kc) * 5 + ky0) * NMMA * 32) >> 4), id);
                } else {
                    // A: pixels at 16-byte rows, the pair's second tap one pixel (16 bytes) on; B: per pair p = kx,
                    // half 0 then half 1 (5 * NMMA rows each)
                    umma_acc(d, desc_plain(row, 16, 128) + (uint64_t)((2 * kx * 16) >> 4),
                             desc_plain(wts, 5 * NMMA * 16, 128) + (uint64_t)(((kx * 10 * NMMA + ky0 * NMMA) * 16) >> 4),
                             id);
                }
            };
            constexpr int KX = L::SWZ ? 5 : 3, KC = L::SWZ ? 2 : 1;
            if constexpr (TC_ORDER) {
                // consecutive MMAs on accumulators that overlap as little as possible (rows 0,7,1,6,2,5,3,4)
#pragma unroll
                for (int kx = 0; kx < KX; kx++)
#pragma unroll
                    for (int kc = 0; kc < KC; kc++)
#pragma unroll
                        for (int j = 0; j < TC_TR + 4; j++) mma((j & 1) ? TC_TR + 3 - j / 2 : j / 2, kx, kc);
            } else {
#pragma unroll
                for (int ir = 0; ir < TC_TR + 4; ir++)
#pragma unroll
                    for (int kx = 0; kx < KX; kx++)
#pragma unroll
                        for (int kc = 0; kc < KC; kc++) mma(ir, kx, kc);
            }
            umma_commit(tfull + 8 * set);
            umma_commit(empty + 8 * (fb % TC_RING));   // no later tile reads this tile's first block
            const bool last_of_run = t + 1 == t1 || !seq.continues(t + 1, t0);
            if (last_of_run) umma_commit(empty + 8 * ((fb + 1) % TC_RING));
        }
        umma_commit(done);   // arrives when every MMA this thread issued has completed
    } else if (warp >= 2) {
        // ---- epilogue: warp w reads tensor-memory lanes 32 (w % 4) .. + 31 (its 32 pixels): with 32 output channels the
        //      tile's four rows, columns hh * 16 .. + 15 (hh = 0 for warps 2-5, 1 for 6-9); with 8, rows 2 hh and 2 hh + 1.
        //      A thread's output of a row is 32 bytes, one sector, written at once (two 16-byte stores of half a sector
        //      each kept the L2 at twice the transactions); a ReLU mask is read before the wait for the MMAs, its four
        //      rows in flight together.
        constexpr int ROWS = NMMA == 32 ? TC_TR : TC_TR / 2;
        const int q = warp & 3, hh = (warp - 2) >> 2;
        const int row0 = NMMA == 32 ? 0 : hh * ROWS, c0 = NMMA == 32 ? hh * CW : 0;
        int i = 0;
        for (int t = t0; t < t1 && !abort_cta; t++, i++) {
            const int set = i & 1;
            int b, x0, y0;
            seq.at(t, b, x0, y0);
            const int px = x0 + q * 32 + lane;
            const int64_t pix0 = ((int64_t)b * H + y0 + row0) * W + px;
            uint32_t mk[MODE == CONV_GRAD_MASK ? ROWS : 1][8];
            if constexpr (MODE == CONV_GRAD_MASK) {
#pragma unroll
                for (int r = 0; r < ROWS; r++)
                    if (px < W && y0 + row0 + r < H) ld_global_32(mk[r], a.mask + (pix0 + (int64_t)r * W) * 32 + c0);
            }
            if (!mbar_wait(tfull + 8 * set, (uint32_t)((i / 2) & 1), &abort_cta, status)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // row orow's accumulator lies at reverse position TC_TR - 1 - orow of the set
            const uint32_t base = tmem + ((uint32_t)(q * 32) << 16) + set * TC_TR * NMMA + c0;
            uint32_t v[ROWS][CW];
#pragma unroll
            for (int r = 0; r < ROWS; r++) tmem_ld_nowait<CW>(base + (TC_TR - 1 - row0 - r) * NMMA, v[r]);
            tmem_wait_ld();
#pragma unroll
            for (int r = 0; r < ROWS; r++) tmem_zero_cols<CW>(base + (TC_TR - 1 - row0 - r) * NMMA);
#pragma unroll
            for (int r = 0; r < ROWS; r++) {
                if (px >= W || y0 + row0 + r >= H) continue;
                const int64_t pix = pix0 + (int64_t)r * W;
                uint32_t o[8];
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    if constexpr (NMMA == 32) {
                        float lo = __uint_as_float(v[r][2 * c]), hi = __uint_as_float(v[r][2 * c + 1]);
                        if constexpr (MODE == CONV_RELU) {
                            lo = fmaxf(lo + bias_s[c0 + 2 * c], 0.0f);
                            hi = fmaxf(hi + bias_s[c0 + 2 * c + 1], 0.0f);
                        } else {
                            if (!(__uint_as_float(mk[r][c] << 16) > 0.0f)) lo = 0.0f;
                            if (!(__uint_as_float(mk[r][c] & 0xffff0000u) > 0.0f)) hi = 0.0f;
                        }
                        const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
                        o[c] = *reinterpret_cast<const uint32_t*>(&p);
                    } else {
                        o[c] = __float_as_uint(__uint_as_float(v[r][c]) + bias_s[c]);
                    }
                }
                if constexpr (NMMA == 32) st_global_32(a.out_b + pix * 32 + c0, o);
                else st_global_32(a.out_f + pix * 8, o);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty + 8 * set);
        }
    }

    // ---- teardown: nothing in flight may outlive the CTA's shared and tensor memory
    __syncwarp();
    if (warp == 0 && lane == 0 && abort_cta) {
        // every issued block's copies land before the shared memory goes (bounded)
        for (int n = max(0, issued_blocks - TC_RING); n < issued_blocks; n++)
            for (int spin = 0; spin < TC_SPINS && !mbar_try(full + 8 * (n % TC_RING), (uint32_t)((n / TC_RING) & 1));
                 spin++) {
            }
    }
    if (warp == 1 && lane == 0) {
        for (int spin = 0; spin < TC_SPINS && !mbar_try(done, 0u); spin++) {
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::TCOLS));
}

const void* conv_tc_kernel(int cin, int cout, int mode) {
    if (cin == 32 && cout == 32 && mode == CONV_RELU) return (const void*)k_conv_tc<32, 32, 32, CONV_RELU>;
    if (cin == 32 && cout == 8 && mode == CONV_LINEAR) return (const void*)k_conv_tc<32, 16, 8, CONV_LINEAR>;
    if (cin == 32 && cout == 32 && mode == CONV_GRAD_MASK) return (const void*)k_conv_tc<32, 32, 32, CONV_GRAD_MASK>;
    if (cin == 8 && cout == 32 && mode == CONV_RELU) return (const void*)k_conv_tc<8, 32, 32, CONV_RELU>;
    if (cin == 8 && cout == 32 && mode == CONV_GRAD_MASK) return (const void*)k_conv_tc<8, 32, 32, CONV_GRAD_MASK>;
    return nullptr;
}

size_t conv_tc_smem(int cin, int cout) {
    if (cin == 8) return TcLayout<8, 32>::SMEM;
    return cout == 8 ? TcLayout<32, 16>::SMEM : TcLayout<32, 32>::SMEM;
}

cudaError_t launch_conv_tc(int cin, int cout, int mode, const ConvArgs& a, uint32_t* status, cudaStream_t s) {
    const void* k = conv_tc_kernel(cin, cout, mode);
    EncodeTiled enc = tensor_map_encoder();
    if (!k || !enc) return cudaErrorInvalidValue;
    // the input as a 4-D tensor (channels, x, y, sample); a box is one plane's channels x the staged pixels of a row
    const bool swz = cin == 32, wide = swz && TC_WIDE;
    CUtensorMap map;
    const cuuint64_t px = (cuuint64_t)cin * 2;
    const cuuint64_t dims[4] = {(cuuint64_t)cin, (cuuint64_t)a.W, (cuuint64_t)a.H, (cuuint64_t)a.B};
    const cuuint64_t strides[3] = {px, (cuuint64_t)a.W * px, (cuuint64_t)a.H * a.W * px};
    const cuuint32_t box[4] = {swz ? (cuuint32_t)TcLayout<32, 32>::CH : (cuuint32_t)TcLayout<8, 32>::CH,
                               swz ? (cuuint32_t)TcLayout<32, 32>::PIX : (cuuint32_t)TcLayout<8, 32>::PIX, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void*)a.in, dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE,
            wide ? CU_TENSOR_MAP_SWIZZLE_64B : swz ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    const int total = a.B * ((a.W + TC_M - 1) / TC_M) * ((a.H + TC_TR - 1) / TC_TR);
    const int grid = total < sm_count() ? total : sm_count();   // one CTA per SM (the register file allows no more)
    void* args[] = {const_cast<ConvArgs*>(&a), &map, &status};
    return cudaLaunchKernel(k, dim3(grid), dim3(TC_THREADS), args, conv_tc_smem(cin, cout), s);
}

}  // namespace vf
