// k_refiner.cu -- kernels of the learned depth refiner.
//
// The convolutions are implicit GEMMs on the 5th-generation tensor cores:
// bf16 operands in shared memory, FP32 accumulators in tensor memory, issued
// by one thread with tcgen05.mma.  Activations are NHWC bf16, so the 16-byte
// "core matrix" rows the tensor core reads are 8 consecutive channels of one
// pixel.
//
// Forward / input gradient (conv3x3_tc_kernel): M = 128 pixels of one image
// row, K = input channels, N = the output channels of up to three output rows:
// an input row is multiplied once per horizontal tap by the weights of all
// three vertical taps side by side, which adds it to the three output rows it
// belongs to.  Rows are staged as planes of 8-channel chunks whose pixels lie
// so that a horizontal tap is an aligned descriptor offset -- no im2col copy.
// The input gradient is the same kernel run on the output gradient with the
// transposed, tap-flipped weights.
//
// Weight gradient (wgrad_tc_kernel): M = (horizontal tap, output channel), N =
// (vertical tap, input channel), K = pixels, with MN-major operands read from
// the staged NHWC data.  Each block accumulates its share of the pixels in
// tensor memory and writes one partial; a reduction kernel sums the partials in
// a fixed order (deterministic).
#include <cuda_bf16.h>

#include <cstddef>
#include <vector>

#include "tde_common.cuh"
#include "tde_refiner.cuh"
#include "tde_tc.cuh"

namespace tde {
namespace refiner {
namespace {

constexpr int kTileM = 128;             // output pixels per MMA tile
// A staged row of a 128-pixel tile and its two halo pixels: core matrix g (8
// rows of 16 bytes, one channel chunk) holds the pixels g, g + 16, ..., g +
// 112, so the tile is core matrices 0..15 and the tile one or two pixels on
// is 1..16 or 2..17: each horizontal tap reads whole 128-byte lines of shared
// memory, where with the pixels in order it would start 16 or 32 bytes into one.
constexpr int kRowGroups = 18;
constexpr int kPlaneBytes = kRowGroups * 128;  // one 8-channel chunk of a staged row
constexpr uint32_t kSmemPerSM = 228 * 1024;

__host__ __device__ constexpr uint32_t tmem_cols(int n) {
    uint32_t c = 32;
    while (c < (uint32_t)n) c <<= 1;
    return c;
}

__device__ __forceinline__ uint4 ldg16(const bf16 *p) { return __ldg(reinterpret_cast<const uint4 *>(p)); }

__device__ __forceinline__ uint32_t bmax2(uint32_t a, uint32_t b) {
    __nv_bfloat162 x = *reinterpret_cast<__nv_bfloat162 *>(&a), y = *reinterpret_cast<__nv_bfloat162 *>(&b);
    __nv_bfloat162 r = __hmax2(x, y);
    return *reinterpret_cast<uint32_t *>(&r);
}
__device__ __forceinline__ uint4 bmax4(uint4 a, uint4 b) {
    return make_uint4(bmax2(a.x, b.x), bmax2(a.y, b.y), bmax2(a.z, b.z), bmax2(a.w, b.w));
}

__device__ __forceinline__ float bf_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf_hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
__device__ __forceinline__ void unpack8(uint4 q, float *f) {
    f[0] = bf_lo(q.x); f[1] = bf_hi(q.x); f[2] = bf_lo(q.y); f[3] = bf_hi(q.y);
    f[4] = bf_lo(q.z); f[5] = bf_hi(q.z); f[6] = bf_lo(q.w); f[7] = bf_hi(q.w);
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 r = __floats2bfloat162_rn(a, b);  // .x = a (low half)
    return *reinterpret_cast<uint32_t *>(&r);
}
__device__ __forceinline__ uint4 pack8(const float *f) {
    return make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
}

// ---------------------------------------------------------------------------
// Forward / input-gradient convolution: a warp-specialised pipeline.
//
// A block owns strips of consecutive output rows of one 128-pixel column
// tile.  Its warps have fixed roles, connected by mbarriers (no block-wide
// barrier in the steady state):
//   warps 0-3 (producers): input row j goes to warp j & 3, which loads
//     the halo row (pixels x0-1 .. x0+128, every 8-channel chunk, as planes)
//     into ring slot j % S once the tensor core has released that slot, and
//     marks it full -- four rows in flight, one per warp;
//   warp 4 (MMA issuer): input row i of a strip belongs to output
//     rows i - 2, i - 1 and i (vertical taps 2, 1, 0).  Their accumulators lie
//     side by side in tensor memory and the three taps' weights side by side
//     in shared memory, so each of the row's 3 x CC/2 MMAs (horizontal tap,
//     K = 16 channels) has N = 3 cout: a third of the MMAs of one per tap to
//     issue (some 70 cycles each, whatever they read, which was most of a row's
//     time), and the pixels are read from shared memory once instead of three
//     times.  An output row still sums its taps in the order (0,0), (0,1), ...
//     (2,2), so its bits are those of one MMA per tap.  The accumulators form a ring of NA rows; the MMAs of
//     a row whose outputs wrap around the ring are split there, and the first
//     MMA of an output row, which overwrites its accumulator, is issued apart;
//   warps 5-8, or 5-12 taking rows in turn (epilogue): a TMEM lane quarter
//     each, one pixel per thread -- wait for the accumulator, read it
//     (tcgen05.ld), release it, apply bias, ReLU, mask or the fused head, store
//     bf16 NHWC.
// Input rows are loaded once per strip; loads, MMAs and epilogues of
// different rows overlap.  At batch 16 of 640x480 the forward pass took 1138 us
// with one MMA per tap, index arithmetic per copied piece and 16-byte stores a
// pixel apart, and takes 792 us (batch 1: 156 and 135 us); what is left per row is
// the issuer's chain of waits and issues (about 1000 cycles a row and block) and,
// at the full resolution, memory (c2 moves 353 MB in 94 us).  Every wait is bounded: on a timeout the block
// raises A.err, all roles leave their loops, the issuer waits (bounded) for
// its MMAs in flight, and the tensor memory is freed.
// ---------------------------------------------------------------------------
constexpr int kConvProdWarps = 4, kConvMmaWarp = kConvProdWarps;
// Epilogue warps follow: one set of four where the output is pooled or the
// input upsampled (the layer's other roles bound it; c4, c6 and c9 took 71, 64
// and 86 us with two sets, 66, 57 and 59 with one, at batch 16 of 640x480), two
// elsewhere (the input gradients of c2 and c10: 134 and 106 us with one, 106
// and 82 with two).
constexpr int conv_epi_sets(int mode, bool pool) { return mode == SRC_UP || pool ? 1 : 2; }
__host__ __device__ constexpr int conv_threads(int sets) { return 32 * (kConvProdWarps + 1 + 4 * sets); }
constexpr int kConvMaxPerSM = 2;  // resident blocks (three or four: the same times)
constexpr int kConvMinAcc = 4;    // accumulator rows: three being summed, one being drained
constexpr int kConvMaxAcc = 8;
constexpr int kConvMaxSlots = 8;  // input-row ring
// No fewer slots than producer warps: a warp's row j - 4 was issued once row
// j - 4 - S had been consumed, so the slot of row j is at most one phase behind
// when it is waited for (a parity wait cannot tell more).
constexpr int kConvMinSlots = kConvProdWarps;
// Ring of the source rows that two input rows share (upsampled sources).
__host__ __device__ constexpr int shared_slots(int slots) { return slots / 2 + 1; }
constexpr int kConvMaxShared = shared_slots(kConvMaxSlots);
constexpr int kStripRowsOneWave = 8;   // longest strip of a one-wave launch
constexpr int kStripRowsBalanced = 16;  // strip length when the work is larger
constexpr uint64_t kConvWaitNs = 2000000000ull;

struct ConvPipe {
    uint64_t full[kConvMaxSlots], empty[kConvMaxSlots];
    uint64_t sfull[kConvMaxShared], sempty[kConvMaxShared];
    uint64_t acc_full[kConvMaxAcc], acc_empty[kConvMaxAcc];
    uint64_t drain;
    uint32_t tmem;
    int abort;
};

// Bounded wait on an mbarrier phase; false when the block aborted (here or
// in another role).
__device__ __forceinline__ bool pipe_wait(uint64_t *bar, uint32_t parity, volatile int *abort, int *err,
                                          uint64_t limit_ns = kConvWaitNs) {
    if (tc::mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = tc::globaltimer_ns();
    // sleeping waits (up to 20 us each) leave the issue slots to the working warps
    while (!tc::mbar_try_wait_sleep(bar, parity, 20000u)) {
        if (*abort) return false;
        if (tc::globaltimer_ns() - t0 > limit_ns) {
            *abort = 1;
            atomicExch(err, 1);
            return false;
        }
    }
    return true;
}
// The bounded wait on its own: one lane waits for a phase that nothing
// completes; after limit_ns it gives up, raises the error flag and the block
// returns normally.  out[0] = the flag, out[1] = nanoseconds waited.
__global__ void wait_selftest_kernel(uint64_t limit_ns, unsigned long long *out) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ int abort_flag;
    __shared__ int err;
    if (threadIdx.x == 0) {
        tc::mbar_init(&bar, 1);
        abort_flag = 0;
        err = 0;
        const uint64_t t0 = tc::globaltimer_ns();
        const bool ok = pipe_wait(&bar, 0u, &abort_flag, &err, limit_ns);
        out[0] = ok ? 0ull : (unsigned long long)err;
        out[1] = tc::globaltimer_ns() - t0;
    }
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}

// Strip `item` of the block's sequence: image, column start, rows [y0, y1).
struct Strip { int img, x0, y0, y1; };
__device__ __forceinline__ Strip strip_of(const ConvArgs &A, int item, int rows_per_item) {
    const int tiles_x = (A.w + kTileM - 1) / kTileM;
    const int chunks = (A.h + rows_per_item - 1) / rows_per_item;
    Strip s;
    s.x0 = (item % tiles_x) * kTileM;
    s.y0 = ((item / tiles_x) % chunks) * rows_per_item;
    s.img = item / (tiles_x * chunks);
    s.y1 = min(A.h, s.y0 + rows_per_item);
    return s;
}

// Copies of CP = 2 or 4 channel chunks (PXE channels a source pixel) of one
// staged row into its planes, read directly or through the nearest 2x
// upsample of a row half as wide; 16-byte cp.async, zeros past the row's ends.
// Eight lanes write the eight pixels of a core matrix (one 128-byte line), the
// four such sets of a warp two or four chunks of one or two pixels (whole
// 32-byte sectors).  Unrolled, every address is a lane's base plus a constant:
// a piece costs a compare, the copy and its zero store (predicated off), where
// index arithmetic per piece made this the longest part of a row.
template <int CP, bool UPS, int PXE>
__device__ __forceinline__ void warp_copy_chunks(const bf16 *row, int x_start, int w, uint32_t dst, int lane) {
    const int k = lane & 7, l3 = lane >> 3;
    const int c = CP == 4 ? l3 : l3 & 1, gl = CP == 4 ? 0 : l3 >> 1;
    const int x = x_start + gl + 16 * k;  // this lane's first pixel; x_start is one left of a multiple of 128
    const int lim = w - x;
    const bf16 *src = row + (UPS ? (x_start + 1) / 2 + 8 * k + ((gl - 1) >> 1) : x) * PXE + 8 * c;
    dst += (uint32_t)(k * 16 + c * kPlaneBytes + gl * 128);
#pragma unroll
    for (int it = 0; it < kRowGroups * CP / 4; ++it) {
        const int g = CP == 4 ? it : 2 * it;
        const int off = UPS ? (CP == 4 ? (it + 1) >> 1 : it) : g;
        if (g < lim && (it > 0 || x >= 0))
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + g * 128), "l"(src + off * PXE) : "memory");
        else
            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(dst + g * 128), "r"(0) : "memory");
    }
}
template <int CC, bool UPS>
__device__ __forceinline__ void warp_copy_source(const bf16 *row, int x_start, int w, uint32_t dst, int lane) {
#pragma unroll
    for (int c = 0; c + 4 <= CC; c += 4)
        warp_copy_chunks<4, UPS, 8 * CC>(row + 8 * c, x_start, w, dst + c * kPlaneBytes, lane);
    if constexpr (CC % 4 != 0)
        warp_copy_chunks<2, UPS, 8 * CC>(row + 8 * (CC - 2), x_start, w, dst + (CC - 2) * kPlaneBytes, lane);
}
// One warp starts the copies of CC chunks of a row (halo pixels x0-1 .. x0+128)
// into the planes at dst, or zeros when the row lies outside the image (null).
template <int CC, bool UPS>
__device__ __forceinline__ void warp_copy_row(const bf16 *row, int x0, int w, uint32_t dst, int lane) {
    if (row) {
        warp_copy_source<CC, UPS>(row, x0 - 1, w, dst, lane);
    } else {
        for (int i = lane; i < CC * kPlaneBytes / 16; i += 32)
            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(dst + i * 16), "r"(0) : "memory");
    }
}

// Pixel of the tile that TMEM lane m holds: row m of a staged tile is element
// m & 7 of core matrix m >> 3.
__device__ __forceinline__ int tile_pixel(int m) { return (m >> 3) + 16 * (m & 7); }

// Bias, ReLU and mask of 16 channels of one pixel, rounded to bf16.
__device__ __forceinline__ void finish16(const ConvArgs &A, float (&v)[16], const float *bias, uint4 m0, uint4 m1, uint4 &q0,
                                         uint4 &q1) {
    if (A.bias) {
#pragma unroll
        for (int k = 0; k < 16; k += 4) {
            const float4 b = *reinterpret_cast<const float4 *>(bias + k);
            v[k] += b.x; v[k + 1] += b.y; v[k + 2] += b.z; v[k + 3] += b.w;
        }
    }
    if (A.relu) {
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = v[k] > 0.f ? v[k] : 0.f;
    }
    if (A.mask) {
        float mk[16];
        unpack8(m0, mk);
        unpack8(m1, mk + 8);
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = mk[k] > 0.f ? v[k] : 0.f;
    }
    q0 = pack8(v);
    q1 = pack8(v + 8);
}
__device__ __forceinline__ void store16(bf16 *o, uint4 q0, uint4 q1) {
    reinterpret_cast<uint4 *>(o)[0] = q0;
    reinterpret_cast<uint4 *>(o)[1] = q1;
}
__device__ __forceinline__ uint4 shfl_xor4(uint4 p, int m) {
    return make_uint4(__shfl_xor_sync(0xffffffffu, p.x, m), __shfl_xor_sync(0xffffffffu, p.y, m),
                      __shfl_xor_sync(0xffffffffu, p.z, m), __shfl_xor_sync(0xffffffffu, p.w, m));
}

// Ring position of an output row's accumulator.
struct AccAt {
    int a;
    uint32_t phase;
    __device__ __forceinline__ void next(int NA) {
        if (++a == NA) {
            a = 0;
            phase ^= 1u;
        }
    }
};

// The epilogue role of one warp: a TMEM lane quarter of every output row, or of every
// other one -- with a pooled output every other pair of rows, whose 2x2
// maximum (the row pair in registers, the pixel pair across lanes 8 apart) goes
// to pool_out, the same bits as a max pool of the stored rows.  With two
// sets of four warps one row's tensor-memory and global latencies overlap the
// next one's.  What does not depend on the sums (the head's input depth, the
// ReLU mask) is fetched before waiting for them, and the accumulator is released
// as soon as it is in registers.
//
// A lane holds one pixel's channels, and its 16-byte stores would write a half
// of a sector at a time, a pixel's stride apart.  The channels of four
// neighbouring pixels are a run of 128 bytes or more: the warp collects its
// eight runs in shared memory and stores them with consecutive lanes.  Of the
// 16-byte units of a run (4 COUT / 8, a multiple of 8), unit u lies at u ^ k, k
// the run, so that the eight lanes of one core matrix write to different banks.
// Where a layer's shared memory has no room for it (conv_plan), each pixel is
// stored directly.
// Shared memory for it: 32 pixels of one row, or of two, per epilogue warp.
__host__ __device__ constexpr size_t conv_stage_bytes(int cout, bool pool) {
    return (size_t)32 * cout * 2 * (pool ? 2 : 1);
}
// The first plane's channels where the output may be two planes (48 channels: the
// input gradient of the full-resolution layer with two sources), else 0.  A constant:
// with the split as a factor of the addresses that convolution took 180 us of 131;
// the layers of 80 and 112 channels, short of registers, lost with it what their
// planes gained.
__host__ __device__ constexpr int conv_split(int cout) { return cout == 48 ? 32 : 0; }
// Channel c of pixel p of a run of pixels that begins at `first` in the first plane
// and at `second` in the second.
template <int COUT>
__device__ __forceinline__ bf16 *split_at(bf16 *first, bf16 *second, int p, int c) {
    constexpr int K = conv_split(COUT);
    return c < K ? first + p * K + c : second + p * (COUT - K) + (c - K);
}
template <int COUT, bool POOL, int SETS>
__device__ __forceinline__ void conv_epilogue(const ConvArgs &A, ConvPipe &pp, const float *s_bias, const float *s_head,
                                           unsigned char *stage, int rows_per_item, int items, int NA, int warp, int lane) {
    constexpr int ROWS = POOL ? 2 : 1;
    constexpr int KS = POOL ? 0 : conv_split(COUT);
    bf16 *const plane2 = A.out + (size_t)A.n * A.h * A.w * KS;
    const bool staged = stage != nullptr;
    constexpr int UNITS = 4 * COUT / 8;  // 16-byte units of one run
    const uint32_t sbase = tc::smem_u32(stage) + (uint32_t)((warp - kConvMmaWarp - 1) * ROWS * 32 * COUT * 2);
    const int run = lane & 7, rpx = lane >> 3;
    // a warp reads the tensor-memory lanes of its number modulo 4; any four
    // consecutive warps cover a row
    const uint32_t set = (uint32_t)(warp - kConvMmaWarp - 1) >> 2, quarter = (uint32_t)warp & 3u;
    const uint32_t tmem = pp.tmem + (quarter << 21);  // lane 32 * quarter in bits 16..
    const int px = tile_pixel(quarter * 32 + lane);
    volatile int *abort = &pp.abort;
    AccAt at{0, 0u};
    uint32_t turn = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
        const Strip st = strip_of(A, item, rows_per_item);
        const int x = st.x0 + px;
        const bool valid = x < A.w;
        for (int y = st.y0; y < st.y1; y += ROWS, ++turn) {
            AccAt row[ROWS];
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                row[r] = at;
                at.next(NA);
            }
            if (SETS > 1 && turn % SETS != set) continue;
            const size_t pix = ((size_t)st.img * A.h + y) * A.w + (valid ? x : 0);
            float din = 0.f;
            if (COUT == 16 && !POOL && A.head_w && valid) din = __ldg(A.depth_in + pix);
            uint4 m0[ROWS], m1[ROWS];
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                m0[r] = m1[r] = make_uint4(0u, 0u, 0u, 0u);
                if (A.mask) {
                    m0[r] = ldg16(A.mask + (pix + (size_t)r * A.w) * COUT);
                    m1[r] = ldg16(A.mask + (pix + (size_t)r * A.w) * COUT + 8);
                }
            }
#pragma unroll
            for (int r = 0; r < ROWS; ++r)
                if (!pipe_wait(&pp.acc_full[row[r].a], row[r].phase, abort, A.err)) return;
            tc::fence_after_sync();
#pragma unroll
            for (int j = 0; j < COUT; j += 16) {
                float v[ROWS][16];
#pragma unroll
                for (int r = 0; r < ROWS; ++r) tc::tmem_ld16_nowait(tmem + (uint32_t)(row[r].a * COUT + j), v[r]);
                tc::tmem_wait_ld();
#pragma unroll
                for (int r = 0; r < ROWS; ++r) tc::tie16(v[r]);
                if (j + 16 >= COUT) {
                    tc::fence_before_sync();
                    __syncwarp();
#pragma unroll
                    for (int r = 0; r < ROWS; ++r)
                        if (lane == 0) mbar_arrive(&pp.acc_empty[row[r].a]);
                }
                uint4 q0[ROWS], q1[ROWS];
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    const uint4 n0 = m0[r], n1 = m1[r];
                    if (A.mask && j + 16 < COUT) {
                        m0[r] = ldg16(A.mask + (pix + (size_t)r * A.w) * COUT + j + 16);
                        m1[r] = ldg16(A.mask + (pix + (size_t)r * A.w) * COUT + j + 24);
                    }
                    finish16(A, v[r], s_bias + j, n0, n1, q0[r], q1[r]);
                    if (staged) {
                        const uint32_t at = sbase + (uint32_t)((r * 8 + run) * UNITS * 16);
                        const int u = rpx * (COUT / 8) + j / 8;
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + ((u ^ run) * 16)), "r"(q0[r].x),
                                     "r"(q0[r].y), "r"(q0[r].z), "r"(q0[r].w) : "memory");
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + (((u + 1) ^ run) * 16)),
                                     "r"(q1[r].x), "r"(q1[r].y), "r"(q1[r].z), "r"(q1[r].w) : "memory");
                    } else if (valid) {
                        const size_t at = pix + (size_t)r * A.w;
                        bf16 *o = A.out + at * COUT + j;
                        if (KS && A.split) o = split_at<COUT>(A.out + at * KS, plane2 + at * (COUT - KS), 0, j);
                        store16(o, q0[r], q1[r]);
                    }
                }
                if constexpr (POOL) {
                    const uint4 p0 = bmax4(q0[0], q0[1]), p1 = bmax4(q1[0], q1[1]);
                    const uint4 n0 = shfl_xor4(p0, 8), n1 = shfl_xor4(p1, 8);
                    if (valid && !(x & 1)) {
                        const size_t ppix = ((size_t)st.img * (A.h >> 1) + (y >> 1)) * (A.w >> 1) + (x >> 1);
                        store16(A.pool_out + ppix * COUT + j, bmax4(p0, n0), bmax4(p1, n1));
                    }
                }
                if constexpr (COUT == 16 && !POOL) {
                    if (A.head_w && valid) {
                        float f[16], r = 0.f;
                        unpack8(q0[0], f);
                        unpack8(q1[0], f + 8);
#pragma unroll
                        for (int k = 0; k < 16; ++k) r = fmaf(s_head[k], f[k], r);
                        const float o = din > 0.f ? din + 0.01f * (r + s_head[16]) : 0.f;  // residual in cm
                        if (A.depth_out) A.depth_out[pix] = o;
                        if (A.depth_mm) {
                            const float mm = fminf(fmaxf(rintf(o * 1000.f), 0.f), (float)TDE_MAX_DEPTH_VALUE);
                            A.depth_mm[pix] = (uint16_t)mm;
                        }
                    }
                }
            }
            if (staged) {
                __syncwarp();
                // pixel 4 * quarter + 16 * k of the tile begins run k
                const size_t first = ((size_t)st.img * A.h + y) * A.w + st.x0 + 4 * (int)quarter;
                const int left = A.w - st.x0 - 4 * (int)quarter;  // pixels of the row from there on
                auto unit = [&](int r, int k, int u) {
                    const uint32_t at = sbase + (uint32_t)((r * 8 + k) * UNITS * 16);
                    uint4 q;
                    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w) : "r"(at + ((u ^ k) * 16)) : "memory");
                    return q;
                };
                if (KS && A.split) {
                    // the units of the first plane, then those of the second
                    constexpr int U1 = KS ? 4 * KS / 8 : 4, U2 = UNITS - U1;
                    bf16 *d1 = A.out + first * KS, *d2 = plane2 + first * (COUT - KS);
#pragma unroll
                    for (int t = 0; t < U1 / 4; ++t) {
                        const int i = t * 32 + lane, k = i / U1, u = i - k * U1, p = u / (U1 / 4);
                        if (16 * k + p < left)
                            *reinterpret_cast<uint4 *>(d1 + 16 * k * KS + u * 8) =
                                unit(0, k, p * (COUT / 8) + u - p * (U1 / 4));
                    }
#pragma unroll
                    for (int t = 0; t < U2 / 4; ++t) {
                        const int i = t * 32 + lane, k = i / U2, u = i - k * U2, p = u / (U2 / 4);
                        if (16 * k + p < left)
                            *reinterpret_cast<uint4 *>(d2 + 16 * k * (COUT - KS) + u * 8) =
                                unit(0, k, p * (COUT / 8) + KS / 8 + u - p * (U2 / 4));
                    }
                } else {
                    bf16 *dst = A.out + first * COUT;
#pragma unroll
                    for (int r = 0; r < ROWS; ++r) {
#pragma unroll
                        for (int t = 0; t < UNITS / 4; ++t) {
                            const int i = t * 32 + lane, k = i / UNITS, u = i - k * UNITS;
                            const uint4 q = unit(r, k, u);
                            if (16 * k + u / (COUT / 8) < left)
                                *reinterpret_cast<uint4 *>(dst + ((size_t)r * A.w + 16 * k) * COUT + u * 8) = q;
                        }
                    }
                }
                __syncwarp();
            }
        }
    }
}

template <int MODE, int CCA, int CCB, int SETS>
__global__ void __launch_bounds__(conv_threads(SETS), kConvMaxPerSM) conv3x3_tc_kernel(const __grid_constant__ ConvArgs A, int rows_per_item,
                                                                        int S, int NA, int staged) {
    constexpr int CC = CCA + CCB;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ ConvPipe pp;
    __shared__ __align__(16) float s_bias[128], s_head[17];  // bias; head weights and head bias
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // A slot holds what only its input row has; an upsampled source's rows,
    // each that of two input rows, lie in a ring of their own.
    constexpr int CS = MODE == SRC_UP ? CCA : 0, CO = CC - CS;
    constexpr uint32_t slot_bytes = (uint32_t)CO * kPlaneBytes, shared_bytes = (uint32_t)CS * kPlaneBytes;
    const int SS = shared_slots(S);
    unsigned char *halo = smem;
    unsigned char *shared_rows = smem + (size_t)S * slot_bytes;
    unsigned char *wsm = shared_rows + (CS ? (size_t)SS * shared_bytes : 0);
    unsigned char *stage = staged ? wsm + (size_t)9 * CC * A.cout * 16 : nullptr;
    const uint32_t ncols = (uint32_t)A.cout;  // tensor-memory columns of one output row
    const uint32_t tcols = tmem_cols(NA * A.cout);
    volatile int *abort = &pp.abort;

    // the next layer may start its prologue; it waits for this grid before
    // reading anything this one writes
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (warp == kConvMmaWarp) tc::tmem_alloc(&pp.tmem, tcols);
    if (tid == 0) {
        for (int s = 0; s < kConvMaxSlots; ++s) {
            tc::mbar_init(&pp.full[s], 1);
            tc::mbar_init(&pp.empty[s], 1);
        }
        for (int s = 0; s < kConvMaxShared; ++s) {
            tc::mbar_init(&pp.sfull[s], 1);
            tc::mbar_init(&pp.sempty[s], 1);
        }
        for (int a = 0; a < kConvMaxAcc; ++a) {
            tc::mbar_init(&pp.acc_full[a], 1);
            tc::mbar_init(&pp.acc_empty[a], 4);  // the four warps that drain a row
        }
        tc::mbar_init(&pp.drain, 1);
        pp.abort = 0;
    }
    if (A.bias && tid < A.cout) s_bias[tid] = A.bias[tid];
    if (A.head_w && tid < 17) s_head[tid] = tid < 16 ? A.head_w[tid] : A.head_b[0];
    // weights: global [co][t][ci] -> planes (dx, chunk) of 3 cout rows x 16 B:
    // the rows of vertical taps 2, 1, 0 (output rows i - 2, i - 1, i of input row i).
    // No kernel launched right before a convolution writes weights, so they
    // are fetched before waiting for the previous grid.
    {
        const int nw = A.cout * 9 * CC;
        for (int i = tid; i < nw; i += (int)blockDim.x) {
            const int c = i % CC, t = (i / CC) % 9, co = i / (9 * CC);
            const int dy = t / 3, dx = t - 3 * dy;
            const uint32_t dst = tc::smem_u32(wsm + ((size_t)((dx * CC + c) * 3 + 2 - dy) * A.cout + co) * 16);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(A.wgt + (size_t)i * 8) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    tc::fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = pp.tmem;
    const int tiles_x = (A.w + kTileM - 1) / kTileM;
    const int items = A.n * tiles_x * ((A.h + rows_per_item - 1) / rows_per_item);

    if (warp < kConvProdWarps) {
        // ---- producers: warp pw loads the input rows j = pw (mod 4), two in
        // flight; a row is marked full once its copies have landed, at the
        // latest before this warp waits for anything ----
        const int pw = warp;
        uint32_t j = 0, js = 0;          // this block's input-row and shared-row sequences
        int pending = -1, spending = -1; // slots of the row issued before the current one
        bool ok = true;
        auto publish = [&](int wait_groups) {
            if (pending < 0) return;
            if (wait_groups) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&pp.full[pending]);
                if (CS && spending >= 0) mbar_arrive(&pp.sfull[spending]);
            }
            pending = spending = -1;
        };
        auto wait_empty = [&](uint64_t *bar, uint32_t k) {
            if (k == 0 || tc::mbar_test_wait(bar, (k - 1) & 1u)) return true;
            publish(0);
            return pipe_wait(bar, (k - 1) & 1u, abort, A.err);
        };
        for (int item = blockIdx.x; item < items && ok && !*abort; item += gridDim.x) {
            const Strip st = strip_of(A, item, rows_per_item);
            const int nin = st.y1 - st.y0 + 2;
            for (int i = 0; i < nin; ++i, ++j) {
                const int y = st.y0 - 1 + i;
                const bool fresh = CS && (i == 0 || !(y & 1));  // the first input row of its shared row
                if ((int)(j % (uint32_t)kConvProdWarps) != pw) {
                    js += fresh;
                    continue;
                }
                const bool row_in = y >= 0 && y < A.h;
                const uint32_t s = j % (uint32_t)S, ss = js % (uint32_t)SS;
                if (!(ok = wait_empty(&pp.empty[s], j / (uint32_t)S))) break;
                if (fresh && !(ok = wait_empty(&pp.sempty[ss], js / (uint32_t)SS))) break;
                const uint32_t dst = tc::smem_u32(halo) + s * slot_bytes;
                if constexpr (MODE == SRC_UP) {
                    if (fresh)
                        warp_copy_row<CCA, true>(
                            row_in ? A.a + ((size_t)st.img * (A.h >> 1) + (y >> 1)) * (A.w >> 1) * (8 * CCA) : nullptr,
                            st.x0, A.w, tc::smem_u32(shared_rows) + ss * shared_bytes, lane);
                    warp_copy_row<CCB, false>(row_in ? A.b + ((size_t)st.img * A.h + y) * A.w * (8 * CCB) : nullptr, st.x0,
                                              A.w, dst, lane);
                } else {
                    warp_copy_row<CCA, false>(row_in ? A.a + ((size_t)st.img * A.h + y) * A.w * (8 * CCA) : nullptr, st.x0,
                                              A.w, dst, lane);
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                publish(1);  // the previous row of this warp, while this one is in flight
                pending = (int)s;
                spending = fresh ? (int)ss : -1;
                js += fresh;
            }
        }
        publish(0);
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == kConvMmaWarp) {
        // ---- MMA issuer ----
        // The whole warp runs this loop (every value in it is the same in all
        // lanes), one elected lane issues, without a branch of its own: a
        // forward pass of batch 16 took 825 us with the MMAs in a branch that
        // the elected lane took, and takes 800 us without.
        const uint32_t halo_s = tc::smem_u32(halo), w_s = tc::smem_u32(wsm);
        const uint32_t s_lo0 = (uint32_t)tc::desc(tc::smem_u32(shared_rows), kPlaneBytes, 128);
        // descriptors: A at a slot's first plane (LBO = plane stride), B at the
        // first weight plane; an MMA adds its byte offset >> 4 to the low word
        const uint64_t a_desc0 = tc::desc(halo_s, kPlaneBytes, 128);
        const uint64_t b_desc0 = tc::desc(w_s, 3 * A.cout * 16, 128);
        const uint32_t a_lo0 = (uint32_t)a_desc0, a_hi = (uint32_t)(a_desc0 >> 32);
        const uint32_t b_lo0 = (uint32_t)b_desc0, b_hi = (uint32_t)(b_desc0 >> 32);
        const uint32_t b_row = (uint32_t)A.cout;                      // one tap's weight rows, 16-byte units
        const int max_rows = 256 / A.cout >= 3 ? 3 : 256 / A.cout;    // output rows of one MMA (N <= 256)
        const uint32_t id1 = tc::idesc_bf16(kTileM, A.cout);
        const uint32_t id_row = tc::idesc_bf16(0, A.cout) - tc::idesc_bf16(0, 0);  // one more output row
        const uint32_t lead = tc::elect_one(), bar0 = tc::smem_u32(&pp);
        uint32_t slot = 0, sphase = 0;      // ring slot and phase of the next input row
        uint32_t sslot = 0, ssphase = 0;    // and of the shared row of the current one
        int acc = 0;                        // accumulator of the next output row to start
        uint32_t aphase = 1;                // its phase: a fresh ring needs no wait (parity of the phase before)
        bool ok = true;
        for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
            const Strip st = strip_of(A, item, rows_per_item);
            const int R = st.y1 - st.y0;
            for (int i = 0; i < R + 2; ++i) {
                const int y = st.y0 - 1 + i;
                ok = pipe_wait(&pp.full[slot], sphase, abort, A.err);
                if (CS && ok && (i == 0 || !(y & 1))) ok = pipe_wait(&pp.sfull[sslot], ssphase, abort, A.err);
                // output rows lo .. hi of the strip; row i, if there is one, starts here
                const int lo = i < 2 ? 0 : i - 2, hi = i < R ? i : R - 1;
                if (ok && i < R) ok = pipe_wait(&pp.acc_empty[acc], aphase, abort, A.err);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc::fence_after_sync();
                // accumulator of row lo: acc is that of row i, or of the one after hi
                int alo = acc - ((i < R ? i : R) - lo);
                if (alo < 0) alo += NA;
                // their accumulators are adjacent but for the ring's end: one or two runs
                const int n = hi - lo + 1;
                const int n0 = min(min(n, NA - alo), max_rows);
                const uint32_t b0 = (uint32_t)(lo - i + 2) * b_row;
                const uint32_t d0 = tmem + (uint32_t)alo * ncols;
                // chunk kc of horizontal tap dx: in the shared row, or in this row's slot
                const uint32_t o_lo = a_lo0 + ((slot * slot_bytes) >> 4), s_lo = s_lo0 + ((sslot * shared_bytes) >> 4);
                auto a_at = [&](int dx, int kc) {
                    return (kc < CS ? s_lo + (uint32_t)((kc * kPlaneBytes + dx * 128) >> 4)
                                    : o_lo + (uint32_t)(((kc - CS) * kPlaneBytes + dx * 128) >> 4));
                };
                const uint32_t a_lo = a_at(0, 0);
                const uint32_t done = alo;   // row lo is complete after this input row when i >= 2
                {
                    if (n0 == n) {
                        const uint32_t id = id1 + (uint32_t)(n - 1) * id_row;
                        // a new output row overwrites its accumulator
                        if (i < R) {
                            tc::mma_bf16<false>(d0 + (uint32_t)(n - 1) * ncols, a_lo, a_hi, b_lo0 + 2 * b_row, b_hi, id1, lead);
                            if (n > 1) tc::mma_bf16<true>(d0, a_lo, a_hi, b_lo0 + b0, b_hi, id - id_row, lead);
                        } else {
                            tc::mma_bf16<true>(d0, a_lo, a_hi, b_lo0 + b0, b_hi, id, lead);
                        }
#pragma unroll
                        for (int m = 1; m < 3 * CC / 2; ++m) {
                            const int dx = m / (CC / 2), kc = 2 * (m % (CC / 2));
                            tc::mma_bf16<true>(d0, a_at(dx, kc), a_hi,
                                               b_lo0 + b0 + (uint32_t)(dx * CC + kc) * 3u * b_row, b_hi, id, lead);
                        }
                    } else {
                        const int n1 = n - n0;
                        const uint32_t d1 = alo + n0 == NA ? tmem : d0 + (uint32_t)n0 * ncols;
                        const uint32_t b1 = b0 + (uint32_t)n0 * b_row;
                        const uint32_t i0 = id1 + (uint32_t)(n0 - 1) * id_row, i1 = id1 + (uint32_t)(n1 - 1) * id_row;
                        tc::mma_bf16<true>(d0, a_lo, a_hi, b_lo0 + b0, b_hi, i0, lead);
                        if (i < R) {
                            if (n1 > 1) tc::mma_bf16<true>(d1, a_lo, a_hi, b_lo0 + b1, b_hi, id1, lead);
                            tc::mma_bf16<false>(d1 + (uint32_t)(n1 - 1) * ncols, a_lo, a_hi, b_lo0 + 2 * b_row, b_hi, id1, lead);
                        } else {
                            tc::mma_bf16<true>(d1, a_lo, a_hi, b_lo0 + b1, b_hi, i1, lead);
                        }
#pragma unroll
                        for (int m = 1; m < 3 * CC / 2; ++m) {
                            const int dx = m / (CC / 2), kc = 2 * (m % (CC / 2));
                            const uint32_t ad = a_at(dx, kc);
                            const uint32_t bd = b_lo0 + (uint32_t)(dx * CC + kc) * 3u * b_row;
                            tc::mma_bf16<true>(d0, ad, a_hi, bd + b0, b_hi, i0, lead);
                            tc::mma_bf16<true>(d1, ad, a_hi, bd + b1, b_hi, i1, lead);
                        }
                    }
                    tc::commit_lead(bar0 + (uint32_t)offsetof(ConvPipe, empty) + 8u * slot, lead);  // this input row is read by no later MMA
                    if (CS && ((y & 1) || i == R + 1)) tc::commit_lead(bar0 + (uint32_t)offsetof(ConvPipe, sempty) + 8u * sslot, lead);
                    if (i >= 2) tc::commit_lead(bar0 + (uint32_t)offsetof(ConvPipe, acc_full) + 8u * done, lead);
                }
                if (++slot == (uint32_t)S) {
                    slot = 0;
                    sphase ^= 1u;
                }
                if (CS && ((y & 1) || i == R + 1) && ++sslot == (uint32_t)SS) {
                    sslot = 0;
                    ssphase ^= 1u;
                }
                if (i < R && ++acc == NA) {
                    acc = 0;
                    aphase ^= 1u;
                }
            }
        }
        // every MMA issued has finished before the tensor memory is freed
        tc::commit_lead(tc::smem_u32(&pp.drain), lead);
        __syncwarp();
        tc::mbar_wait(&pp.drain, 0u, kConvWaitNs);
        __syncwarp();
    } else {
        // ---- epilogue ----
        // (the output channels that the network's layers and their gradients
        // have with this many input channels)
#define TDE_EPILOGUE(N, P) \
    conv_epilogue<N, P, SETS>(A, pp, s_bias, s_head, stage, rows_per_item, items, NA, warp, lane)
        if constexpr (MODE == SRC_UP) {
            TDE_EPILOGUE(8 * CCB, false);
        } else if constexpr (SETS == 1) {
            TDE_EPILOGUE(8 * CCA, true);
        } else if constexpr (CCA == 2) {
            if (A.cout == 16) TDE_EPILOGUE(16, false);
            else if (A.cout == 32) TDE_EPILOGUE(32, false);
            else TDE_EPILOGUE(48, false);
        } else if constexpr (CCA == 4) {
            if (A.cout == 16) TDE_EPILOGUE(16, false);
            else if (A.cout == 32) TDE_EPILOGUE(32, false);
            else if (A.cout == 48) TDE_EPILOGUE(48, false);
            else TDE_EPILOGUE(80, false);
        } else if constexpr (CCA == 6) {
            if (A.cout == 32) TDE_EPILOGUE(32, false);
            else if (A.cout == 48) TDE_EPILOGUE(48, false);
            else if (A.cout == 64) TDE_EPILOGUE(64, false);
            else TDE_EPILOGUE(112, false);
        } else {
            if (A.cout == 48) TDE_EPILOGUE(48, false);
            else TDE_EPILOGUE(64, false);
        }
#undef TDE_EPILOGUE
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == kConvMmaWarp) tc::tmem_dealloc(tmem, tcols);
}

// (mode, input chunks) pairs the network uses: forward c2..c11 (the encoder's
// pooled inputs come precomputed from the epilogue of the layer before) and
// the input gradients of c2..c11 (direct sources with cout/8 chunks)
#define TDE_CONV_VARIANTS(X) \
    X(SRC_DIRECT, 2, 0) X(SRC_DIRECT, 4, 0) X(SRC_DIRECT, 6, 0) X(SRC_DIRECT, 8, 0) \
    X(SRC_UP, 4, 2) X(SRC_UP, 6, 4) X(SRC_UP, 8, 6)

// The kernel for a source mode, the input chunks of sources A and B, and
// whether the output is pooled as well.
const void *conv_kernel_fn(int mode, int cca, int ccb, bool pool) {
#define TDE_CONV_FN(M, A, B) \
    if (mode == M && cca == A && ccb == B && !pool) return (const void *)conv3x3_tc_kernel<M, A, B, conv_epi_sets(M, false)>;
    TDE_CONV_VARIANTS(TDE_CONV_FN)
#undef TDE_CONV_FN
#define TDE_CONV_FN(A) \
    if (mode == SRC_DIRECT && cca == A && ccb == 0 && pool) return (const void *)conv3x3_tc_kernel<SRC_DIRECT, A, 0, 1>;
    TDE_CONV_FN(2) TDE_CONV_FN(4) TDE_CONV_FN(6)
#undef TDE_CONV_FN
    return nullptr;
}

// ---------------------------------------------------------------------------
// Weight gradient
//
// dW[co][dy][dx][ci] = sum over output pixels of dZ[y][x][co] X[y+dy-1][x+dx-1][ci],
// as D = A B with K = pixels, both operands MN-major: the tensor core reads the
// staged NHWC data as it lies, as planes of 8 channels (16 bytes a pixel).  For
// output row y and input pixels q of a column of KP = 128 pixels (64 in the
// layers whose rings would not fit):
//   A, M = (dx, co): three copies of dZ's row y, copy dx shifted so that pixel q
//     holds dZ[y][q + 1 - dx];
//   B, N = (dy, ci): X's rows y - 1, y, y + 1, neighbours in a ring of rows.
// One MMA per 16 pixels then does all nine taps of a layer whose 3 cout fit in
// M = 128 (two MMAs beyond; two more where the ring wraps), and each row of X is
// staged once for the three output rows it belongs to.  Before, an MMA did one
// horizontal tap and 128 rows (dy, ci) of X -- 28 MMAs where this takes 4, at some
// 100 cycles of issue each -- and X was staged three times; wgrad of c11 and c2 at
// batch 16 of 640x480: 811 and 576 us then, 238 and 156 us now, of all layers
// together 2230 and 940 (about 1800 cycles a step of 128 pixels remain).
// Rows of A past 3 cout read whatever follows in shared memory; their rows of D
// are not used.  The bias gradient is summed on the CUDA cores from copy dx = 1.
// Without swizzling, a descriptor's LBO is the stride between 8-element groups
// along K and its SBO the stride along M (or N), for MN-major operands as for
// K-major ones.
//
// A block takes a contiguous share of all (image, column, row) steps, rows
// fastest; each stretch of one column is a run of n output rows and n + 2 rows
// of X, staged as units: unit u holds X row u and dZ row u - 2 of the run.
//   warps 0-3 (producers): unit j goes to warp j & 3, two in flight each;
//   warp 4 (MMA issuer): at unit u >= 2 the MMAs of output row u - 2, committed to
//     the dZ slot and to the slot of the X row no later step reads;
//   warps 5-8: sum dZ for the bias, waiting for dZ rows alone: a slot of X is
//     released without them, so its phases could pass them by, where a dZ slot is
//     filled again only after they have read it; at the end drain the accumulators,
//     which stay in tensor memory across all the block's steps, into its partial.
// Bounded waits as in the convolution.
// ---------------------------------------------------------------------------
constexpr int kWgProdWarps = 4, kWgMmaWarp = 4, kWgBiasWarps = 4;
constexpr int kWgThreads = 32 * (kWgProdWarps + 1 + kWgBiasWarps);
constexpr int kWgMaxFlight = 8;
// Pixels of a step, and units in flight beside the step being multiplied, for
// cc input and cz output chunks: what one block's shared memory holds.  The dZ
// ring has no fewer slots than producer warps (as the convolution's ring).
__host__ __device__ constexpr uint32_t wg_smem(int cc, int cz, int kp, int flight) {
    return (uint32_t)(((flight + 1) * 3 * cz + (flight + 3) * cc) * kp * 16);
}
constexpr uint32_t kWgSmem = 224 * 1024;
__host__ __device__ constexpr int wg_kp(int cc, int cz) { return wg_smem(cc, cz, 128, 3) <= kWgSmem ? 128 : 64; }
__host__ __device__ constexpr int wg_flight(int cc, int cz) {
    int f = 3;
    while (f < kWgMaxFlight && wg_smem(cc, cz, wg_kp(cc, cz), f + 1) <= kWgSmem) ++f;
    return f;
}

// MN-major kind::f16 instruction descriptor (bits 15, 16 = 1).
__host__ __device__ constexpr uint32_t idesc_bf16_mn(int M, int N) {
    return tc::idesc_bf16(M, N) | (1u << 15) | (1u << 16);
}
__host__ __device__ constexpr int wg_mtiles(int cout) { return (3 * cout + 127) / 128; }
// Floats of one block's partial: [3 cout][3 cin], then the bias.
__host__ __device__ constexpr int wg_partial(int cin, int cout) { return 9 * cin * cout + cout; }

struct WgPipe {
    uint64_t full[kWgMaxFlight + 3], empty[kWgMaxFlight + 3], zfull[kWgMaxFlight + 1], zempty[kWgMaxFlight + 1], drain;
    uint32_t tmem;
    int abort;
};

// Copies of CP = 2 or 4 channel chunks of KP pixels of a row (PXE channels a
// pixel) from pixel x_start on, read directly or through the nearest 2x
// upsample (x_start even then), into planes; zeros past the row's ends.  Eight
// lanes take eight neighbouring pixels of one chunk, the four such sets of a
// warp the chunks of the same pixels.
template <int KP, int CP, bool UPS, int PXE>
__device__ __forceinline__ void wg_copy_chunks(const bf16 *row, int x_start, int w, uint32_t dst, int lane) {
    const int k = lane & 7, l3 = lane >> 3;
    const int c = CP == 4 ? l3 : l3 & 1, bl = CP == 4 ? 0 : l3 >> 1;
    const int x = x_start + 8 * bl + k, lim = w - x;
    const bf16 *src = row + (UPS ? (x_start >> 1) + 4 * bl + (k >> 1) : x) * PXE + 8 * c;
    dst += (uint32_t)(c * KP * 16 + (8 * bl + k) * 16);
#pragma unroll
    for (int it = 0; it < KP * CP / 32; ++it) {
        const int px = (CP == 4 ? 8 : 16) * it;
        if (px < lim && (it > 0 || x >= 0))
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + px * 16), "l"(src + (UPS ? px / 2 : px) * PXE)
                         : "memory");
        else
            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(dst + px * 16), "r"(0) : "memory");
    }
}
template <int KP, int CC, bool UPS>
__device__ __forceinline__ void wg_copy_row(const bf16 *row, int x_start, int w, uint32_t dst, int lane) {
    if (row) {
#pragma unroll
        for (int c = 0; c + 4 <= CC; c += 4)
            wg_copy_chunks<KP, 4, UPS, 8 * CC>(row + 8 * c, x_start, w, dst + c * KP * 16, lane);
        if constexpr (CC % 4 != 0)
            wg_copy_chunks<KP, 2, UPS, 8 * CC>(row + 8 * (CC - 2), x_start, w, dst + (CC - 2) * KP * 16, lane);
    } else {
        for (int i = lane; i < CC * KP; i += 32)
            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(dst + i * 16), "r"(0) : "memory");
    }
}

// A stretch of one column: image, first pixel, output rows [y0, y1).
struct WgRun { int img, x0, y0, y1; };
template <int KP> __device__ __forceinline__ WgRun wg_run(const WgradArgs &A, int step, int last) {
    const int tiles_x = (A.w + KP - 1) / KP;
    const int col = step / A.h;
    WgRun r;
    r.img = col / tiles_x;
    r.x0 = (col - r.img * tiles_x) * KP;
    r.y0 = step - col * A.h;
    r.y1 = min(A.h, r.y0 + last - step);
    return r;
}

template <int MODE, int CCA, int CCB, int CZ>
__global__ void __launch_bounds__(kWgThreads, 1) wgrad_tc_kernel(const WgradArgs A) {
    constexpr int CC = CCA + CCB, CIN = 8 * CC, COUT = 8 * CZ, MT = wg_mtiles(COUT), N = 3 * CIN;
    constexpr int KP = wg_kp(CC, CZ), kRowSlots = wg_flight(CC, CZ) + 3, kDzSlots = wg_flight(CC, CZ) + 1;
    constexpr int kPlane = KP * 16;  // one 8-channel plane of a row
    constexpr uint32_t xbytes = CC * kPlane, zbytes = 3 * CZ * kPlane;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ WgPipe pp;
    __shared__ float s_bias[kWgBiasWarps][COUT];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr uint32_t tcols = tmem_cols(MT * N);
    // dZ ring first: the rows of A that a tile of 128 reads past it are X's
    unsigned char *zring = smem, *xring = smem + kDzSlots * zbytes;
    volatile int *abort = &pp.abort;
    if (warp == kWgMmaWarp) tc::tmem_alloc(&pp.tmem, tcols);
    if (tid == 0) {
        for (int s = 0; s < kRowSlots; ++s) {
            tc::mbar_init(&pp.full[s], 1);
            tc::mbar_init(&pp.empty[s], 1);
        }
        for (int s = 0; s < kDzSlots; ++s) {
            tc::mbar_init(&pp.zfull[s], 1);
            tc::mbar_init(&pp.zempty[s], 1 + kWgBiasWarps);
        }
        tc::mbar_init(&pp.drain, 1);
        pp.abort = 0;
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = pp.tmem;
    const long steps = (long)A.n * A.h * ((A.w + KP - 1) / KP);
    const int s0 = (int)(steps * blockIdx.x / gridDim.x), s1 = (int)(steps * (blockIdx.x + 1) / gridDim.x);

    if (warp < kWgProdWarps) {
        // ---- producers ----
        uint32_t j = 0, jz = 0;  // units and dZ rows of this block so far
        int pending = -1, zpending = -1;  // slots of the unit issued before the current one
        bool ok = true;
        auto publish = [&](int wait_groups) {
            if (pending < 0) return;
            if (wait_groups) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&pp.full[pending]);
                if (zpending >= 0) mbar_arrive(&pp.zfull[zpending]);
            }
            pending = zpending = -1;
        };
        auto wait_empty = [&](uint64_t *bar, uint32_t k) {
            if (k == 0 || tc::mbar_test_wait(bar, (k - 1) & 1u)) return true;
            publish(0);
            return pipe_wait(bar, (k - 1) & 1u, abort, A.err);
        };
        for (int step = s0; step < s1 && ok && !*abort;) {
            const WgRun run = wg_run<KP>(A, step, s1);
            const int n = run.y1 - run.y0;
            for (int u = 0; u < n + 2; ++u, ++j) {
                const bool has_z = u >= 2;
                if ((int)(j % (uint32_t)kWgProdWarps) != warp) {
                    jz += has_z;
                    continue;
                }
                const uint32_t s = j % (uint32_t)kRowSlots, sz = jz % (uint32_t)kDzSlots;
                if (!(ok = wait_empty(&pp.empty[s], j / (uint32_t)kRowSlots))) break;
                if (has_z && !(ok = wait_empty(&pp.zempty[sz], jz / (uint32_t)kDzSlots))) break;
                const int y = run.y0 - 1 + u;
                const bool row_in = y >= 0 && y < A.h;
                const uint32_t xd = tc::smem_u32(xring) + s * xbytes;
                if constexpr (MODE == SRC_UP)
                    wg_copy_row<KP, CCA, true>(
                        row_in ? A.a + ((size_t)run.img * (A.h >> 1) + (y >> 1)) * (A.w >> 1) * (8 * CCA) : nullptr, run.x0,
                        A.w, xd, lane);
                else
                    wg_copy_row<KP, CCA, false>(row_in ? A.a + ((size_t)run.img * A.h + y) * A.w * (8 * CCA) : nullptr, run.x0,
                                            A.w, xd, lane);
                if constexpr (CCB > 0)
                    wg_copy_row<KP, CCB, false>(row_in ? A.b + ((size_t)run.img * A.h + y) * A.w * (8 * CCB) : nullptr, run.x0,
                                            A.w, xd + CCA * kPlane, lane);
                if (has_z) {
                    const bf16 *zrow = A.dz + ((size_t)run.img * A.h + y - 1) * A.w * COUT;
                    const uint32_t zd = tc::smem_u32(zring) + sz * zbytes;
#pragma unroll 1
                    for (int dx = 0; dx < 3; ++dx)
                        wg_copy_row<KP, CZ, false>(zrow, run.x0 + 1 - dx, A.w, zd + (uint32_t)(dx * CZ * kPlane), lane);
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                publish(1);
                pending = (int)s;
                zpending = has_z ? (int)sz : -1;
                jz += has_z;
            }
            step += n;
        }
        publish(0);
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == kWgMmaWarp) {
        // ---- MMA issuer (the whole warp runs the loop, one lane issues) ----
        const uint64_t z0 = tc::desc(tc::smem_u32(zring), 128, kPlane), x0 = tc::desc(tc::smem_u32(xring), 128, kPlane);
        const uint32_t z_lo = (uint32_t)z0, z_hi = (uint32_t)(z0 >> 32), x_lo = (uint32_t)x0, x_hi = (uint32_t)(x0 >> 32);
        const uint32_t id1 = idesc_bf16_mn(128, CIN), id_row = tc::idesc_bf16(0, CIN) - tc::idesc_bf16(0, 0);
        const uint32_t lead = tc::elect_one(), bar0 = tc::smem_u32(&pp);
        const uint32_t empty0 = bar0 + (uint32_t)offsetof(WgPipe, empty), zempty0 = bar0 + (uint32_t)offsetof(WgPipe, zempty);
        uint32_t slot = 0, sphase = 0, zslot = 0, acc = 0;
        bool ok = true;
        for (int step = s0; step < s1 && ok;) {
            const WgRun run = wg_run<KP>(A, step, s1);
            const int n = run.y1 - run.y0;
            const int nk = (min(KP, A.w - run.x0) + 15) / 16;  // K steps with pixels of the image
            for (int u = 0; u < n + 2; ++u) {
                ok = __all_sync(0xffffffffu, pipe_wait(&pp.full[slot], sphase, abort, A.err));
                if (!ok) break;
                if (u >= 2) {
                    tc::fence_after_sync();
                    // X rows u - 2 .. u: one run of the ring, or two
                    const uint32_t first = slot >= 2 ? slot - 2 : slot + kRowSlots - 2;
                    const uint32_t r0 = min(3u, (uint32_t)kRowSlots - first);
                    const uint32_t al = z_lo + ((zslot * zbytes) >> 4), b0 = x_lo + ((first * xbytes) >> 4);
                    const uint32_t i0 = id1 + (r0 - 1) * id_row, i1 = id1 + (2 - r0) * id_row;
                    for (int kk = 0; kk < nk; ++kk) {
                        const uint32_t ko = (uint32_t)(kk * 16);  // 16 pixels, in 16-byte units
#pragma unroll
                        for (int mt = 0; mt < MT; ++mt) {
                            const uint32_t a = al + ko + (uint32_t)(mt * 16 * kPlane >> 4), d = tmem + (uint32_t)(mt * N);
                            tc::mma_bf16(d, a, z_hi, b0 + ko, x_hi, i0, acc, lead);
                            if (r0 < 3) tc::mma_bf16(d + r0 * CIN, a, z_hi, x_lo + ko, x_hi, i1, acc, lead);
                        }
                        acc = 1;
                    }
                    tc::commit_lead(zempty0 + 8u * zslot, lead);
                    tc::commit_lead(empty0 + 8u * first, lead);
                    if (++zslot == (uint32_t)kDzSlots) zslot = 0;
                    if (u == n + 1) {  // the run's last two rows are read by no later step either
                        tc::commit_lead(empty0 + 8u * (slot >= 1 ? slot - 1 : (uint32_t)kRowSlots - 1), lead);
                        tc::commit_lead(empty0 + 8u * slot, lead);
                    }
                }
                if (++slot == (uint32_t)kRowSlots) {
                    slot = 0;
                    sphase ^= 1u;
                }
            }
            step += n;
        }
        // every MMA issued has finished before the accumulators are read
        tc::commit_lead(tc::smem_u32(&pp.drain), lead);
        __syncwarp();
        if (!tc::mbar_wait(&pp.drain, 0u, kConvWaitNs) && lane == 0) {
            *abort = 1;
            atomicExch(A.err, 1);
        }
        __syncwarp();
    } else {
        // ---- bias: thread t sums pixel t % KP of chunks t / KP, + 128 / KP, ... ----
        constexpr int GR = 128 / KP, CT = CZ / GR;
        const int t = tid - 32 * (kWgMmaWarp + 1), px = t % KP, c0 = t / KP;
        float sum[CT][8];
#pragma unroll
        for (int c = 0; c < CT; ++c)
#pragma unroll
            for (int e = 0; e < 8; ++e) sum[c][e] = 0.f;
        uint32_t zslot = 0, zphase = 0;
        for (int step = s0; step < s1; ++step) {
            if (!pipe_wait(&pp.zfull[zslot], zphase, abort, A.err)) break;
            const unsigned char *z = zring + zslot * zbytes + CZ * kPlane + px * 16;  // copy dx = 1
#pragma unroll
            for (int c = 0; c < CT; ++c) {
                float f[8];
                unpack8(*reinterpret_cast<const uint4 *>(z + (c0 + GR * c) * kPlane), f);
#pragma unroll
                for (int e = 0; e < 8; ++e) sum[c][e] += f[e];
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&pp.zempty[zslot]);
            if (++zslot == (uint32_t)kDzSlots) {
                zslot = 0;
                zphase ^= 1u;
            }
        }
        // over the warp's 32 pixels (the warps of a chunk are added below)
        const int wb = warp - kWgMmaWarp - 1;
#pragma unroll
        for (int c = 0; c < CT; ++c)
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                float v = sum[c][e];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) s_bias[wb][8 * (c0 + GR * c) + e] = v;
            }
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (!*abort && warp > kWgMmaWarp) {
        // D row m = (dx, co), column n = (dy, ci)
        float *dst = A.partial + (size_t)blockIdx.x * wg_partial(CIN, COUT);
        const int q = warp & 3;  // a warp reads the tensor-memory lanes of its number modulo 4
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            const int m = mt * 128 + q * 32 + lane;
            for (int j = 0; j < N; j += 16) {
                float v[16];
                tc::tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(mt * N + j), v);
                if (m >= 3 * COUT) continue;
                float4 *o = reinterpret_cast<float4 *>(dst + (size_t)m * N + j);
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    o[e] = s0 < s1 ? make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3])
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        const int t = tid - 32 * (kWgMmaWarp + 1);
        if (t < COUT) {  // chunk t / 8 was summed by KP / 32 warps
            const int wb = ((t >> 3) % (128 / KP)) * (KP / 32);
            float v = s_bias[wb][t];
#pragma unroll
            for (int k = 1; k < KP / 32; ++k) v += s_bias[wb + k][t];
            dst[3 * COUT * N + t] = v;
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == kWgMmaWarp) tc::tmem_dealloc(tmem, tcols);
}

// The weight-gradient kernel for a source mode, the input chunks of sources A
// and B and the output chunks: c2 .. c8, c10, c11, and c9 as two (its 112 input
// channels' accumulators exceed the tensor memory).
#define TDE_WG_VARIANTS(X) \
    X(SRC_DIRECT, 2, 0, 2) X(SRC_DIRECT, 2, 0, 4) X(SRC_DIRECT, 4, 0, 4) X(SRC_DIRECT, 4, 0, 6) X(SRC_DIRECT, 6, 0, 6) \
    X(SRC_DIRECT, 6, 0, 8) X(SRC_DIRECT, 8, 0, 8) X(SRC_UP, 8, 0, 6) X(SRC_UP, 6, 4, 4) X(SRC_UP, 4, 2, 2)
const void *wgrad_kernel_fn(int mode, int cca, int ccb, int cz) {
#define TDE_WG_FN(M, A, B, Z) \
    if (mode == M && cca == A && ccb == B && cz == Z) return (const void *)wgrad_tc_kernel<M, A, B, Z>;
    TDE_WG_VARIANTS(TDE_WG_FN)
#undef TDE_WG_FN
    return nullptr;
}

// Fixed-order sum of `blocks` partial vectors of n floats ([blocks][n]): a
// block takes 32 consecutive elements (coalesced); warp w sums the partials
// w, w + 8, ... with eight loads in flight, then the eight warp sums are added
// in warp order.  Deterministic; the partials' latency is paid about
// blocks / 64 times instead of `blocks` times.
__device__ __forceinline__ bool sum_partials(const float *__restrict__ partial, int blocks, int n, int &e,
                                             float &total) {
    __shared__ float part[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    e = blockIdx.x * 32 + lane;
    float a[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = 0.f;
    if (e < n) {
        int b = w;
        for (; b + 56 < blocks; b += 64) {
#pragma unroll
            for (int k = 0; k < 8; ++k) a[k] += __ldg(partial + (size_t)(b + 8 * k) * n + e);
        }
        for (int k = 0; b < blocks; b += 8, ++k) a[k & 7] += __ldg(partial + (size_t)b * n + e);
    }
    part[w][lane] = ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
    __syncthreads();
    if (w != 0 || e >= n) return false;
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += part[k][lane];
    total = t;
    return true;
}

// Weight gradients from the per-block partials [blocks][(dx, co)][(dy, ci)] and
// their bias; this part's cin channels lie at ci0 of the layer's cin_all:
// dw[(co * 9 + 3 dy + dx) * cin_all + ci0 + ci].
__global__ void __launch_bounds__(256) wgrad_reduce_kernel(const float *__restrict__ partial, int blocks, int cin,
                                                           int cin_all, int ci0, int cout, float *__restrict__ dw,
                                                           float *__restrict__ db) {
    int e;
    float t;
    if (!sum_partials(partial, blocks, wg_partial(cin, cout), e, t)) return;
    const int m = e / (3 * cin), n = e - m * (3 * cin);
    if (m >= 3 * cout) {  // (the bias is shorter than a row of D)
        if (db) db[n] = t;
        return;
    }
    const int dx = m / cout, co = m - dx * cout, dy = n / cin, ci = n - dy * cin;
    dw[((size_t)co * 9 + 3 * dy + dx) * cin_all + ci0 + ci] = t;
}

// ---------------------------------------------------------------------------
// First convolution (2 -> 16, FP32) and its weight gradient
// ---------------------------------------------------------------------------
// Input features of tap t (3x3 window around the pixel, t = 3*dy + dx):
// [100 (d_t - d_c) if both valid else 0, valid_t, d_t], d in metres (0 where
// invalid).  Differences in centimetres keep millimetre noise representable
// once the first layer's output is stored as bf16.
constexpr int kInCh = 3, kInK = 9 * kInCh;
// Two FP32 values in one 64-bit register and their fused multiply-adds (each
// rounded as fmaf): half the instructions of the two scalar ones.
__device__ __forceinline__ uint64_t f2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unf2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The three features of one tap, for the pixel with depth dc.
__device__ __forceinline__ void tap_features(float d, float dc, float (&f)[kInCh]) {
    const bool v = d > 0.f;
    f[0] = (v && dc > 0.f) ? (d - dc) * 100.f : 0.f;
    f[1] = v ? 1.f : 0.f;
    f[2] = d;
}

// A thread makes kInRows pixels of one column, so that a weight read from shared
// memory serves four fused multiply-adds (one pixel a thread waited for those
// reads: 193 us at batch 16 of 640x480, 115 us now; the arithmetic alone is
// 57 us).  Each output channel's sum runs over the features in order.
constexpr int kInRows = 4;
__global__ void __launch_bounds__(128) conv_in_kernel(const uint16_t *__restrict__ raw, float *__restrict__ depth_m,
                                                      const float *__restrict__ w1, const float *__restrict__ b1,
                                                      bf16 *__restrict__ e0a, int n, int h, int w) {
    __shared__ __align__(16) float sw[kInK + 1][16];  // by feature, then the bias
    for (int i = threadIdx.x; i < 16 * kInK; i += blockDim.x) sw[i % kInK][i / kInK] = w1[i];
    if (threadIdx.x < 16) sw[kInK][threadIdx.x] = b1[threadIdx.x];
    __syncthreads();
    // rows are multiples of kInRows; lanes run over w, a multiple of 8
    const unsigned p = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned x = p % (unsigned)w, strip = p / (unsigned)w, strips = (unsigned)h / kInRows;
    const bool live = strip < (unsigned)n * strips;
    const int img = live ? (int)(strip / strips) : 0, y0 = live ? (int)(strip % strips) * kInRows : 0;
    float d[kInRows + 2][3];
#pragma unroll
    for (int r = 0; r < kInRows + 2; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int yy = y0 + r - 1, xx = (int)x + c - 1;
            d[r][c] = 0.f;
            if (yy >= 0 && yy < h && xx >= 0 && xx < w) d[r][c] = (float)__ldg(raw + ((size_t)img * h + yy) * w + xx) * 0.001f;
        }
    uint64_t o2[kInRows][8];  // channel pairs
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int r = 0; r < kInRows; ++r) o2[r][c] = f2(sw[kInK][2 * c], sw[kInK][2 * c + 1]);
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        float f[kInRows][kInCh];
#pragma unroll
        for (int r = 0; r < kInRows; ++r) tap_features(d[r + t / 3][t % 3], d[r + 1][1], f[r]);
#pragma unroll
        for (int k = 0; k < kInCh; ++k) {
            uint64_t ff[kInRows];
#pragma unroll
            for (int r = 0; r < kInRows; ++r) ff[r] = f2(f[r][k], f[r][k]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 wv = *reinterpret_cast<const float4 *>(&sw[kInCh * t + k][4 * q]);
                const uint64_t wa = f2(wv.x, wv.y), wb = f2(wv.z, wv.w);
#pragma unroll
                for (int r = 0; r < kInRows; ++r) {
                    o2[r][2 * q] = fma2(wa, ff[r], o2[r][2 * q]);
                    o2[r][2 * q + 1] = fma2(wb, ff[r], o2[r][2 * q + 1]);
                }
            }
        }
    }
    // Stores in whole sectors: an even lane and the odd one after it (the next
    // pixel of the row: w is even) swap halves, so that a store's neighbouring
    // lanes write the two halves of one pixel.
    const bool odd = threadIdx.x & 1;
#pragma unroll
    for (int r = 0; r < kInRows; ++r) {
        float o[16];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float2 v = unf2(o2[r][c]);
            o[2 * c] = v.x > 0.f ? v.x : 0.f;
            o[2 * c + 1] = v.y > 0.f ? v.y : 0.f;
        }
        const size_t pix = ((size_t)img * h + y0 + r) * w + x;
        const uint4 q0 = pack8(o), q1 = pack8(o + 8);
        const uint4 give = odd ? q0 : q1, got = shfl_xor4(give, 1);
        if (live) {
            depth_m[pix] = d[r + 1][1];
            uint4 *dst = reinterpret_cast<uint4 *>(e0a + (pix - odd) * 16);  // the even pixel
            dst[odd] = odd ? got : q0;
            dst[2 + odd] = odd ? q1 : got;
        }
    }
}

// Gradient of the first convolution: C[16 channels][28 features] += G F over the
// pixels (the 28th feature is 1: the bias).  A block stages 64 pixels of a row at
// a time as feature and gradient rows in shared memory; thread (kg, cq, fq) takes
// the pixels 4 kg .. 4 kg + 3, the channels cq + 4 i and the features 7 fq + j: 11
// 16-byte reads for 112 multiply-adds.  (One channel a thread, each forming the
// pixel's features again: 413 us at batch 16 of 640x480; 212 us now.)
// Row strides of 72 words put a warp's eight distinct reads into different banks.
constexpr int kInPartial = 16 * (kInK + 1);
constexpr int kInTile = 64, kInStride = 72, kInBlocksPerSM = 4;
__global__ void __launch_bounds__(256, kInBlocksPerSM) conv_in_wgrad_kernel(const float *__restrict__ depth_m,
                                                            const bf16 *__restrict__ dz1, int n, int h, int w,
                                                            float *__restrict__ partial) {
    __shared__ __align__(16) float F[kInK + 1][kInStride], G[16][kInStride];
    __shared__ float red[8][kInPartial];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kg = tid >> 4, cq = (tid >> 2) & 3, fq = tid & 3;
    float s[4][7];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 7; ++j) s[i][j] = 0.f;
    if (tid < kInTile) F[kInK][tid] = 1.f;
    const int tiles_x = (w + kInTile - 1) / kInTile;
    const long tiles = (long)n * h * tiles_x;
    const int px = tid & 63, part = tid >> 6;
    // taps 3 part .. 3 part + 2 (one kernel row) by the first 192 threads, the
    // gradients by the last 64; a tile is fetched while the one before is summed
    float d[3], dc = 0.f;
    uint4 gv[2];
    auto fetch = [&](long tile) {
        const long rowi = tile / tiles_x;
        const int y = (int)(rowi % h), x = (int)(tile - rowi * tiles_x) * kInTile + px;
        const bool in = tile < tiles && x < w;
        if (part < 3) {
            const float *row = depth_m + rowi * w;
            const int yy = y + part - 1;
            dc = in ? __ldg(row + x) : 0.f;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int xx = x + c - 1;
                d[c] = in && yy >= 0 && yy < h && xx >= 0 && xx < w ? __ldg(row + (part - 1) * w + xx) : 0.f;
            }
        } else {
            gv[0] = in ? ldg16(dz1 + (rowi * w + x) * 16) : make_uint4(0u, 0u, 0u, 0u);
            gv[1] = in ? ldg16(dz1 + (rowi * w + x) * 16 + 8) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    fetch(blockIdx.x);
    for (long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        __syncthreads();  // the previous tile has been read
        if (part < 3) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                float f[kInCh];
                tap_features(d[c], dc, f);
#pragma unroll
                for (int k = 0; k < kInCh; ++k) F[kInCh * (3 * part + c) + k][px] = f[k];
            }
        } else {
            float f[16];
            unpack8(gv[0], f);
            unpack8(gv[1], f + 8);
#pragma unroll
            for (int c = 0; c < 16; ++c) G[c][px] = f[c];
        }
        __syncthreads();
        fetch(tile + gridDim.x);
        float4 g[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) g[i] = *reinterpret_cast<const float4 *>(&G[cq + 4 * i][4 * kg]);
#pragma unroll
        for (int j = 0; j < 7; ++j) {
            const float4 f = *reinterpret_cast<const float4 *>(&F[7 * fq + j][4 * kg]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s[i][j] = fmaf(g[i].x, f.x, s[i][j]);
                s[i][j] = fmaf(g[i].y, f.y, s[i][j]);
                s[i][j] = fmaf(g[i].z, f.z, s[i][j]);
                s[i][j] = fmaf(g[i].w, f.w, s[i][j]);
            }
        }
    }
    // the warp's two pixel groups, then the warps in order
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 7; ++j) {
            const float v = s[i][j] + __shfl_xor_sync(0xffffffffu, s[i][j], 16);
            if (lane < 16) red[warp][(cq + 4 * i) * (kInK + 1) + 7 * fq + j] = v;
        }
    __syncthreads();
    for (int i = tid; i < kInPartial; i += blockDim.x) {
        float t = red[0][i];
#pragma unroll
        for (int k = 1; k < 8; ++k) t += red[k][i];
        partial[(size_t)blockIdx.x * kInPartial + i] = t;
    }
}

__global__ void __launch_bounds__(256) conv_in_wgrad_reduce_kernel(const float *__restrict__ partial, int blocks,
                                                                   float *__restrict__ dw1, float *__restrict__ db1) {
    int i;  // c * 28 + k
    float t;
    if (!sum_partials(partial, blocks, kInPartial, i, t)) return;
    const int c = i / (kInK + 1), k = i % (kInK + 1);
    if (k == kInK) db1[c] = t;
    else dw1[c * kInK + k] = t;
}

// ---------------------------------------------------------------------------
// Loss, head gradient and the gradient entering the last convolution
// ---------------------------------------------------------------------------
constexpr int kLossThreads = 256;
__global__ void __launch_bounds__(kLossThreads) loss_kernel(const float *__restrict__ out_m,
                                                            const float *__restrict__ depth_m,
                                                            const uint16_t *__restrict__ target,
                                                            const bf16 *__restrict__ d0,
                                                            const float *__restrict__ head_w, size_t npix, float inv,
                                                            bf16 *__restrict__ dz11, float *__restrict__ partial) {
    // per thread: loss, count, 16 head-weight sums, head-bias sum
    float acc[19];
#pragma unroll
    for (int k = 0; k < 19; ++k) acc[k] = 0.f;
    float hw[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) hw[c] = __ldg(head_w + c);
    for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += (size_t)gridDim.x * blockDim.x) {
        const float t = (float)target[p] * 0.001f;
        const bool m = depth_m[p] > 0.f && target[p] != 0;
        const float diff = out_m[p] - t;
        float dr = 0.f;
        if (m) {
            acc[0] += fabsf(diff) * inv;
            acc[1] += 1.f;
            // gradient with respect to the head output r (out = d + 0.01 r)
            dr = 0.01f * (diff > 0.f ? inv : diff < 0.f ? -inv : 0.f);
        }
        float f[16];
        unpack8(ldg16(d0 + p * 16), f);
        unpack8(ldg16(d0 + p * 16 + 8), f + 8);
        float g[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            acc[2 + c] = fmaf(dr, f[c], acc[2 + c]);
            g[c] = f[c] > 0.f ? dr * hw[c] : 0.f;
        }
        acc[18] += dr;
        uint4 *o = reinterpret_cast<uint4 *>(dz11 + p * 16);
        o[0] = pack8(g);
        o[1] = pack8(g + 8);
    }
    __shared__ float red[kLossThreads / 32][19];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 19; ++k) {
        float v = acc[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[warp][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < 19) {
        float v = 0.f;
        for (int w = 0; w < kLossThreads / 32; ++w) v += red[w][threadIdx.x];
        partial[(size_t)blockIdx.x * 19 + threadIdx.x] = v;
    }
}

// One block per reduced quantity; a fixed-shape tree over the block partials.
__global__ void loss_reduce_kernel(const float *__restrict__ partial, int blocks, float *__restrict__ dhead_w,
                                   float *__restrict__ dhead_b, double *__restrict__ loss2) {
    __shared__ double red[256];
    const int k = blockIdx.x;
    double t = 0.0;
    for (int b = threadIdx.x; b < blocks; b += blockDim.x) t += (double)partial[(size_t)b * 19 + k];
    red[threadIdx.x] = t;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (k < 2) loss2[k] = red[0];
        else if (k < 18) dhead_w[k - 2] = (float)red[0];
        else dhead_b[0] = (float)red[0];
    }
}

// ---------------------------------------------------------------------------
// Gradient routing through upsampling, pooling and skips
// ---------------------------------------------------------------------------
// A block takes kRouteThreads of the (pixel, 8 channels) items of one low-resolution
// row, a thread one of them with its four full-resolution pixels.  Memory bounds
// these kernels.  Of an interleaved gradient of two sources each kernel wants some
// 32-byte sectors of each pixel, and DRAM moves 64 bytes, so the largest lies in two
// planes.  Batch 16 of 640x480, that level: up_back 101 -> 73 us (470 MB),
// pool_back_add 121 -> 69 us (510 MB).
constexpr int kRouteThreads = 128;
struct LowPixel {
    int c, x, y, img;  // channel group, column, row, image
    size_t q;          // raster index over the images
};
__device__ __forceinline__ bool low_pixel(int hl, int wl, int cch, LowPixel &t) {
    const unsigned items = (unsigned)wl * (unsigned)cch, per_row = (items + kRouteThreads - 1) / kRouteThreads;
    const unsigned row = blockIdx.x / per_row, i = (blockIdx.x - row * per_row) * kRouteThreads + threadIdx.x;
    if (i >= items) return false;
    t.x = (int)(i / (unsigned)cch);
    t.c = (int)(i - (unsigned)t.x * (unsigned)cch);
    t.img = (int)(row / (unsigned)hl);
    t.y = (int)(row - (unsigned)t.img * (unsigned)hl);
    t.q = (size_t)row * wl + t.x;
    return true;
}

__global__ void __launch_bounds__(kRouteThreads) up_back_kernel(const bf16 *__restrict__ g, int cu, int ca,
                                                                const bf16 *__restrict__ y_low, bf16 *__restrict__ dz,
                                                                int h, int w) {
    const int hl = h >> 1, wl = w >> 1;
    LowPixel t;
    if (!low_pixel(hl, wl, ca >> 3, t)) return;
    const int c = t.c, xl = t.x, yl = t.y, img = t.img;
    const size_t q = t.q;
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int y = 2 * yl + (k >> 1), x = 2 * xl + (k & 1);
        float f[8];
        unpack8(ldg16(g + (((size_t)img * h + y) * w + x) * cu + 8 * c), f);
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] += f[j];
    }
    float mk[8];
    unpack8(ldg16(y_low + q * ca + 8 * c), mk);
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] = mk[j] > 0.f ? s[j] : 0.f;
    *reinterpret_cast<uint4 *>(dz + q * ca + 8 * c) = pack8(s);
}

__global__ void __launch_bounds__(kRouteThreads) pool_back_add_kernel(const bf16 *__restrict__ e,
                                                                      const bf16 *__restrict__ gp,
                                                                      const bf16 *__restrict__ skip, int cu, int ch,
                                                                      bf16 *__restrict__ dz, int h, int w) {
    const int hl = h >> 1, wl = w >> 1;
    LowPixel t;
    if (!low_pixel(hl, wl, ch >> 3, t)) return;
    const int c = t.c, xl = t.x, yl = t.y, img = t.img;
    const size_t q = t.q;
    float ev[4][8], mx[8];
    size_t pix[4];
    uint4 sk[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        pix[k] = ((size_t)img * h + 2 * yl + (k >> 1)) * w + 2 * xl + (k & 1);
        unpack8(ldg16(e + pix[k] * ch + 8 * c), ev[k]);
        sk[k] = ldg16(skip + pix[k] * cu + 8 * c);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) mx[j] = fmaxf(fmaxf(ev[0][j], ev[1][j]), fmaxf(ev[2][j], ev[3][j]));
    float gv[8];
    unpack8(ldg16(gp + q * ch + 8 * c), gv);
    int first[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) first[j] = ev[0][j] == mx[j] ? 0 : ev[1][j] == mx[j] ? 1 : ev[2][j] == mx[j] ? 2 : 3;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float s[8];
        unpack8(sk[k], s);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float v = s[j] + (first[j] == k ? gv[j] : 0.f);
            s[j] = ev[k][j] > 0.f ? v : 0.f;
        }
        *reinterpret_cast<uint4 *>(dz + pix[k] * ch + 8 * c) = pack8(s);
    }
}

// ---------------------------------------------------------------------------
// Optimiser and weight packing
// ---------------------------------------------------------------------------
__global__ void adamw_kernel(float *__restrict__ theta, const float *__restrict__ grad, float *__restrict__ m,
                             float *__restrict__ v, const uint8_t *__restrict__ decay, size_t count, float lr,
                             float b1, float b2, float eps, float wd, float bc1, float bc2) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float g = grad[i];
    const float mi = b1 * m[i] + (1.f - b1) * g;
    const float vi = b2 * v[i] + (1.f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float upd = (mi / bc1) / (sqrtf(vi / bc2) + eps);
    const float th = theta[i];
    theta[i] = th - lr * (upd + (decay[i] ? wd : 0.f) * th);
}

__global__ void pack_weights_kernel(const float *__restrict__ w, int cout, int cin, bf16 *__restrict__ wq,
                                    bf16 *__restrict__ wt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;  // i = (co * 9 + t) * cin + ci
    if (i >= cout * 9 * cin) return;
    const int ci = i % cin, t = (i / cin) % 9, co = i / (9 * cin);
    const bf16 q = __float2bfloat16_rn(w[i]);
    wq[i] = q;
    wt[((size_t)ci * 9 + (8 - t)) * cout + co] = q;
}

}  // namespace

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
static uint32_t smem_floor_for_tmem(uint32_t ncols) {
    // at most 512 / ncols blocks per SM may hold TMEM at once; a block asks
    // for enough shared memory that no more than that fit
    const uint32_t kmax = 512u / ncols;
    return kSmemPerSM / (kmax + 1) - 1024u + 16u;
}

int prepare_kernels() {
    // allow the largest dynamic shared memory a block may have, once, so that
    // launches (also inside stream capture) make no other runtime call
    std::vector<const void *> fns;
#define TDE_CONV_FN(M, A, B) \
    fns.push_back(conv_kernel_fn(M, A, B, false));
    TDE_CONV_VARIANTS(TDE_CONV_FN)
#undef TDE_CONV_FN
#define TDE_WG_FN(M, A, B, Z) fns.push_back((const void *)wgrad_tc_kernel<M, A, B, Z>);
    TDE_WG_VARIANTS(TDE_WG_FN)
#undef TDE_WG_FN
    for (int cca = 2; cca <= 6; cca += 2) fns.push_back(conv_kernel_fn(SRC_DIRECT, cca, 0, true));
    for (const void *fn : fns) {
        cudaFuncAttributes fa;
        TDE_CUDA(cudaFuncGetAttributes(&fa, fn), "refiner: kernel attributes");
        TDE_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(227 * 1024 - fa.sharedSizeBytes)),
                 "refiner: shared memory limit");
    }
    return TDE_OK;
}

int conv_plan(int mode, int ca, int cin, int cout, bool pool, ConvPlan *out) {
    // Two resident blocks per SM when the tensor memory, the registers and the
    // shared memory allow them at least kConvMinSlots input rows each, else
    // one; the ring takes as many rows (up to kConvMaxSlots) as then fit.  The
    // shared memory is padded so that no further block becomes resident.
    const void *fn = conv_kernel_fn(mode, ca / 8, (cin - ca) / 8, pool);
    if (!fn) return set_error(TDE_ERR_UNSUPPORTED, "refiner conv: no kernel for mode %d with %d + %d input channels", mode,
                              ca, cin - ca);
    cudaFuncAttributes fa;
    TDE_CUDA(cudaFuncGetAttributes(&fa, fn), "refiner: kernel attributes");
    const size_t shared = mode == SRC_UP ? (size_t)(ca / 8) * kPlaneBytes : 0;
    const size_t slot = (size_t)(cin / 8) * kPlaneBytes - shared;
    const int sets = conv_epi_sets(mode, pool), threads = conv_threads(sets);
    const size_t weights = (size_t)9 * (cin / 8) * cout * 16, stage = 4 * sets * conv_stage_bytes(cout, pool);
    size_t fixed = 0;
    auto need = [&](size_t S) { return S * slot + (shared ? (size_t)shared_slots((int)S) * shared : 0) + fixed; };
    const int by_tmem = (int)(512u / tmem_cols(kConvMinAcc * cout));
    const int by_regs = 65536 / (((fa.numRegs + 7) / 8) * 8 * threads);
    int bps = by_tmem < by_regs ? by_tmem : by_regs;
    bps = bps > kConvMaxPerSM ? kConvMaxPerSM : bps;
    for (; bps >= 1; --bps) {
        const size_t budget = kSmemPerSM / bps - 1024 - fa.sharedSizeBytes;
        fixed = weights + stage;
        out->staged = budget >= need(kConvMinSlots);
        if (!out->staged) fixed = weights;
        if (budget < need(kConvMinSlots)) continue;
        size_t S = kConvMinSlots;
        while (S < (size_t)kConvMaxSlots && need(S + 1) <= budget) ++S;
        size_t smem = need(S);
        const size_t floor = kSmemPerSM / (bps + 1) - 1024 - fa.sharedSizeBytes + 16;
        if (smem < floor) smem = floor;
        out->per_sm = bps;
        out->threads = threads;
        out->slots = (int)S;
        // as many accumulator rows as the block's share of tensor memory holds
        int acc = kConvMaxAcc;
        while (tmem_cols(acc * cout) * (uint32_t)bps > 512u) --acc;
        out->acc = acc;
        out->smem = smem;
        return TDE_OK;
    }
    return set_error(TDE_ERR_UNSUPPORTED, "refiner conv: cin=%d cout=%d does not fit an SM", cin, cout);
}

// Whether conv3x3_tc_kernel has an epilogue for these channels.
static bool epilogue_for(int mode, int cca, int ccb, int cout, bool pool) {
    if (mode == SRC_UP) return cout == 8 * ccb && !pool;
    if (pool) return cca < 8 && cout == 8 * cca;
    switch (cca) {
    case 2: return cout == 16 || cout == 32 || cout == 48;
    case 4: return cout == 16 || cout == 32 || cout == 48 || cout == 80;
    case 6: return cout == 32 || cout == 48 || cout == 64 || cout == 112;
    default: return cca == 8 && (cout == 48 || cout == 64);
    }
}

int launch_conv(const ConvArgs &a, const ConvPlan &plan, int num_sms, cudaStream_t s) {
    const int cin = a.ca + a.cb;
    if (a.split && a.split != conv_split(a.cout))
        return set_error(TDE_ERR_INVALID_ARG, "refiner conv: %d channels in planes of %d", a.cout, a.split);
    if (cin % 16 || a.ca % 8 || a.cout % 16 || a.cout < 16 || a.cout > 128 || cin > 128 || a.w <= 0 || a.h <= 0 ||
        a.n <= 0 || (a.head_w && a.cout != 16) || (a.mode_a == SRC_UP && (a.h % 2 || a.w % 2)) ||
        (a.pool_out && (a.h % 2 || a.w % 2 || a.mask)) ||
        !epilogue_for(a.mode_a, a.ca / 8, a.cb / 8, a.cout, a.pool_out != nullptr))
        return set_error(TDE_ERR_INVALID_ARG, "refiner conv: unsupported shape cin=%d cout=%d", cin, a.cout);
    if (plan.slots < kConvMinSlots || plan.slots > kConvMaxSlots || plan.per_sm < 1 || plan.smem > 227 * 1024 - 256 ||
        plan.acc < kConvMinAcc || plan.acc > kConvMaxAcc || tmem_cols(plan.acc * a.cout) * plan.per_sm > 512)
        return set_error(TDE_ERR_INVALID_ARG, "refiner conv: bad launch plan");
    // rows per block: as many as keep every resident block busy
    const int tiles_x = (a.w + kTileM - 1) / kTileM;
    const long row_tiles = (long)a.n * a.h * tiles_x;
    const long slots = (long)num_sms * plan.per_sm;
    // rows per strip: enough that the strips do not outnumber the resident
    // blocks (no second wave), even when the epilogue pools row pairs; with
    // more work than that (training batches), short strips that the resident
    // blocks take in turn, which balances their load better than long ones
    int rows = (int)((row_tiles + slots - 1) / slots);
    rows = rows < 1 ? 1 : rows > kStripRowsOneWave ? kStripRowsBalanced : rows;
    if (a.pool_out) rows += rows & 1;
    const long items = (long)a.n * tiles_x * ((a.h + rows - 1) / rows);
    const int grid = (int)(items < slots ? items : slots);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(plan.threads);
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const void *fn = conv_kernel_fn(a.mode_a, a.ca / 8, a.cb / 8, a.pool_out != nullptr);
    if (!fn) return set_error(TDE_ERR_UNSUPPORTED, "refiner conv: no kernel for mode %d with %d + %d input channels",
                              a.mode_a, a.ca, a.cb);
    int S = plan.slots, NA = plan.acc, staged = plan.staged;
    void *args[] = {(void *)&a, (void *)&rows, (void *)&S, (void *)&NA, (void *)&staged};
    cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
    if (e != cudaSuccess) return set_error(TDE_ERR_CUDA, "refiner conv: %s", cudaGetErrorString(e));
    return check_launch("refiner conv");
}

// One block per SM.  Two blocks of 64-pixel steps took as long (912 against
// 940 us for all layers at batch 16 of 640x480) with half as many additions into
// each accumulator; the sums then differ by 3e-5 of a gradient's norm from those
// of one block, which differ by 3e-6 from the per-tap form's.
int wgrad_blocks(int num_sms) { return num_sms; }

size_t wgrad_partial_floats(int blocks, int cin, int cout) { return (size_t)blocks * wg_partial(cin, cout); }

int launch_wgrad(const WgradArgs &a, int blocks, cudaStream_t s) {
    const int cin = a.ca + a.cb;
    const void *fn = wgrad_kernel_fn(a.mode_a, a.ca / 8, a.cb / 8, a.cout / 8);
    if (!fn) return set_error(TDE_ERR_UNSUPPORTED, "refiner wgrad: no kernel for mode %d with %d + %d input, %d output channels",
                              a.mode_a, a.ca, a.cb, a.cout);
    const int kp = wg_kp(cin / 8, a.cout / 8);
    if ((long)a.n * a.h * ((a.w + kp - 1) / kp) > 0x7fffffffL)
        return set_error(TDE_ERR_UNSUPPORTED, "refiner wgrad: %d images of %dx%d are too many", a.n, a.w, a.h);
    WgradArgs args = a;
    void *kargs[] = {(void *)&args};
    // never more blocks than fit in tensor memory: pad the shared memory
    size_t smem = wg_smem(cin / 8, a.cout / 8, kp, wg_flight(cin / 8, a.cout / 8));
    const size_t fl = smem_floor_for_tmem(tmem_cols(wg_mtiles(a.cout) * 3 * cin));
    if (smem < fl) smem = fl;
    cudaError_t e = cudaLaunchKernel(fn, dim3(blocks), dim3(kWgThreads), kargs, smem, s);
    if (e != cudaSuccess) return set_error(TDE_ERR_CUDA, "refiner wgrad: %s", cudaGetErrorString(e));
    return check_launch("refiner wgrad");
}

int launch_wait_selftest(uint64_t limit_ns, unsigned long long *out, cudaStream_t s) {
    wait_selftest_kernel<<<1, 32, 0, s>>>(limit_ns, out);
    return check_launch("wait selftest");
}

int launch_wgrad_reduce(const float *partial, int blocks, int cin, int cin_all, int ci0, int cout, float *dw, float *db,
                        cudaStream_t s) {
    wgrad_reduce_kernel<<<div_up(wg_partial(cin, cout), 32), 256, 0, s>>>(partial, blocks, cin, cin_all, ci0, cout, dw, db);
    return check_launch("refiner wgrad reduce");
}

int launch_conv_in(const uint16_t *raw, float *depth_m, const float *w1, const float *b1, bf16 *e0a, int n, int h,
                   int w, cudaStream_t s) {
    if (h % kInRows || w % 2) return set_error(TDE_ERR_INVALID_ARG, "refiner conv_in: %dx%d", w, h);
    const size_t items = (size_t)n * (h / kInRows) * w;
    if (items > 0x7fffff00u) return set_error(TDE_ERR_UNSUPPORTED, "refiner conv_in: %d images of %dx%d are too many", n, w, h);
    conv_in_kernel<<<(unsigned)((items + 127) / 128), 128, 0, s>>>(raw, depth_m, w1, b1, e0a, n, h, w);
    return check_launch("refiner conv_in");
}

int conv_in_wgrad_blocks(int num_sms, int n, int h, int w) {
    const size_t tiles = (size_t)n * h * ((w + kInTile - 1) / kInTile), resident = (size_t)num_sms * kInBlocksPerSM;
    return (int)(tiles < resident ? tiles : resident);
}

int launch_conv_in_wgrad(const float *depth_m, const bf16 *dz1, int n, int h, int w, float *partial, int blocks,
                         float *dw1, float *db1, cudaStream_t s) {
    conv_in_wgrad_kernel<<<blocks, 256, 0, s>>>(depth_m, dz1, n, h, w, partial);
    TDE_TRY(check_launch("refiner conv_in wgrad"));
    conv_in_wgrad_reduce_kernel<<<div_up(kInPartial, 32), 256, 0, s>>>(partial, blocks, dw1, db1);
    return check_launch("refiner conv_in wgrad reduce");
}

int loss_blocks(int n, int h, int w) {
    const size_t np = (size_t)n * h * w;
    size_t b = (np + kLossThreads * 8 - 1) / (kLossThreads * 8);
    return (int)(b < 1 ? 1 : b > 4096 ? 4096 : b);
}

int launch_loss(const float *out_m, const float *depth_m, const uint16_t *target, const bf16 *d0, const float *head_w,
                int n, int h, int w, bf16 *dz11, float *partial, int blocks, float *dhead_w, float *dhead_b,
                double *loss2, cudaStream_t s) {
    const size_t np = (size_t)n * h * w;
    loss_kernel<<<blocks, kLossThreads, 0, s>>>(out_m, depth_m, target, d0, head_w, np, 1.f / (float)np, dz11,
                                                partial);
    TDE_TRY(check_launch("refiner loss"));
    loss_reduce_kernel<<<19, 256, 0, s>>>(partial, blocks, dhead_w, dhead_b, loss2);
    return check_launch("refiner loss reduce");
}

int conv_planes(int cout) { return conv_split(cout); }

static unsigned route_blocks(int n, int hl, int wl, int cch) {
    return (unsigned)(n * hl) * div_up(wl * cch, kRouteThreads);
}

int launch_up_back(const bf16 *g, int cu, int ca, const bf16 *y_low, bf16 *dz, int n, int h, int w, cudaStream_t s) {
    up_back_kernel<<<route_blocks(n, h / 2, w / 2, ca / 8), kRouteThreads, 0, s>>>(g, cu, ca, y_low, dz, h, w);
    return check_launch("refiner up_back");
}

int launch_pool_back_add(const bf16 *e, const bf16 *gp, const bf16 *skip, int cu, int c, bf16 *dz, int n, int h, int w,
                         cudaStream_t s) {
    pool_back_add_kernel<<<route_blocks(n, h / 2, w / 2, c / 8), kRouteThreads, 0, s>>>(e, gp, skip, cu, c, dz, h, w);
    return check_launch("refiner pool_back_add");
}

int launch_adamw(float *theta, const float *grad, float *m, float *v, const uint8_t *decay_mask, size_t count,
                 float lr, float beta1, float beta2, float eps, float wd, float bc1, float bc2, cudaStream_t s) {
    adamw_kernel<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(theta, grad, m, v, decay_mask, count, lr, beta1,
                                                                 beta2, eps, wd, bc1, bc2);
    return check_launch("refiner adamw");
}

int launch_pack_weights(const float *w, int cout, int cin, bf16 *wq, bf16 *wt, cudaStream_t s) {
    const int n = cout * 9 * cin;
    pack_weights_kernel<<<div_up(n, 256), 256, 0, s>>>(w, cout, cin, wq, wt);
    return check_launch("refiner pack weights");
}

}  // namespace refiner
}  // namespace tde
