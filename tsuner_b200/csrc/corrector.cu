// corrector.cu -- learned corrector: a 6-layer, 32-channel 3x3 convolutional
// network that lifts coarse-grid maximum-depth / bed-change maps to the fine
// grid.  Its convolutions (forward, input gradient, weight gradient) run on
// the 5th-generation tensor cores (tcgen05.mma, BF16 operands from shared
// memory, FP32 accumulators in TMEM); the rest of the training loop
// (feature assembly, loss, Adam) is small elementwise kernels.
// No counterpart in the reference.
//
// Tensors: activations NHWC BF16 with 32 channels ([img][y][x][32]);
// weights BF16 Wk[cout][tap][cin], tap = (dy+1)*3 + (dx+1) (so that
// Y[y][x] = sum W[tap] X[y+dy][x+dx], zero padding); FP32 master weights,
// bias and Adam moments.
//
// Both convolution kernels read their shifted operands in place: a tile of
// pixels lies in shared memory as TMA writes it, one pixel's 32 channels per
// 64-byte row with the 64-byte swizzle, and an MMA operand is a start address
// and two strides into it (sdesc64).
//
// Forward / input-gradient convolution (conv3x3_fwd_kernel): implicit GEMM
// whose M = 128 rows are 16 groups of 8 pixels of one image row each and whose
// N = 96 columns are the contributions of an input row to the three output
// rows around it, 6 MMAs (3 column offsets x 2 channel halves, K = 16) per
// input row.  8 x 528^2 pixels, BF16 with ReLU: 103 -> 64 us from HBM (the 285
// MB it reads and writes take 44 us).
//
// Weight gradient (conv3x3_wgrad_kernel): dW[cout][tap][cin] =
//   sum_p dZ[p][cout] X[p + off(tap)][cin], a GEMM with the pixels as the
// reduction dimension; all nine taps in one MMA per 16 pixels (M = the three
// row offsets x cin, N = the three column offsets x cout).  8 x 528^2: kernel
// 100 -> 50 us, the call with its reduction 187 -> 74 us.  The bias gradient
// is summed from the dZ tile on the CUDA cores.
//
// Every mbarrier wait is bounded (globaltimer); on expiry the kernel sets
// the error word, waits once more (bounded) for its MMAs, frees its TMEM and
// returns.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

#include "hostio.h"
#include "async.cuh"
#include "tsuner_b200.h"

namespace tsu {
namespace corr {

typedef __nv_bfloat16 bf16;

constexpr int C = 32;        // channels
constexpr int kPix = C * 2;  // one pixel: 64 B, the span of the 64-byte swizzle
constexpr int KROWS = 9 * C; // 288

// forward (conv3x3_fwd_kernel)
constexpr int GX = 8, NG = 16;               // columns of a group, groups of a tile row (M = 128 pixels)
constexpr int GW = GX + 2;                   // columns loaded per group
constexpr int kCRows = 4;                    // input rows per chunk
constexpr int kGRow = GW * kPix;             // one group's row: 640 B
constexpr int kGrpBytes = kCRows * kGRow;    // 2560 B
constexpr int kChunk = NG * kGrpBytes;       // 40960 B
constexpr int kChunks = 2;                   // chunk ring
constexpr int kWBytes = 9 * 4 * 32 * 16;     // weights: 18432 B
constexpr int kWBlk = 96 * 16;               // one (dx, channel quarter): 3 dy x 32 cout rows of 16 B
constexpr int kAcc = 8;                      // TMEM accumulators (output rows) of 32 columns
constexpr int kEpiWarps = 8;
constexpr int kFwdCtas = 2;                  // CTAs per SM: one's issuing covers the other's
constexpr int kFwdThreads = 64 + 32 * kEpiWarps;
constexpr int kFwdBars = (2 * kChunks + 2 * kAcc + 1) * 8 + 32;
constexpr int kFwdSmem = 1024 + kWBytes + kChunks * kChunk + kFwdBars;
static_assert(kGrpBytes % 512 == 0 && kWBytes % 512 == 0, "swizzled TMA destinations");
static_assert(kFwdCtas * (kFwdSmem + 1024) <= 228 * 1024 && kFwdCtas * 32 * kAcc <= 512, "residency");

// weight gradient (conv3x3_wgrad_kernel)
constexpr int TYP = 16;                          // tile: 8 columns x 16 rows (K = 128 pixels)
constexpr int kXRow = GX * kPix;                 // 512 B
constexpr int kXBytes = (TYP + 2) * kXRow;       // 9216 B loaded
constexpr int kXBuf = (TYP + 3) * kXRow;         // + the row read by the ignored rows 96..127 of A
constexpr int kZBytes = TYP * kGRow;             // 10240 B
constexpr int kWgStage = kXBuf + kZBytes;        // 19968 B
constexpr int kWgStages = 8;
constexpr int kWgThreads = 192;
// tiles summed in TMEM before the sum moves to registers: the tensor cores add
// to an FP32 accumulator with truncation, whose bias grows with the number of
// additions.  Relative error of dW against 64 bits at 8 x 528^2 / 1 x 428 x 330:
// all of a CTA's tiles in one accumulator 1.4e-5, batches of 24 2.3e-6 /
// 6.3e-7, of 8 6.5e-7 / 6.3e-7, of 6 4.9e-7 / 4.3e-7 (592 CTAs with an
// accumulator each 3.2e-6 / 4.8e-7); 62-63 us warm for any of them
constexpr int kWgFlush = 6;
constexpr int kWgSmem = 1024 + kWgStages * kWgStage + (2 * kWgStages + 5) * 8 + 32;
static_assert(kXBuf % 512 == 0 && kWgStage % 512 == 0, "swizzled TMA destinations");
static_assert(kWgSmem + 1024 <= 228 * 1024, "one CTA per SM");

__device__ int g_corr_err;  // set by a kernel whose wait expired

// UMMA shared-memory descriptor, no swizzle, sm100 version field
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46);
}

// the same with the 64-byte swizzle.  K-major operands: rows of 64 B, sbo = the
// stride of 8-row groups (lbo unused).  MN-major operands: lbo = the stride of
// 32-element blocks along M or N, sbo = the stride of 8-row groups along K.
// The hardware swizzles the final shared-memory address (16-byte chunk index
// ^= address bits 7-8), as TMA does when it writes, so an operand may start
// at any pixel of a tile and its blocks may overlap: a convolution's shifted
// operands are start addresses and strides into one tile.
__device__ __forceinline__ uint64_t sdesc64(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return sdesc(addr, lbo, sbo) | ((uint64_t)4 << 61);
}

// kind::f16 instruction descriptor: D FP32, A/B BF16, majors, N, M
__host__ __device__ constexpr uint32_t idesc(int M, int N, int a_mn, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t id, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        :
        : "r"(tmem_d), "l"(da), "l"(db), "r"(id), "r"(accum)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
// true in one lane of a converged warp.  A role's loop runs in the whole warp,
// so that its counters and descriptors stay in uniform registers, which the
// MMA takes its operands from; only the issuing itself is one lane's.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// thread `lane` of the warp receives TMEM lane (base + lane), 32 columns
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&h);
}

// The forward kernel's work: the images' columns in groups of 8, 16 groups to
// a set (one tile row of a set is M = 128 pixels, of any images), and the sets'
// rows, numbered set by set, shared out evenly among the CTAs.  Where the images
// have no more than 8 groups in all and more than two rows for each of 148 SMs,
// their rows are cut into bands that lie side by side in the set, so that it is
// not mostly empty (1 x 1000 x 8: 9.3 -> 6.1 us, 1 x 1056 x 48: 9.5 -> 8.3; with
// two rows a CTA or fewer it only makes a CTA's work longer, 1 x 48 x 48: 5.2 -> 5.5).
struct FwdGeom {
    int ntx, bands, H;       // groups per image row, bands per image, rows of a band
    int groups, sets, rows;  // groups in all, sets, rows of all sets
    // group g: its image, first column and first row
    __host__ __device__ __forceinline__ void place(int g, int &img, int &x0, int &y0) const {
        img = g / (ntx * bands);
        const int r = g - img * ntx * bands, band = r / ntx;
        x0 = (r - band * ntx) * GX;
        y0 = band * H;
    }
};
__host__ __device__ inline FwdGeom fwd_geom(int nimg, int H, int W) {
    FwdGeom g;
    g.ntx = (W + GX - 1) / GX;
    g.bands = (nimg * g.ntx <= NG / 2 && H > 2 * 148) ? NG / (nimg * g.ntx) : 1;
    g.H = (H + g.bands - 1) / g.bands;
    g.groups = nimg * g.ntx * g.bands;
    g.sets = (g.groups + NG - 1) / NG;
    g.rows = g.sets * g.H;
    return g;
}

struct ConvArgs {
    const bf16 *X;
    int nimg, H, W;
    const bf16 *Wk;      // [cout][tap][cin]
    const float *bias;   // [32] or null
    int relu;            // apply max(., 0)
    const bf16 *gate;    // optional: zero output channel n where gate[p][n] <= 0
    bf16 *Ybf;           // BF16 output, or
    float *Yf;           // FP32 output, or
    float *Y2;           // FP32 output of channels 0 and 1 only, [pixel][2] (the corrector's last layer)
    int wide;            // output and gate lie on 32-byte boundaries
};

// A CTA's run of rows [b, e) of FwdGeom::rows, one segment (a range of rows of
// one set) at a time.
struct Segments {
    int H, at, end, set, y0, y1;
    __device__ __forceinline__ Segments(int H_, int rows, int cta, int nctas) : H(H_) {
        at = (int)((long long)rows * cta / nctas);
        end = (int)((long long)rows * (cta + 1) / nctas);
        set = y0 = y1 = 0;
    }
    __device__ __forceinline__ bool next() {
        if (at >= end) return false;
        set = at / H;
        y0 = at - set * H;
        y1 = min(H, y0 + (end - at));
        at += y1 - y0;
        return true;
    }
};

// 32 bytes of a pixel at once (the base 32-byte aligned), or as two halves
__device__ __forceinline__ void store32(void *p, const uint32_t (&v)[8], bool wide) {
    if (wide) {
        asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                     "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                     : "memory");
    } else {
        reinterpret_cast<uint4 *>(p)[0] = make_uint4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<uint4 *>(p)[1] = make_uint4(v[4], v[5], v[6], v[7]);
    }
}
__device__ __forceinline__ void load32(const void *p, uint32_t (&v)[8], bool wide) {
    if (wide) {
        asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                     : "l"(p));
    } else {
        const uint4 a = __ldg(reinterpret_cast<const uint4 *>(p)), b = __ldg(reinterpret_cast<const uint4 *>(p) + 1);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    }
}

// Epilogue of 32 pixels (4 groups of 8) of an output row: TMEM accumulators
// (lane = pixel, column = output channel) + bias, ReLU, optional gate, then
// the store of this lane's own pixel at element offset px (-1: outside the
// image).  A pixel's channels are whole 32-byte sectors, so each lane stores
// them itself, 32 bytes an instruction: staging them through shared memory
// for contiguous 512-byte stores took twice the instructions and was what the
// kernel waited for (8 x 528^2 with the gate: 95 us, now 78).
// g: the pixel's gate, requested before the accumulator was waited for.
__device__ __forceinline__ void conv_epilogue(const ConvArgs &a, uint32_t taddr, int lane, const float *sBias,
                                              const long long px, const uint32_t (&g)[2][8], uint64_t *release) {
    float acc[32];
    tmem_ld32(taddr, acc);
    fence_before();  // the accumulator is in registers: hand its TMEM columns back to the MMA issuer
    __syncwarp();
    if (lane == 0) mbar_arrive(release);
    if (px < 0) return;
    const float4 *b4 = reinterpret_cast<const float4 *>(sBias);
#pragma unroll
    for (int n = 0; n < 8; n++) {
        const float4 b = b4[n];
        acc[4 * n] += b.x;
        acc[4 * n + 1] += b.y;
        acc[4 * n + 2] += b.z;
        acc[4 * n + 3] += b.w;
    }
    if (a.relu) {
#pragma unroll
        for (int n = 0; n < 32; n++) acc[n] = fmaxf(acc[n], 0.f);
    }
    if (a.gate) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162 *>(&g[k][j]);
                if (!(__low2float(h) > 0.f)) acc[16 * k + 2 * j] = 0.f;
                if (!(__high2float(h) > 0.f)) acc[16 * k + 2 * j + 1] = 0.f;
            }
        }
    }
    if (a.Y2) {  // the two used channels: 8 B per pixel
        *reinterpret_cast<float2 *>(a.Y2 + px / C * 2) = make_float2(acc[0], acc[1]);
    } else if (a.Yf) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            uint32_t v[8];
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = __float_as_uint(acc[8 * k + j]);
            store32(a.Yf + px + 8 * k, v, a.wide);
        }
    } else {
#pragma unroll
        for (int k = 0; k < 2; k++) {
            uint32_t v[8];
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = pack2(acc[16 * k + 2 * j], acc[16 * k + 2 * j + 1]);
            store32(a.Ybf + px + 16 * k, v, a.wide);
        }
    }
}

// Forward convolution.  Persistent, two CTAs per SM; a CTA's rows come in
// segments.
//   warp 0: input rows of the segment, kCRows at a time: lane i loads group i's
//     box (10 columns x 4 rows x 32 channels) into the chunk ring;
//   warp 1 (lane 0): for each input row r, the MMAs A_dx,h[128 x 16] .
//     B_dx,h[16 x 96] of the 3 column offsets and 2 channel halves: N = 96 are
//     the contributions to output rows r - 1, r, r + 1, whose accumulators are
//     neighbours in a ring of kAcc TMEM column blocks.  An output row thus
//     collects its taps in the order (dy, dx, half).  The first MMA of a row's
//     first input overwrites (N = 32 of its own); at a segment's ends and
//     where the ring wraps N is 32 or 64;
//   warps 2-9: epilogue, a quarter of the pixels of every other output row.
// What bounded the one-tap form (18 MMAs of N = 32 per 128 pixels, the patch
// as four 16-byte channel planes): each MMA reads 4 KB of A for 131 kFLOP, and
// TMA writes 16 bytes at a time.  Here 6-7 MMAs read A once for three taps,
// and a TMA row is a pixel's 64 bytes.  No role waits at a CTA barrier inside
// its loop.  Every wait is bounded; a role whose wait expires sets the error
// word and leaves its loop, the others' waits then expire in turn, and before
// TMEM is freed the issued MMAs and loads are waited for.
__global__ void __launch_bounds__(kFwdThreads, kFwdCtas)
    conv3x3_fwd_kernel(const __grid_constant__ ConvArgs a, const __grid_constant__ CUtensorMap tmX) {
    extern __shared__ unsigned char sm_raw[];
    unsigned char *sm = smem_align<1024>(sm_raw);
    unsigned char *sW = sm;
    unsigned char *sP = sm + kWBytes;                  // chunk ring
    uint64_t *full = reinterpret_cast<uint64_t *>(sP + kChunks * kChunk);  // [kChunks] chunk landed
    uint64_t *empty = full + kChunks;                                      // [kChunks] chunk's MMAs done
    uint64_t *accf = empty + kChunks;                                      // [kAcc] accumulator ready
    uint64_t *acce = accf + kAcc;                                          // [kAcc] accumulator read
    uint64_t *fin = acce + kAcc;                                           // all MMAs done
    uint32_t *tslot = reinterpret_cast<uint32_t *>(fin + 1);
    int *sCount = reinterpret_cast<int *>(tslot + 1);  // [0] chunks issued, [1] chunks waited for
    __shared__ __align__(16) float sBias[32];
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const FwdGeom G = fwd_geom(a.nimg, a.H, a.W);

    // warp 0: input rows r .. r + kCRows - 1 of the segment into chunk slot b
    Segments seg(G.H, G.rows, blockIdx.x, gridDim.x);
    auto load_chunk = [&](const Segments &s, int r, int b) {
        const int ng = min(NG, G.groups - s.set * NG);
        int img, x0, y0;
        G.place(s.set * NG + lane, img, x0, y0);
        if (lane == 0) mbar_expect_tx(&full[b], ng * kGrpBytes);
        __syncwarp();
        if (lane < ng) tma_load_4d(sP + b * kChunk + lane * kGrpBytes, &tmX, 0, x0 - 1, y0 + r, img, &full[b]);
    };
    if (warp == 0) {
        // the barriers and the first chunk before anything else: it travels while
        // the weights and the TMEM are fetched (1 x 48 x 48: 7.1 -> 6.6 us)
        if (lane == 0) {
            for (int k = 0; k < kChunks; k++) {
                mbar_init(&full[k], 1);
                mbar_init(&empty[k], 1);
            }
            for (int k = 0; k < kAcc; k++) {
                mbar_init(&accf[k], 1);
                mbar_init(&acce[k], 4);  // one arrival per lane quarter
            }
            mbar_init(fin, 1);
            sCount[0] = sCount[1] = 0;
            mbar_init_fence();
        }
        __syncwarp();
        Segments first = seg;
        if (first.next()) load_chunk(first, first.y0 - 1, 0);
    }
    // weights -> [dx][quarter][dy = +1, 0, -1][cout] rows of 16 B (K-major B operand, no swizzle)
    for (int c = tid; c < 32 * 36; c += kFwdThreads) {
        const int n = c / 36, r = c - n * 36, tap = r >> 2, q = r & 3;
        const int dy = tap / 3, dx = tap - dy * 3;
        cp_async16(sW + (dx * 4 + q) * kWBlk + ((2 - dy) * 32 + n) * 16, a.Wk + n * KROWS + r * 8, 16);
    }
    cp_async_commit();
    if (tid < 32) sBias[tid] = a.bias ? a.bias[tid] : 0.f;
    if (warp == 1) tmem_alloc(tslot, 32 * kAcc);
    cp_async_wait_all();
    fence_async_smem();  // the weights, written by cp.async, are read by the MMAs (async proxy)
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tslot;

    if (warp == 0) {
        int c = 0;  // chunks issued
        bool ok = true;
        while (ok && seg.next()) {
            for (int r = seg.y0 - 1; r <= seg.y1 && ok; r += kCRows, c++) {
                if (c == 0) continue;  // on its way
                const int b = c % kChunks;
                if (c >= kChunks) ok = mbar_wait_first(&empty[b], ((c / kChunks) - 1) & 1);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                load_chunk(seg, r, b);
            }
        }
        if (lane == 0) {
            if (!ok) atomicExch(&g_corr_err, 1);
            sCount[0] = c;
        }
    } else if (warp == 1) {
        const uint64_t db0 = sdesc(smem_u32(sW), kWBlk, 128);
        const uint64_t dp0 = sdesc64(smem_u32(sP), 16, kGrpBytes);  // an address is the descriptor's low bits
        int cb = -1, chunks = 0;  // current chunk's ring slot, chunks waited for
        unsigned cph = 1;         // parity of the current pass over the chunk ring
        int sh = 0;               // accumulator slot of the next fresh output row
        unsigned aph = 1;         // parity of a read accumulator on this pass (1 at first: a fresh barrier)
        bool ok = true;
        while (ok && seg.next()) {
            int in = kCRows;  // row of the current chunk
            for (int r = seg.y0 - 1; r <= seg.y1; r++, in++) {
                if (in == kCRows) {
                    in = 0;
                    cb = (cb == kChunks - 1) ? 0 : cb + 1;
                    if (cb == 0) cph ^= 1;
                    ok = mbar_wait_first(&full[cb], cph);
                    if (__any_sync(0xffffffffu, !ok)) {
                        ok = false;
                        break;
                    }
                    chunks++;
                }
                // output rows lo .. hi take part; hi is fresh (no contribution yet) if it is r + 1
                const int lo = max(r - 1, seg.y0), hi = min(r + 1, seg.y1 - 1), nl = hi - lo + 1;
                const bool fresh = hi == r + 1;
                const int sl = (sh - (fresh ? nl - 1 : nl)) & (kAcc - 1);  // slot of lo
                if (fresh) {
                    ok = mbar_wait_first(&acce[sh], aph);
                    if (__any_sync(0xffffffffu, !ok)) {
                        ok = false;
                        break;
                    }
                    sh = (sh + 1) & (kAcc - 1);
                    if (sh == 0) aph ^= 1;
                }
                fence_after();
                const uint64_t da0 = dp0 + (uint64_t)(uint32_t)((cb * kChunk + in * kGRow) >> 4);
                // outputs lo + [i, j) of this input row, whose accumulators
                // start at slot s; dx, h: column offset and channel half; blk:
                // lo's block of the weights
                auto mma = [&](int blk, int dx, int h, int i, int j, int s, uint32_t acc) {
                    mma_bf16(tmem + (uint32_t)(s * 32), da0 + (uint64_t)((dx * kPix + h * 32) >> 4),
                             db0 + (uint64_t)(((dx * 4 + 2 * h) * kWBlk + (blk + i) * 512) >> 4),
                             idesc(128, 32 * (j - i), 0, 0), acc);
                };
                if (elect_one()) {
                    // the usual cases straight: the issuing lane's instructions
                    // are what the tensor pipe waits for
                    if (fresh && nl == 3 && sl <= kAcc - 3) {
                        mma(0, 0, 0, 0, 2, sl, 1u);
                        mma(0, 0, 0, 2, 3, sl + 2, 0u);
#pragma unroll
                        for (int t = 1; t < 6; t++) mma(0, t >> 1, t & 1, 0, 3, sl, 1u);
                    } else if (fresh && nl == 3 && sl == kAcc - 2) {
#pragma unroll
                        for (int t = 0; t < 6; t++) {
                            mma(0, t >> 1, t & 1, 0, 2, sl, 1u);
                            mma(0, t >> 1, t & 1, 2, 3, 0, t ? 1u : 0u);
                        }
                    } else if (fresh && nl == 3) {
                        mma(0, 0, 0, 0, 1, sl, 1u);
                        mma(0, 0, 0, 1, 2, 0, 1u);
                        mma(0, 0, 0, 2, 3, 1, 0u);
#pragma unroll
                        for (int t = 1; t < 6; t++) {
                            mma(0, t >> 1, t & 1, 0, 1, sl, 1u);
                            mma(0, t >> 1, t & 1, 1, 3, 0, 1u);
                        }
                    } else if (nl == 1) {  // a segment's first and last rows (straight too: 6.6 -> 5.2 us)
                        const int blk = lo - (r - 1);
#pragma unroll
                        for (int t = 0; t < 6; t++) mma(blk, t >> 1, t & 1, 0, 1, sl, (fresh && t == 0) ? 0u : 1u);
                    } else if (nl == 2 && sl <= kAcc - 2) {  // its second and last but one
                        const int blk = lo - (r - 1);
                        if (fresh) {
                            mma(blk, 0, 0, 0, 1, sl, 1u);
                            mma(blk, 0, 0, 1, 2, sl + 1, 0u);
                        } else {
                            mma(blk, 0, 0, 0, 2, sl, 1u);
                        }
#pragma unroll
                        for (int t = 1; t < 6; t++) mma(blk, t >> 1, t & 1, 0, 2, sl, 1u);
                    } else {  // the same at the ring's end: row by row
                        const int blk = lo - (r - 1);
#pragma unroll 1
                        for (int t = 0; t < 6; t++)
#pragma unroll 1
                            for (int i = 0; i < nl; i++)
                                mma(blk, t >> 1, t & 1, i, i + 1, (sl + i) & (kAcc - 1),
                                    (fresh && t == 0 && i == nl - 1) ? 0u : 1u);
                    }
                    if (in == kCRows - 1 || r == seg.y1) mma_commit(&empty[cb]);
                    if (r - 1 >= seg.y0) mma_commit(&accf[sl]);  // output row r - 1 is complete
                }
                __syncwarp();
            }
        }
        if (elect_one()) {
            if (!ok) atomicExch(&g_corr_err, 1);
            sCount[1] = chunks;
            mma_commit(fin);
            mbar_wait(fin, 0);
        }
    } else {
        const int q = warp & 3;                  // TMEM lane quarter this warp may read
        const int par = (warp - 2) >> 2;         // output rows this warp takes: k % (kEpiWarps / 4)
        int k = 0;
        bool ok = true;
        while (ok && seg.next()) {
            // this lane's pixel of groups 4 q .. 4 q + 3 of the set
            const int g = seg.set * NG + 4 * q + (lane >> 3);
            int img, x, top;
            G.place(g, img, x, top);
            x += lane & 7;
            const int rows = (g < G.groups && x < a.W) ? a.H - top : 0;  // of its image from the band's first
            const long long p0 = (((long long)img * a.H + top) * a.W + x) * C;
            for (int y = seg.y0; y < seg.y1; y++, k++) {
                if (k % (kEpiWarps / 4) != par) continue;
                const int ac = k % kAcc;
                const long long px = y < rows ? p0 + (long long)y * a.W * C : -1;
                uint32_t g[2][8];
                if (a.gate && px >= 0) {  // on its way while the MMAs run
                    load32(a.gate + px, g[0], a.wide);
                    load32(a.gate + px + 16, g[1], a.wide);
                }
                // every lane waits; the warp leaves together if any lane's wait
                // expired (the TMEM load below is a warp-wide instruction)
                ok = mbar_wait_first(&accf[ac], (k / kAcc) & 1);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                fence_after();
                conv_epilogue(a, tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(ac * 32), lane, sBias, px, g,
                              &acce[ac]);
            }
        }
        if (!ok && lane == 0) atomicExch(&g_corr_err, 1);
    }
    __syncwarp();
    fence_before();
    __syncthreads();
    if (tid == 0) {  // chunks issued but never waited for (an expired wait): let them land
        for (int c = sCount[1]; c < sCount[0]; c++) mbar_wait(&full[c % kChunks], (c / kChunks) & 1);
    }
    __syncthreads();
    fence_after();
    if (warp == 1) tmem_dealloc(tmem, 32 * kAcc);
}

struct TileGeom {
    int ntx, nty, per_img, total;
};
__host__ __device__ inline TileGeom tile_geom(int nimg, int H, int W) {
    TileGeom g;
    g.ntx = (W + GX - 1) / GX;
    g.nty = (H + TYP - 1) / TYP;
    g.per_img = g.ntx * g.nty;
    g.total = nimg * g.per_img;
    return g;
}

// Weight (and bias) gradient partials of this CTA's tiles, written to its row
// of `part` ([gridDim.x][kWgPart]: dW[cout][288], then the 4 warps' bias sums
// [4][32], then whether one of them is not finite); wgrad_reduce_kernel adds the rows to dW and db in a fixed order, so
// the gradient does not depend on which CTA finishes first.
//   warp 0: tile k (8 x 16 pixels) of X with one row of halo above and below,
//     and of dZ with one column left and right, into a ring of kWgStages;
//   warp 1 (lane 0): per 16 pixels (two tile rows) one MMA of
//     D[dy * 32 + cin (+ 32 ignored rows)][j * 32 + cout], j = 1 - dx:
//     A = X shifted by dy rows (blocks one tile row apart), B = dZ shifted by j
//     columns (blocks one pixel apart: overlapping windows of the same tile).
//     X[p'] dZ[p' - dx] summed over p' is the tap's gradient: both operands
//     are zero outside the image;
//   warps 2-5: the bias gradient on the CUDA cores, a pixel per thread.
constexpr int kWgFlags = 32 * KROWS + 4 * 32;
constexpr int kWgPart = kWgFlags + 32;  // rows of whole 128-byte lines
__global__ void __launch_bounds__(kWgThreads, 1)
    conv3x3_wgrad_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmZ, int nimg,
                         int H, int W, float *__restrict__ part) {
    extern __shared__ unsigned char sm_raw[];
    unsigned char *sm = smem_align<1024>(sm_raw);
    uint64_t *full = reinterpret_cast<uint64_t *>(sm + kWgStages * kWgStage);  // [kWgStages] stage loaded
    uint64_t *empty = full + kWgStages;  // [kWgStages] stage's MMAs and bias sums done
    uint64_t *accf = empty + kWgStages;  // [2] accumulator set's batch summed
    uint64_t *acce = accf + 2;           // [2] accumulator set read
    uint64_t *fin = acce + 2;            // all MMAs done
    uint32_t *tslot = reinterpret_cast<uint32_t *>(fin + 1);
    int *sCount = reinterpret_cast<int *>(tslot + 1);  // [0] stages issued, [1] stages waited for by the MMA warp
    int *sFail = sCount + 2, *sOdd = sCount + 3;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const TileGeom G = tile_geom(nimg, H, W);
    const int ntile = (int)blockIdx.x < G.total ? (G.total - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

    if (tid == 0) {
        for (int k = 0; k < 2; k++) {
            mbar_init(&accf[k], 1);
            mbar_init(&acce[k], 4);
        }
        for (int k = 0; k < kWgStages; k++) {
            mbar_init(&full[k], 1);
            mbar_init(&empty[k], 5);  // the MMAs and four bias warps
        }
        mbar_init(fin, 1);
        sCount[0] = sCount[1] = 0;
        *sFail = *sOdd = 0;
        mbar_init_fence();
    }
    // TMEM is taken only now: a grid that holds some while it waits could starve
    // the one it waits for, if that one lets it start before it has its own
    prior_grids_done();
    if (warp == 1) tmem_alloc(tslot, 256);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tslot;
    next_grid_may_start();
    float db[32];      // bias gradient of this thread's pixels
    float sum[3][32];  // this lane's row of D (j, cout), summed over the batches
#pragma unroll
    for (int n = 0; n < 32; n++) db[n] = sum[0][n] = sum[1][n] = sum[2][n] = 0.f;

    if (warp == 0) {
        if (lane == 0) {
            int k = 0;
            for (; k < ntile; k++) {
                const int b = k % kWgStages;
                if (k >= kWgStages && !mbar_wait_first(&empty[b], ((k / kWgStages) - 1) & 1)) {
                    atomicExch(sFail, 1);
                    break;
                }
                const int t = (int)blockIdx.x + k * (int)gridDim.x;
                const int img = t / G.per_img, r = t - img * G.per_img;
                const int tyi = r / G.ntx, x0 = (r - tyi * G.ntx) * GX, y0 = tyi * TYP;
                unsigned char *stg = sm + b * kWgStage;
                mbar_expect_tx(&full[b], kXBytes + kZBytes);
                tma_load_4d(stg, &tmX, 0, x0, y0 - 1, img, &full[b]);
                tma_load_4d(stg + kXBuf, &tmZ, 0, x0 - 1, y0, img, &full[b]);
            }
            sCount[0] = k;
        }
    } else if (warp == 1) {
        const uint32_t id = idesc(128, 96, 1, 1);
        const uint64_t dx0 = sdesc64(smem_u32(sm), kXRow, kXRow);  // an address is the descriptor's low bits
        const uint64_t dz0 = sdesc64(smem_u32(sm) + kXBuf, kPix, kGRow);
        int b = 0, first = 0, f = 0, k = 0;  // ring slot; tile of the batch, batch; tile
        unsigned ph = 0;
        bool ok = true;
        for (; k < ntile; k++) {
            ok = mbar_wait_first(&full[b], ph);
            if (first == 0 && f >= 2) ok &= mbar_wait_first(&acce[f & 1], ((f >> 1) - 1) & 1);
            if (__any_sync(0xffffffffu, !ok)) break;
            fence_after();
            const uint64_t st = (uint64_t)(uint32_t)((b * kWgStage) >> 4), da = dx0 + st, dz = dz0 + st;
            const uint32_t d = tmem + (uint32_t)((f & 1) * 128);
            if (elect_one()) {
                mma_bf16(d, da, dz, id, first ? 1u : 0u);
#pragma unroll
                for (int s = 1; s < TYP / 2; s++)
                    mma_bf16(d, da + (uint64_t)((2 * s * kXRow) >> 4), dz + (uint64_t)((2 * s * kGRow) >> 4), id, 1u);
                mma_commit(&empty[b]);
                if (first == kWgFlush - 1 || k == ntile - 1) mma_commit(&accf[f & 1]);
            }
            __syncwarp();
            if (++b == kWgStages) {
                b = 0;
                ph ^= 1;
            }
            if (++first == kWgFlush) {
                first = 0;
                f++;
            }
        }
        if (elect_one()) {
            if (k < ntile) atomicExch(sFail, 1);
            sCount[1] = k;
            mma_commit(fin);
            mbar_wait(fin, 0);
        }
    } else {
        const int p = tid - 64;  // pixel of the tile: 8 per row
        const uint32_t off = (p >> 3) * kGRow + ((p & 7) + 1) * kPix;
        const int dy = warp & 3;  // TMEM lanes 32 dy ..: rows dy * 32 + cin; dy = 3 is ignored
        // adds batch f's accumulators to `sum` and hands them back
        auto flush = [&](int f) {
            const bool ok = mbar_wait_first(&accf[f & 1], (f >> 1) & 1);
            if (__any_sync(0xffffffffu, !ok)) return false;
            fence_after();
            if (dy < 3) {
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    float v[32];
                    tmem_ld32(tmem + ((uint32_t)(dy * 32) << 16) + (uint32_t)((f & 1) * 128 + j * 32), v);
#pragma unroll
                    for (int n = 0; n < 32; n++) sum[j][n] += v[n];
                }
            }
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acce[f & 1]);
            return true;
        };
        int flushed = 0;  // batches
        bool good = true;
        for (int k = 0; k < ntile; k++) {
            const int b = k % kWgStages;
            // the batch before this one's, once the MMAs are well into this one
            if (k >= flushed * kWgFlush + kWgFlush + kWgFlush / 2) good = flush(flushed++);
            const bool ok = good && mbar_wait_first(&full[b], (k / kWgStages) & 1);
            if (__any_sync(0xffffffffu, !ok)) {
                if (lane == 0) atomicExch(sFail, 1);
                good = false;
                break;
            }
            const unsigned char *z = sm + b * kWgStage + kXBuf + off;
            const uint32_t swz = (smem_u32(z) >> 7) & 3;
            uint4 v[4];
#pragma unroll
            for (int c = 0; c < 4; c++) v[c] = *reinterpret_cast<const uint4 *>(z + ((c ^ swz) << 4));
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const uint32_t w[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162 *>(&w[j]);
                    db[8 * c + 2 * j] += __low2float(h);
                    db[8 * c + 2 * j + 1] += __high2float(h);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[b]);
        }
        while (good && flushed * kWgFlush < ntile) good = flush(flushed++);
        if (!good && lane == 0) atomicExch(sFail, 1);
    }
    __syncwarp();
    fence_before();
    __syncthreads();
    if (tid == 0) {
        if (*sFail) atomicExch(&g_corr_err, 1);
        // stages issued but never waited for (an expired wait): let them land
        for (int k = sCount[1]; k < sCount[0]; k++) mbar_wait(&full[k % kWgStages], (k / kWgStages) & 1);
    }
    __syncthreads();
    fence_after();
    float *prow = part + (size_t)blockIdx.x * kWgPart;
    if (*sFail || ntile == 0) {  // no partials from this CTA
        for (int k = tid; k < kWgPart; k += kWgThreads) prow[k] = 0.f;
    } else if (warp >= 2) {
        const int dy = warp & 3;
        if (dy < 3) {
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const int m = (dy * 3 + 2 - j) * 32 + lane;  // tap * 32 + cin
#pragma unroll
                for (int n = 0; n < 32; n++) prow[n * KROWS + m] = sum[j][n];
            }
        }
        float mine = 0.f;  // channel `lane` summed over the warp's 32 pixels
#pragma unroll
        for (int n = 0; n < 32; n++) {
            float v = db[n];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == n) mine = v;
        }
        prow[32 * KROWS + (warp - 2) * 32 + lane] = mine;
        if (!isfinite(mine)) atomicExch(sOdd, 1);
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (tid == 0) prow[kWgFlags] = *sOdd ? 1.f : 0.f;
    if (warp == 1) tmem_dealloc(tmem, 256);
}

// ---------------------------------------------------------------- training
// Feature scales (metres per unit)
constexpr float kSh = 2.0f;    // maximum depth
constexpr float kSb = 0.05f;   // bed change
constexpr float kSH = 50.0f;   // bathymetry
constexpr float kSdH = 2.0f;   // sub-grid bathymetry detail

// bilinear sample of a coarse [hc][wc] plane at fine cell (x, y), factor f,
// cell-centred, clamped at the edges
__device__ __forceinline__ float up_bilinear(const float *__restrict__ p, int hc, int wc, int f, int x, int y) {
    const float cx = (x + 0.5f) / f - 0.5f, cy = (y + 0.5f) / f - 0.5f;
    const float fx = fminf(fmaxf(cx, 0.f), (float)(wc - 1)), fy = fminf(fmaxf(cy, 0.f), (float)(hc - 1));
    const int x0 = min((int)fx, wc - 1), y0 = min((int)fy, hc - 1);
    const int x1 = min(x0 + 1, wc - 1), y1 = min(y0 + 1, hc - 1);
    const float ax = fx - x0, ay = fy - y0;
    const float a = p[y0 * wc + x0], b = p[y0 * wc + x1], c = p[y1 * wc + x0], d = p[y1 * wc + x1];
    // the fused operations spelled out, so that the maps do not depend on what
    // the compiler contracts in which kernel
    const float lo = __fmaf_rn(ax, b, __fmul_rn(1.f - ax, a)), hi = __fmaf_rn(ax, d, __fmul_rn(1.f - ax, c));
    return __fmaf_rn(1.f - ay, lo, __fmul_rn(ay, hi));
}

// The network runs on a canvas padded by kPad pixels on each side: a
// padded pixel holds the features of the nearest fine cell (edge
// replication), so that no fine cell is within the 6-layer network's
// receptive radius (6 pixels) of the convolutions' zero padding, which would
// otherwise read as dry, flat land at the image border.  Targets and the
// loss cover the fine cells only.
constexpr int kPad = 8;

struct Canvas {
    int H, W, Hp, Wp;  // fine image, padded canvas
};
__host__ __device__ inline Canvas canvas(int H, int W) { return Canvas{H, W, H + 2 * kPad, W + 2 * kPad}; }
// padded pixel (xp, yp) -> its fine cell (x, y); true if it is that cell
__device__ __forceinline__ bool unpad(const Canvas &cv, int xp, int yp, int &x, int &y) {
    x = min(max(xp - kPad, 0), cv.W - 1);
    y = min(max(yp - kPad, 0), cv.H - 1);
    return x == xp - kPad && y == yp - kPad;
}

// Builds the 32-channel BF16 input of sample idx[b] on the padded canvas
// and, when targets are requested, the normalised residual targets
// T[b][pp][2] (0 outside the fine image); base[b][pp][2] = the interpolated
// coarse maps.
//   coarse: [nsamples][3][hc*wc] = maximum depth, bed change, bathymetry H
//   fineT:  [nsamples][2][H*W]   = maximum depth, bed change (or null)
// A warp's unit is 32 consecutive pixels of a canvas row; their 64-byte records
// are written as four runs of 512 contiguous bytes (chunk 0 of a pixel holds
// its 8 features, the others are zeros).
// 8 x 528^2: 62 -> 47 us, the loss below 44 -> 29 us (a pixel's 64 B per lane
// and 64-bit divisions per pixel before).
__device__ __forceinline__ void put_pixels32(bf16 *row, int xp0, int Wp, uint4 mine) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int from = i * 8 + (lane >> 2);
        uint4 v;
        v.x = __shfl_sync(0xffffffffu, mine.x, from);
        v.y = __shfl_sync(0xffffffffu, mine.y, from);
        v.z = __shfl_sync(0xffffffffu, mine.z, from);
        v.w = __shfl_sync(0xffffffffu, mine.w, from);
        if (lane & 3) v = make_uint4(0, 0, 0, 0);
        if (xp0 + from < Wp) reinterpret_cast<uint4 *>(row + (size_t)(xp0 + from) * C)[lane & 3] = v;
    }
}
// the units of nb canvases, one warp after another
struct Units {
    int segs, total;  // units per canvas row, units
};
__host__ __device__ inline Units units(const Canvas &cv, int nb) {
    const int segs = (cv.Wp + 31) / 32;
    return Units{segs, nb * cv.Hp * segs};
}
__global__ void __launch_bounds__(256)
    features_kernel(const int *__restrict__ idx, int nb, const float *__restrict__ coarse, const float *__restrict__ fineT,
                    const float *__restrict__ Hf, Canvas cv, int hc, int wc, int f, bf16 *__restrict__ X0,
                    float *__restrict__ T, float *__restrict__ base) {
    const long long npix = (long long)cv.H * cv.W;
    const Units U = units(cv, nb);
    for (int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < U.total; u += gridDim.x * blockDim.x >> 5) {
        const int r = u / U.segs, b = r / cv.Hp, yp = r - b * cv.Hp;
        const int xp = (u - r * U.segs) * 32 + (threadIdx.x & 31);
        const long long row = (long long)r * cv.Wp;
        uint4 mine = make_uint4(0, 0, 0, 0);
        if (xp < cv.Wp) {
            int x, y;
            const bool inside = unpad(cv, xp, yp, x, y);
            const long long p = (long long)y * cv.W + x;
            const int s = idx[b];
            const float *cs = coarse + (long long)s * 3 * hc * wc;
            const float hm = up_bilinear(cs, hc, wc, f, x, y);
            const float dbv = up_bilinear(cs + hc * wc, hc, wc, f, x, y);
            const float Hc = up_bilinear(cs + 2 * hc * wc, hc, wc, f, x, y);
            const float Hfine = Hf[p];
            const int xi = min(x / f, wc - 1), yi = min(y / f, hc - 1);  // coarse cell containing the fine cell
            const float wet = cs[yi * wc + xi] > 0.f ? 1.f : 0.f;
            // channel 5 is 1 everywhere (a bias input); 6 and 7 locate the cell
            // (the source enters through the west boundary)
            const float v[8] = {hm / kSh, dbv / kSb, Hfine / kSH, (Hfine - Hc) / kSdH, wet, 1.f,
                                (float)x / (float)max(cv.W - 1, 1), (float)y / (float)max(cv.H - 1, 1)};
            mine = make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
            if (base) reinterpret_cast<float2 *>(base)[row + xp] = make_float2(hm, dbv);
            if (T && fineT) {
                const float *ft = fineT + (long long)s * 2 * npix;
                reinterpret_cast<float2 *>(T)[row + xp] =
                    inside ? make_float2((ft[p] - hm) / kSh, (ft[npix + p] - dbv) / kSb) : make_float2(0.f, 0.f);
            }
        }
        put_pixels32(X0 + row * C, xp & ~31, cv.Wp, mine);
    }
}

// Mean-square loss over the 2 output channels of the fine cells, each
// cell's maximum-depth term weighted by 1 + wbig * T^2 (T: the normalised
// residual target), so that the few large residuals at run-up fronts weigh
// more than their share of cells; dY = d(loss)/d(output) in BF16 (channels
// 2..31 and the padding zero); loss sum accumulated in FP64.
__global__ void __launch_bounds__(256)
    loss_kernel(const float *__restrict__ Y, const float *__restrict__ T, int nb, Canvas cv, float wbig,
                bf16 *__restrict__ dY, double *__restrict__ loss) {
    __shared__ double sred[8];
    const float scale = 1.f / (float)((long long)nb * cv.H * cv.W);  // d/dy of sum(w d^2) / (2 cells)
    const Units U = units(cv, nb);
    double acc = 0.0;
    for (int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < U.total; u += gridDim.x * blockDim.x >> 5) {
        const int r = u / U.segs, yp = r % cv.Hp;
        const int xp = (u - r * U.segs) * 32 + (threadIdx.x & 31);
        const long long row = (long long)r * cv.Wp;
        uint4 mine = make_uint4(0, 0, 0, 0);
        int x, y;
        if (xp < cv.Wp && unpad(cv, xp, yp, x, y)) {
            const float2 t = reinterpret_cast<const float2 *>(T)[row + xp];
            const float2 o = reinterpret_cast<const float2 *>(Y)[row + xp];
            const float w0 = 1.f + wbig * t.x * t.x;
            const float d0 = o.x - t.x, d1 = o.y - t.y;
            acc += (double)w0 * d0 * d0 + (double)d1 * d1;
            mine.x = pack2(scale * w0 * d0, scale * d1);
        }
        put_pixels32(dY + row * C, xp & ~31, cv.Wp, mine);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) sred[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < 8; w++) s += sred[w];
        atomicAdd(loss, s);
    }
}

// Adam on the FP32 master weights and biases of all layers; refreshes the
// BF16 weights and their tap-flipped transpose (the input-gradient weights:
// Wt[cin][8 - tap][cout] = W[cout][tap][cin]).
__global__ void adam_kernel(float *__restrict__ Wm, float *__restrict__ mW, float *__restrict__ vW,
                            const float *__restrict__ gW, float *__restrict__ Bm, float *__restrict__ mB,
                            float *__restrict__ vB, const float *__restrict__ gB, int nlayers, float lr, float b1,
                            float b2, float c1, float c2, float eps, bf16 *__restrict__ Wbf, bf16 *__restrict__ Wt) {
    const int nw = nlayers * 32 * KROWS;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nw + nlayers * 32; k += gridDim.x * blockDim.x) {
        if (k < nw) {
            const float g = gW[k];
            const float m = b1 * mW[k] + (1.f - b1) * g, v = b2 * vW[k] + (1.f - b2) * g * g;
            mW[k] = m;
            vW[k] = v;
            const float w = Wm[k] - lr * (m / c1) / (sqrtf(v / c2) + eps);
            Wm[k] = w;
            const int l = k / (32 * KROWS), r = k - l * 32 * KROWS, co = r / KROWS, kk = r - co * KROWS;
            const int tap = kk / 32, ci = kk - tap * 32;
            Wbf[k] = __float2bfloat16_rn(w);
            Wt[l * 32 * KROWS + ci * KROWS + (8 - tap) * 32 + co] = __float2bfloat16_rn(w);
        } else {
            const int j = k - nw;
            const float g = gB[j];
            const float m = b1 * mB[j] + (1.f - b1) * g, v = b2 * vB[j] + (1.f - b2) * g * g;
            mB[j] = m;
            vB[j] = v;
            Bm[j] -= lr * (m / c1) / (sqrtf(v / c2) + eps);
        }
    }
}

// The BF16 weights and their tap-flipped transpose (as adam_kernel refreshes
// them) from new master weights, and Adam's moments to zero.
__global__ void load_weights_kernel(const float *__restrict__ Wm, int nlayers, bf16 *__restrict__ Wbf,
                                    bf16 *__restrict__ Wt, float *__restrict__ mW, float *__restrict__ vW,
                                    float *__restrict__ mB, float *__restrict__ vB) {
    const int nw = nlayers * 32 * KROWS;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nw; k += gridDim.x * blockDim.x) {
        const int l = k / (32 * KROWS), r = k - l * 32 * KROWS, co = r / KROWS, kk = r - co * KROWS;
        const int tap = kk / 32, ci = kk - tap * 32;
        const bf16 w = __float2bfloat16_rn(Wm[k]);
        Wbf[k] = w;
        Wt[l * 32 * KROWS + ci * KROWS + (8 - tap) * 32 + co] = w;
        mW[k] = vW[k] = 0.f;
        if (k < nlayers * 32) mB[k] = vB[k] = 0.f;
    }
}

// Per-cell envelope of the training targets: E[c][p] = max over the batch
// (and earlier batches) of |T[b][p][c]| over the fine cells p.  Non-negative
// floats order like their bit patterns, so the maximum is an integer
// atomicMax.
__global__ void envelope_kernel(const float *__restrict__ T, int nb, Canvas cv, float *__restrict__ E) {
    const long long npix = (long long)cv.H * cv.W;
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < nb * npix;
         g += (long long)gridDim.x * blockDim.x) {
        const int b = (int)(g / npix);
        const long long p = g - (long long)b * npix;
        const int y = (int)(p / cv.W), x = (int)(p - (long long)y * cv.W);
        const long long gp = (long long)b * cv.Hp * cv.Wp + (long long)(y + kPad) * cv.Wp + (x + kPad);
        atomicMax(reinterpret_cast<int *>(E) + p, __float_as_int(fabsf(T[gp * 2])));
        atomicMax(reinterpret_cast<int *>(E) + npix + p, __float_as_int(fabsf(T[gp * 2 + 1])));
    }
}

// Corrected fields of one image's fine cells: base + scale * output channel.
// With an envelope E, each channel's residual is first clamped to
// +-k E[c][p], k times the largest residual the training pairs needed at
// that cell.  A maximum depth is not negative (0 = never wet), so the
// corrected one is clipped at 0 when asked.  out = [4][H*W]: corrected
// maximum depth and bed change, then the interpolated ones.
__global__ void apply_kernel(const float *__restrict__ Y, const float *__restrict__ base, Canvas cv, int clip_depth,
                             const float *__restrict__ E, float k, float *__restrict__ out) {
    const long long npix = (long long)cv.H * cv.W;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < npix;
         p += (long long)gridDim.x * blockDim.x) {
        const int y = (int)(p / cv.W), x = (int)(p - (long long)y * cv.W);
        const long long gp = (long long)(y + kPad) * cv.Wp + (x + kPad);
        float y0 = Y[gp * 2], y1 = Y[gp * 2 + 1];
        if (E) {
            const float e0 = k * E[p], e1 = k * E[npix + p];
            y0 = fminf(fmaxf(y0, -e0), e0);
            y1 = fminf(fmaxf(y1, -e1), e1);
        }
        const float hb = base[gp * 2], bb = base[gp * 2 + 1];
        const float hc = hb + kSh * y0;
        out[p] = clip_depth ? fmaxf(hc, 0.f) : hc;
        out[npix + p] = bb + kSb * y1;
        out[2 * npix + p] = hb;
        out[3 * npix + p] = bb;
    }
}

// tensor map of an NHWC BF16 32-channel tensor [nimg][H][W][32] with boxes of
// 32 channels x bx x by pixels, 64-byte swizzle (dst multiples of 512 B)
cudaError_t make_map(CUtensorMap *m, const void *base, int nimg, int H, int W, int bx, int by) {
    EncodeTiledFn f = tensor_map_encoder();
    if (!f) return cudaErrorNotSupported;
    const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)nimg};
    const cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)C * 2 * W, (cuuint64_t)C * 2 * W * H};
    const cuuint32_t box[4] = {C, (cuuint32_t)bx, (cuuint32_t)by, 1};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    const CUresult r = f(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(base), dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// What is set up or looked up once per device: the kernels' shared-memory
// attribute, the SM count, the pool of the calls that bring no scratch.
constexpr int kMaxDevices = 64;
struct DeviceState {
    std::atomic<bool> ready{false};
    std::atomic<int> sms{0};
    cudaMemPool_t pool = nullptr;  // under g_dev_mu
};
std::mutex g_dev_mu;
DeviceState g_dev[kMaxDevices];
// the current device's entry, or null (a device beyond the table: looked up on each call)
DeviceState *device_state() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    return &g_dev[dev];
}

// the kernels' shared memory on the current device
cudaError_t prepare() {
    DeviceState *d = device_state();
    if (d && d->ready.load(std::memory_order_acquire)) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(conv3x3_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(conv3x3_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgSmem);
    if (e == cudaSuccess && d) d->ready.store(true, std::memory_order_release);
    return e;
}

// SMs of the current device
int num_sms() {
    DeviceState *d = device_state();
    if (d)
        if (const int k = d->sms.load(std::memory_order_relaxed)) return k;
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 148;
    if (d) d->sms.store(n, std::memory_order_relaxed);
    return n;
}

cudaError_t conv_launch(ConvArgs a, cudaStream_t st) {
    cudaError_t e = prepare();
    if (e != cudaSuccess) return e;
    if (reinterpret_cast<uintptr_t>(a.X) % 16) return cudaErrorInvalidValue;
    a.wide = (reinterpret_cast<uintptr_t>(a.Ybf) | reinterpret_cast<uintptr_t>(a.Yf) |
              reinterpret_cast<uintptr_t>(a.gate)) % 32 == 0;
    CUtensorMap mx;
    e = make_map(&mx, a.X, a.nimg, a.H, a.W, GW, kCRows);
    if (e != cudaSuccess) return e;
    // persistent CTAs; at least two output rows each (every segment also reads
    // the rows above and below it)
    const int ctas = std::max(1, std::min(fwd_geom(a.nimg, a.H, a.W).rows / 2, kFwdCtas * num_sms()));
    conv3x3_fwd_kernel<<<ctas, kFwdThreads, kFwdSmem, st>>>(a, mx);
    return cudaGetLastError();
}

// One tap's gradient of 32 input channels and output channel co by its
// definition, sum over the pixels p of the images of dZ[p] X[p + off] with zeros
// around X: what the tensor cores' products cannot give where an operand is not
// finite, because they also multiply X by the zeros around dZ and leave out
// those around X.  Lane: input channel; warp w of nw takes every nw-th row.
__device__ __noinline__ double wgrad_direct(const bf16 *X, const bf16 *dZ, int nimg, int H, int W, int co, int tap,
                                            int w, int nw) {
    const int lane = threadIdx.x & 31, dy = tap / 3 - 1, dx = tap % 3 - 1;
    double s = 0.0;
    for (int r = w; r < nimg * H; r += nw) {
        const int y = r % H + dy;
        const bool in = y >= 0 && y < H;
        const bf16 *z = dZ + (long long)r * W * C + co;
        const bf16 *v = X + ((long long)(r + dy) * W + dx) * C + lane;
#pragma unroll 8
        for (int x = 0; x < W; x++) {
            const float a = (in && x + dx >= 0 && x + dx < W) ? __bfloat162float(v[(long long)x * C]) : 0.f;
            s += (double)__bfloat162float(z[(long long)x * C]) * (double)a;
        }
        if (__all_sync(0xffffffffu, isnan(s))) break;  // nothing changes a NaN
    }
    return s;
}

// dW[k] (+)= sum over CTAs of part[b][k]; db[n] (+)= sum over CTAs and the 4
// warps of the bias partials; added to what is there, or in its place.  A block
// owns 32 elements; each of its kRedWarps warps takes every kRedWarps-th row
// (all loads in flight together: the kernel is a latency, not a bandwidth), then
// the sums are added in order.
constexpr int kRedWarps = 16, kRedRows = 10;  // one pass covers 160 rows
__global__ void __launch_bounds__(32 * kRedWarps)
    wgrad_reduce_kernel(const float *part, int nctas, const bf16 *X, const bf16 *dZ, int nimg, int H, int W, float *dW,
                        float *db, bool add) {
    __shared__ float sSum[kRedWarps][32];
    __shared__ double sDirect[kRedWarps][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int k = blockIdx.x * 32 + lane;
    const bool bias = k >= 32 * KROWS;  // the last block
    const int n = bias ? 4 * nctas : nctas;
    float acc = 0.f;
    prior_grids_done();
    next_grid_may_start();
    float flags = 0.f;  // first, so that they arrive with the sums
    for (int b = threadIdx.x; b < nctas && !bias; b += 32 * kRedWarps)
        flags += tsu::load_written(part + (size_t)b * kWgPart + kWgFlags);
    for (int b0 = w; b0 < n; b0 += kRedWarps * kRedRows) {
        float v[kRedRows];
#pragma unroll
        for (int i = 0; i < kRedRows; i++) {
            const int b = b0 + i * kRedWarps;
            const float *p = bias ? part + (size_t)(b >> 2) * kWgPart + 32 * KROWS + (b & 3) * 32 + lane
                                  : part + (size_t)b * kWgPart + k;
            v[i] = (b < n) ? tsu::load_written(p) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < kRedRows; i++) acc += v[i];
    }
    sSum[w][lane] = acc;
    bool odd = flags != 0.f;  // a gradient (below: or an element of X) that is not finite
    __syncthreads();
    if (w == 0) {
#pragma unroll
        for (int q = 1; q < kRedWarps; q++) acc += sSum[q][lane];
        odd |= !bias && !isfinite(acc);
    }
    if (__syncthreads_or(odd)) {
        sDirect[w][lane] = wgrad_direct(X, dZ, nimg, H, W, blockIdx.x / 9, blockIdx.x % 9, w, kRedWarps);
        __syncthreads();
        if (w == 0) {
            double s = sDirect[0][lane];
            for (int q = 1; q < kRedWarps; q++) s += sDirect[q][lane];
            acc = (float)s;
        }
    }
    if (w == 0) {
        if (!bias) dW[k] = add ? dW[k] + acc : acc;
        else if (db) db[lane] = add ? db[lane] + acc : acc;
    }
}

// CTAs of a weight-gradient launch
int wgrad_ctas(int nimg, int H, int W) { return std::min(tile_geom(nimg, H, W).total, num_sms()); }

// Stream-ordered scratch of the calls that bring none.  The device's default
// pool gives its memory back at every synchronisation, and the next call then
// maps it again (600 us against 80 us for the gradient itself); this pool
// keeps up to kKeep bytes (one unit of its growth).  tsu_corr_destroy returns them.
constexpr unsigned long long kKeep = 32ull << 20;

cudaError_t scratch_alloc(float **p, size_t bytes, cudaStream_t st) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (st && cudaStreamIsCapturing(st, &cap) != cudaSuccess) cudaGetLastError();
    cudaMemPool_t pool = nullptr;
    std::unique_lock<std::mutex> g(g_dev_mu);
    DeviceState *d = device_state();
    if (cap == cudaStreamCaptureStatusNone && d) {
        if (!d->pool) {
            cudaMemPoolProps props{};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = (int)(d - g_dev);
            unsigned long long keep = kKeep;
            if (cudaMemPoolCreate(&d->pool, &props) != cudaSuccess) {
                cudaGetLastError();
                d->pool = nullptr;
            } else {
                cudaMemPoolSetAttribute(d->pool, cudaMemPoolAttrReleaseThreshold, &keep);
            }
        }
        pool = d->pool;
    }
    g.unlock();
    return pool ? cudaMallocFromPoolAsync((void **)p, bytes, pool, st) : cudaMallocAsync((void **)p, bytes, st);
}
void scratch_trim(int dev) {
    std::lock_guard<std::mutex> g(g_dev_mu);
    if (dev >= 0 && dev < kMaxDevices && g_dev[dev].pool) cudaMemPoolTrimTo(g_dev[dev].pool, 0);
}

// part: wgrad_ctas(...) * kWgPart floats of device scratch, or null (then
// allocated on the stream for this call)
cudaError_t wgrad_launch(const bf16 *X, const bf16 *dZ, int nimg, int H, int W, float *dW, float *db, bool add,
                         float *part, cudaStream_t st) {
    cudaError_t e = prepare();
    if (e != cudaSuccess) return e;
    if (reinterpret_cast<uintptr_t>(X) % 16 || reinterpret_cast<uintptr_t>(dZ) % 16) return cudaErrorInvalidValue;
    CUtensorMap mx, mz;
    e = make_map(&mx, X, nimg, H, W, GX, TYP + 2);
    if (e == cudaSuccess) e = make_map(&mz, dZ, nimg, H, W, GW, TYP);
    if (e != cudaSuccess) return e;
    const int ctas = wgrad_ctas(nimg, H, W);
    float *own = nullptr;
    if (!part) {
        e = scratch_alloc(&own, (size_t)ctas * kWgPart * sizeof(float), st);
        if (e != cudaSuccess) return e;
        part = own;
    }
    // programmatic dependent launches: the reduction's blocks are in place when
    // the partials are complete (8 images of 528^2: 76.2 -> 73.5 us; the same for
    // the forward kernel cost it 1 %)
    launch_after(conv3x3_wgrad_kernel, dim3(ctas), dim3(kWgThreads), kWgSmem, st, mx, mz, nimg, H, W, part);
    e = cudaGetLastError();
    if (e == cudaSuccess) {
        launch_after(wgrad_reduce_kernel, dim3(KROWS + 1), dim3(32 * kRedWarps), 0, st, part, ctas, X, dZ, nimg, H, W, dW,
                     db, add);
        e = cudaGetLastError();
    }
    if (own) {
        const cudaError_t f = cudaFreeAsync(own, st);
        if (e == cudaSuccess) e = f;
    }
    return e;
}

}  // namespace corr

cudaError_t set_wait_limit_corrector(unsigned long long ns) {
    return cudaMemcpyToSymbol(g_wait_limit_ns, &ns, sizeof(ns));
}

}  // namespace tsu

using namespace tsu::corr;

// ------------------------------------------------------------ the corrector
struct TsuCorrector {
    int device = 0;
    int H = 0, W = 0, f = 1, hc = 0, wc = 0, max_batch = 0;
    Canvas cv{};  // the padded canvas the network runs on
    static constexpr int L = 6;
    cudaStream_t st = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    // parameters
    float *Wm = nullptr, *mW = nullptr, *vW = nullptr, *gW = nullptr;  // [L][32][288]
    float *Bm = nullptr, *mB = nullptr, *vB = nullptr, *gB = nullptr;  // [L][32]
    bf16 *Wbf = nullptr, *Wt = nullptr;
    long adam_t = 0;
    // activations [max_batch][Hp][Wp][32] on the padded canvas: act[0] = features, act[l] = output of layer l-1
    bf16 *act[L] = {};
    float *Yout = nullptr;  // the last layer's output channels 0 and 1 [max_batch][Hp][Wp][2]
    bf16 *g0 = nullptr, *g1 = nullptr;
    float *T = nullptr, *base = nullptr;  // [max_batch][Hp][Wp][2]
    int *d_idx = nullptr;
    double *d_loss = nullptr;
    // data set
    float *Hf = nullptr;                       // fine bathymetry
    float *coarse = nullptr, *fine = nullptr;  // [n][3][hc*wc], [n][2][H*W]
    int nsamples = 0, cap = 0;
    double last_ms = 0.0;
    long last_convs = 0;
    // options (tsu_corr_set_options)
    float wbig = 0.f;
    int clip_depth = 0;
    float envelope = 0.f;
    // per-pixel envelope of the normalised residual targets of samples
    // [0, env_n) ([2][H*W]); ntrain = the training set of the last tsu_corr_train
    float *E = nullptr;
    int env_n = 0, ntrain = 0;
    float *wg_part = nullptr;  // weight-gradient partials of one layer ([CTAs][kWgPart])
    // predictions: a map of one sample ([4][H*W]), made at the first prediction,
    // and a second one at the first of several samples, so that one is copied
    // to the host (on cp) while the next is computed
    float *out[2] = {};
    cudaStream_t cp = nullptr;
    cudaEvent_t done[2] = {};
    double *h_loss = nullptr;  // pinned, one per training iteration, grown when needed
    int h_loss_cap = 0;
};

namespace {
thread_local char g_corr_msg[256] = "";
#define CCK(call)                                                                                \
    do {                                                                                         \
        cudaError_t _e = (call);                                                                 \
        if (_e != cudaSuccess) {                                                                 \
            snprintf(g_corr_msg, sizeof(g_corr_msg), "%s: %s", #call, cudaGetErrorString(_e));   \
            return _e == cudaErrorMemoryAllocation ? TSU_ERR_GPU_OOM : TSU_ERR_CUDA;             \
        }                                                                                        \
    } while (0)

uint64_t splitmix(uint64_t &s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
double uniform01(uint64_t &s) { return (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0); }

void free_all(TsuCorrector *c) {
    float *fp[] = {c->Wm, c->mW, c->vW, c->gW, c->Bm, c->mB, c->vB, c->gB, c->Yout, c->T, c->base, c->Hf, c->coarse, c->fine,
                   c->E, c->wg_part, c->out[0], c->out[1]};
    for (float *p : fp) cudaFree(p);
    if (c->h_loss) cudaFreeHost(c->h_loss);
    for (cudaEvent_t ev : c->done)
        if (ev) cudaEventDestroy(ev);
    if (c->cp) cudaStreamDestroy(c->cp);
    cudaFree(c->Wbf);
    cudaFree(c->Wt);
    for (bf16 *p : c->act) cudaFree(p);
    cudaFree(c->g0);
    cudaFree(c->g1);
    cudaFree(c->d_idx);
    cudaFree(c->d_loss);
    if (c->e0) cudaEventDestroy(c->e0);
    if (c->e1) cudaEventDestroy(c->e1);
    if (c->st) cudaStreamDestroy(c->st);
}

int upload_weights(TsuCorrector *c, const float *W, const float *B) {
    const int L = TsuCorrector::L;
    const size_t nw = (size_t)L * 32 * KROWS;
    CCK(cudaMemcpyAsync(c->Wm, W, nw * sizeof(float), cudaMemcpyHostToDevice, c->st));
    CCK(cudaMemcpyAsync(c->Bm, B, (size_t)L * 32 * sizeof(float), cudaMemcpyHostToDevice, c->st));
    load_weights_kernel<<<(int)((nw + 255) / 256), 256, 0, c->st>>>(c->Wm, L, c->Wbf, c->Wt, c->mW, c->vW, c->mB, c->vB);
    CCK(cudaGetLastError());
    CCK(cudaStreamSynchronize(c->st));
    c->adam_t = 0;
    return TSU_OK;
}

int check_kernel_flag() {
    int flag = 0;
    CCK(cudaMemcpyFromSymbol(&flag, g_corr_err, sizeof(int)));
    if (flag) {
        snprintf(g_corr_msg, sizeof(g_corr_msg), "corrector: a tensor-core wait expired");
        int z = 0;
        cudaMemcpyToSymbol(g_corr_err, &z, sizeof(int));
        return TSU_ERR_CUDA;
    }
    return TSU_OK;
}

// forward pass of `nb` images already in act[0]; the last layer's two used
// output channels in Yout ([pixel][2], FP32)
int forward(TsuCorrector *c, int nb) {
    const int L = TsuCorrector::L;
    for (int l = 0; l < L; l++) {
        ConvArgs a;
        a.X = c->act[l];
        a.nimg = nb;
        a.H = c->cv.Hp;
        a.W = c->cv.Wp;
        a.Wk = c->Wbf + (size_t)l * 32 * KROWS;
        a.bias = c->Bm + l * 32;
        a.relu = (l < L - 1);
        a.gate = nullptr;
        a.Ybf = (l < L - 1) ? c->act[l + 1] : nullptr;
        a.Yf = nullptr;
        a.Y2 = (l < L - 1) ? nullptr : c->Yout;
        CCK(conv_launch(a, c->st));
    }
    return TSU_OK;
}

int load_batch(TsuCorrector *c, const int *idx, int nb, bool targets) {
    CCK(cudaMemcpyAsync(c->d_idx, idx, nb * sizeof(int), cudaMemcpyHostToDevice, c->st));
    features_kernel<<<8 * num_sms(), 256, 0, c->st>>>(c->d_idx, nb, c->coarse, targets ? c->fine : nullptr, c->Hf,
                                                               c->cv, c->hc, c->wc, c->f, c->act[0],
                                                               targets ? c->T : nullptr, c->base);
    CCK(cudaGetLastError());
    return TSU_OK;
}

// the residual envelope of training samples [0, n)
int compute_envelope(TsuCorrector *c, int n) {
    const long long npix = (long long)c->H * c->W;
    CCK(cudaMemsetAsync(c->E, 0, 2 * npix * sizeof(float), c->st));
    std::vector<int> idx(c->max_batch);
    for (int s0 = 0; s0 < n; s0 += c->max_batch) {
        const int nb = std::min(c->max_batch, n - s0);
        for (int b = 0; b < nb; b++) idx[b] = s0 + b;
        const int rc = load_batch(c, idx.data(), nb, true);
        if (rc) return rc;
        envelope_kernel<<<4 * num_sms(), 256, 0, c->st>>>(c->T, nb, c->cv, c->E);
        CCK(cudaGetLastError());
    }
    c->env_n = n;
    return TSU_OK;
}
}  // namespace

extern "C" int tsu_corr_create(TsuCorrector **out, int ny, int nx, int factor, int max_batch, unsigned long long seed,
                               int device) {
    if (!out || ny < 1 || nx < 1 || factor < 1 || ny % factor || nx % factor || max_batch < 1) return TSU_ERR_INVALID;
    *out = nullptr;
    TsuCorrector *c = new (std::nothrow) TsuCorrector();
    if (!c) return TSU_ERR_HOST_OOM;
    c->device = device;
    c->H = ny;
    c->W = nx;
    c->cv = canvas(ny, nx);
    c->f = factor;
    c->hc = ny / factor;
    c->wc = nx / factor;
    c->max_batch = max_batch;
    const int L = TsuCorrector::L;
    const size_t nw = (size_t)L * 32 * KROWS, nbias = (size_t)L * 32;
    const size_t npix = (size_t)max_batch * c->cv.Hp * c->cv.Wp;  // padded canvas
    cudaError_t e = cudaSetDevice(device);
#define CAL(p, bytes) \
    if (e == cudaSuccess) e = cudaMalloc((void **)&(p), (bytes))
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreate(&c->e0);
    if (e == cudaSuccess) e = cudaEventCreate(&c->e1);
    CAL(c->Wm, nw * 4);
    CAL(c->mW, nw * 4);
    CAL(c->vW, nw * 4);
    CAL(c->gW, nw * 4);
    CAL(c->Bm, nbias * 4);
    CAL(c->mB, nbias * 4);
    CAL(c->vB, nbias * 4);
    CAL(c->gB, nbias * 4);
    CAL(c->Wbf, nw * 2);
    CAL(c->Wt, nw * 2);
    for (int l = 0; l < L; l++) CAL(c->act[l], npix * C * 2);
    CAL(c->Yout, npix * 2 * 4);
    CAL(c->g0, npix * C * 2);
    CAL(c->g1, npix * C * 2);
    CAL(c->T, npix * 2 * 4);
    CAL(c->base, npix * 2 * 4);
    CAL(c->d_idx, (size_t)max_batch * 4);
    CAL(c->d_loss, 8);
    CAL(c->Hf, (size_t)ny * nx * 4);
    CAL(c->E, (size_t)2 * ny * nx * 4);
    CAL(c->wg_part, (size_t)wgrad_ctas(max_batch, c->cv.Hp, c->cv.Wp) * kWgPart * 4);
#undef CAL
    if (e == cudaSuccess) e = prepare();
    if (e != cudaSuccess) {
        snprintf(g_corr_msg, sizeof(g_corr_msg), "tsu_corr_create: %s", cudaGetErrorString(e));
        free_all(c);
        delete c;
        return e == cudaErrorMemoryAllocation ? TSU_ERR_GPU_OOM : TSU_ERR_CUDA;
    }
    // He-normal initialisation (SplitMix64 + Box-Muller); the last layer is
    // zero, so the untrained corrector returns the interpolated coarse fields
    std::vector<float> W(nw, 0.f), B(nbias, 0.f);
    uint64_t s = seed;
    const double sd = std::sqrt(2.0 / (9.0 * 32.0));
    for (int l = 0; l < L - 1; l++)
        for (size_t k = 0; k < (size_t)32 * KROWS; k++) {
            const double u1 = uniform01(s), u2 = uniform01(s);
            W[(size_t)l * 32 * KROWS + k] = (float)(sd * std::sqrt(-2.0 * std::log1p(-u1)) * std::cos(2.0 * M_PI * u2));
        }
    int rc = upload_weights(c, W.data(), B.data());
    if (rc) {
        free_all(c);
        delete c;
        return rc;
    }
    *out = c;
    return TSU_OK;
}

extern "C" int tsu_corr_destroy(TsuCorrector *c) {
    if (!c) return TSU_OK;
    cudaSetDevice(c->device);
    if (c->st) cudaStreamSynchronize(c->st);
    free_all(c);
    scratch_trim(c->device);
    delete c;
    return TSU_OK;
}

extern "C" int tsu_corr_set_site(TsuCorrector *c, const float *fine_H) {
    if (!c || !fine_H) return TSU_ERR_INVALID;
    CCK(cudaSetDevice(c->device));
    CCK(cudaMemcpyAsync(c->Hf, fine_H, (size_t)c->H * c->W * 4, cudaMemcpyHostToDevice, c->st));
    CCK(cudaStreamSynchronize(c->st));
    return TSU_OK;
}

extern "C" int tsu_corr_add_samples(TsuCorrector *c, int n, const float *coarse, const float *fine) {
    if (!c || n < 1 || !coarse) return TSU_ERR_INVALID;
    CCK(cudaSetDevice(c->device));
    const size_t cs = (size_t)3 * c->hc * c->wc, fs = (size_t)2 * c->H * c->W;
    if (c->nsamples + n > c->cap) {
        const int ncap = std::max(c->nsamples + n, 2 * c->cap);
        float *nc = nullptr, *nf = nullptr;
        CCK(cudaMalloc((void **)&nc, ncap * cs * 4));
        if (cudaMalloc((void **)&nf, ncap * fs * 4) != cudaSuccess) {
            cudaFree(nc);
            snprintf(g_corr_msg, sizeof(g_corr_msg), "tsu_corr_add_samples: out of device memory");
            return TSU_ERR_GPU_OOM;
        }
        if (c->nsamples) {
            CCK(cudaMemcpyAsync(nc, c->coarse, c->nsamples * cs * 4, cudaMemcpyDeviceToDevice, c->st));
            CCK(cudaMemcpyAsync(nf, c->fine, c->nsamples * fs * 4, cudaMemcpyDeviceToDevice, c->st));
        }
        CCK(cudaStreamSynchronize(c->st));
        cudaFree(c->coarse);
        cudaFree(c->fine);
        c->coarse = nc;
        c->fine = nf;
        c->cap = ncap;
    }
    CCK(tsu::bytes_h2d(c->coarse + c->nsamples * cs, coarse, n * cs * 4, c->st));
    if (fine)
        CCK(tsu::bytes_h2d(c->fine + c->nsamples * fs, fine, n * fs * 4, c->st));
    else
        CCK(cudaMemsetAsync(c->fine + c->nsamples * fs, 0, n * fs * 4, c->st));
    CCK(cudaStreamSynchronize(c->st));
    c->nsamples += n;
    return TSU_OK;
}

extern "C" int tsu_corr_num_samples(TsuCorrector *c, int *n) {
    if (!c || !n) return TSU_ERR_INVALID;
    *n = c->nsamples;
    return TSU_OK;
}

extern "C" int tsu_corr_set_options(TsuCorrector *c, float large_residual_weight, int clip_depth, float envelope) {
    if (!c || !(large_residual_weight >= 0.f) || (clip_depth != 0 && clip_depth != 1) || !(envelope >= 0.f))
        return TSU_ERR_INVALID;
    c->wbig = large_residual_weight;
    c->clip_depth = clip_depth;
    c->envelope = envelope;
    return TSU_OK;
}

extern "C" int tsu_corr_get_weights(TsuCorrector *c, float *W, float *B) {
    if (!c || !W || !B) return TSU_ERR_INVALID;
    CCK(cudaSetDevice(c->device));
    CCK(cudaMemcpyAsync(W, c->Wm, (size_t)TsuCorrector::L * 32 * KROWS * 4, cudaMemcpyDeviceToHost, c->st));
    CCK(cudaMemcpyAsync(B, c->Bm, (size_t)TsuCorrector::L * 32 * 4, cudaMemcpyDeviceToHost, c->st));
    CCK(cudaStreamSynchronize(c->st));
    return TSU_OK;
}

extern "C" int tsu_corr_set_weights(TsuCorrector *c, const float *W, const float *B) {
    if (!c || !W || !B) return TSU_ERR_INVALID;
    CCK(cudaSetDevice(c->device));
    return upload_weights(c, W, B);
}

// `iters` Adam steps on mini-batches drawn (seeded) from samples [0, ntrain)
extern "C" int tsu_corr_train(TsuCorrector *c, int ntrain, int iters, int batch, float lr, unsigned long long seed,
                              float *loss) {
    if (!c || ntrain < 1 || ntrain > c->nsamples || iters < 0 || batch < 1 || batch > c->max_batch)
        return TSU_ERR_INVALID;
    CCK(cudaSetDevice(c->device));
    c->ntrain = ntrain;
    const int L = TsuCorrector::L;
    const size_t nw = (size_t)L * 32 * KROWS;
    const long long npix = (long long)batch * c->H * c->W;
    uint64_t s = seed;
    std::vector<int> idx(batch);
    if (iters > c->h_loss_cap) {  // kept between calls: page-locking memory costs more than an iteration
        if (c->h_loss) cudaFreeHost(c->h_loss);
        c->h_loss = nullptr;
        c->h_loss_cap = 0;
        CCK(cudaMallocHost((void **)&c->h_loss, sizeof(double) * iters));
        c->h_loss_cap = iters;
    }
    double *const h_loss = c->h_loss;
    int rc = TSU_OK;
    cudaError_t e = cudaEventRecord(c->e0, c->st);
    for (int it = 0; it < iters && !rc && e == cudaSuccess; it++) {
        for (int b = 0; b < batch; b++) idx[b] = (int)(splitmix(s) % (uint64_t)ntrain);
        rc = load_batch(c, idx.data(), batch, true);
        if (!rc) rc = forward(c, batch);
        if (rc) break;
        e = cudaMemsetAsync(c->d_loss, 0, 8, c->st);
        if (e != cudaSuccess) break;
        loss_kernel<<<8 * num_sms(), 256, 0, c->st>>>(c->Yout, c->T, batch, c->cv, c->wbig, c->g0, c->d_loss);
        if ((e = cudaGetLastError()) != cudaSuccess) break;
        if ((e = cudaMemcpyAsync(h_loss + it, c->d_loss, 8, cudaMemcpyDeviceToHost, c->st)) != cudaSuccess) break;
        bf16 *dZ = c->g0, *dX = c->g1;
        for (int l = L - 1; l >= 0 && e == cudaSuccess; l--) {
            e = wgrad_launch(c->act[l], dZ, batch, c->cv.Hp, c->cv.Wp, c->gW + (size_t)l * 32 * KROWS, c->gB + l * 32,
                             false, c->wg_part, c->st);
            if (e == cudaSuccess && l > 0) {  // dZ_{l-1} = conv(dZ_l, flipped W_l), zero where act[l] <= 0
                ConvArgs a;
                a.X = dZ;
                a.nimg = batch;
                a.H = c->cv.Hp;
                a.W = c->cv.Wp;
                a.Wk = c->Wt + (size_t)l * 32 * KROWS;
                a.bias = nullptr;
                a.relu = 0;
                a.gate = c->act[l];
                a.Ybf = dX;
                a.Yf = nullptr;
                a.Y2 = nullptr;
                e = conv_launch(a, c->st);
                std::swap(dZ, dX);
            }
        }
        if (e != cudaSuccess) break;
        c->adam_t++;
        const float b1 = 0.9f, b2 = 0.999f;
        const float c1 = 1.f - powf(b1, (float)c->adam_t), c2 = 1.f - powf(b2, (float)c->adam_t);
        adam_kernel<<<(int)((nw + 255) / 256), 256, 0, c->st>>>(c->Wm, c->mW, c->vW, c->gW, c->Bm, c->mB, c->vB, c->gB,
                                                              L, lr, b1, b2, c1, c2, 1e-8f, c->Wbf, c->Wt);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && !rc) e = cudaEventRecord(c->e1, c->st);
    if (e == cudaSuccess && !rc) e = cudaStreamSynchronize(c->st);
    if (e != cudaSuccess && !rc) {
        snprintf(g_corr_msg, sizeof(g_corr_msg), "tsu_corr_train: %s", cudaGetErrorString(e));
        rc = TSU_ERR_CUDA;
    }
    if (!rc) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, c->e0, c->e1);
        c->last_ms = ms;
        c->last_convs = (long)iters * (3 * L - 1);
        if (loss)
            for (int it = 0; it < iters; it++) loss[it] = (float)(h_loss[it] / (2.0 * (double)npix));
    }
    if (rc) return rc;
    return check_kernel_flag();
}

// corrected (and interpolated baseline) fine fields of samples
// [first, first + n): out_* are [n][H][W]; base_* may be null
extern "C" int tsu_corr_predict(TsuCorrector *c, int first, int n, float *out_hmax, float *out_db, float *base_hmax,
                                float *base_db) {
    if (!c || first < 0 || n < 1 || first + n > c->nsamples || !out_hmax || !out_db) return TSU_ERR_INVALID;
    CCK(cudaSetDevice(c->device));
    const size_t np = (size_t)c->H * c->W;
    // the envelope clamp needs the training set's targets (none before training)
    const bool clamp = c->envelope > 0.f && c->ntrain > 0;
    if (clamp && c->env_n != c->ntrain) {
        const int r = compute_envelope(c, c->ntrain);
        if (r) return r;
    }
    if (!c->out[0]) CCK(cudaMalloc((void **)&c->out[0], 4 * np * 4));
    if (n > 1 && !c->out[1] && cudaMalloc((void **)&c->out[1], 4 * np * 4) != cudaSuccess) {
        cudaGetLastError();  // no room for it: one sample after the other
        c->out[1] = nullptr;
    }
    const bool two = n > 1 && c->out[1];
    if (two && !c->cp) {
        for (int q = 0; q < 2; q++)
            if (!c->done[q]) CCK(cudaEventCreateWithFlags(&c->done[q], cudaEventDisableTiming));
        CCK(cudaStreamCreateWithFlags(&c->cp, cudaStreamNonBlocking));
    }
    const cudaStream_t copy = two ? c->cp : c->st;
    auto map = [&](int k) { return two ? k & 1 : 0; };
    auto compute = [&](int k) -> int {  // sample first + k -> its map
        const int s = first + k;
        int r = load_batch(c, &s, 1, false);
        if (!r) r = forward(c, 1);
        if (r) return r;
        apply_kernel<<<2 * num_sms(), 256, 0, c->st>>>(c->Yout, c->base, c->cv, c->clip_depth, clamp ? c->E : nullptr,
                                                         c->envelope, c->out[map(k)]);
        CCK(cudaGetLastError());
        if (two) CCK(cudaEventRecord(c->done[map(k)], c->st));
        return TSU_OK;
    };
    int rc = compute(0);
    for (int k = 0; k < n && !rc; k++) {
        // the other map's copy (of sample k - 1) has ended: planes_d2h waits for it
        if (two && k + 1 < n) rc = compute(k + 1);
        if (rc) break;
        float *want[4] = {out_hmax, out_db, base_hmax, base_db};
        void *outs[4];
        const void *ins[4];
        int m = 0;
        for (int q = 0; q < 4; q++)
            if (want[q]) {
                outs[m] = want[q] + k * np;
                ins[m++] = c->out[map(k)] + q * np;
            }
        if ((two && cudaStreamWaitEvent(copy, c->done[map(k)], 0) != cudaSuccess) ||
            tsu::planes_d2h(m, outs, (size_t)c->W * 4, ins, (size_t)c->W * 4, (size_t)c->W * 4, c->H, copy) != cudaSuccess ||
            cudaStreamSynchronize(copy) != cudaSuccess) {
            snprintf(g_corr_msg, sizeof(g_corr_msg), "tsu_corr_predict: CUDA error");
            rc = TSU_ERR_CUDA;
            break;
        }
        if (!two && k + 1 < n) rc = compute(k + 1);
    }
    if (cudaStreamSynchronize(c->st) != cudaSuccess && !rc) {
        snprintf(g_corr_msg, sizeof(g_corr_msg), "tsu_corr_predict: CUDA error");
        rc = TSU_ERR_CUDA;
    }
    if (rc) return rc;
    return check_kernel_flag();
}

// times `iters` forward convolutions of one layer over `nimg` images of the
// first sample's features: device ms per convolution and TFLOP/s
// (2 x pixels x 288 x 32 FLOPs per convolution)
extern "C" int tsu_corr_bench_conv(TsuCorrector *c, int nimg, int iters, double *ms_per_conv, double *tflops) {
    if (!c || nimg < 1 || nimg > c->max_batch || iters < 1 || c->nsamples < 1) return TSU_ERR_INVALID;
    CCK(cudaSetDevice(c->device));
    std::vector<int> idx(nimg, 0);
    int rc = load_batch(c, idx.data(), nimg, false);
    if (rc) return rc;
    ConvArgs a;
    a.X = c->act[0];
    a.nimg = nimg;
    a.H = c->cv.Hp;  // the padded canvas the network runs on
    a.W = c->cv.Wp;
    a.Wk = c->Wbf;
    a.bias = c->Bm;
    a.relu = 1;
    a.gate = nullptr;
    a.Ybf = c->act[1];
    a.Yf = nullptr;
    a.Y2 = nullptr;
    for (int k = 0; k < 3; k++) CCK(conv_launch(a, c->st));
    CCK(cudaEventRecord(c->e0, c->st));
    for (int k = 0; k < iters; k++) CCK(conv_launch(a, c->st));
    CCK(cudaEventRecord(c->e1, c->st));
    CCK(cudaEventSynchronize(c->e1));
    float ms = 0.f;
    CCK(cudaEventElapsedTime(&ms, c->e0, c->e1));
    const double per = ms / iters;
    if (ms_per_conv) *ms_per_conv = per;
    if (tflops) *tflops = 2.0 * nimg * (double)c->cv.Hp * c->cv.Wp * KROWS * 32 / (per * 1e-3) / 1e12;
    return check_kernel_flag();
}

extern "C" int tsu_corr_last_train_ms(TsuCorrector *c, double *ms, long *convs) {
    if (!c || !ms) return TSU_ERR_INVALID;
    *ms = c->last_ms;
    if (convs) *convs = c->last_convs;
    return TSU_OK;
}

// ---- raw kernels on caller-owned device buffers (stream: a cudaStream_t or null)
extern "C" int tsu_corr_conv3x3(const void *X, int nimg, int H, int W, const void *Wk, const float *bias, int relu,
                                const void *gate, void *Ybf, float *Yf, void *stream) {
    if (!X || !Wk || nimg < 1 || H < 1 || W < 1 || (!Ybf && !Yf)) return TSU_ERR_INVALID;
    ConvArgs a;
    a.X = static_cast<const bf16 *>(X);
    a.nimg = nimg;
    a.H = H;
    a.W = W;
    a.Wk = static_cast<const bf16 *>(Wk);
    a.bias = bias;
    a.relu = relu;
    a.gate = static_cast<const bf16 *>(gate);
    a.Ybf = static_cast<bf16 *>(Ybf);
    a.Yf = Yf;
    a.Y2 = nullptr;
    CCK(conv_launch(a, static_cast<cudaStream_t>(stream)));
    return TSU_OK;
}

extern "C" int tsu_corr_conv3x3_wgrad(const void *X, const void *dZ, int nimg, int H, int W, float *dW, float *db,
                                      void *stream) {
    if (!X || !dZ || !dW || nimg < 1 || H < 1 || W < 1) return TSU_ERR_INVALID;
    CCK(wgrad_launch(static_cast<const bf16 *>(X), static_cast<const bf16 *>(dZ), nimg, H, W, dW, db, true, nullptr,
                     static_cast<cudaStream_t>(stream)));
    return TSU_OK;
}

// synchronises the device and reports (and clears) an expired kernel wait
extern "C" int tsu_corr_status(void) {
    CCK(cudaDeviceSynchronize());
    return check_kernel_flag();
}

extern "C" const char *tsu_corr_last_error(void) { return g_corr_msg; }
