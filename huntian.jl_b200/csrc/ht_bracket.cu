// Learned walk-length bracket: a 12 -> 64 -> 64 -> 64 -> 2 MLP (BF16 weights and
// activations, FP32 accumulation on the tensor cores) that predicts,
// for every peak, a low and a high quantile of the radius at which its shell walk stops.
// The shell collapse itself never reads the prediction: it only orders the work (peaks with
// similar predicted walks share a warp, longest first), so every result is identical to the
// unordered path.  No counterpart in the reference.
//
// Features (per peak, all known before the walk):
//   0 Rf / alatt          1 sqrt(ir2min)         2 delta_s at the peak (FcRf)
//   3 fcrit               4 ZZon                 5 delta at the peak cell
//   6..9 mean delta over the in-tile cells of shells 2, 3, 4, 5 (radii 1, sqrt2, sqrt3, 2)
//   10 rad[m0_init]       11 Rf / alatt + 2 (how far the walk must reach at least: the
//                            first shell past ir2min and the gradient window at Rf)
//   12..15 zero padding (K = 16 for the first tensor-core layer)
// Features are standardised with the model's mean / std before the first layer.
//
// Kernels:
//   features_kernel      one thread per peak
//   mlp_infer_tc_kernel  inference, 128 peaks per CTA tile: every layer a tcgen05.mma chain
//                        from shared memory into tensor memory, read back per row
//                        (tcgen05.ld), bias + ReLU + BF16 as the next layer's operand
//   train_grad_kernel    training (offline, not on the step): forward, pinball loss,
//                        backward and the weight gradients of 128-sample tiles, one CTA
//                        partial each; train_reduce_kernel adds the partials
//   adam_kernel          the optimiser step
#include <cuda_bf16.h>
#include <math.h>

#include <cub/device/device_radix_sort.cuh>
#include <string>

#include "ht_async.cuh"
#include "ht_internal.cuh"

namespace {

constexpr int kIn = 16, kHid = 64;

__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);   // .x = lo (low half)
    unsigned u;
    memcpy(&u, &v, 4);
    return u;
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const unsigned (&a)[4], unsigned b0,
                                         unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ---------------------------------------------------------------- features ----

struct FeatArgs {
    const float4* rec;        // packed records of the bound tile (nullable)
    const float* delta;       // or the delta field
    int n1, n2, n3;
    long long s2;
    const char4* off;
    const int32_t* start;
    const int32_t* count;
    const int32_t* r2;
    const double* rad;
    int nshells;
    const int32_t* pi;
    const int32_t* pj;
    const int32_t* pk;
    const double* Rf;
    const int32_t* ir2min;
    const float* ZZon;
    const float* fcrit;
    const float* peak_delta;  // delta_s at each peak (nullable: 0)
    long long npeaks;
    double alatt;
};

__global__ void __launch_bounds__(256) features_kernel(const FeatArgs a, float* __restrict__ F) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.npeaks) return;
    const int ci = a.pi[p], cj = a.pj[p], ck = a.pk[p];
    float f[kIn];
#pragma unroll
    for (int i = 0; i < kIn; ++i) f[i] = 0.f;
    const double Rf = a.Rf[p];
    const int ir2 = a.ir2min[p];
    f[0] = (float)(Rf / a.alatt);
    f[1] = sqrtf((float)max(ir2, 0));
    f[2] = a.peak_delta ? a.peak_delta[p] : 0.f;
    f[3] = a.fcrit[p];
    f[4] = a.ZZon[p];
    auto value = [&](int i, int j, int k, float& v) {
        if (i < 1 || i > a.n1 || j < 1 || j > a.n2 || k < 1 || k > a.n3) return false;
        const long long idx = (long long)(i - 1) + (long long)a.n1 * (j - 1) + a.s2 * (k - 1);
        v = a.rec ? __ldg(a.rec + 2 * idx).x : __ldg(a.delta + idx);
        return true;
    };
    float v;
    if (value(ci, cj, ck, v)) f[5] = v;
    // shells 2-5 (r^2 = 1, 2, 3, 4) hold 6, 12, 8 and 6 cells, the table's first 32 after the
    // centre: a peak at least two cells inside the tile has every one of them, so all 32
    // loads go out before any is summed (same sums, same order as the loop below)
    const bool inner2 = a.nshells >= 5 && ci > 2 && ci + 2 <= a.n1 && cj > 2 &&
                        cj + 2 <= a.n2 && ck > 2 && ck + 2 <= a.n3;
    if (inner2) {
        const long long c0 = (long long)(ci - 1) + (long long)a.n1 * (cj - 1) + a.s2 * (ck - 1);
        const int st2 = __ldg(a.start + 2);
        float w[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) {
            const char4 o = __ldg(a.off + st2 + c);
            const long long idx = c0 + o.x + (long long)a.n1 * o.y + a.s2 * o.z;
            w[c] = a.rec ? __ldg(reinterpret_cast<const float*>(a.rec + 2 * idx))
                         : __ldg(a.delta + idx);
        }
        constexpr int kFirst[5] = {0, 6, 18, 26, 32};
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            float sum = 0.f;
#pragma unroll
            for (int c = kFirst[s]; c < kFirst[s + 1]; ++c) sum += w[c];
            const int nin = kFirst[s + 1] - kFirst[s];
            f[6 + s] = sum / nin;
        }
    }
    for (int s = 2; !inner2 && s <= 5 && s <= a.nshells; ++s) {
        const int st = __ldg(a.start + s), cnt = __ldg(a.count + s);
        float sum = 0.f;
        int nin = 0;
        for (int c = st; c < st + cnt; ++c) {
            const char4 o = __ldg(a.off + c);
            if (value(ci + o.x, cj + o.y, ck + o.z, v)) { sum += v; ++nin; }
        }
        f[4 + s] = nin ? sum / nin : 0.f;
    }
    // data-independent walk bounds: first shell with r2 > ir2min, and where the gradient
    // window at the filter radius ends
    int lo = 1, hi = a.nshells - 1, m0 = a.nshells - 1;
    while (lo <= hi) {
        const int mid = (lo + hi) >> 1;
        if (a.r2[mid] > ir2) { m0 = mid; hi = mid - 1; } else { lo = mid + 1; }
    }
    f[10] = (float)a.rad[m0];
    const double RR = Rf / a.alatt;
    f[11] = (float)(RR + 2.0);
    float* out = F + p * kIn;
#pragma unroll
    for (int i = 0; i < kIn; i += 4) *reinterpret_cast<float4*>(out + i) = make_float4(f[i], f[i + 1], f[i + 2], f[i + 3]);
}

// --------------------------------------------------------- fused inference ----

struct MlpW {
    const __nv_bfloat16* W1;   // [64][16]
    const __nv_bfloat16* W2;   // [64][64]
    const __nv_bfloat16* W3;   // [64][64]
    const __nv_bfloat16* W4;   // [8][64] (rows 2..7 zero)
    const float* b1;           // [64]
    const float* b2;
    const float* b3;
    const float* b4;           // [8]
    const float* mean;         // [16] feature standardisation
    const float* istd;         // [16]
};

// ------------------------------------------------- fused inference, tcgen05 ----
//
// The same four layers on the 5th-generation tensor cores.  A CTA of 128 threads takes
// tiles of 128 peaks (M = 128), persistent over the tiles.  Every layer is a chain of
// tcgen05.mma (kind::f16, BF16 x BF16 -> FP32, one elected thread issues them) from shared
// memory into a 64-column accumulator in tensor memory: the activations A [128 x K] and the
// layer's weights W [N x K] (the row-major weights are K-major already) sit in the
// no-swizzle K-major layout of 8-row x 16-byte core matrices.  The MMAs of a layer are
// committed to an mbarrier; every thread then reads its own row back (tcgen05.ld 32x32b:
// warp w owns lanes 32w .. 32w + 31, and row r of an M = 128 accumulator is lane r), adds
// the bias, applies ReLU, rounds to BF16 and writes the row as the next layer's A.  The
// output layer is padded to N = 16 (weight rows 2 .. 15 zero).  Waits are bounded; a wait
// that gives up records the status, and the CTA still frees its tensor memory.

constexpr int kTcRows = 128;    // peaks per tile (the MMA's M)
constexpr int kTcN4 = 16;       // the output layer's N (2 used)
constexpr int kTcCols = 64;     // tensor-memory columns per CTA (FP32 accumulator, N <= 64)

// Byte offset of element (r, k) in a K-major operand of R rows: core matrices of 8 rows x
// 8 K-values (16 bytes a row, 128 bytes each), row groups 128 bytes apart (the descriptor's
// stride offset), the two K halves of a 16-wide K step R x 16 bytes apart (its leading
// offset), K steps R x 32 bytes apart.
__host__ __device__ constexpr int umma_off(int R, int r, int k) {
    return (k >> 4) * (R * 32) + ((k >> 3) & 1) * (R * 16) + (r >> 3) * 128 + (r & 7) * 16 +
           (k & 7) * 2;
}

// Shared-memory matrix descriptor of such an operand (R rows) starting at shared address
// saddr: start >> 4 in bits [0, 14), leading offset >> 4 in [16, 30), stride offset >> 4
// in [32, 46), version 1 in [46, 48), no swizzle, base offset 0.
__device__ __forceinline__ unsigned long long umma_desc(unsigned saddr, int R) {
    const unsigned long long lbo = (unsigned long long)(R * 16) >> 4, sbo = 128ull >> 4;
    return (unsigned long long)((saddr >> 4) & 0x3FFFu) | (lbo << 16) | (sbo << 32) |
           (1ull << 46);
}

// Instruction descriptor: FP32 accumulator, BF16 A and B, both K-major, N >> 3 in bits
// [17, 23), M >> 4 in bits [24, 29).
__host__ __device__ constexpr unsigned umma_idesc(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(N >> 3) << 17) |
           ((unsigned)(M >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(unsigned tmem_d, unsigned long long da,
                                          unsigned long long db, unsigned idesc,
                                          unsigned accumulate) {
    const unsigned z = 0u;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
        :: "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(z), "r"(z), "r"(z),
           "r"(z));
}

__device__ __forceinline__ void umma_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"(htasync::smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// 16 consecutive accumulator columns of this thread's lane.
__device__ __forceinline__ void tmem_ld16(unsigned taddr, float (&v)[16]) {
    unsigned u[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]),
          "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]),
          "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(u[i]);
}

// Shared-memory layout of the tcgen05 inference kernel (bytes from the dynamic base).
constexpr int kTcOffA = 0;                                  // A [128 x 64] BF16
constexpr int kTcOffW1 = kTcOffA + kTcRows * kHid * 2;      // W1 [64 x 16]
constexpr int kTcOffW2 = kTcOffW1 + kHid * kIn * 2;         // W2 [64 x 64]
constexpr int kTcOffW3 = kTcOffW2 + kHid * kHid * 2;        // W3 [64 x 64]
constexpr int kTcOffW4 = kTcOffW3 + kHid * kHid * 2;        // W4 [16 x 64]
constexpr int kTcOffB = kTcOffW4 + kTcN4 * kHid * 2;        // b1 b2 b3 [64] b4 [8], FP32
constexpr int kTcSmem = kTcOffB + (3 * kHid + 8) * 4;

// Copy the row-major weights W [rows x K] (global, BF16) into the K-major layout with Rpad
// rows (rows >= rows zero).
__device__ __forceinline__ void stage_weights(unsigned char* dst, const __nv_bfloat16* W,
                                              int rows, int Rpad, int K, int tid, int nthr) {
    for (int e = tid; e < Rpad * (K / 2); e += nthr) {
        const int r = e / (K / 2), k = 2 * (e % (K / 2));
        const unsigned v = r < rows ? __ldg(reinterpret_cast<const unsigned*>(W + (size_t)r * K + k))
                                    : 0u;
        *reinterpret_cast<unsigned*>(dst + umma_off(Rpad, r, k)) = v;
    }
}

// Bias, ReLU and BF16 rounding of the 64 columns of this thread's row, written as row r of
// the next layer's A.
__device__ __forceinline__ void hidden_out(unsigned tmem_row, const float* bias,
                                           unsigned char* A, int r) {
#pragma unroll
    for (int q = 0; q < kHid / 16; ++q) {
        float v[16];
        tmem_ld16(tmem_row + 16 * q, v);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint4 u;
            unsigned* pu = reinterpret_cast<unsigned*>(&u);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c = 8 * h + 2 * j;
                pu[j] = pack_bf16(fmaxf(v[c] + bias[16 * q + c], 0.f),
                                  fmaxf(v[c + 1] + bias[16 * q + c + 1], 0.f));
            }
            *reinterpret_cast<uint4*>(A + umma_off(kTcRows, r, 16 * q + 8 * h)) = u;
        }
    }
}

__global__ void __launch_bounds__(kTcRows) mlp_infer_tc_kernel(const MlpW w,
                                                               const float* __restrict__ F,
                                                               long long n,
                                                               float* __restrict__ Y,
                                                               int32_t* status,
                                                               long long wait_ns) {
    extern __shared__ __align__(128) unsigned char tsm[];
    __shared__ __align__(8) unsigned long long bar;
    __shared__ unsigned tmem_slot;
    const int tid = threadIdx.x, warp = tid >> 5;
    unsigned char* A = tsm + kTcOffA;
    float* bias = reinterpret_cast<float*>(tsm + kTcOffB);
    stage_weights(tsm + kTcOffW1, w.W1, kHid, kHid, kIn, tid, kTcRows);
    stage_weights(tsm + kTcOffW2, w.W2, kHid, kHid, kHid, tid, kTcRows);
    stage_weights(tsm + kTcOffW3, w.W3, kHid, kHid, kHid, tid, kTcRows);
    stage_weights(tsm + kTcOffW4, w.W4, 2, kTcN4, kHid, tid, kTcRows);
    for (int i = tid; i < kHid; i += kTcRows) {
        bias[i] = __ldg(w.b1 + i);
        bias[kHid + i] = __ldg(w.b2 + i);
        bias[2 * kHid + i] = __ldg(w.b3 + i);
    }
    if (tid < 8) bias[3 * kHid + tid] = __ldg(w.b4 + tid);
    if (tid == 0) {
        htasync::bar_init(&bar, 1);
        htasync::bar_init_fence();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(htasync::smem_addr(&tmem_slot)), "r"(kTcCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    htasync::fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tmem_slot;
    const unsigned tmem_row = tmem + ((unsigned)(32 * warp) << 16);   // this warp's lanes
    const unsigned sA = htasync::smem_addr(A);
    const unsigned sW1 = htasync::smem_addr(tsm + kTcOffW1), sW2 = htasync::smem_addr(tsm + kTcOffW2),
                   sW3 = htasync::smem_addr(tsm + kTcOffW3), sW4 = htasync::smem_addr(tsm + kTcOffW4);
    const float* mean = w.mean;
    const float* istd = w.istd;
    const long long ntiles = (n + kTcRows - 1) / kTcRows;
    unsigned parity = 0;
    bool ok = true;
    // one layer: the MMAs over nk K steps, committed; every thread waits for them
    auto layer = [&](unsigned sB, int RB, int nk, int N) -> bool {
        htasync::fence_async_smem();   // this thread's A writes, seen by the tensor cores
        tc_fence_before();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            const unsigned idesc = umma_idesc(kTcRows, N);
            for (int s = 0; s < nk; ++s)
                umma_bf16(tmem, umma_desc(sA + s * (kTcRows * 32), kTcRows),
                          umma_desc(sB + s * (RB * 32), RB), idesc, s > 0 ? 1u : 0u);
            umma_commit(&bar);
        }
        const bool done = htasync::bar_wait(&bar, parity, wait_ns);
        parity ^= 1u;
        tc_fence_after();
        return !__syncthreads_or(!done);
    };
    for (long long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const long long row = tile * kTcRows + tid;
        {   // layer-1 input: the standardised features of this thread's peak, BF16
            float x[kIn];
#pragma unroll
            for (int c = 0; c < kIn; c += 4) {
                const float4 f4 = row < n ? __ldg(reinterpret_cast<const float4*>(F + row * kIn + c))
                                          : make_float4(0.f, 0.f, 0.f, 0.f);
                x[c] = f4.x; x[c + 1] = f4.y; x[c + 2] = f4.z; x[c + 3] = f4.w;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint4 u;
                unsigned* pu = reinterpret_cast<unsigned*>(&u);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = 8 * h + 2 * j;
                    const float a0 = row < n ? (x[c] - __ldg(mean + c)) * __ldg(istd + c) : 0.f;
                    const float a1 = row < n ? (x[c + 1] - __ldg(mean + c + 1)) * __ldg(istd + c + 1)
                                             : 0.f;
                    pu[j] = pack_bf16(a0, a1);
                }
                *reinterpret_cast<uint4*>(A + umma_off(kTcRows, tid, 8 * h)) = u;
            }
        }
        if (!(ok = layer(sW1, kHid, 1, kHid))) break;
        hidden_out(tmem_row, bias, A, tid);
        if (!(ok = layer(sW2, kHid, kHid / 16, kHid))) break;
        hidden_out(tmem_row, bias + kHid, A, tid);
        if (!(ok = layer(sW3, kHid, kHid / 16, kHid))) break;
        hidden_out(tmem_row, bias + 2 * kHid, A, tid);
        if (!(ok = layer(sW4, kTcN4, kHid / 16, kTcN4))) break;
        {
            unsigned u0, u1;
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];"
                         : "=r"(u0), "=r"(u1) : "r"(tmem_row));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (row < n) {
                Y[row * 2] = __uint_as_float(u0) + bias[3 * kHid];
                Y[row * 2 + 1] = __uint_as_float(u1) + bias[3 * kHid + 1];
            }
        }
    }
    if (!ok && tid == 0) {
        // record the timeout, then give the MMAs in flight a bounded time to finish
        atomicExch(status, kStatusWaitTimeout);
        htasync::bar_wait(&bar, parity ^ 1u, wait_ns);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     :: "r"(tmem), "r"(kTcCols));
    }
}

// --------------------------------------------------------------- training ----
//
// Gradient of the mean pinball loss in one kernel.  A CTA of 8 warps takes tiles of 128
// samples, persistent over the tiles; a warp carries 16 samples through the whole network
// in registers (mma.sync m16n8k16: the accumulator of one layer is, rounded to BF16, the A
// operand of the next), forward and back, and leaves the BF16 activations and dZ of its
// rows in shared memory.  The CTA then adds dZ^T H of the tile to the weight gradients,
// which stay in the warps' accumulators over all tiles (16 x 32 of dW2 and dW3, 16 x 8 of
// dW1 and dW4 each; ldmatrix.trans gives both operands with the samples as K).  Every CTA
// writes one partial gradient and train_reduce_kernel adds them in CTA order, so the
// result does not depend on timing.  What bounds it is the chain of dependent layers of a
// tile, not bytes (68 B a sample) or MMAs.
//
// The samples are the K of the weight gradients: a GEMM tiled over the 64 x 64 output ran
// them on one CTA, 26.1 ms of the 26.3 ms of a 65,536-sample gradient and Adam step; that
// step takes 44 us with this kernel (four tiles per CTA, one CTA per SM: 175 KB of shared
// memory and 255 registers hold a tile's matrices and every accumulator).

constexpr int kTrRows = 128, kTrWarps = 8, kTrThreads = 32 * kTrWarps;
constexpr int kTrS = 72, kTrSn = 24;      // row strides (BF16) of 64- and 16-wide matrices:
                                          // 36 and 12 words, conflict-free fragment reads
constexpr int kTrPart = HT_BRACKET_NPARAMS + 8;   // a CTA's partial: gradient, then the loss

// Shared-memory layout (bytes from the dynamic base).
constexpr int kTrBig = kTrRows * kTrS * 2, kTrNarrow = kTrRows * kTrSn * 2;
constexpr int kTrOffX = 0, kTrOffY = kTrOffX + kTrNarrow, kTrOffH = kTrOffY + kTrNarrow,
              kTrOffD = kTrOffH + 3 * kTrBig, kTrOffW1 = kTrOffD + 3 * kTrBig,
              kTrOffW = kTrOffW1 + kHid * kTrSn * 2,          // W2, W3 [out][in]
              kTrOffWT = kTrOffW + 2 * kHid * kTrS * 2,       // W2, W3 [in][out]
              kTrOffW4 = kTrOffWT + 2 * kHid * kTrS * 2,      // W4 [8][in]
              kTrOffW4T = kTrOffW4 + 8 * kTrS * 2,            // W4 [in][16]
              kTrOffB = kTrOffW4T + kHid * kTrSn * 2,         // b1 b2 b3 [64] b4 [8] FP32
              kTrOffR = kTrOffB + 200 * 4,                    // [8 warps][200] bias sums
              kTrSmem = kTrOffR + kTrWarps * 200 * 4;
static_assert(kTrSmem <= 227 * 1024, "one CTA per SM");

__device__ __forceinline__ void ldmatrix4_trans(unsigned (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(htasync::smem_addr(p)) : "memory");
}

__device__ __forceinline__ unsigned ld32(const __nv_bfloat16* p) {
    return *reinterpret_cast<const unsigned*>(p);
}

// c[j] (8 columns 8 j .. 8 j + 7, j < NJ) += A B over KS steps of 16, B (k, n) at
// W[n * stride + k].
template <int KS, int NJ>
__device__ __forceinline__ void warp_gemm(float (&c)[NJ][4], const unsigned (&a)[KS][4],
                                          const __nv_bfloat16* W, int stride, int g, int t) {
#pragma unroll
    for (int s = 0; s < KS; ++s)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const __nv_bfloat16* p = W + (8 * j + g) * stride + 16 * s + 2 * t;
            mma_bf16(c[j], a[s], ld32(p), ld32(p + 8));
        }
}

// The warp's 16 x 64 values c, rounded to BF16, as the next product's A operand and in
// rows g and g + 8 of S.
__device__ __forceinline__ void to_operand(const float (&c)[8][4], unsigned (&a)[4][4],
                                           __nv_bfloat16* S, int g, int t) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const unsigned lo = pack_bf16(c[j][0], c[j][1]), hi = pack_bf16(c[j][2], c[j][3]);
        a[j >> 1][2 * (j & 1)] = lo;
        a[j >> 1][2 * (j & 1) + 1] = hi;
        *reinterpret_cast<unsigned*>(S + g * kTrS + 8 * j + 2 * t) = lo;
        *reinterpret_cast<unsigned*>(S + (g + 8) * kTrS + 8 * j + 2 * t) = hi;
    }
}

// z = c + b, kept positions of z > 0, relu; then as to_operand.
__device__ __forceinline__ unsigned activate(float (&c)[8][4], const float* b,
                                             unsigned (&a)[4][4], __nv_bfloat16* S, int g,
                                             int t) {
    unsigned pos = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float z = c[j][e] + b[8 * j + 2 * t + (e & 1)];
            if (z > 0.f) pos |= 1u << (4 * j + e);
            c[j][e] = fmaxf(z, 0.f);
        }
    to_operand(c, a, S, g, t);
    return pos;
}

// dZ = dH where z > 0, added to the column sums; then as to_operand.
__device__ __forceinline__ void relu_back(float (&c)[8][4], unsigned pos, float (&db)[16],
                                          unsigned (&a)[4][4], __nv_bfloat16* S, int g,
                                          int t) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (!((pos >> (4 * j + e)) & 1u)) c[j][e] = 0.f;
        db[2 * j] += c[j][0] + c[j][2];
        db[2 * j + 1] += c[j][1] + c[j][3];
    }
    to_operand(c, a, S, g, t);
}

template <int NJ>
__device__ __forceinline__ void clear(float (&c)[NJ][4]) {
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) c[j][e] = 0.f;
}

__global__ void __launch_bounds__(kTrThreads, 1) train_grad_kernel(
    const MlpW w, const float* __restrict__ F, const float* __restrict__ tgt, long long n,
    float* __restrict__ part) {
    extern __shared__ __align__(128) unsigned char tsm[];
    auto mat = [&](int off) { return reinterpret_cast<__nv_bfloat16*>(tsm + off); };
    __nv_bfloat16 *Xs = mat(kTrOffX), *Ys = mat(kTrOffY), *W1 = mat(kTrOffW1),
                  *W4 = mat(kTrOffW4), *W4T = mat(kTrOffW4T);
    auto Hs = [&](int l) { return mat(kTrOffH + l * kTrBig); };
    auto Ds = [&](int l) { return mat(kTrOffD + l * kTrBig); };
    auto Wm = [&](int l) { return mat(kTrOffW + (l - 1) * kHid * kTrS * 2); };   // l = 1, 2
    auto WT = [&](int l) { return mat(kTrOffWT + (l - 1) * kHid * kTrS * 2); };
    float* bias = reinterpret_cast<float*>(tsm + kTrOffB);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const __nv_bfloat16 zero = __float2bfloat16(0.f);
    for (int e = tid; e < kHid * kHid; e += kTrThreads) {
        const int o = e / kHid, i = e % kHid;
        const __nv_bfloat16 v2 = w.W2[e], v3 = w.W3[e];
        Wm(1)[o * kTrS + i] = v2;
        WT(1)[i * kTrS + o] = v2;
        Wm(2)[o * kTrS + i] = v3;
        WT(2)[i * kTrS + o] = v3;
    }
    for (int e = tid; e < kHid * kIn; e += kTrThreads) {
        const int o = e / kIn, i = e % kIn;
        W1[o * kTrSn + i] = w.W1[e];
        W4T[o * kTrSn + i] = i < 2 ? w.W4[i * kHid + o] : zero;   // (in, out): two outputs
    }
    for (int e = tid; e < 8 * kHid; e += kTrThreads)
        W4[(e / kHid) * kTrS + e % kHid] = e < 2 * kHid ? w.W4[e] : zero;
    for (int e = tid; e < kTrRows * kTrSn; e += kTrThreads) Ys[e] = zero;
    if (tid < kHid) {
        bias[tid] = w.b1[tid];
        bias[kHid + tid] = w.b2[tid];
        bias[2 * kHid + tid] = w.b3[tid];
    }
    if (tid < 2) bias[3 * kHid + tid] = w.b4[tid];
    __syncthreads();

    // weight-gradient accumulators of this warp: rows (outputs) 16 mi .. 16 mi + 15
    const int mi = warp >> 1, nh = warp & 1;
    float g2[4][4], g3[4][4], g1[1][4], g4[1][4];   // columns 32 nh.., 32 nh.., 8 nh.., 8 warp..
    clear(g2);
    clear(g3);
    clear(g1);
    clear(g4);
    float db[3][16], db4[2] = {0.f, 0.f}, loss = 0.f;
#pragma unroll
    for (int l = 0; l < 3; ++l)
#pragma unroll
        for (int i = 0; i < 16; ++i) db[l][i] = 0.f;
    const float inv = 1.0f / (float)n;
    const int r0 = 16 * warp;                       // the warp's rows of the tile
    const long long ntiles = (n + kTrRows - 1) / kTrRows;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const long long ra = tile * kTrRows + r0 + g, rb = ra + 8;   // this thread's samples
        unsigned a[4][4], x[1][4];
        float c[8][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {               // x[0][q]: row ra / rb, inputs k, k + 1
            const long long r = (q & 1) ? rb : ra;
            const int k = 2 * t + 8 * (q >> 1);
            float v0 = 0.f, v1 = 0.f;
            if (r < n) {
                v0 = (__ldg(F + r * kIn + k) - __ldg(w.mean + k)) * __ldg(w.istd + k);
                v1 = (__ldg(F + r * kIn + k + 1) - __ldg(w.mean + k + 1)) * __ldg(w.istd + k + 1);
            }
            x[0][q] = pack_bf16(v0, v1);
            *reinterpret_cast<unsigned*>(Xs + (r0 + g + 8 * (q & 1)) * kTrSn + k) = x[0][q];
        }
        // forward
        unsigned pos[3];
        clear(c);
        warp_gemm<1, 8>(c, x, W1, kTrSn, g, t);
        pos[0] = activate(c, bias, a, Hs(0) + r0 * kTrS, g, t);
        clear(c);
        warp_gemm<4, 8>(c, a, Wm(1), kTrS, g, t);
        pos[1] = activate(c, bias + kHid, a, Hs(1) + r0 * kTrS, g, t);
        clear(c);
        warp_gemm<4, 8>(c, a, Wm(2), kTrS, g, t);
        pos[2] = activate(c, bias + 2 * kHid, a, Hs(2) + r0 * kTrS, g, t);
        float y[1][4];
        clear(y);
        warp_gemm<4, 1>(y, a, W4, kTrS, g, t);
        // pinball loss of the two quantiles (tau 0.1 and 0.9): columns 0, 1 sit in lanes t = 0
        unsigned dy[1][4] = {{0u, 0u, 0u, 0u}};
        if (t == 0) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const long long r = h ? rb : ra;
                float gq[2] = {0.f, 0.f};
                if (r < n) {
                    const float target = __ldg(tgt + r);
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const float tau = q ? 0.9f : 0.1f;
                        const float d = target - (y[0][2 * h + q] + bias[3 * kHid + q]);
                        loss += d > 0.f ? tau * d : (tau - 1.f) * d;
                        gq[q] = (d > 0.f ? -tau : 1.f - tau) * inv;
                        db4[q] += gq[q];
                    }
                }
                dy[0][h] = pack_bf16(gq[0], gq[1]);
                *reinterpret_cast<unsigned*>(Ys + (r0 + g + 8 * h) * kTrSn) = dy[0][h];
            }
        }
        __syncwarp();
        // backward
        clear(c);
        warp_gemm<1, 8>(c, dy, W4T, kTrSn, g, t);
        relu_back(c, pos[2], db[2], a, Ds(2) + r0 * kTrS, g, t);
        clear(c);
        warp_gemm<4, 8>(c, a, WT(2), kTrS, g, t);
        relu_back(c, pos[1], db[1], a, Ds(1) + r0 * kTrS, g, t);
        clear(c);
        warp_gemm<4, 8>(c, a, WT(1), kTrS, g, t);
        relu_back(c, pos[0], db[0], a, Ds(0) + r0 * kTrS, g, t);
        __syncthreads();
        // weight gradients: K = the tile's 128 samples
        const int lr = lane & 7, q = lane >> 3;
        const int ka = lr + 8 * (q >> 1), ma = 8 * (q & 1);   // A: (k, m) blocks 00 01 10 11
        const int kb = lr + 8 * (q & 1), nb = 8 * (q >> 1);   // B: (k, n) blocks 00 10 01 11
#pragma unroll 2
        for (int k0 = 0; k0 < kTrRows; k0 += 16) {
            unsigned A[4], B[4];
#pragma unroll
            for (int l = 1; l < 3; ++l) {
                ldmatrix4_trans(A, Ds(l) + (k0 + ka) * kTrS + 16 * mi + ma);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    ldmatrix4_trans(B, Hs(l - 1) + (k0 + kb) * kTrS + 32 * nh + 16 * h + nb);
                    auto& acc = l == 1 ? g2 : g3;
                    mma_bf16(acc[2 * h], A, B[0], B[1]);
                    mma_bf16(acc[2 * h + 1], A, B[2], B[3]);
                }
            }
            ldmatrix4_trans(A, Ds(0) + (k0 + ka) * kTrS + 16 * mi + ma);
            ldmatrix4_trans(B, Xs + (k0 + kb) * kTrSn + nb);
            mma_bf16(g1[0], A, nh ? B[2] : B[0], nh ? B[3] : B[1]);
            ldmatrix4_trans(A, Ys + (k0 + ka) * kTrSn + ma);
            ldmatrix4_trans(B, Hs(2) + (k0 + kb) * kTrS + 16 * (warp >> 1) + nb);
            mma_bf16(g4[0], A, nh ? B[2] : B[0], nh ? B[3] : B[1]);
        }
        __syncthreads();   // the tile's matrices have been read
    }

    // this CTA's partial gradient: W1 [64x16] W2 W3 [64x64] W4 [8x64] b1 b2 b3 [64] b4 [8]
    float* P = part + (size_t)blockIdx.x * kTrPart;
    auto put = [&](float* M, int ld, int m0, int n0, const float (&v)[4], int rows) {
        if (m0 + g < rows)
            *reinterpret_cast<float2*>(M + (m0 + g) * ld + n0 + 2 * t) = make_float2(v[0], v[1]);
        if (m0 + g + 8 < rows)
            *reinterpret_cast<float2*>(M + (m0 + g + 8) * ld + n0 + 2 * t) =
                make_float2(v[2], v[3]);
    };
    put(P, kIn, 16 * mi, 8 * nh, g1[0], kHid);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        put(P + 1024, kHid, 16 * mi, 32 * nh + 8 * j, g2[j], kHid);
        put(P + 5120, kHid, 16 * mi, 32 * nh + 8 * j, g3[j], kHid);
    }
    if (g >= 2) g4[0][0] = g4[0][1] = 0.f;   // W4's padding rows, whatever the activations
    put(P + 9216, kHid, 0, 8 * warp, g4[0], 8);
    // bias gradients and the loss: over the rows of the warp, then over the warps in order
    float* R = reinterpret_cast<float*>(tsm + kTrOffR) + warp * 200;
#pragma unroll
    for (int l = 0; l < 3; ++l)
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float v = db[l][i];
            for (int o = 4; o <= 16; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (g == 0) R[l * kHid + 8 * (i >> 1) + 2 * t + (i & 1)] = v;
        }
    float v[3] = {db4[0], db4[1], loss};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        for (int o = 4; o <= 16; o <<= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
        if (lane == 0) R[192 + i] = v[i];
    }
    __syncthreads();
    const float* R0 = reinterpret_cast<const float*>(tsm + kTrOffR);
    if (tid < 195) {
        float s = 0.f;
        for (int k = 0; k < kTrWarps; ++k) s += R0[k * 200 + tid];
        P[tid < 194 ? 9728 + tid : HT_BRACKET_NPARAMS] = s;
    } else if (tid < 201) {
        P[9728 + tid - 1] = 0.f;   // b4's padding
    }
}

// grads[i] = the sum of the CTAs' partials in order (8 strided sums, then those in order);
// loss = its sum / n.  A block takes 32 neighbouring values.
__global__ void __launch_bounds__(256) train_reduce_kernel(const float* __restrict__ part,
                                                           int ctas, long long n,
                                                           float* __restrict__ grads,
                                                           float* __restrict__ loss) {
    __shared__ float red[8][33];
    const int c = threadIdx.x & 31, k = threadIdx.x >> 5, i = blockIdx.x * 32 + c;
    float s = 0.f;
    if (i <= HT_BRACKET_NPARAMS)
        for (int b = k; b < ctas; b += 8) s += __ldg(part + (size_t)b * kTrPart + i);
    red[k][c] = s;
    __syncthreads();
    if (k == 0 && i <= HT_BRACKET_NPARAMS) {
        s = 0.f;
#pragma unroll
        for (int q = 0; q < 8; ++q) s += red[q][c];
        if (i < HT_BRACKET_NPARAMS) grads[i] = s;
        else *loss = s / (float)n;
    }
}

// Adam on the packed FP32 parameters; writes the BF16 weights and FP32 biases of `out`.
struct PackedModel {
    __nv_bfloat16* W[4];
    float* b[4];
};

__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ gr,
                            float* __restrict__ m, float* __restrict__ v, int n, float lr,
                            float b1t, float b2t, PackedModel out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float g = gr[i];
    const float mi = 0.9f * m[i] + 0.1f * g;
    const float vi = 0.999f * v[i] + 0.001f * g * g;
    m[i] = mi;
    v[i] = vi;
    const float mh = mi / (1.f - b1t), vh = vi / (1.f - b2t);
    const float pi = p[i] - lr * mh / (sqrtf(vh) + 1e-8f);
    p[i] = pi;
    // packed layout: W1 [64x16] W2 [64x64] W3 [64x64] W4 [8x64] b1 b2 b3 [64] b4 [8]
    const int off[9] = {0, 1024, 5120, 9216, 9728, 9792, 9856, 9920, 9928};
    for (int s = 0; s < 8; ++s) {
        if (i >= off[s] && i < off[s + 1]) {
            if (s < 4) out.W[s][i - off[s]] = __float2bfloat16(pi);
            else out.b[s - 4][i - off[s]] = pi;
        }
    }
}

}  // namespace

// ------------------------------------------------------------------ C ABI ----

namespace {

int check_model(const ht_bracket_model* m, const char* who) {
    if (!m || !m->W1 || !m->W2 || !m->W3 || !m->W4 || !m->b1 || !m->b2 || !m->b3 || !m->b4 ||
        !m->mean || !m->istd)
        return ht_fail(HT_ERR_INVALID, std::string(who) + ": NULL model array");
    return HT_OK;
}

MlpW mlp_of(const ht_bracket_model* m) {
    MlpW w;
    w.W1 = (const __nv_bfloat16*)m->W1; w.W2 = (const __nv_bfloat16*)m->W2;
    w.W3 = (const __nv_bfloat16*)m->W3; w.W4 = (const __nv_bfloat16*)m->W4;
    w.b1 = m->b1; w.b2 = m->b2; w.b3 = m->b3; w.b4 = m->b4;
    w.mean = m->mean; w.istd = m->istd;
    return w;
}

unsigned blocks_for(long long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

extern "C" HT_API int ht_bracket_features(ht_ctx* ctx, const ht_peak_batch* b,
                                          const float* d_peak_delta, double alatt,
                                          float* d_feat, void* stream) {
    HT_RANGE("ht_bracket_features");
    if (!ctx || !b || !d_feat) return ht_fail(HT_ERR_INVALID, "ht_bracket_features: NULL argument");
    if (!ctx->bound) return ht_fail(HT_ERR_STATE, "ht_bracket_features: no tile bound (ht_fields_pack)");
    if (b->npeaks < 0) return ht_fail(HT_ERR_INVALID, "ht_bracket_features: npeaks < 0");
    if (!(alatt > 0.0)) return ht_fail(HT_ERR_INVALID, "ht_bracket_features: alatt must be > 0");
    if (b->npeaks == 0) return HT_OK;
    if (!b->pi || !b->pj || !b->pk || !b->Rf || !b->ir2min || !b->ZZon || !b->fcrit)
        return ht_fail(HT_ERR_INVALID, "ht_bracket_features: NULL peak array");
    HT_CUDA_TRY(cudaSetDevice(ctx->device), "cudaSetDevice");
    FeatArgs a;
    const ht_fields& f = ctx->fields;
    a.rec = ctx->d_rec; a.delta = f.delta;
    a.n1 = f.n1; a.n2 = f.n2; a.n3 = f.n3; a.s2 = (long long)f.n1 * f.n2;
    a.off = ctx->d_off; a.start = ctx->d_start; a.count = ctx->d_count; a.r2 = ctx->d_r2;
    a.rad = ctx->d_rad; a.nshells = ctx->nshells;
    a.pi = b->pi; a.pj = b->pj; a.pk = b->pk; a.Rf = b->Rf; a.ir2min = b->ir2min;
    a.ZZon = b->ZZon; a.fcrit = b->fcrit; a.peak_delta = d_peak_delta;
    a.npeaks = b->npeaks; a.alatt = alatt;
    features_kernel<<<blocks_for(b->npeaks, 256), 256, 0, (cudaStream_t)stream>>>(a, d_feat);
    HT_CUDA_TRY(cudaGetLastError(), "features_kernel launch");
    ctx->last_kernels = 1;
    return HT_OK;
}

extern "C" HT_API int ht_bracket_predict(ht_ctx* ctx, const ht_bracket_model* m,
                                         const float* d_feat, int64_t n, float* d_pred,
                                         void* stream) {
    HT_RANGE("ht_bracket_predict");
    if (!ctx || !d_feat || !d_pred) return ht_fail(HT_ERR_INVALID, "ht_bracket_predict: NULL argument");
    int rc = check_model(m, "ht_bracket_predict");
    if (rc != HT_OK) return rc;
    if (n < 0) return ht_fail(HT_ERR_INVALID, "ht_bracket_predict: n < 0");
    if (n == 0) return HT_OK;
    if (((uintptr_t)d_feat & 15u) != 0)
        return ht_fail(HT_ERR_INVALID, "ht_bracket_predict: d_feat must be 16-byte aligned");
    HT_CUDA_TRY(cudaSetDevice(ctx->device), "cudaSetDevice");
    // persistent CTAs of 128 peaks, four per SM (each holds 64 tensor-memory columns)
    const long long tiles = (n + kTcRows - 1) / kTcRows;
    const unsigned grid = (unsigned)std::min<long long>(tiles, 4LL * ctx->num_sms);
    mlp_infer_tc_kernel<<<grid, kTcRows, kTcSmem, (cudaStream_t)stream>>>(
        mlp_of(m), d_feat, n, d_pred, ht_status_word(ctx), ctx->wait_ns);
    HT_CUDA_TRY(cudaGetLastError(), "mlp_infer_tc_kernel launch");
    ctx->last_kernels = 1;
    return HT_OK;
}

extern "C" HT_API int ht_bracket_grad(ht_ctx* ctx, const ht_bracket_model* m,
                                      const float* d_feat, const float* d_target, int64_t n,
                                      float* d_grads, float* d_loss, void* stream) {
    HT_RANGE("ht_bracket_grad");
    if (!ctx || !d_feat || !d_target || !d_grads || !d_loss)
        return ht_fail(HT_ERR_INVALID, "ht_bracket_grad: NULL argument");
    int rc = check_model(m, "ht_bracket_grad");
    if (rc != HT_OK) return rc;
    if (n < 1 || n > (1LL << 24)) return ht_fail(HT_ERR_INVALID, "ht_bracket_grad: need 1 <= n <= 2^24");
    HT_CUDA_TRY(cudaSetDevice(ctx->device), "cudaSetDevice");
    cudaStream_t st = (cudaStream_t)stream;
    const long long tiles = (n + kTrRows - 1) / kTrRows;
    const int ctas = (int)std::min<long long>(tiles, ctx->num_sms);
    rc = ht_grow(&ctx->d_mlp_ws, &ctx->mlp_ws_bytes, (size_t)ctas * kTrPart * sizeof(float),
                 "bracket training workspace");
    if (rc != HT_OK) return rc;
    float* part = (float*)ctx->d_mlp_ws;
    HT_CUDA_TRY(cudaFuncSetAttribute(train_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrSmem), "train_grad smem");
    train_grad_kernel<<<ctas, kTrThreads, kTrSmem, st>>>(mlp_of(m), d_feat, d_target, n, part);
    HT_CUDA_TRY(cudaGetLastError(), "train_grad_kernel launch");
    train_reduce_kernel<<<blocks_for(HT_BRACKET_NPARAMS + 1, 32), 256, 0, st>>>(part, ctas, n,
                                                                               d_grads, d_loss);
    HT_CUDA_TRY(cudaGetLastError(), "train_reduce_kernel launch");
    ctx->last_kernels = 2;
    return HT_OK;
}

extern "C" HT_API int ht_bracket_adam(ht_ctx* ctx, float* d_params, const float* d_grads,
                                      float* d_m, float* d_v, int32_t step, float lr,
                                      const ht_bracket_model* out, void* stream) {
    HT_RANGE("ht_bracket_adam");
    if (!ctx || !d_params || !d_grads || !d_m || !d_v)
        return ht_fail(HT_ERR_INVALID, "ht_bracket_adam: NULL argument");
    int rc = check_model(out, "ht_bracket_adam");
    if (rc != HT_OK) return rc;
    if (step < 1) return ht_fail(HT_ERR_INVALID, "ht_bracket_adam: step counts from 1");
    HT_CUDA_TRY(cudaSetDevice(ctx->device), "cudaSetDevice");
    PackedModel pm;
    pm.W[0] = (__nv_bfloat16*)out->W1; pm.W[1] = (__nv_bfloat16*)out->W2;
    pm.W[2] = (__nv_bfloat16*)out->W3; pm.W[3] = (__nv_bfloat16*)out->W4;
    pm.b[0] = out->b1; pm.b[1] = out->b2; pm.b[2] = out->b3; pm.b[3] = out->b4;
    const float b1t = powf(0.9f, (float)step), b2t = powf(0.999f, (float)step);
    adam_kernel<<<blocks_for(HT_BRACKET_NPARAMS, 256), 256, 0, (cudaStream_t)stream>>>(
        d_params, d_grads, d_m, d_v, HT_BRACKET_NPARAMS, lr, b1t, b2t, pm);
    HT_CUDA_TRY(cudaGetLastError(), "adam_kernel launch");
    ctx->last_kernels = 1;
    return HT_OK;
}
