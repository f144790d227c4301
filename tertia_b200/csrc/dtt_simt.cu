// dtt_simt.cu — half-integer DCT-IV / DST-IV transforms as batched dense
// GEMMs, exact FP32 or FP64.
//
// Replaces the reference's FFTW REDFT11/RODFT11 plans
// (movefieldshydrolinlayersplit.cpp:389-427) and the dead cuFFT twin
// CUDA_WRAP_fourierHalfInteger2D (half_integer2D.cu:583).  The design is the
// reference's own dense-matrix attempt (surfaceFFT.cu:108-164) scaled up:
// Y = A_z X A_y, computed as two passes of out = (in . A)^T so each pass
// reads its operand row-major and the transpose lands in the epilogue.
// This is the plain FP64 path and the exact-FP32 path; the split-precision
// tensor-core path is dtt_tc.cu.
#include <algorithm>
#include <cstdint>

#include "qs_common.cuh"
#include "qs_internal.h"
#include "pdl.cuh"

namespace qs {

namespace {

constexpr int kBM = 32, kBN = 32;   // output tile of a block
constexpr int kKC = 64;             // k values per stage
constexpr int kLD = kKC + 4;        // stage row: 4 mod 16 doubles (4 mod 32 floats) apart, so
                                    // that a fragment's 8 rows fall on distinct banks
constexpr int kStages = 2;
constexpr int kWarps = 4;           // the warps split a stage's k values

template <class T>
constexpr size_t stage_bytes() { return (size_t)(kBM + kBN) * kLD * sizeof(T); }

template <int BYTES>
__device__ __forceinline__ void cp_async(void* s, const void* g, bool ok) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(s);
    const int n = ok ? BYTES : 0;   // 0: the slot is filled with zeros, nothing is read
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(g), "r"(n)
                     : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(g), "n"(BYTES),
                     "r"(n)
                     : "memory");
}

// rows row0 .. row0+31 (below nrows) x columns k0 .. k0+63 (below K) of a
// row-major matrix of K columns into a stage; K is a multiple of 8, so whole
// 16-byte pieces are in or out
template <class T, int BYTES>
__device__ __forceinline__ void load_rows(T* S, const T* __restrict__ g, int row0, int nrows,
                                          int k0, int K) {
    constexpr int E = BYTES / (int)sizeof(T);   // values per copy
    constexpr int PER = kKC / E;
    for (int i = threadIdx.x; i < kBM * PER; i += 32 * kWarps) {
        const int r = i / PER, c = (i % PER) * E;
        const bool ok = row0 + r < nrows && k0 + c < K;
        cp_async<BYTES>(S + r * kLD + c, ok ? g + (size_t)(row0 + r) * K + k0 + c : g, ok);
    }
}

// one 8x8x4 FP64 tensor-core product: lane (g = lane/4, t = lane%4) holds
// a(g, t), b(t, g) and c(g, 2t), c(g, 2t+1)
__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// a warp's share of a stage: acc += in rows x matrix rows over its 16 k values
struct TileF64 {
    double c[4][4][2];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) c[i][j][0] = c[i][j][1] = 0.0;
    }
    __device__ __forceinline__ void add(const double* A, const double* B, int kw, int lane) {
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int k = 0; k < kKC / kWarps; k += 4) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                a[i] = A[(8 * i + g) * kLD + kw + k + t];
                b[i] = B[(8 * i + g) * kLD + kw + k + t];
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) mma_f64(c[i][j], a[i], b[j]);
        }
    }
    // partial sums as [col][row] with rows 33 apart
    __device__ __forceinline__ void put(double* P, int lane) const {
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int e = 0; e < 2; e++) P[(8 * j + 2 * t + e) * 33 + 8 * i + g] = c[i][j][e];
    }
};

struct TileF32 {
    float c[4][8];   // rows lr + 8 i, columns lc + 4 j
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) c[i][j] = 0.f;
    }
    __device__ __forceinline__ void add(const float* A, const float* B, int kw, int lane) {
        const int lr = lane & 7, lc = lane >> 3;
#pragma unroll
        for (int k = 0; k < kKC / kWarps; k += 4) {
            float4 a[4];
#pragma unroll
            for (int i = 0; i < 4; i++)
                a[i] = *reinterpret_cast<const float4*>(A + (lr + 8 * i) * kLD + kw + k);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float4 b = *reinterpret_cast<const float4*>(B + (lc + 4 * j) * kLD + kw + k);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    c[i][j] = fmaf(a[i].x, b.x, c[i][j]);
                    c[i][j] = fmaf(a[i].y, b.y, c[i][j]);
                    c[i][j] = fmaf(a[i].z, b.z, c[i][j]);
                    c[i][j] = fmaf(a[i].w, b.w, c[i][j]);
                }
            }
        }
    }
    __device__ __forceinline__ void put(float* P, int lane) const {
        const int lr = lane & 7, lc = lane >> 3;
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) P[(lc + 4 * j) * 33 + lr + 8 * i] = c[i][j];
    }
};

template <class T> struct TileOf;
template <> struct TileOf<double> { using type = TileF64; };
template <> struct TileOf<float> { using type = TileF32; };

// A pass over planes of 100 to 250 cells a side is a few output tiles per SM
// at most, so its time is one block's serial chain: with 64 x 64 (FP64) and
// 128 x 128 (FP32) tiles and 8 k values per step a 128 x 128 pass of 6 planes
// kept 24 blocks busy for 21.7 us.  A block therefore takes a 32 x 32 tile
// with 128 k values in flight (two stages of 64, 16-byte cp.async), and its
// four warps split the k values of every stage and add their partial tiles in
// a fixed order at the end.  FP64 products run on the FP64 tensor cores
// (8 x 8 x 4, IEEE FMA), whose fragments need an eighth of the shared-memory
// reads of a SIMT tile.  Two stages (70 KB in FP64) keep three blocks on an
// SM; four stages leave one and lose at every size from 128 up.  `mat` is
// symmetric, so its rows serve as its columns.  Two passes of 6 planes, 64x64 or
// 128x128 tiles before -> this kernel: FP64 128^2 45.1 -> 12.4 us, 256^2
// 77.9 -> 28.7 us, 512^2 377 -> 151 us (22 TFLOP/s); FP32 96 x 160
// 56.5 -> 14.4 us, 768 x 640 507 -> 290 us.
template <class T>
__global__ void __launch_bounds__(32 * kWarps) dtt_dense_kernel(DttPassArgs<T> a, int nbuf,
                                                               int aligned) {
    extern __shared__ __align__(16) unsigned char smem_dense[];
    T* S = reinterpret_cast<T*>(smem_dense);
    constexpr int STAGE = (kBM + kBN) * kLD;
    const int f = blockIdx.z;
    const T* __restrict__ A = a.in[f];
    const T* __restrict__ B = a.mat[f];
    T* __restrict__ O = a.out[f];
    const int R = a.R, K = a.K;
    const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * kBN;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nk = (K + kKC - 1) / kKC;
    auto load_mat = [&](int kt) {
        T* Sb = S + (kt % nbuf) * STAGE + kBM * kLD;
        if (kt < nk) load_rows<T, 16>(Sb, B, n0, K, kt * kKC, K);
    };
    auto load_in = [&](int kt) {
        T* Sa = S + (kt % nbuf) * STAGE;
        if (kt < nk) {
            if (aligned) load_rows<T, 16>(Sa, A, m0, R, kt * kKC, K);
            else load_rows<T, (int)sizeof(T)>(Sa, A, m0, R, kt * kKC, K);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the matrix does not depend on the kernel before this one
    for (int kt = 0; kt < kStages; kt++) load_mat(kt);
    pdl_wait();
    for (int kt = 0; kt < kStages; kt++) load_in(kt);
    typename TileOf<T>::type acc;
    acc.zero();
    for (int kt = 0; kt < nk; kt++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
        __syncthreads();
        const T* Sa = S + (kt % nbuf) * STAGE;
        acc.add(Sa, Sa + kBM * kLD, w * (kKC / kWarps), lane);
        __syncthreads();   // the stage is free
        load_mat(kt + kStages);
        load_in(kt + kStages);
    }
    pdl_trigger();
    // the warps' partial tiles, added in warp order; out[n][m] (transposed),
    // consecutive threads cover consecutive m
    acc.put(S + w * (kBN * 33), lane);
    __syncthreads();
    const T s = a.scale;
    const int gm = m0 + lane;
    if (gm >= R) return;
#pragma unroll
    for (int q = 0; q < kBN / kWarps; q++) {
        const int c = w + kWarps * q, gn = n0 + c;
        T v = S[c * 33 + lane];
#pragma unroll
        for (int p = 1; p < kWarps; p++) v += S[p * (kBN * 33) + c * 33 + lane];
        if (gn < K) O[(size_t)gn * R + gm] = v * s;
    }
}

}  // namespace

template <class T>
cudaError_t dtt_dense_setup() {
    return cudaFuncSetAttribute(dtt_dense_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(kStages * stage_bytes<T>()));
}
template cudaError_t dtt_dense_setup<float>();
template cudaError_t dtt_dense_setup<double>();

template <class T>
static void launch_pass(const DttPassArgs<T>& a, int nf, cudaStream_t st) {
    static_assert(kWarps * kBN * 33 <= (kBM + kBN) * kLD, "the partial tiles fit one stage");
    // 16-byte copies where every plane starts on one (its rows are multiples
    // of 8 values), else one value at a time
    uintptr_t bits = 0;
    for (int f = 0; f < nf; f++) bits |= (uintptr_t)a.in[f];
    const dim3 grid((a.R + kBM - 1) / kBM, (a.K + kBN - 1) / kBN, nf);
    const int nbuf = std::min((a.K + kKC - 1) / kKC, kStages);
    launch_pdl(dtt_dense_kernel<T>, grid, dim3(32 * kWarps), (size_t)nbuf * stage_bytes<T>(), st, a,
               nbuf, (int)((bits & 15) == 0));
}

template <class T>
int run_dtt_simt_pass(int pass, const DttJob<T>& job, int ny, int nz, const DttMats<T>& my,
                      const DttMats<T>& mz, T* scratch, cudaStream_t st) {
    if (job.nf <= 0) return 0;
    const size_t plane = (size_t)ny * nz;
    DttPassArgs<T> a{};
    for (int f = 0; f < job.nf; f++) {
        if (pass == 0) {
            a.in[f] = job.in[f];
            a.mat[f] = my.m[job.ky[f]];
            a.out[f] = scratch + f * plane;
        } else {
            a.in[f] = scratch + f * plane;
            a.mat[f] = mz.m[job.kz[f]];
            a.out[f] = job.out[f];
        }
    }
    if (pass == 0) { a.R = nz; a.K = ny; a.scale = T(1); }
    else { a.R = ny; a.K = nz; a.scale = job.scale; }
    launch_pass<T>(a, job.nf, st);
    return 1;
}

template <class T>
int run_dtt_simt(const DttJob<T>& job, int ny, int nz, const DttMats<T>& my,
                 const DttMats<T>& mz, T* scratch, cudaStream_t st) {
    return run_dtt_simt_pass<T>(0, job, ny, nz, my, mz, scratch, st) +
           run_dtt_simt_pass<T>(1, job, ny, nz, my, mz, scratch, st);
}

template int run_dtt_simt_pass<float>(int, const DttJob<float>&, int, int, const DttMats<float>&,
                                      const DttMats<float>&, float*, cudaStream_t);
template int run_dtt_simt_pass<double>(int, const DttJob<double>&, int, int,
                                       const DttMats<double>&, const DttMats<double>&, double*,
                                       cudaStream_t);
template int run_dtt_simt<float>(const DttJob<float>&, int, int, const DttMats<float>&,
                                 const DttMats<float>&, float*, cudaStream_t);
template int run_dtt_simt<double>(const DttJob<double>&, int, int, const DttMats<double>&,
                                  const DttMats<double>&, double*, cudaStream_t);

}  // namespace qs
