// aphid_unet.cu -- the initial-guess network's device side: the tcgen05 BF16
// GEMM launcher and (below) the layers: convolutions as implicit GEMMs
// (unet_conv.cuh) and the memory-bound passes between them.  Activations are BF16 in
// planes of 8 channels [C/8][Vp][8], gradients FP32 channels last [Vp][C].
// C ABI in include/aphid_unet.h.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <random>
#include <string>
#include <vector>

#include "../../include/aphid_unet.h"
#include "unet_conv.cuh"
#include "unet_gemm.cuh"

namespace aphid {
namespace unet {

namespace {

thread_local std::string g_last_error = "no error";

int set_err(int code, const std::string &msg) {
  g_last_error = msg;
  return code;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess) f = nullptr;
    return (EncodeTiledFn)f;
  }();
  return fn;
}

// a row-major BF16 matrix (rows x cols, leading dimension ld elements) as a
// 2-D tensor of box cols_box x rows_box, 128-byte swizzle
int bf16_map(CUtensorMap *m, const __nv_bfloat16 *base, int rows, int cols, int ld, int rows_box) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return set_err(APHID_UNET_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)rows_box}, es[2] = {1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16 *>(base), dims, strides, box,
                        es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return set_err(APHID_UNET_ERR_CUDA, "cuTensorMapEncodeTiled (gemm): " + std::to_string((int)r));
  return APHID_UNET_OK;
}

template <int BN, int OUT>
int launch_gemm_t(const __nv_bfloat16 *A, int lda, const __nv_bfloat16 *B, int ldb, void *C, int ldc,
                  const float *bias, int M, int N, int K, int splitk, cudaStream_t st, int *err) {
  const size_t shm = TmaShm<BN>::bytes;
  static bool attr = false;  // once per instantiation and process
  if (!attr) {
    if (cudaFuncSetAttribute(k_gemm_tma<BN, OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm) !=
        cudaSuccess)
      return set_err(APHID_UNET_ERR_CUDA, "cudaFuncSetAttribute (gemm)");
    attr = true;
  }
  CUtensorMap ma, mb;
  int rc;
  if ((rc = bf16_map(&ma, A, M, K, lda, kBM)) || (rc = bf16_map(&mb, B, N, K, ldb, BN))) return rc;
  const int nkb = K / kBK;
  const int per = (nkb + splitk - 1) / splitk;
  // 16-byte output stores where every row start is 16-byte aligned
  const size_t es = (OUT == OUT_BF16_RELU || OUT == OUT_BF16) ? 2 : 4;
  const int vec = (reinterpret_cast<uintptr_t>(C) % 16 == 0) && ((size_t)ldc * es) % 16 == 0;
  dim3 grid((unsigned)(M / kBM), (unsigned)(N / BN), (unsigned)((nkb + per - 1) / per));
  k_gemm_tma<BN, OUT><<<grid, kGemmThreads, shm, st>>>(ma, mb, C, ldc, bias, K, per * kBK, vec, err);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_err(APHID_UNET_ERR_CUDA, std::string("gemm launch: ") + cudaGetErrorString(e));
  return APHID_UNET_OK;
}

template <int OUT>
int launch_gemm_o(const __nv_bfloat16 *A, int lda, const __nv_bfloat16 *B, int ldb, void *C, int ldc,
                  const float *bias, int M, int N, int K, int splitk, cudaStream_t st, int *err) {
  if (N % 128 == 0) return launch_gemm_t<128, OUT>(A, lda, B, ldb, C, ldc, bias, M, N, K, splitk, st, err);
  if (N % 64 == 0) return launch_gemm_t<64, OUT>(A, lda, B, ldb, C, ldc, bias, M, N, K, splitk, st, err);
  if (N % 32 == 0) return launch_gemm_t<32, OUT>(A, lda, B, ldb, C, ldc, bias, M, N, K, splitk, st, err);
  return launch_gemm_t<16, OUT>(A, lda, B, ldb, C, ldc, bias, M, N, K, splitk, st, err);
}

}  // namespace

// C (op)= A B^T on the tensor cores; see unet_gemm.cuh for the shapes
int gemm_bf16(const __nv_bfloat16 *A, int lda, const __nv_bfloat16 *B, int ldb, void *C, int ldc,
              const float *bias, int M, int N, int K, int out, int splitk, cudaStream_t st, int *err) {
  if (M <= 0 || N <= 0 || K <= 0 || M % kBM || N % 16 || K % kBK || lda % 8 || ldb % 8 || lda < K || ldb < K ||
      ldc < N || splitk < 1)
    return set_err(APHID_UNET_ERR_BADARG, "gemm: M % 128, N % 16, K % 64 and the leading dimensions");
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15)
    return set_err(APHID_UNET_ERR_BADARG, "gemm: A and B must be 16-byte aligned");
  if (splitk > 1 && out != OUT_F32_ATOMIC)
    return set_err(APHID_UNET_ERR_BADARG, "gemm: split-K needs the atomic output");
  switch (out) {
    case OUT_F32: return launch_gemm_o<OUT_F32>(A, lda, B, ldb, C, ldc, bias, M, N, K, splitk, st, err);
    case OUT_BF16_RELU: return launch_gemm_o<OUT_BF16_RELU>(A, lda, B, ldb, C, ldc, bias, M, N, K, splitk, st, err);
    case OUT_BF16: return launch_gemm_o<OUT_BF16>(A, lda, B, ldb, C, ldc, bias, M, N, K, splitk, st, err);
    case OUT_F32_ATOMIC: return launch_gemm_o<OUT_F32_ATOMIC>(A, lda, B, ldb, C, ldc, bias, M, N, K, splitk, st, err);
  }
  return set_err(APHID_UNET_ERR_BADARG, "gemm: unknown output operation");
}

}  // namespace unet
}  // namespace aphid


namespace aphid {
namespace unet {
namespace {

constexpr int kT = 256;  // threads of the elementwise kernels

__host__ __device__ inline long long rup(long long a, long long b) { return (a + b - 1) / b * b; }
inline unsigned nblk(long long n) { return (unsigned)std::min<long long>((n + kT - 1) / kT, 148LL * 64); }

struct Vol {
  int X, Y, Z;
  long long V, Vp;  // voxels, rows padded to 128
};

// ---------------------------------------------------------------- kernels
// features [V][3] (original volume) -> [Vp][8] BF16 on the padded volume
// (a voxel index fits 32 bits: 2^32 voxels would be 400 GB of activations; a
// 64-bit division per value made these passes 2 to 8 x their memory time)
struct Xyz { int x, y, z; };
__device__ __forceinline__ Xyz xyz(unsigned r, int X, int Y) {
  const unsigned q = r / (unsigned)X, z = q / (unsigned)Y;
  return {(int)(r - q * X), (int)(q - z * Y), (int)z};
}
__global__ void k_pack_in(const float *__restrict__ x, int X, int Y, int Z, Vol v, __nv_bfloat16 *__restrict__ a) {
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < v.Vp; r += (long long)gridDim.x * blockDim.x) {
    float f[3] = {};
    if (r < v.V) {
      const Xyz p = xyz((unsigned)r, v.X, v.Y);
      if (p.x < X && p.y < Y && p.z < Z) {
        const float *s = x + (p.x + (long long)X * (p.y + (long long)Y * p.z)) * 3;
        f[0] = s[0], f[1] = s[1], f[2] = s[2];
      }
    }
    auto b = [](float q) { return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(q)); };
    reinterpret_cast<uint4 *>(a)[r] = make_uint4(b(f[0]) | (b(f[1]) << 16), b(f[2]), 0, 0);
  }
}
// head output [Vp][16] FP32 -> [V][8] on the original volume
__global__ void k_unpack_out(const float *__restrict__ y, int X, int Y, int Z, Vol v, float *__restrict__ o) {
  const long long n = (long long)X * Y * Z * 2;
  const bool vec = ((uintptr_t)o & 15) == 0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const Xyz p = xyz((unsigned)(t >> 1), X, Y);
    const float4 f = reinterpret_cast<const float4 *>(y)[(p.x + (long long)v.X * (p.y + (long long)v.Y * p.z)) * 4 + (t & 1)];
    if (vec)
      reinterpret_cast<float4 *>(o)[t] = f;
    else
      o[4 * t] = f.x, o[4 * t + 1] = f.y, o[4 * t + 2] = f.z, o[4 * t + 3] = f.w;
  }
}

// dz = g * (act > 0) (relu) or g; dZ in planes of 8 channels, BF16, rows past the
// volume zero, and gb[c] += sum_r dz[r][c] before the rounding.  A thread takes 8
// channels (plane blockIdx.y) of its voxels; gb has room for whole planes.
__global__ void k_relu_back(const float *__restrict__ g, const __nv_bfloat16 *__restrict__ act, int C, int relu, Vol v,
                            __nv_bfloat16 *__restrict__ dZ, float *__restrict__ gb) {
  const int c8 = blockIdx.y;
  float sum[8] = {};
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < v.Vp; r += (long long)gridDim.x * blockDim.x) {
    float d[8] = {};
    if (r < v.V) {
      const float4 *s = reinterpret_cast<const float4 *>(g + r * C + c8 * 8);
      const float4 a = s[0], b = s[1];
      d[0] = a.x, d[1] = a.y, d[2] = a.z, d[3] = a.w, d[4] = b.x, d[5] = b.y, d[6] = b.z, d[7] = b.w;
      if (relu) {
        const uint4 w = reinterpret_cast<const uint4 *>(act)[c8 * v.Vp + r];
        const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(&w);
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (!(__bfloat162float(e[j]) > 0.f)) d[j] = 0.f;
      }
    }
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; j++)
      o[j] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(d[2 * j])) |
             ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(d[2 * j + 1])) << 16);
    reinterpret_cast<uint4 *>(dZ)[c8 * v.Vp + r] = make_uint4(o[0], o[1], o[2], o[3]);
#pragma unroll
    for (int j = 0; j < 8; j++) sum[j] += d[j];
  }
  __shared__ float sh[kT / 32][8];
#pragma unroll
  for (int j = 0; j < 8; j++) {
    for (int o = 16; o; o >>= 1) sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5][j] = sum[j];
  }
  __syncthreads();
  if (threadIdx.x < 8) {
    float t = 0.f;
    for (int q = 0; q < kT / 32; q++) t += sh[q][threadIdx.x];
    atomicAdd(gb + c8 * 8 + threadIdx.x, t);
  }
}
// 2x2x2 mean: fine volume f -> coarse volume o, plane blockIdx.y of 8 channels
__global__ void k_pool(const __nv_bfloat16 *__restrict__ in, Vol f, Vol o, __nv_bfloat16 *__restrict__ out) {
  const int c8 = blockIdx.y;
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < o.V; r += (long long)gridDim.x * blockDim.x) {
    const Xyz p = xyz((unsigned)r, o.X, o.Y);
    float s[8] = {};
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const long long fr = (2 * p.x + (q & 1)) + (long long)f.X * ((2 * p.y + ((q >> 1) & 1)) + (long long)f.Y * (2 * p.z + (q >> 2)));
      const uint4 w = reinterpret_cast<const uint4 *>(in)[c8 * f.Vp + fr];
      const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(&w);
#pragma unroll
      for (int c = 0; c < 8; c++) s[c] += __bfloat162float(e[c]);
    }
    uint4 w;
    __nv_bfloat16 *e = reinterpret_cast<__nv_bfloat16 *>(&w);
#pragma unroll
    for (int c = 0; c < 8; c++) e[c] = __float2bfloat16_rn(s[c] * 0.125f);
    reinterpret_cast<uint4 *>(out)[c8 * o.Vp + r] = w;
  }
}
// gf[child][c] += go[parent][c] / 8
__global__ void k_pool_back(const float *__restrict__ go, int C, Vol f, Vol o, float *__restrict__ gf) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < f.V * C; t += (long long)gridDim.x * blockDim.x) {
    const long long r = t / C;
    const int c = (int)(t % C);
    const int x = (int)(r % f.X), y = (int)((r / f.X) % f.Y), z = (int)(r / ((long long)f.X * f.Y));
    gf[t] += 0.125f * go[((x >> 1) + (long long)o.X * ((y >> 1) + (long long)o.Y * (z >> 1))) * C + c];
  }
}
// the upper half of a concatenation, cat[r] = up(low)[r], plane blockIdx.y of 8
// channels (the skip's planes follow in the same array and are written there by
// the layer that computes them)
__global__ void k_up(const __nv_bfloat16 *__restrict__ low, Vol f, Vol o, __nv_bfloat16 *__restrict__ cat) {
  const int c8 = blockIdx.y;
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < f.V; r += (long long)gridDim.x * blockDim.x) {
    const Xyz p = xyz((unsigned)r, f.X, f.Y);
    reinterpret_cast<uint4 *>(cat)[c8 * f.Vp + r] =
        reinterpret_cast<const uint4 *>(low)[c8 * o.Vp + (p.x >> 1) + (long long)o.X * ((p.y >> 1) + (long long)o.Y * (p.z >> 1))];
  }
}
// the gradient of the concatenation: glow[p][c] += sum over the 8 children, gskip += tail
__global__ void k_upcat_back_low(const float *__restrict__ gcat, int Cu, int Cs, Vol f, Vol o, float *__restrict__ glow) {
  const int C = Cu + Cs;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < o.V * Cu; t += (long long)gridDim.x * blockDim.x) {
    const long long p = t / Cu;
    const int c = (int)(t % Cu);
    const int x = (int)(p % o.X), y = (int)((p / o.X) % o.Y), z = (int)(p / ((long long)o.X * o.Y));
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const long long fr = (2 * x + (q & 1)) + (long long)f.X * ((2 * y + ((q >> 1) & 1)) + (long long)f.Y * (2 * z + (q >> 2)));
      s += gcat[fr * C + c];
    }
    glow[t] += s;
  }
}
__global__ void k_upcat_back_skip(const float *__restrict__ gcat, int Cu, int Cs, Vol f, float *__restrict__ gskip) {
  const int C = Cu + Cs;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < f.V * Cs; t += (long long)gridDim.x * blockDim.x) {
    const long long r = t / Cs;
    const int c = (int)(t % Cs);
    gskip[t] += gcat[r * C + Cu + c];
  }
}
// weighted squared error of the head output against [V][8] targets:
// sums[0] += sum w, sums[1] += sum w r^2 (w per voxel, 8 channels each)
__global__ void k_loss_sums(const float *__restrict__ y, const float *__restrict__ tgt, const float *__restrict__ w,
                            int X, int Y, int Z, Vol v, double *__restrict__ sums) {
  const long long n = (long long)X * Y * Z;
  double sw = 0.0, se = 0.0;
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < n; r += (long long)gridDim.x * blockDim.x) {
    const int px = (int)(r % X), py = (int)((r / X) % Y), pz = (int)(r / ((long long)X * Y));
    const long long q = px + (long long)v.X * (py + (long long)v.Y * pz);
    const float wr = w ? w[r] : 1.f;
    float e = 0.f;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const float d = y[q * 16 + c] - tgt[r * 8 + c];
      e += d * d;
    }
    sw += 8.0 * wr;
    se += (double)wr * e;
  }
  for (int o = 16; o; o >>= 1) {
    sw += __shfl_xor_sync(0xffffffffu, sw, o);
    se += __shfl_xor_sync(0xffffffffu, se, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(sums, sw);
    atomicAdd(sums + 1, se);
  }
}
// dy = 2 w (y - t) / sum w on the padded head output (pads zero)
__global__ void k_loss_grad(const float *__restrict__ y, const float *__restrict__ tgt, const float *__restrict__ w,
                            int X, int Y, int Z, Vol v, const double *__restrict__ sums, float *__restrict__ gy) {
  const float inv = (float)(2.0 / fmax(sums[0], 1e-30));
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < v.Vp * 16; t += (long long)gridDim.x * blockDim.x) {
    const long long q = t >> 4;
    const int c = (int)(t & 15);
    float g = 0.f;
    if (q < v.V && c < 8) {
      const int px = (int)(q % v.X), py = (int)((q / v.X) % v.Y), pz = (int)(q / ((long long)v.X * v.Y));
      if (px < X && py < Y && pz < Z) {
        const long long r = px + (long long)X * (py + (long long)Y * pz);
        g = inv * (w ? w[r] : 1.f) * (y[t] - tgt[r * 8 + c]);
      }
    }
    gy[t] = g;
  }
}
// device copies of one layer's weights in BF16: Wf, the forward stream [K chunk
// (tap, 8 input channels)][cn][8] with a zero chunk when their number is odd, and
// Wd, the data gradient's [group of nc input channels][tap][cn / 8][nc][8]
__global__ void k_cast_w(const float *__restrict__ W, int cin, int cg, int cout, int cn, int nc,
                         __nv_bfloat16 *__restrict__ Wf, __nv_bfloat16 *__restrict__ Wd) {
  const int ch = cg / 8, chunks = (27 * ch + 1) / 2 * 2;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)chunks * cn * 8; t += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(t & 7), co = (int)((t >> 3) % cn), k = (int)((t >> 3) / cn);
    const int tap = k / ch, ci = (k - tap * ch) * 8 + j;
    float w = 0.f;
    if (co < cout && tap < 27 && ci < cin) w = W[(long long)co * 27 * cin + tap * cin + ci];
    const __nv_bfloat16 b = __float2bfloat16_rn(w);
    Wf[t] = b;
    if (nc && tap < 27) Wd[((((long long)(ci / nc) * 27 + tap) * (cn / 8) + co / 8) * nc + ci % nc) * 8 + co % 8] = b;
  }
}
// Adam on one layer (FP32 master weights), gradient of W from gWT [27 cg][cn]
__global__ void k_adam(float *__restrict__ W, float *__restrict__ m, float *__restrict__ v2, const float *__restrict__ gWT,
                       int cin, int cg, int cout, int cn, float *__restrict__ b, float *__restrict__ mb,
                       float *__restrict__ vb, const float *__restrict__ gb, float lr, float c1, float c2) {
  const long long nw = (long long)cout * 27 * cin;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nw + cout; t += (long long)gridDim.x * blockDim.x) {
    float g, *p, *pm, *pv;
    if (t < nw) {
      const int co = (int)(t / (27 * cin)), k = (int)(t % (27 * cin));
      const int tap = k / cin, ci = k % cin;
      g = gWT[(long long)(tap * cg + ci) * cn + co];
      p = W + t, pm = m + t, pv = v2 + t;
    } else {
      const int co = (int)(t - nw);
      g = gb[co];
      p = b + co, pm = mb + co, pv = vb + co;
    }
    const float mt = 0.9f * *pm + 0.1f * g, vt = 0.999f * *pv + 0.001f * g * g;
    *pm = mt;
    *pv = vt;
    *p -= lr * (mt * c1) / (sqrtf(vt * c2) + 1e-8f);
  }
}
// the gradient in the parameter layout
__global__ void k_grad_out(const float *__restrict__ gWT, const float *__restrict__ gb, int cin, int cg, int cout, int cn,
                           float *__restrict__ out) {
  const long long nw = (long long)cout * 27 * cin;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nw + cout; t += (long long)gridDim.x * blockDim.x) {
    if (t < nw) {
      const int co = (int)(t / (27 * cin)), k = (int)(t % (27 * cin));
      out[t] = gWT[(long long)((k / cin) * cg + k % cin) * cn + co];
    } else {
      out[t] = gb[t - nw];
    }
  }
}

}  // namespace

// ----------------------------------------------------------------- network
struct Layer {
  int cin, cg, cout, cn, nc, level, relu;  // cg: cin rounded to 8; cn: cout rounded to 16; nc: see k_conv_dx
  float *W = nullptr, *b = nullptr, *mW = nullptr, *vW = nullptr, *mb = nullptr, *vb = nullptr;
  float *gWT = nullptr, *gb = nullptr;
  __nv_bfloat16 *Wf = nullptr, *Wd = nullptr;
  long long nparam() const { return 27LL * cin * cout + cout; }
};

// activations: index, level, channels
enum {
  A_IN, A0, S1, P1, A2, S2, P2, A4, S3, P3, A6, A7, CAT3, A8, A9, CAT2, A10, A11, CAT1, A12, A13, A_COUNT
};

}  // namespace unet
}  // namespace aphid

struct aphid_unet {
  int X, Y, Z, train;
  aphid::unet::Vol vol[4];
  std::vector<aphid::unet::Layer> L;
  __nv_bfloat16 *act[aphid::unet::A_COUNT] = {};
  float *grad[aphid::unet::A_COUNT] = {};
  int ach[aphid::unet::A_COUNT], alev[aphid::unet::A_COUNT];
  float *y = nullptr, *gy = nullptr;               // head output / its gradient [Vp][16]
  __nv_bfloat16 *dZ = nullptr;
  float *grad_all = nullptr, *gout = nullptr;  // all gradients (zeroed in one pass); the copy in the parameter layout
  size_t grad_bytes = 0, nparam = 0;
  double *sums = nullptr;
  int *err = nullptr;
  long long step = 0;
  std::vector<void *> owned;
};

namespace aphid {
namespace unet {
namespace {

const int kLayerDef[15][4] = {  // cin, cout, level, relu
    {3, 16, 0, 1},  {16, 16, 0, 1},  {16, 32, 1, 1},  {32, 32, 1, 1},  {32, 64, 2, 1},
    {64, 64, 2, 1}, {64, 128, 3, 1}, {128, 128, 3, 1}, {192, 64, 2, 1}, {64, 64, 2, 1},
    {96, 32, 1, 1}, {32, 32, 1, 1},  {48, 16, 0, 1},  {16, 16, 0, 1},  {16, 8, 0, 0}};
// input activation and output activation of each layer (-1: head output)
const int kLayerIO[15][2] = {{A_IN, A0}, {A0, S1}, {P1, A2}, {A2, S2}, {P2, A4}, {A4, S3}, {P3, A6}, {A6, A7},
                             {CAT3, A8}, {A8, A9}, {CAT2, A10}, {A10, A11}, {CAT1, A12}, {A12, A13}, {A13, -1}};

template <class T>
int dalloc(aphid_unet *n, T **p, size_t count) {
  void *q = nullptr;
  if (cudaMalloc(&q, std::max<size_t>(count, 1) * sizeof(T)) != cudaSuccess) {
    cudaGetLastError();
    return set_err(APHID_UNET_ERR_NOMEM, "unet: device allocation failed");
  }
  if (cudaMemset(q, 0, std::max<size_t>(count, 1) * sizeof(T)) != cudaSuccess)
    return set_err(APHID_UNET_ERR_CUDA, "unet: cudaMemset");
  n->owned.push_back(q);
  *p = static_cast<T *>(q);
  return APHID_UNET_OK;
}

#define UK(call)                                                      \
  do {                                                                \
    cudaError_t e_ = (call);                                          \
    if (e_ != cudaSuccess)                                            \
      return set_err(APHID_UNET_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)
#define UR(call)        \
  do {                  \
    int r_ = (call);    \
    if (r_) return r_;  \
  } while (0)

int cast_weights(aphid_unet *n, cudaStream_t st) {
  for (auto &l : n->L)
    k_cast_w<<<nblk(28LL * l.cg * l.cn), kT, 0, st>>>(l.W, l.cin, l.cg, l.cout, l.cn, n->train ? l.nc : 0, l.Wf, l.Wd);
  UK(cudaGetLastError());
  return APHID_UNET_OK;
}

// an activation (or dZ) of C channels in planes of 8 as a tensor with boxes of
// bx x by x bz voxels of bc planes
int act_map(CUtensorMap *m, const __nv_bfloat16 *base, int C, const Vol &v, int bx, int by, int bz, int bc) {
  const cuuint64_t dims[4] = {8 * (cuuint64_t)v.X, (cuuint64_t)v.Y, (cuuint64_t)v.Z, (cuuint64_t)(C / 8)};
  const cuuint64_t strides[3] = {16 * (cuuint64_t)v.X, 16 * (cuuint64_t)v.X * v.Y, 16 * (cuuint64_t)v.Vp};
  const cuuint32_t box[4] = {(cuuint32_t)(8 * bx), (cuuint32_t)by, (cuuint32_t)bz, (cuuint32_t)bc}, es[4] = {1, 1, 1, 1};
  EncodeTiledFn fn = encode_fn();
  if (!fn) return set_err(APHID_UNET_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<__nv_bfloat16 *>(base), dims, strides, box, es,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return set_err(APHID_UNET_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
  return APHID_UNET_OK;
}
template <class Kernel, class... Args>
int launch_conv(Kernel kernel, const __nv_bfloat16 *in, int C, const Vol &v, int bz, int groups, size_t shm, cudaStream_t st,
                Args... args) {
  ConvArgs a{v.X, v.Y, v.Z, v.Vp, (v.X + kTX - 1) / kTX, (v.Y + kTY - 1) / kTY};
  CUtensorMap m;
  UR(act_map(&m, in, C, v, kTX + 2, kTY + 2, bz + 2, C / 8));
  UK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
  kernel<<<dim3((unsigned)(a.tx * a.ty * ((v.Z + bz - 1) / bz)), (unsigned)groups), kConvThreads, shm, st>>>(m, a, args...);
  UK(cudaGetLastError());
  return APHID_UNET_OK;
}
template <int CH, int BN, int BZ, int PER, int ST, bool RELU = true>
int conv_fwd_t(aphid_unet *n, const Layer &l, const __nv_bfloat16 *in, void *out, cudaStream_t st) {
  return launch_conv(k_conv_fwd<CH, BN, BZ, PER, ST, RELU>, in, CH * 8, n->vol[l.level], BZ, 1,
                     conv_shm(CH, BZ, ST * PER * BN * 16), st, l.Wf, l.b, out, n->err);
}
template <int CH, int NC, int BZ, int PER, int ST>
int conv_dx_t(aphid_unet *n, const Layer &l, float *gin, cudaStream_t st) {
  return launch_conv(k_conv_dx<CH, NC, BZ, PER, ST>, n->dZ, CH * 8, n->vol[l.level], BZ, l.cg / NC,
                     conv_shm(CH, BZ, ST * PER * CH * NC * 16), st, l.Wd, l.cg, gin, n->err);
}

// One convolution of the forward pass.  The z-planes per block and the weight
// stages are the fastest of a sweep over both at the levels of a 168 x 168 x 136
// and a 72 x 72 x 56 volume: deep tiles save halo and weight traffic while two
// blocks still fit an SM (one block's copies run under the other's products).
// Per layer of the larger volume, before -> after the issuing warp's loop and
// these tiles: 48 -> 16 channels 1468 -> 479 us (4 planes; 1 to 8: 479 to 572),
// 96 -> 32 654 -> 183 (1 to 4: 285 to 183), 192 -> 64 376 -> 115, 16 -> 16
// 175 -> 130, 128 -> 128 54 -> 20.
// A forward pass of the 161 x 161 x 129 volume took 22.9 ms with a column
// matrix and a GEMM per layer, 14.9 of them in writing the column matrices.  The
// outputs are the same bit for bit: so is the order of the products.
int conv_fwd(aphid_unet *n, int li, cudaStream_t st) {
  const Layer &l = n->L[li];
  const __nv_bfloat16 *in = n->act[kLayerIO[li][0]];
  if (kLayerIO[li][1] < 0) return conv_fwd_t<2, 16, 4, 54, 1, false>(n, l, in, n->y, st);
  __nv_bfloat16 *out = n->act[kLayerIO[li][1]];
  switch (l.cg * 1000 + l.cn) {
    case 8016: return conv_fwd_t<1, 16, 4, 28, 1>(n, l, in, out, st);
    case 16016: return conv_fwd_t<2, 16, 4, 54, 1>(n, l, in, out, st);
    case 16032: return conv_fwd_t<2, 32, 2, 18, 2>(n, l, in, out, st);
    case 32032: return conv_fwd_t<4, 32, 2, 12, 4>(n, l, in, out, st);
    case 32064: return conv_fwd_t<4, 64, 1, 12, 2>(n, l, in, out, st);
    case 64064: return conv_fwd_t<8, 64, 1, 8, 4>(n, l, in, out, st);
    case 64128: return conv_fwd_t<8, 128, 1, 8, 4>(n, l, in, out, st);
    case 128128: return conv_fwd_t<16, 128, 1, 8, 4>(n, l, in, out, st);
    case 192064: return conv_fwd_t<24, 64, 1, 8, 2>(n, l, in, out, st);
    case 96032: return conv_fwd_t<12, 32, 4, 12, 2>(n, l, in, out, st);
    case 48016: return conv_fwd_t<6, 16, 4, 18, 2>(n, l, in, out, st);
  }
  return set_err(APHID_UNET_ERR_BADARG, "no convolution kernel for this layer");
}

// The data gradient of one layer into gin.  Few planes per block here: the
// epilogue's sums take BZ x NC registers, and three or four blocks per SM hide
// its reads of tensor memory (a 72 x 72 x 56 volume, 16 -> 16 channels: 25, 31,
// 37 us at 2, 4, 8 planes; 32 of 96 channels at half of it: 33, 46 at 1, 2).
int conv_dx(aphid_unet *n, int li, float *gin, cudaStream_t st) {
  const Layer &l = n->L[li];
  switch (l.nc * 1000 + l.cn) {
    case 16016: return conv_dx_t<2, 16, 2, 27, 1>(n, l, gin, st);
    case 16032: return conv_dx_t<4, 16, 1, 27, 1>(n, l, gin, st);
    case 32032: return conv_dx_t<4, 32, 1, 3, 2>(n, l, gin, st);
    case 32064: return conv_dx_t<8, 32, 1, 3, 2>(n, l, gin, st);
    case 32128: return conv_dx_t<16, 32, 1, 1, 2>(n, l, gin, st);
    case 48016: return conv_dx_t<2, 48, 1, 3, 4>(n, l, gin, st);
  }
  return set_err(APHID_UNET_ERR_BADARG, "no data-gradient kernel for this layer");
}

template <int CH, int CN>
int conv_dw_t(aphid_unet *n, const Layer &l, const __nv_bfloat16 *in, cudaStream_t st) {
  using D = DwShape<CH, CN>;
  const Vol &v = n->vol[l.level];
  const ConvArgs a{v.X, v.Y, v.Z, v.Vp, (v.X + kTX - 1) / kTX, (v.Y + kTY - 1) / kTY};
  CUtensorMap mi, mz;
  UR(act_map(&mi, in, l.cg, v, kTX + 2, kTY, 1, 1));
  UR(act_map(&mz, n->dZ, l.cn, v, kTX, kTY, 1, 1));
  UK(cudaFuncSetAttribute(k_conv_dw<CH, CN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)D::shm));
  const int tiles = a.tx * a.ty * v.Z;
  // one wave: two blocks per SM up to 32 outputs, else one
  const int split = std::max(1, std::min(tiles, (CN <= 32 ? 296 : 148) / D::kGroups));
  k_conv_dw<CH, CN><<<dim3(D::kGroups, (unsigned)split), kConvThreads, D::shm, st>>>(mi, mz, a, tiles, l.gWT, n->err);
  UK(cudaGetLastError());
  return APHID_UNET_OK;
}
// The weight gradient of one layer into gWT (zeroed).
int conv_dw(aphid_unet *n, int li, cudaStream_t st) {
  const Layer &l = n->L[li];
  const __nv_bfloat16 *in = n->act[kLayerIO[li][0]];
  switch (l.cg * 1000 + l.cn) {
    case 8016: return conv_dw_t<1, 16>(n, l, in, st);
    case 16016: return conv_dw_t<2, 16>(n, l, in, st);
    case 16032: return conv_dw_t<2, 32>(n, l, in, st);
    case 32032: return conv_dw_t<4, 32>(n, l, in, st);
    case 32064: return conv_dw_t<4, 64>(n, l, in, st);
    case 64064: return conv_dw_t<8, 64>(n, l, in, st);
    case 64128: return conv_dw_t<8, 128>(n, l, in, st);
    case 128128: return conv_dw_t<16, 128>(n, l, in, st);
    case 192064: return conv_dw_t<24, 64>(n, l, in, st);
    case 96032: return conv_dw_t<12, 32>(n, l, in, st);
    case 48016: return conv_dw_t<6, 16>(n, l, in, st);
  }
  return set_err(APHID_UNET_ERR_BADARG, "no weight-gradient kernel for this layer");
}

// gOut: gradient of this layer's output (FP32 [Vp][cn]); adds into the input's gradient
int conv_back(aphid_unet *n, int li, const float *gout, const __nv_bfloat16 *out, cudaStream_t st) {
  const Layer &l = n->L[li];
  const Vol &v = n->vol[l.level];
  const int io = kLayerIO[li][0];
  k_relu_back<<<dim3((unsigned)std::min<long long>((v.Vp + kT - 1) / kT, 296), (unsigned)(l.cn / 8)), kT, 0, st>>>(
      gout, out, l.cn, l.relu, v, n->dZ, l.gb);
  UK(cudaGetLastError());
  UR(conv_dw(n, li, st));
  if (li == 0) return APHID_UNET_OK;  // no gradient for the input features
  return conv_dx(n, li, n->grad[io], st);
}

int forward(aphid_unet *n, const float *x, cudaStream_t st) {
  const Vol *V = n->vol;
  k_pack_in<<<nblk(V[0].Vp), kT, 0, st>>>(x, n->X, n->Y, n->Z, V[0], n->act[A_IN]);
  UK(cudaGetLastError());
  auto pool = [&](int a, int b, int lev) {
    k_pool<<<dim3((unsigned)nblk(V[lev + 1].V), (unsigned)(n->ach[a] / 8)), kT, 0, st>>>(n->act[a], V[lev], V[lev + 1], n->act[b]);
  };
  auto up = [&](int low, int cat, int lev) {
    k_up<<<dim3((unsigned)nblk(V[lev].V), (unsigned)(n->ach[low] / 8)), kT, 0, st>>>(n->act[low], V[lev], V[lev + 1], n->act[cat]);
  };
  UR(conv_fwd(n, 0, st));
  UR(conv_fwd(n, 1, st));
  pool(S1, P1, 0);
  UR(conv_fwd(n, 2, st));
  UR(conv_fwd(n, 3, st));
  pool(S2, P2, 1);
  UR(conv_fwd(n, 4, st));
  UR(conv_fwd(n, 5, st));
  pool(S3, P3, 2);
  UR(conv_fwd(n, 6, st));
  UR(conv_fwd(n, 7, st));
  up(A7, CAT3, 2);
  UR(conv_fwd(n, 8, st));
  UR(conv_fwd(n, 9, st));
  up(A9, CAT2, 1);
  UR(conv_fwd(n, 10, st));
  UR(conv_fwd(n, 11, st));
  up(A11, CAT1, 0);
  UR(conv_fwd(n, 12, st));
  UR(conv_fwd(n, 13, st));
  UR(conv_fwd(n, 14, st));
  UK(cudaGetLastError());
  return APHID_UNET_OK;
}

int backward(aphid_unet *n, cudaStream_t st) {
  const Vol *V = n->vol;
  UK(cudaMemsetAsync(n->grad_all, 0, n->grad_bytes, st));
  auto back = [&](int li) {
    const int o = kLayerIO[li][1];
    return o < 0 ? conv_back(n, li, n->gy, nullptr, st) : conv_back(n, li, n->grad[o], n->act[o], st);
  };
  auto split = [&](int cat, int low, int skip, int lev) {
    const int cu = n->ach[low], cs = n->ach[skip];
    k_upcat_back_low<<<nblk(V[lev + 1].V * cu), kT, 0, st>>>(n->grad[cat], cu, cs, V[lev], V[lev + 1], n->grad[low]);
    k_upcat_back_skip<<<nblk(V[lev].V * cs), kT, 0, st>>>(n->grad[cat], cu, cs, V[lev], n->grad[skip]);
  };
  auto pool_back = [&](int pooled, int fine, int lev) {
    k_pool_back<<<nblk(V[lev].V * n->ach[fine]), kT, 0, st>>>(n->grad[pooled], n->ach[fine], V[lev], V[lev + 1],
                                                              n->grad[fine]);
  };
  UR(back(14));
  UR(back(13));
  UR(back(12));
  split(CAT1, A11, S1, 0);
  UR(back(11));
  UR(back(10));
  split(CAT2, A9, S2, 1);
  UR(back(9));
  UR(back(8));
  split(CAT3, A7, S3, 2);
  UR(back(7));
  UR(back(6));
  pool_back(P3, S3, 2);
  UR(back(5));
  UR(back(4));
  pool_back(P2, S2, 1);
  UR(back(3));
  UR(back(2));
  pool_back(P1, S1, 0);
  UR(back(1));
  UR(back(0));
  UK(cudaGetLastError());
  return APHID_UNET_OK;
}

int check_err(aphid_unet *n, cudaStream_t st) {
  int e = 0;
  UK(cudaMemcpyAsync(&e, n->err, sizeof(int), cudaMemcpyDeviceToHost, st));
  UK(cudaStreamSynchronize(st));
  if (e) return set_err(APHID_UNET_ERR_CUDA, "unet: a bounded wait in the tensor-core GEMM gave up");
  return APHID_UNET_OK;
}

}  // namespace
}  // namespace unet
}  // namespace aphid

using namespace aphid::unet;

extern "C" {

const char *aphid_unet_last_error(void) { return g_last_error.c_str(); }

long long aphid_unet_param_count(void) {
  long long n = 0;
  for (auto &d : kLayerDef) n += 27LL * d[0] * d[1] + d[1];
  return n;
}

int aphid_unet_create(aphid_unet **out, int X, int Y, int Z, int train, unsigned long long seed) {
  if (!out || X < 1 || Y < 1 || Z < 1) return set_err(APHID_UNET_ERR_BADARG, "unet_create: bad volume");
  *out = nullptr;
  aphid_unet *n = new aphid_unet();
  n->X = X, n->Y = Y, n->Z = Z, n->train = train ? 1 : 0;
  int dims[3] = {(int)rup(X, 8), (int)rup(Y, 8), (int)rup(Z, 8)};
  for (int l = 0; l < 4; l++) {
    Vol &v = n->vol[l];
    v.X = dims[0] >> l, v.Y = dims[1] >> l, v.Z = dims[2] >> l;
    v.V = (long long)v.X * v.Y * v.Z;
    v.Vp = rup(v.V, kBM);
  }
  const int ach[A_COUNT] = {8, 16, 16, 16, 32, 32, 32, 64, 64, 64, 128, 128, 192, 64, 64, 96, 32, 32, 48, 16, 16};
  const int alev[A_COUNT] = {0, 0, 0, 1, 1, 1, 2, 2, 2, 3, 3, 3, 2, 2, 2, 1, 1, 1, 0, 0, 0};
  int rc = APHID_UNET_OK;
  std::mt19937_64 rng(seed);
  for (int li = 0; li < 15 && !rc; li++) {
    Layer l;
    l.cin = kLayerDef[li][0], l.cout = kLayerDef[li][1], l.level = kLayerDef[li][2], l.relu = kLayerDef[li][3];
    l.cg = (int)rup(l.cin, 8), l.cn = (int)rup(l.cout, 16);
    l.nc = l.cg % 32 == 0 ? 32 : l.cg % 48 == 0 ? 48 : 16;
    const size_t nw = 27ULL * l.cin * l.cout;
    if ((rc = dalloc(n, &l.W, nw)) || (rc = dalloc(n, &l.b, l.cn)) || (rc = dalloc(n, &l.Wf, 28ULL * l.cg * l.cn)))
      break;
    if (train && ((rc = dalloc(n, &l.mW, nw)) || (rc = dalloc(n, &l.vW, nw)) || (rc = dalloc(n, &l.mb, l.cout)) ||
                  (rc = dalloc(n, &l.vb, l.cout)) || (rc = dalloc(n, &l.Wd, 27ULL * rup(l.cg, 16) * l.cn))))
      break;
    // He-normal initial weights, zero biases
    std::normal_distribution<float> nd(0.f, std::sqrt(2.f / (27.f * l.cin)));
    std::vector<float> h(nw);
    for (auto &w : h) w = nd(rng);
    if (cudaMemcpy(l.W, h.data(), nw * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess) {
      rc = set_err(APHID_UNET_ERR_CUDA, "unet_create: weight upload");
      break;
    }
    n->L.push_back(l);
  }
  size_t gn = 0;  // gradients: activations, then weights and biases
  for (int a = 0; a < A_COUNT && !rc; a++) {
    n->ach[a] = ach[a], n->alev[a] = alev[a];
    const size_t cnt = (size_t)n->vol[alev[a]].Vp * ach[a];
    if (a != S1 && a != S2 && a != S3) rc = dalloc(n, &n->act[a], cnt);
    if (a != A_IN) gn += cnt;
  }
  // a skip is the lower planes of its concatenation
  for (auto &sc : {std::pair<int, int>{S1, CAT1}, {S2, CAT2}, {S3, CAT3}})
    if (!rc) n->act[sc.first] = n->act[sc.second] + (size_t)n->vol[alev[sc.second]].Vp * (ach[sc.second] - ach[sc.first]);
  for (auto &l : n->L) gn += 27ULL * l.cg * l.cn + l.cn, n->nparam += l.nparam();
  if (!rc && train && !(rc = dalloc(n, &n->grad_all, gn)) && !(rc = dalloc(n, &n->gout, n->nparam))) {
    n->grad_bytes = gn * sizeof(float);
    float *g = n->grad_all;
    for (int a = 0; a < A_COUNT; a++)
      if (a != A_IN) n->grad[a] = g, g += (size_t)n->vol[alev[a]].Vp * ach[a];
    for (auto &l : n->L) l.gWT = g, g += 27ULL * l.cg * l.cn, l.gb = g, g += l.cn;
  }
  if (!rc) rc = dalloc(n, &n->y, (size_t)n->vol[0].Vp * 16);
  if (!rc) rc = dalloc(n, &n->err, 1);
  if (!rc) rc = dalloc(n, &n->sums, 2);
  if (!rc && train) {
    size_t dzmax = 0;
    for (auto &l : n->L) {
      dzmax = std::max(dzmax, (size_t)n->vol[l.level].Vp * l.cn);
    }
    if (!rc) rc = dalloc(n, &n->gy, (size_t)n->vol[0].Vp * 16);
    if (!rc) rc = dalloc(n, &n->dZ, dzmax);
  }
  if (!rc) rc = cast_weights(n, 0);
  if (!rc && cudaDeviceSynchronize() != cudaSuccess) rc = set_err(APHID_UNET_ERR_CUDA, "unet_create: initialisation");
  if (rc) {
    aphid_unet_destroy(n);
    return rc;
  }
  *out = n;
  return APHID_UNET_OK;
}

int aphid_unet_destroy(aphid_unet *n) {
  if (!n) return APHID_UNET_OK;
  for (void *p : n->owned) cudaFree(p);
  delete n;
  return APHID_UNET_OK;
}

int aphid_unet_get_params(aphid_unet *n, float *host) {
  if (!n || !host) return set_err(APHID_UNET_ERR_BADARG, "unet_get_params: null");
  size_t o = 0;
  for (auto &l : n->L) {
    const size_t nw = 27ULL * l.cin * l.cout;
    UK(cudaMemcpy(host + o, l.W, nw * sizeof(float), cudaMemcpyDeviceToHost));
    UK(cudaMemcpy(host + o + nw, l.b, l.cout * sizeof(float), cudaMemcpyDeviceToHost));
    o += nw + l.cout;
  }
  return APHID_UNET_OK;
}

int aphid_unet_set_params(aphid_unet *n, const float *host) {
  if (!n || !host) return set_err(APHID_UNET_ERR_BADARG, "unet_set_params: null");
  size_t o = 0;
  for (auto &l : n->L) {
    const size_t nw = 27ULL * l.cin * l.cout;
    UK(cudaMemcpy(l.W, host + o, nw * sizeof(float), cudaMemcpyHostToDevice));
    UK(cudaMemcpy(l.b, host + o + nw, l.cout * sizeof(float), cudaMemcpyHostToDevice));
    if (n->train) {  // a new starting point: the optimiser forgets its moments
      UK(cudaMemset(l.mW, 0, nw * sizeof(float)));
      UK(cudaMemset(l.vW, 0, nw * sizeof(float)));
      UK(cudaMemset(l.mb, 0, l.cout * sizeof(float)));
      UK(cudaMemset(l.vb, 0, l.cout * sizeof(float)));
    }
    o += nw + l.cout;
  }
  n->step = 0;
  UR(cast_weights(n, 0));
  UK(cudaDeviceSynchronize());
  return APHID_UNET_OK;
}

int aphid_unet_forward(aphid_unet *n, const float *x, float *y, void *stream) {
  if (!n || !x || !y) return set_err(APHID_UNET_ERR_BADARG, "unet_forward: null");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  UR(forward(n, x, st));
  k_unpack_out<<<nblk((long long)n->X * n->Y * n->Z * 2), kT, 0, st>>>(n->y, n->X, n->Y, n->Z, n->vol[0], y);
  UK(cudaGetLastError());
  return check_err(n, st);
}

int aphid_unet_train_step(aphid_unet *n, const float *x, const float *target, const float *weight, float lr,
                          int update, double *loss, void *stream) {
  if (!n || !x || !target) return set_err(APHID_UNET_ERR_BADARG, "unet_train_step: null");
  if (!n->train) return set_err(APHID_UNET_ERR_BADARG, "unet_train_step: created without training buffers");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  UR(forward(n, x, st));
  UK(cudaMemsetAsync(n->sums, 0, 2 * sizeof(double), st));
  k_loss_sums<<<nblk((long long)n->X * n->Y * n->Z), kT, 0, st>>>(n->y, target, weight, n->X, n->Y, n->Z, n->vol[0],
                                                                  n->sums);
  k_loss_grad<<<nblk(n->vol[0].Vp * 16), kT, 0, st>>>(n->y, target, weight, n->X, n->Y, n->Z, n->vol[0], n->sums,
                                                      n->gy);
  UK(cudaGetLastError());
  UR(backward(n, st));
  if (update) {
    n->step++;
    const float c1 = 1.f / (1.f - std::pow(0.9f, (float)n->step)), c2 = 1.f / (1.f - std::pow(0.999f, (float)n->step));
    for (auto &l : n->L)
      k_adam<<<nblk(27LL * l.cin * l.cout + l.cout), kT, 0, st>>>(l.W, l.mW, l.vW, l.gWT, l.cin, l.cg, l.cout, l.cn, l.b,
                                                                   l.mb, l.vb, l.gb, lr, c1, c2);
    UK(cudaGetLastError());
    UR(cast_weights(n, st));
  }
  double s[2] = {0, 0};
  UK(cudaMemcpyAsync(s, n->sums, sizeof(s), cudaMemcpyDeviceToHost, st));
  UR(check_err(n, st));
  if (loss) *loss = s[1] / std::max(s[0], 1e-30);
  return APHID_UNET_OK;
}

int aphid_unet_get_grads(aphid_unet *n, float *host) {
  if (!n || !host || !n->train) return set_err(APHID_UNET_ERR_BADARG, "unet_get_grads: no training buffers");
  size_t o = 0;
  for (auto &l : n->L) {
    k_grad_out<<<nblk(l.nparam()), kT>>>(l.gWT, l.gb, l.cin, l.cg, l.cout, l.cn, n->gout + o);
    o += l.nparam();
  }
  UK(cudaGetLastError());
  UK(cudaMemcpy(host, n->gout, o * sizeof(float), cudaMemcpyDeviceToHost));
  return APHID_UNET_OK;
}


int aphid_unet_gemm_bf16(const void *A, int lda, const void *B, int ldb, void *C, int ldc, const float *bias, int M,
                         int N, int K, int out, int splitk, void *stream, int *err_flag) {
  return gemm_bf16(static_cast<const __nv_bfloat16 *>(A), lda, static_cast<const __nv_bfloat16 *>(B), ldb, C, ldc,
                   bias, M, N, K, out, splitk, static_cast<cudaStream_t>(stream), err_flag);
}

}  // extern "C"
