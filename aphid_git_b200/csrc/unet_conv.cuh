// unet_conv.cuh -- the 3 x 3 x 3 convolutions of the initial-guess network as
// implicit GEMMs on the sm_100a tensor cores (tcgen05): forward, data gradient
// and weight gradient.  No column matrix: a block brings the voxels of its tile with a
// one-voxel halo into shared memory once, and every tap's operand is the same
// memory read from a shifted start address.
//
// Activations are stored in planes of 8 channels, [C/8][Vp][8] BF16 (16 bytes
// per voxel and plane, x fastest).  A tile is 8 x 16 voxels of BZ z-planes; one
// 4-D TMA box (10 x 8 channels, 18, BZ + 2, C/8) lands as [C/8][z][y][x][8], zero
// outside the volume.  In it 8 voxels of a row are 128 contiguous bytes -- an
// unswizzled K-major core matrix (8 rows x 16 bytes) -- rows lie 160 bytes apart
// (the stride between the 16 core matrices of the 128-row operand) and the
// planes of 8 channels a fixed stride apart (the two core matrices of K = 16),
// so the operand of tap (dx, dy, dz) starts 16 dx + 160 dy + 2880 dz bytes on.
//
// What bounds them: each K = 16 step reads 4 KB of operand A from shared memory
// (32 cycles at 128 B per cycle) for 128 x 16 to 128 x 128 outputs, and the tile
// comes in once instead of 27 times.  The column matrix of the same layers cost
// 27 x the activations in and out of memory; see conv_fwd for the figures.
//
// Every wait is bounded: one that gives up sets the error flag, the later ones
// are skipped, and the kernel still frees its tensor memory before it returns.
#pragma once
#include "unet_gemm.cuh"

namespace aphid {
namespace unet {

constexpr int kTX = 8, kTY = 16, kRowB = (kTX + 2) * 16, kPlaneB = (kTY + 2) * kRowB;  // tile, bytes of a staged row, plane
constexpr int kConvThreads = 192;  // warps 0-3: epilogue, 4: producer, 5: MMA issuer
constexpr int kMaxStages = 4;
constexpr uint32_t kLast = 2 * (16 + kRowB + kPlaneB);  // the last tap's offset in the staged tile

struct ConvArgs {
  int X, Y, Z;    // volume
  long long Vp;   // voxels per plane of 8 channels
  int tx, ty;     // tiles along x, y
};

// shared-memory descriptor of an unswizzled K-major operand: lbo between the
// two core matrices of K = 16, sbo between 8-row core matrices (bytes)
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.b32 %0, 1, 0, q;\n}\n" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void g_mbar_init_n(uint32_t bar, uint32_t n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(n) : "memory");
}
__device__ __forceinline__ void g_mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// 1-D bulk copy into this block's shared memory (16-byte multiples)
__device__ __forceinline__ void g_bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void g_tma_load4(uint32_t dst, const CUtensorMap *map, int x, int y, int z, int c, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];\n" ::"r"(dst),
      "l"((unsigned long long)map), "r"(x), "r"(y), "r"(z), "r"(c), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t a, float *x) {
  uint32_t v[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(a));
#pragma unroll
  for (int q = 0; q < 8; q++) x[q] = __uint_as_float(v[q]);
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

// shared memory: the input tile, the weight stages, the barriers
// (with one plane of 8 channels the last K = 16 step has no second tap: its
// operand is a plane of zeros behind the tile, not a neighbour's value times a
// zero weight, which an infinity would turn into NaN)
__host__ __device__ constexpr uint32_t conv_tile_bytes(int ch, int bz) {
  return ((ch * (bz + 2) + (ch & 1)) * kPlaneB + 127) / 128 * 128;
}
__host__ __device__ constexpr uint32_t conv_shm(int ch, int bz, uint32_t weight_bytes) {
  return 128 + conv_tile_bytes(ch, bz) + weight_bytes + 256;
}

struct ConvShm {
  unsigned char *tile, *w;
  uint64_t *full, *empty, *tile_in, *tfull, *tempty;  // [kMaxStages] x 2, 1, 2, 2
  uint32_t *tslot;
};
// carve the dynamic shared memory (WB bytes of weight stages), allocate COLS of
// tensor memory, arm the barriers
template <int CH, int BZ, uint32_t WB, uint32_t COLS>
__device__ __forceinline__ ConvShm conv_init(unsigned char *raw, uint32_t &tmem) {
  ConvShm s;
  s.tile = raw + ((128u - (gsm(raw) & 127u)) & 127u);
  s.w = s.tile + conv_tile_bytes(CH, BZ);
  s.full = reinterpret_cast<uint64_t *>(s.w + WB);
  s.empty = s.full + kMaxStages;
  s.tile_in = s.empty + kMaxStages;
  s.tfull = s.tile_in + 1;
  s.tempty = s.tfull + 2;
  s.tslot = reinterpret_cast<uint32_t *>(s.tempty + 2);
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(gsm(s.tslot)), "r"(COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (threadIdx.x == 32) {
    for (int q = 0; q < kMaxStages; q++) {
      g_mbar_init(gsm(&s.full[q]));
      g_mbar_init(gsm(&s.empty[q]));
    }
    g_mbar_init(gsm(s.tile_in));
    for (int q = 0; q < 2; q++) {
      g_mbar_init(gsm(&s.tfull[q]));
      g_mbar_init_n(gsm(&s.tempty[q]), 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  if (CH & 1) {
    uint4 *z = reinterpret_cast<uint4 *>(s.tile + CH * (BZ + 2) * kPlaneB);
    for (int q = threadIdx.x; q < kPlaneB / 16; q += kConvThreads) z[q] = make_uint4(0, 0, 0, 0);
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  tmem = *s.tslot;
  return s;
}
__device__ __forceinline__ void conv_exit(uint32_t tmem, uint32_t cols) {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(cols) : "memory");
}
__host__ __device__ constexpr uint32_t tmem_cols(int n) { return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : n <= 256 ? 256 : 512; }

// offset of the tap after the one at (dx, dy) in the staged tile
__device__ __forceinline__ void next_tap(uint32_t &at, int &dx, int &dy) {
  at += 16;
  if (++dx == 3) {
    dx = 0, at += kRowB - 48;
    if (++dy == 3) dy = 0, at += kPlaneB - 3 * kRowB;
  }
}

// Forward: out = act(conv(in) + bias) from CH planes of 8 channels to BN output
// channels, BZ z-planes per block.  Weights: the stream [K chunk][BN][8] (K = tap
// x channels, in that order), read once per block through a ring of ST stages of
// PER chunks.  The products are added in the order of K, 16 at a time.  RELU:
// BF16 planes of 8 channels; else FP32 rows [Vp][BN] (the head).
// The issuing warp runs its loop as a whole, with every extent a constant, and
// elects a lane for the instruction alone: one diverged lane with run-time
// extents spent 160 cycles on the indexes of each K = 16 step and 630 on each
// weight stage, against the 64 of a 128 x 128 x 16 product.
template <int CH, int BN, int BZ, int PER, int ST, bool RELU>
__global__ void __launch_bounds__(kConvThreads) k_conv_fwd(const __grid_constant__ CUtensorMap map, const ConvArgs a,
                                                           const __nv_bfloat16 *__restrict__ wgt,
                                                           const float *__restrict__ bias, void *__restrict__ out, int *err) {
  extern __shared__ unsigned char cs_raw[];
  static_assert(CH == 1 || CH % 2 == 0, "K = 16: two planes of a tap, or two taps of one plane");
  static_assert(PER % 2 == 0 && ST <= kMaxStages, "weight stages");
  constexpr int kChunks = (27 * CH + 1) / 2 * 2, kStages = (kChunks + PER - 1) / PER;
  constexpr uint32_t kCols = tmem_cols(BN * BZ), chunk_b = BN * 16, stage_b = PER * chunk_b, plane_b = (BZ + 2) * kPlaneB;
  uint32_t tmem;
  const ConvShm s = conv_init<CH, BZ, ST * stage_b, kCols>(cs_raw, tmem);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  int b = blockIdx.x;
  const int x0 = b % a.tx * kTX;
  b /= a.tx;
  const int y0 = b % a.ty * kTY, z0 = b / a.ty * BZ;
  bool ok = true;
  if (warp == 4) {
    if (lane == 0) {
      g_mbar_expect(gsm(s.tile_in), CH * plane_b);
      g_tma_load4(gsm(s.tile), &map, (x0 - 1) * 8, y0 - 1, z0 - 1, 0, gsm(s.tile_in));
      int st = 0, lap = 0;
      for (int q = 0; q < kStages; q++) {
        if (lap > 0 && ok) ok = g_mbar_wait(gsm(&s.empty[st]), (uint32_t)((lap - 1) & 1));
        const uint32_t bytes = min(PER, kChunks - q * PER) * chunk_b;
        g_mbar_expect(gsm(&s.full[st]), bytes);
        g_bulk_load(gsm(s.w) + st * stage_b, wgt + (size_t)q * stage_b / 2, bytes, gsm(&s.full[st]));
        if (++st == ST) st = 0, lap++;
      }
    }
  } else if (warp == 5) {
    constexpr uint32_t idesc = idesc_bf16(kBM, BN);
    const bool lead = elect_one();
    ok = g_mbar_wait(gsm(s.tile_in), 0u);
    const uint64_t da0 = smem_desc(gsm(s.tile), plane_b, kRowB), db0 = smem_desc(gsm(s.w), chunk_b, 128);
    uint32_t at = 0, c_at = 0;  // tap, channel plane: bytes from the tile's start
    int dx = 0, dy = 0, st = 0, lap = 0;
#pragma unroll 1
    for (int q = 0; q < kStages; q++) {
      if (ok) ok = g_mbar_wait(gsm(&s.full[st]), (uint32_t)(lap & 1));
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const int steps = min(PER, kChunks - q * PER) / 2;
      uint64_t db = db0 + (uint64_t)((uint32_t)st * stage_b >> 4);
#pragma unroll(PER <= 16 ? PER / 2 : 4)
      for (int k = 0; k < steps; k++) {
        const uint32_t acc = q > 0 || k > 0;
        uint64_t da = da0 + (uint64_t)((at + c_at) >> 4);
        uint32_t lbo = plane_b;  // two planes of one tap
        if (CH == 1) {           // two taps, the last with zeros
          const uint32_t t0 = at;
          next_tap(at, dx, dy);
          lbo = at - t0;
          da = smem_desc(gsm(s.tile) + t0, lbo, kRowB);
          if (q * PER / 2 + k == kChunks / 2 - 1) lbo = 0;
        }
        if (lead) {
#pragma unroll
          for (int p = 0; p < BZ; p++) {
            if (CH == 1 && lbo == 0)
              mma_f16(tmem + p * BN, smem_desc(gsm(s.tile) + kLast + p * kPlaneB, plane_b - kLast - p * kPlaneB, kRowB), db, idesc, acc);
            else
              mma_f16(tmem + p * BN, da + p * (kPlaneB >> 4), db, idesc, acc);
          }
        }
        db += 2 * chunk_b >> 4;
        if (CH == 1) {
          next_tap(at, dx, dy);
        } else if ((c_at += 2 * plane_b) == CH * plane_b) {
          c_at = 0;
          next_tap(at, dx, dy);
        }
      }
      if (lead) mma_commit(gsm(&s.empty[st]));
      if (++st == ST) st = 0, lap++;
    }
    if (lead) mma_commit(gsm(s.tfull));
  }
  __syncwarp();
  if (warp < 4) {
    ok = g_mbar_wait(gsm(s.tfull), 0u) && ok;
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    // lane = row of the tile: x fastest
    const int x = x0 + (lane & 7), y = y0 + warp * 4 + (lane >> 3);
    const uint32_t acc = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
    for (int p = 0; p < BZ; p++) {
      const int z = z0 + p;
      const long long v = x + (long long)a.X * (y + (long long)a.Y * z);
      const bool in = x < a.X && y < a.Y && z < a.Z;
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += 16) {
        float f[16];
        __syncwarp();
        tmem_ld8(acc + p * BN + c0, f);
        tmem_ld8(acc + p * BN + c0 + 8, f + 8);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 16; q++) f[q] += __ldg(bias + c0 + q);
        if (in && RELU) {
#pragma unroll
          for (int h = 0; h < 2; h++) {
            uint32_t u[4];
#pragma unroll
            for (int q = 0; q < 4; q++)
              u[q] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(fmaxf(f[8 * h + 2 * q], 0.f))) |
                     ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(fmaxf(f[8 * h + 2 * q + 1], 0.f))) << 16);
            reinterpret_cast<uint4 *>(out)[(c0 / 8 + h) * a.Vp + v] = make_uint4(u[0], u[1], u[2], u[3]);
          }
        } else if (in) {
          float4 *o = reinterpret_cast<float4 *>(reinterpret_cast<float *>(out) + v * BN + c0);
#pragma unroll
          for (int q = 0; q < 4; q++) o[q] = make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]);
        }
      }
    }
  }
  if (!ok && err) atomicExch(err, 1);
  conv_exit(tmem, kCols);
}

// Data gradient: gin[u][c] += sum over the taps t = 0 .. 26 of
// sum_co dz[u - d_t][co] W[co][t][c], NC input channels of group blockIdx.y, CH
// planes of dz, BZ z-planes per block.  Each tap's products are formed in tensor
// memory on their own and added in FP32 registers in the order of the taps, as a
// column matrix and its gather would add them: a sum over the taps inside tensor
// memory would round differently, and the next layer's BF16 rounding turns that
// into steps.  Two tensor-memory buffers: the tap after the one being added is in
// flight.  Weights: [group][tap][co / 8][NC][8], ST stages of PER taps.
template <int CH, int NC, int BZ, int PER, int ST>
__global__ void __launch_bounds__(kConvThreads) k_conv_dx(const __grid_constant__ CUtensorMap map, const ConvArgs a,
                                                          const __nv_bfloat16 *__restrict__ wgt, int C,
                                                          float *__restrict__ gin, int *err) {
  extern __shared__ unsigned char cs_raw[];
  static_assert(CH % 2 == 0 && ST <= kMaxStages, "K = 16, weight stages");
  constexpr int kTaps = 27, kStages = (kTaps + PER - 1) / PER;
  constexpr uint32_t kCols = tmem_cols(2 * NC * BZ), tap_b = CH * NC * 16, stage_b = PER * tap_b, plane_b = (BZ + 2) * kPlaneB;
  uint32_t tmem;
  const ConvShm s = conv_init<CH, BZ, ST * stage_b, kCols>(cs_raw, tmem);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  int b = blockIdx.x;
  const int x0 = b % a.tx * kTX;
  b /= a.tx;
  const int y0 = b % a.ty * kTY, z0 = b / a.ty * BZ;
  bool ok = true;
  if (warp == 4) {
    if (lane == 0) {
      const __nv_bfloat16 *w = wgt + (size_t)blockIdx.y * kTaps * tap_b / 2;
      g_mbar_expect(gsm(s.tile_in), CH * plane_b);
      g_tma_load4(gsm(s.tile), &map, (x0 - 1) * 8, y0 - 1, z0 - 1, 0, gsm(s.tile_in));
      int st = 0, lap = 0;
      for (int q = 0; q < kStages; q++) {
        if (lap > 0 && ok) ok = g_mbar_wait(gsm(&s.empty[st]), (uint32_t)((lap - 1) & 1));
        const uint32_t bytes = min(PER, kTaps - q * PER) * tap_b;
        g_mbar_expect(gsm(&s.full[st]), bytes);
        g_bulk_load(gsm(s.w) + st * stage_b, w + (size_t)q * stage_b / 2, bytes, gsm(&s.full[st]));
        if (++st == ST) st = 0, lap++;
      }
    }
  } else if (warp == 5) {
    constexpr uint32_t idesc = idesc_bf16(kBM, NC);
    const bool lead = elect_one();
    ok = g_mbar_wait(gsm(s.tile_in), 0u);
    const uint64_t da0 = smem_desc(gsm(s.tile), plane_b, kRowB), db0 = smem_desc(gsm(s.w), NC * 16, 128);
    uint32_t at = 0;
    int dx = 0, dy = 0, st = 0, lap = 0, left = PER;
#pragma unroll 1
    for (int t = 0; t < kTaps; t++) {
      const int buf = t & 1;
      if (left == PER && ok) ok = g_mbar_wait(gsm(&s.full[st]), (uint32_t)(lap & 1));
      if (t >= 2 && ok) ok = g_mbar_wait(gsm(&s.tempty[buf]), (uint32_t)((t / 2 - 1) & 1));
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      // u - d_t: the staged voxel 1 - d_t on
      const uint64_t da = da0 + (uint64_t)((kLast - at) >> 4);
      const uint64_t db = db0 + (uint64_t)(((uint32_t)st * stage_b + (uint32_t)(PER - left) * tap_b) >> 4);
      if (lead) {
#pragma unroll
        for (int c = 0; c < CH; c += 2)
#pragma unroll
          for (int p = 0; p < BZ; p++)
            mma_f16(tmem + (buf * BZ + p) * NC, da + ((c * plane_b + p * kPlaneB) >> 4), db + (c * NC), idesc, c > 0);
        mma_commit(gsm(&s.tfull[buf]));
      }
      next_tap(at, dx, dy);
      if (--left == 0 || t + 1 == kTaps) {
        if (lead) mma_commit(gsm(&s.empty[st]));
        left = PER;
        if (++st == ST) st = 0, lap++;
      }
    }
  }
  __syncwarp();
  if (warp < 4) {
    float sum[BZ * NC];
#pragma unroll
    for (int q = 0; q < BZ * NC; q++) sum[q] = 0.f;
    const uint32_t acc = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
    for (int t = 0; t < kTaps; t++) {
      const int buf = t & 1;
      if (ok) ok = g_mbar_wait(gsm(&s.tfull[buf]), (uint32_t)((t / 2) & 1));
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
      for (int q = 0; q < BZ * NC; q += 16) {
        float f[16];
        tmem_ld8(acc + buf * BZ * NC + q, f);
        tmem_ld8(acc + buf * BZ * NC + q + 8, f + 8);
        tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < 16; h++) sum[q + h] += f[h];
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) g_mbar_arrive(gsm(&s.tempty[buf]));
    }
    const int x = x0 + (lane & 7), y = y0 + warp * 4 + (lane >> 3);
#pragma unroll
    for (int p = 0; p < BZ; p++) {
      const int z = z0 + p;
      if (x >= a.X || y >= a.Y || z >= a.Z) continue;
      const long long v = x + (long long)a.X * (y + (long long)a.Y * z);
      float4 *g = reinterpret_cast<float4 *>(gin + v * C + (int)blockIdx.y * NC);
#pragma unroll
      for (int q = 0; q < NC / 4; q++) {
        float4 o = g[q];
        o.x += sum[p * NC + 4 * q];
        o.y += sum[p * NC + 4 * q + 1];
        o.z += sum[p * NC + 4 * q + 2];
        o.w += sum[p * NC + 4 * q + 3];
        g[q] = o;
      }
    }
  }
  if (!ok && err) atomicExch(err, 1);
  conv_exit(tmem, kCols);
}

// Weight gradient: gW[tap * C + c][n] += sum over the voxels of in[r + d_tap][c]
// dz[r][n], CH planes of 8 input channels, CN outputs.  The voxels are the K
// dimension, so both operands are MN-major: 8 voxels x 8 channels of a plane are
// 128 contiguous bytes, one core matrix.  The 128 rows of a block are 16 slots of 8
// channels, a slot being a (dy, dz) shift of a plane, staged as 16 rows of 10
// voxels; the three dx are three products from start addresses 16 bytes apart into
// three accumulators, so a staged slot serves three taps (single taps staged at 8
// voxels a row copy 2.4 x the bytes).  Blocks along y split the tiles of the
// volume and add their sums with vector reductions, as a split-K GEMM would.
// It is bound by the copies of the shifted slots from L2 (9 x the activations).
// Against 64-bit sums of the same operands (16 -> 16 channels of 72 x 72 x 56) it
// is off by 4.0e-6 where all terms are positive and by 1.4e-6 where their signs
// are mixed; the GEMM over a transposed column matrix by 1.1e-5 and 2.8e-6 (tensor
// memory truncates: the error grows with the terms of one accumulator).  The 15
// weight gradients of a training step take 0.25 ms; 1.2 with the column matrices.
template <int CH, int CN>
struct DwShape {
  static constexpr int kSlots = 9 * CH, kGroups = (kSlots + 15) / 16;
  static constexpr uint32_t slot_b = kTY * kRowB, plane_b = kTX * kTY * 16;
  static constexpr uint32_t stage_b = 16 * slot_b + CN / 8 * plane_b;
  static constexpr int ST = CN <= 32 ? 2 : 3;  // two blocks per SM, or one with a deeper ring
  static constexpr size_t shm = 128 + ST * stage_b + 256;
};
template <int CH, int CN>
__global__ void __launch_bounds__(kConvThreads) k_conv_dw(const __grid_constant__ CUtensorMap map_in,
                                                          const __grid_constant__ CUtensorMap map_dz, const ConvArgs a,
                                                          int tiles, float *__restrict__ gw, int *err) {
  using D = DwShape<CH, CN>;
  extern __shared__ unsigned char cs_raw[];
  constexpr uint32_t kCols = tmem_cols(3 * CN);
  uint32_t tmem;
  const ConvShm s = conv_init<0, 0, D::ST * D::stage_b, kCols>(cs_raw, tmem);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int slot0 = blockIdx.x * 16, used = min(16, D::kSlots - slot0);
  bool ok = true;
  if (warp == 4) {
    // lane q < used copies slot q, the next CN / 8 lanes the planes of dz
    const int c = lane < used ? (slot0 + lane) % CH : lane - used, sh = (slot0 + lane) / CH;
    const int sy = lane < used ? sh % 3 - 1 : 0, sz = lane < used ? sh / 3 - 1 : 0, sx = lane < used ? 1 : 0;
    int st = 0, lap = 0;
    for (int i = blockIdx.y; i < tiles; i += gridDim.y) {
      if (lap > 0 && ok) ok = g_mbar_wait(gsm(&s.empty[st]), (uint32_t)((lap - 1) & 1));
      const int x = i % a.tx * kTX, y = i / a.tx % a.ty * kTY, z = i / (a.tx * a.ty);
      const uint32_t base = gsm(s.w) + st * D::stage_b, bar = gsm(&s.full[st]);
      if (lane == 0) g_mbar_expect(bar, used * D::slot_b + CN / 8 * D::plane_b);
      __syncwarp();
      if (lane < used)
        g_tma_load4(base + lane * D::slot_b, &map_in, (x - sx) * 8, y + sy, z + sz, c, bar);
      else if (lane < used + CN / 8)
        g_tma_load4(base + 16 * D::slot_b + c * D::plane_b, &map_dz, x * 8, y, z, c, bar);
      if (++st == D::ST) st = 0, lap++;
    }
  } else if (warp == 5) {
    // both operands MN-major (bits 15, 16)
    constexpr uint32_t idesc = idesc_bf16(kBM, CN) | (1u << 15) | (1u << 16);
    const bool lead = elect_one();
    int st = 0, lap = 0;
    uint32_t acc = 0;
    for (int i = blockIdx.y; i < tiles; i += gridDim.y) {
      if (ok) ok = g_mbar_wait(gsm(&s.full[st]), (uint32_t)(lap & 1));
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t base = gsm(s.w) + st * D::stage_b;
      const uint64_t da = smem_desc(base, kRowB, D::slot_b), db = smem_desc(base + 16 * D::slot_b, kTX * 16, D::plane_b);
      if (lead) {
#pragma unroll
        for (int k = 0; k < kTY / 2; k++) {  // 16 voxels: two rows of 8
#pragma unroll
          for (int dx = 0; dx < 3; dx++)
            mma_f16(tmem + dx * CN, da + ((k * 2 * kRowB + dx * 16) >> 4), db + (k * 2 * kTX * 16 >> 4), idesc, acc | (k > 0));
        }
        mma_commit(gsm(&s.empty[st]));
      }
      acc = 1;
      if (++st == D::ST) st = 0, lap++;
    }
    if (lead) mma_commit(gsm(s.tfull));
  }
  __syncwarp();
  if (warp < 4) {
    ok = g_mbar_wait(gsm(s.tfull), 0u) && ok;
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const int row = warp * 32 + lane, slot = slot0 + row / 8;
    const uint32_t at = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
    for (int dx = 0; dx < 3; dx++) {
      float *o = gw + ((long long)((slot / CH) * 3 + dx) * (CH * 8) + slot % CH * 8 + row % 8) * CN;
#pragma unroll 1
      for (int c0 = 0; c0 < CN; c0 += 8) {
        float f[8];
        __syncwarp();
        tmem_ld8(at + dx * CN + c0, f);
        tmem_ld_wait();
        if (slot < D::kSlots && ok) {
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(o + c0), "f"(f[0]), "f"(f[1]), "f"(f[2]), "f"(f[3]) : "memory");
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(o + c0 + 4), "f"(f[4]), "f"(f[5]), "f"(f[6]), "f"(f[7]) : "memory");
        }
      }
    }
  }
  if (!ok && err) atomicExch(err, 1);
  conv_exit(tmem, kCols);
}

}  // namespace unet
}  // namespace aphid
