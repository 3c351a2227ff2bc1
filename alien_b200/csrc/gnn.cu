// gnn.cu -- the learned preconditioner: a message-passing network on the
// matrix graph, its training kernels, and flexible CG with ILU(0) fallback.
// No counterpart in the reference; the network is defined (and checked) by
// oracle/gnn_oracle.py.  It works on the diagonal-scaled system
// D^-1/2 A D^-1/2, so neither inputs nor outputs carry the coefficients'
// orders of magnitude:
//   xr_i = r_i / sqrt(a_ii), s = rms(xr); x0_i = [xr_i/s, log(a_ii)/10]
//   h1 = relu(W0 x0 + b0)                                                      (2 -> 64)
//   4 x { g_ij = sigmoid(u e_ij + c), e_ij = log|a_ij| - (log a_ii + log a_jj)/2 ;
//         m_i = sum_j g_ij h_j ; h <- relu(W [h; m] + b) }                       (128 -> 64)
//   z_i = s (wd . h5_i + bd + ws x0_i) / sqrt(a_ii)       (ws: the Jacobi skip)
// Activations are stored in BF16 ([n][64], 128 B per node); h1 by a kernel of its
// own.  Each layer is one fused kernel, neighbour sums, dense layer on the tensor
// cores (BF16 x BF16 -> FP32) and bias/relu epilogue, of two: on 3-D 7-point graphs
// the grid layer (k_gnn_layer_grid: neighbours by bulk copy, tcgen05.mma), on others
// the gather layer (k_gnn_layer: neighbours by index, mma.sync m16n8k16, a warp 16
// nodes x 64 outputs over K = 128).  The last one applies the decoder in its
// epilogue, so inference moves about 2 x 128 B per node and layer.  Training: hand-written backward kernels (loss
// (z-e)^T A (z-e) / e^T A e on (residual, error) pairs), per-block partial
// sums reduced in a fixed order (deterministic), Adam on FP32 master weights
// with BF16 copies for the forward.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <random>
#include <type_traits>
#include <vector>

#include "ab2_internal.cuh"
#include "precond.cuh"
#include "reduce.cuh"
#include "sentinel.cuh"
#include "spmv_view.cuh"
#include "tcgen05.cuh"

namespace ab2 {
namespace {

constexpr int kH = 64;          // hidden width
constexpr int kLayers = 4;
constexpr int kIn = 2 * kH;     // dense layer input [h ; m]
constexpr int kWStride = kIn + 8;  // padded smem row (bf16): conflict-free fragment loads
// flat parameter layout (oracle/gnn_oracle.py Params.flat)
constexpr int kOffW0 = 0;
constexpr int kOffB0 = kOffW0 + kH * 2;
constexpr int kOffW = kOffB0 + kH;
constexpr int kOffB = kOffW + kLayers * kH * kIn;
constexpr int kOffU = kOffB + kLayers * kH;
constexpr int kOffC = kOffU + kLayers;
constexpr int kOffWd = kOffC + kLayers;
constexpr int kOffBd = kOffWd + kH;
constexpr int kOffWs = kOffBd + 1;
constexpr int kParams = kOffWs + 1;

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<unsigned*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16(unsigned u) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}
__device__ __forceinline__ float sigmoidf(float t) { return 1.f / (1.f + expf(-t)); }

// D = A B + D, m16n8k16, A row-major BF16 (4 regs), B col-major BF16 (2 regs), FP32 accumulators.
__device__ __forceinline__ void mma_bf16(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ------------------------------------------------------------------ graph features
// Per row: 1/sqrt(a_ii) and log(a_ii)/10; per CSR entry the edge feature
// log|a_ij| - (log a_ii + log a_jj)/2 (the entry of D^-1/2 A D^-1/2) and the
// position of the transposed entry (the pattern must be structurally
// symmetric).  bad |= 1: a row without a positive diagonal; |= 2: no (j, i).
__device__ __forceinline__ bool diag_of(int r, const int* __restrict__ rp, const int* __restrict__ ci,
                                        const double* __restrict__ v, const int* __restrict__ dcol, double* d) {
  const int dk = dcol[r];
  if (dk < rp[r + 1] && ci[dk] == r && v[dk] > 0) {
    *d = v[dk];
    return true;
  }
  return false;
}

__global__ void k_gnn_prep(int n, const int* __restrict__ rp, const int* __restrict__ ci, const double* __restrict__ v,
                           const int* __restrict__ dcol, float* __restrict__ isd, float* __restrict__ logd10,
                           float* __restrict__ efeat, int* __restrict__ tidx, int* bad) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double d = 1.0;
    if (!diag_of(i, rp, ci, v, dcol, &d)) {
      atomicOr(bad, 1);
      continue;
    }
    isd[i] = (float)(1.0 / sqrt(d));
    logd10[i] = (float)(log(d) / 10.0);
    for (int k = rp[i]; k < rp[i + 1]; ++k) {
      const int j = ci[k];
      if (j == i) {
        efeat[k] = 0.f;
        tidx[k] = -1;
        continue;
      }
      double dj = 1.0;
      if (!diag_of(j, rp, ci, v, dcol, &dj)) atomicOr(bad, 1);
      efeat[k] = (float)(log(fabs(v[k])) - 0.5 * (log(d) + log(dj)));
      int t = -1;  // (j, i) in row j (columns sorted: binary search)
      int lo = rp[j], hi = rp[j + 1] - 1;
      while (lo <= hi) {
        const int mid = (lo + hi) >> 1;
        if (ci[mid] == i) {
          t = mid;
          break;
        }
        if (ci[mid] < i) lo = mid + 1;
        else hi = mid - 1;
      }
      tidx[k] = t;
      if (t < 0) atomicOr(bad, 2);
    }
  }
}

// The forward pass reads the graph as a padded neighbour table: per node nbw
// (a multiple of 8) slots of (column, edge feature) in CSR order, -1 marking
// padding -- one 32-byte load per 8 neighbours instead of a row-pointer load
// followed by dependent column loads.
__global__ void k_gnn_nbr(int n, const int* __restrict__ rp, const int* __restrict__ ci, const float* __restrict__ efeat,
                          int nbw, int* __restrict__ nb_idx, float* __restrict__ nb_ef) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int w = 0;
    for (int k = rp[i]; k < rp[i + 1]; ++k) {
      if (ci[k] == i) continue;
      nb_idx[(size_t)i * nbw + w] = ci[k];
      nb_ef[(size_t)i * nbw + w] = efeat[k];
      ++w;
    }
    for (; w < nbw; ++w) {
      nb_idx[(size_t)i * nbw + w] = -1;
      nb_ef[(size_t)i * nbw + w] = 0.f;
    }
  }
}

// The grid layer's edge features: per node (rows padded to whole 128-node
// tiles) the feature of each direction -nx ny, -nx, -1, +1, +nx, +nx ny (the
// CSR column order), NaN where the row has no entry there.
__global__ void k_gnn_dir_table(int n, long long rows, int nx, int sxy, const int* __restrict__ rp,
                                const int* __restrict__ ci, const float* __restrict__ efeat, float* __restrict__ tab) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < rows; i += (long long)gridDim.x * blockDim.x) {
    float e[6];
#pragma unroll
    for (int d = 0; d < 6; ++d) e[d] = __int_as_float(0x7fc00000);
    if (i < n) {
      for (int k = rp[i]; k < rp[i + 1]; ++k) {
        const long long off = (long long)ci[k] - i;
        const int d = off == -sxy ? 0 : off == -nx ? 1 : off == -1 ? 2 : off == 1 ? 3 : off == nx ? 4 : off == sxy ? 5 : -1;
        if (d >= 0) e[d] = efeat[k];
      }
    }
#pragma unroll
    for (int d = 0; d < 6; ++d) tab[i * 6 + d] = e[d];
  }
}

// ------------------------------------------------------------------ forward
// xr_i = r_i / sqrt(a_ii) (FP32) and s = rms(xr): s2[0] = s, s2[1] = 1/s (0 if s = 0).
__global__ void __launch_bounds__(kThreads) k_gnn_scale(int n, const double* __restrict__ r, const float* __restrict__ isd,
                                                        float* __restrict__ xr, double* partials, unsigned* counter,
                                                        double* red_out, double* s2) {
  double acc[1] = {0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float t = (float)(r[i] * (double)isd[i]);
    xr[i] = t;
    acc[0] = fma((double)t, (double)t, acc[0]);
  }
  if (grid_reduce<1>(acc, partials, counter, red_out)) {
    const double s = sqrt(red_out[0] / (double)max(n, 1));
    s2[0] = s;
    s2[1] = s > 0 ? 1.0 / s : 0.0;
  }
}

// One message-passing layer, fused, on tensor cores for both of its products:
//   m = G H_nb       (G: the 16 nodes' gates as a 16 x K BF16 matrix, one
//                     nonzero run per row; H_nb: the K = 16 nbw neighbour rows)
//   h_out = relu(W [h ; m] + b)
// A warp takes 16 nodes at a time (persistent: it walks the tiles with a
// stride).  The neighbour rows (padding slots zero-filled) are copied into the
// warp's shared memory with cp.async, 8 lanes per 128-byte row so that every
// copy instruction moves 4 whole rows.  The neighbour-table entries of the
// warp's next tile are loaded while the current one computes, so a tile waits
// on one memory latency.  Gates are computed one (node, slot) pair per lane
// and shuffled straight into A fragments (G is block diagonal: row g of a
// 16-column chunk is nonzero only where the chunk's pairs belong to node g).
// The aggregation is K/16 mma.sync m16n8k16 steps (B from the neighbour rows
// via ldmatrix.trans); its FP32 accumulators, rounded to BF16, are already in
// the A-fragment layout of the dense layer's last four k-steps; the own rows'
// fragments are read from global memory.  W (64 x 128, BF16) is staged once
// per CTA and read with ldmatrix.  Epilogue: bias, relu, BF16, 128-byte row
// stores through shared memory; LAST fuses the decoder
// z_i = s (wd . h5_i + bd + ws x0_i) / sqrt(a_ii).
// Optional stores (training): m_out, h_out (LAST).
struct LayerArgs {
  int n;
  int nbw;              // neighbour slots per node (even, <= kMaxNbw)
  const int* nb_idx;    // [n][nbw], -1 = padding
  const float* nb_ef;   // [n][nbw] edge features
  const float* P;       // FP32 parameters
  const bf16* W;        // this layer's W in BF16 (64 x 128, row = output)
  int layer;
  const bf16* h_in;     // h_l
  const float* xr;      // r_i / sqrt(a_ii)
  const float* isd;
  const double* s2;     // s, 1/s
  bf16* m_out;          // m_l (or null)
  bf16* h_out;          // h_{l+1} (or null when LAST)
  double* z;            // LAST: the network's output
};

constexpr int kMaxNbw = 16;
constexpr int kMaxRounds = kMaxNbw / 2;  // 32 (node, slot) pairs a round
constexpr int kLayerWarps = 4;
constexpr int kRowStride = kH + 8;       // bf16: 144-byte rows, conflict-free ldmatrix
__host__ __device__ constexpr int agg_k(int nbw) { return 16 * nbw; }  // nbw even: a multiple of 32
size_t layer_smem_bytes(int nbw) {
  return sizeof(bf16) * ((size_t)kH * kWStride + (size_t)kLayerWarps * agg_k(nbw) * kRowStride) +
         sizeof(float) * 2 * kH;
}

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool fill) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(dst)), "l"(src), "r"(fill ? 16 : 0));
}
__device__ __forceinline__ void ldsm_x4(unsigned (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}
__device__ __forceinline__ void ldsm_x4_t(unsigned (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}
__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
// Two FP32 values in one 64-bit register pair, and acc += g * (lo(w), hi(w)) as
// one packed FP32 FMA (fma.rn.f32x2): a BF16 value is the high half of its FP32
// value, so the halves of w unpack with a shift and a mask; each product is exact
// and each sum rounds once.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 make_f32x2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void split_f32x2(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 unpack_f32x2(unsigned w) {
  return make_f32x2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
__device__ __forceinline__ void fma_f32x2(f32x2& acc, f32x2 g, f32x2 x) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(g), "l"(x));
}
__device__ __forceinline__ f32x2 add_f32x2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned pack_f32x2(f32x2 v) {  // rounded to BF16
  float lo, hi;
  split_f32x2(v, lo, hi);
  return pack_bf16(lo, hi);
}
// max(x, 0) of two BF16 values (NaN: 0, as fmaxf)
__device__ __forceinline__ unsigned relu_bf16x2(unsigned w) {
  unsigned r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(w), "r"(0u));
  return r;
}
// Shared-memory words at 32-bit shared addresses.
__device__ __forceinline__ float lds_f32(unsigned a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint4 lds128(unsigned a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
}

template <bool LAST>
__global__ void __launch_bounds__(kLayerWarps * 32) k_gnn_layer(const LayerArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  bf16* Ws = reinterpret_cast<bf16*>(smem);
  float* bs = reinterpret_cast<float*>(Ws + kH * kWStride);
  float* wds = bs + kH;
  for (int t = threadIdx.x; t < kH * kIn / 8; t += blockDim.x)
    *reinterpret_cast<uint4*>(Ws + (t >> 4) * kWStride + (t & 15) * 8) = reinterpret_cast<const uint4*>(a.W)[t];
  for (int t = threadIdx.x; t < kH; t += blockDim.x) {
    bs[t] = a.P[kOffB + a.layer * kH + t];
    wds[t] = a.P[kOffWd + t];
  }
  __syncthreads();
  const unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nbw = a.nbw, K = agg_k(nbw), rounds = K / 32;
  bf16* Nb = reinterpret_cast<bf16*>(wds + kH) + warp * K * kRowStride;  // neighbour rows [K][kRowStride]
  const float u = a.P[kOffU + a.layer], c = a.P[kOffC + a.layer];
  const int g = lane >> 2, t = lane & 3;
  const int lrow = (lane & 7) + ((lane >> 3) & 1) * 8, lcol = (lane >> 4) * 8;  // ldmatrix x4 lane address
  const int wrow = (lane & 7) + (lane >> 4) * 8, wcol = ((lane >> 3) & 1) * 8;  // W fragments
  const int ntiles = (a.n + 15) / 16;
  const int stride = gridDim.x * kLayerWarps;
  // neighbour-table entries of pair 32 r + lane of a tile
  int pidx[kMaxRounds];
  float pef[kMaxRounds];
  auto fetch = [&](int tile) {
#pragma unroll
    for (int r = 0; r < kMaxRounds; ++r) {
      pidx[r] = -1;
      pef[r] = 0.f;
      const long long e = (long long)tile * 16 * nbw + 32 * r + lane;
      if (r < rounds && tile < ntiles && e < (long long)a.n * nbw) {
        pidx[r] = a.nb_idx[e];
        pef[r] = a.nb_ef[e];
      }
    }
  };
  fetch(blockIdx.x * kLayerWarps + warp);
  for (int tile = blockIdx.x * kLayerWarps + warp; tile < ntiles; tile += stride) {
    const int base = tile * 16;
    // ---- neighbour rows into shared memory; gates of this lane's pairs
    float gr[kMaxRounds];
#pragma unroll
    for (int r = 0; r < kMaxRounds; ++r) {
      gr[r] = 0.f;
      if (r < rounds) {
        const int j = pidx[r];
        if (j >= 0) gr[r] = bf16r(sigmoidf(fmaf(u, pef[r], c)));
#pragma unroll
        for (int q = 0; q < 8; ++q) {  // rows 32 r + 4 q .. + 3, 8 lanes each
          const int src = q * 4 + (lane >> 3);
          const int jj = __shfl_sync(kFull, j, src);
          cp_async16(Nb + (32 * r + src) * kRowStride + (lane & 7) * 8,
                     a.h_in + (size_t)max(jj, 0) * kH + (lane & 7) * 8, jj >= 0);
        }
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    fetch(tile + stride);  // the next tile's table entries, in flight during this tile
    // own rows' A fragments (k-steps 0..3) straight from global memory
    unsigned hA[4][4];
    {
      const unsigned* hv = reinterpret_cast<const unsigned*>(a.h_in);
      const int r0 = base + g, r1 = r0 + 8;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        const int col = ks * 16 + 2 * t;
        hA[ks][0] = r0 < a.n ? __ldg(hv + (((size_t)r0 * kH + col) >> 1)) : 0u;
        hA[ks][1] = r1 < a.n ? __ldg(hv + (((size_t)r1 * kH + col) >> 1)) : 0u;
        hA[ks][2] = r0 < a.n ? __ldg(hv + (((size_t)r0 * kH + col + 8) >> 1)) : 0u;
        hA[ks][3] = r1 < a.n ? __ldg(hv + (((size_t)r1 * kH + col + 8) >> 1)) : 0u;
      }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncwarp();
    // ---- aggregation m = G H_nb on tensor cores
    float accm[8][4];
#pragma unroll
    for (int nb = 0; nb < 8; ++nb) accm[nb][0] = accm[nb][1] = accm[nb][2] = accm[nb][3] = 0.f;
#pragma unroll
    for (int r = 0; r < kMaxRounds; ++r) {
      if (r < rounds) {
#pragma unroll
        for (int hlf = 0; hlf < 2; ++hlf) {
          const int k0 = 32 * r + 16 * hlf;
          // pairs k0 + 2t (+1) and k0 + 2t + 8 (+1): gates from lanes 16 hlf + 2t + {0, 1, 8, 9}
          const float g0 = __shfl_sync(kFull, gr[r], 16 * hlf + 2 * t);
          const float g1 = __shfl_sync(kFull, gr[r], 16 * hlf + 2 * t + 1);
          const float g8 = __shfl_sync(kFull, gr[r], 16 * hlf + 2 * t + 8);
          const float g9 = __shfl_sync(kFull, gr[r], 16 * hlf + 2 * t + 9);
          const int na = (k0 + 2 * t) / nbw, nc = (k0 + 2 * t + 8) / nbw;  // their nodes
          const unsigned pa = pack_bf16(g0, g1), pc = pack_bf16(g8, g9);
          const unsigned af[4] = {na == g ? pa : 0u, na == g + 8 ? pa : 0u, nc == g ? pc : 0u, nc == g + 8 ? pc : 0u};
#pragma unroll
          for (int n0 = 0; n0 < kH; n0 += 16) {
            unsigned bf[4];
            ldsm_x4_t(bf, Nb + (k0 + lrow) * kRowStride + n0 + lcol);
            mma_bf16(accm[n0 / 8], af, bf[0], bf[1]);
            mma_bf16(accm[n0 / 8 + 1], af, bf[2], bf[3]);
          }
        }
      }
    }
    // m in BF16, already laid out as the A fragments of k-steps 4..7
    unsigned mA[4][4];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      mA[ks][0] = pack_bf16(accm[2 * ks][0], accm[2 * ks][1]);
      mA[ks][1] = pack_bf16(accm[2 * ks][2], accm[2 * ks][3]);
      mA[ks][2] = pack_bf16(accm[2 * ks + 1][0], accm[2 * ks + 1][1]);
      mA[ks][3] = pack_bf16(accm[2 * ks + 1][2], accm[2 * ks + 1][3]);
    }
    // ---- dense layer [h ; m] W^T on tensor cores
    float acc[8][4];
#pragma unroll
    for (int nb = 0; nb < 8; ++nb) acc[nb][0] = acc[nb][1] = acc[nb][2] = acc[nb][3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
#pragma unroll
      for (int n0 = 0; n0 < kH; n0 += 16) {
        unsigned bf[4];
        ldsm_x4(bf, Ws + (n0 + wrow) * kWStride + ks * 16 + wcol);
        const unsigned(&af)[4] = ks < 4 ? hA[ks] : mA[ks - 4];
        mma_bf16(acc[n0 / 8], af, bf[0], bf[1]);
        mma_bf16(acc[n0 / 8 + 1], af, bf[2], bf[3]);
      }
    }
    __syncwarp();  // every lane is done with the neighbour rows: rows 0..31 stage the outputs
    bf16* Ms = Nb;
    bf16* Hs = Nb + 16 * kRowStride;
    if (a.m_out) {
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        *reinterpret_cast<unsigned*>(Ms + g * kRowStride + ks * 16 + 2 * t) = mA[ks][0];
        *reinterpret_cast<unsigned*>(Ms + (g + 8) * kRowStride + ks * 16 + 2 * t) = mA[ks][1];
        *reinterpret_cast<unsigned*>(Ms + g * kRowStride + ks * 16 + 8 + 2 * t) = mA[ks][2];
        *reinterpret_cast<unsigned*>(Ms + (g + 8) * kRowStride + ks * 16 + 8 + 2 * t) = mA[ks][3];
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int idx = q * 32 + lane, row = idx >> 3, c8 = idx & 7;
        if (base + row < a.n)
          reinterpret_cast<uint4*>(a.m_out + (size_t)(base + row) * kH)[c8] =
              *reinterpret_cast<const uint4*>(Ms + row * kRowStride + c8 * 8);
      }
    }
    // ---- epilogue: bias, relu, BF16
    float y0 = 0.f, y1 = 0.f;
    unsigned o0[8], o1[8];
#pragma unroll
    for (int nb = 0; nb < 8; ++nb) {
      const int cc = nb * 8 + 2 * t;
      const float h00 = bf16r(fmaxf(acc[nb][0] + bs[cc], 0.f)), h01 = bf16r(fmaxf(acc[nb][1] + bs[cc + 1], 0.f));
      const float h10 = bf16r(fmaxf(acc[nb][2] + bs[cc], 0.f)), h11 = bf16r(fmaxf(acc[nb][3] + bs[cc + 1], 0.f));
      o0[nb] = pack_bf16(h00, h01);
      o1[nb] = pack_bf16(h10, h11);
      if constexpr (LAST) {
        y0 = fmaf(wds[cc], h00, fmaf(wds[cc + 1], h01, y0));
        y1 = fmaf(wds[cc], h10, fmaf(wds[cc + 1], h11, y1));
      }
    }
    if (a.h_out) {
#pragma unroll
      for (int nb = 0; nb < 8; ++nb) {
        *reinterpret_cast<unsigned*>(Hs + g * kRowStride + nb * 8 + 2 * t) = o0[nb];
        *reinterpret_cast<unsigned*>(Hs + (g + 8) * kRowStride + nb * 8 + 2 * t) = o1[nb];
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int idx = q * 32 + lane, row = idx >> 3, c8 = idx & 7;
        if (base + row < a.n)
          reinterpret_cast<uint4*>(a.h_out + (size_t)(base + row) * kH)[c8] =
              *reinterpret_cast<const uint4*>(Hs + row * kRowStride + c8 * 8);
      }
    }
    if constexpr (LAST) {
      y0 += __shfl_xor_sync(kFull, y0, 1);
      y0 += __shfl_xor_sync(kFull, y0, 2);
      y1 += __shfl_xor_sync(kFull, y1, 1);
      y1 += __shfl_xor_sync(kFull, y1, 2);
      if (t == 0) {
        const double s = a.s2[0], is = a.s2[1];
        const float bd = a.P[kOffBd], ws = a.P[kOffWs];
        const int r0 = base + g, r1 = r0 + 8;
        if (r0 < a.n) a.z[r0] = s * (double)(y0 + bd + ws * (float)(a.xr[r0] * is)) * (double)a.isd[r0];
        if (r1 < a.n) a.z[r1] = s * (double)(y1 + bd + ws * (float)(a.xr[r1] * is)) * (double)a.isd[r1];
      }
    }
    __syncwarp();  // the staging rows are refilled by the next tile's copies
  }
}

// ------------------------------------------------------------------ layer on a 3-D grid (tcgen05)
// The same layer for a matrix whose graph is a 3-D 7-point grid in
// lexicographic order (row i + nx (j + ny k), off-diagonal columns at -nx ny,
// -nx, -1, +1, +nx, +nx ny where inside the grid): 128 consecutive nodes a
// tile, so each direction's neighbour rows form one contiguous block of h and
// nothing is gathered by index.  A persistent CTA (one an SM) walks tiles with
// its warps in four roles that hand on through mbarriers:
//   - copies (one thread): a step's inputs (64 nodes, half a tile) by bulk copy
//     (cp.async.bulk, no multicast) into a ring of three stages -- the step's own
//     rows with one row either side (the +-1 neighbours), the four +-nx / +-nx ny
//     blocks, and the edge features in direction order (NaN where no neighbour);
//   - aggregation (16 warps, each four nodes a step and a lane one 8-feature chunk
//     of one node): the gates sigmoid(u e + c) once per (node, direction), a lane
//     each, handed round by shuffles, m = sum_d g_d h_nbr(d) (BF16 x BF16 products,
//     FP32 sums in the CSR column order, rounded to BF16 as the tensor-core
//     aggregation of k_gnn_layer is; 0 for absent neighbours), then [h ; m] written
//     as A (128 x 128 BF16, 128-byte swizzle) into one of two buffers;
//   - MMA (one thread): once a tile's A operand is complete and an accumulator is
//     free, eight tcgen05.mma (M = 128, N = 64, K = 16) into it (two 128 x 64 FP32
//     accumulators in tensor memory); B is W (64 x 128 BF16), staged once per CTA;
//   - epilogue (4 warps, one a tensor-memory lane quarter): a row a thread, bias,
//     BF16, relu, turned through shared memory so that h is stored in whole
//     sectors (LAST: the decoder's z instead).
// Beside the MMA the work a tile is about 7,500 warp instructions and 3,000 turns of
// the shared-memory port (inputs copied in, seven rows read a node, A written and
// read, the output turned), and that port, 81 % busy, is what bounds it: 1.72 million nodes take 180 us a layer (the last one 190), 227 (192)
// before, when the aggregation warps went in step through a tile (gates, a barrier,
// sums, a wait for the one A buffer) and the epilogue stored a row a thread, 16 bytes
// at a time.  Also measured there: the neighbour rows by registers from global
// memory instead of the ring 219 to 293 us (too few bytes in flight for L2's
// latency), the last reader refilling a stage behind an atomic and a fence instead of
// a warp of its own 300, the epilogue's first warp issuing the MMA 222.
// Every wait is bounded: on expiry the kernel sets *err, every role stops at
// its next tile, and the CTA waits (bounded) for the copies and the MMA it
// issued and frees its tensor memory before it returns.
constexpr int kTcAggWarps = 16;
constexpr int kTcEpiWarps = 4;
constexpr int kTcThreads = (kTcAggWarps + kTcEpiWarps + 2) * 32;  // + the MMA's and the copies' warps
constexpr int kTcTile = 128;
constexpr int kTcHalf = kTcAggWarps * 4;                     // nodes the aggregation warps take at a time: a step
constexpr int kTcStages = 3;
constexpr unsigned kTcRowB = kH * 2;                         // bytes of one h row
constexpr unsigned kTcW = 0;                                 // B: 2 regions x 64 rows x 128 B
constexpr unsigned kTcA = kTcW + 2 * kH * kTcRowB;           // A: 2 buffers x 2 regions x 128 rows x 128 B
constexpr unsigned kTcARegion = kTcTile * kTcRowB;
constexpr unsigned kTcABuf = 2 * kTcARegion;
constexpr unsigned kTcStage = kTcA + 2 * kTcABuf;            // a step's inputs:
constexpr unsigned kTcBlockB = kTcHalf * kTcRowB;
constexpr unsigned kTcXOff = 0;                              //   rows b-1 .. b+64
constexpr unsigned kTcYmOff = kTcXOff + (kTcHalf + 2) * kTcRowB;
constexpr unsigned kTcYpOff = kTcYmOff + kTcBlockB;
constexpr unsigned kTcZmOff = kTcYpOff + kTcBlockB;
constexpr unsigned kTcZpOff = kTcZmOff + kTcBlockB;
constexpr unsigned kTcEfOff = kTcZpOff + kTcBlockB;          //   64 x 6 floats
constexpr unsigned kTcEfBytes = kTcHalf * 6 * 4;
constexpr unsigned kTcStageB = kTcEfOff + kTcEfBytes;
constexpr unsigned kTcOut = kTcStage + kTcStages * kTcStageB;  // the epilogue's half rows: 4 warps x 32 x 64 B
constexpr unsigned kTcOutB = 32 * kTcRowB / 2;
constexpr unsigned kTcBias = kTcOut + kTcEpiWarps * kTcOutB;  // bias, wd: 2 x 64 floats
constexpr unsigned kTcBar = kTcBias + 2 * kH * 4;            // 14 mbarriers, tensor-memory address, abort flag
constexpr unsigned kTcSmem = kTcBar + 128 + 1024;            // + slack to align the base to 1024 bytes
constexpr unsigned kTcCols = 2 * kH;                         // tensor-memory columns: two accumulators
static_assert(kTcSmem <= 227 * 1024, "grid layer: shared memory");
static_assert(kTcA % 1024 == 0 && kTcABuf % 1024 == 0 && kTcStageB % 16 == 0, "grid layer: alignment");
static_assert(kTcBias - kTcOut == 4 * 32 * 64, "grid layer: one staging buffer an epilogue warp");
static_assert(2 * kTcHalf == kTcTile && kTcHalf % 8 == 0, "grid layer: two steps a tile, one swizzle for both");

struct GridLayerArgs {
  LayerArgs a;
  int nx, sxy;           // grid strides along j and k
  const float* dir_ef;   // [ceil(n/128) * 128][6] edge features by direction, NaN = none
  int* err;              // set when a bounded wait gives up
};

template <bool LAST>
__global__ void __launch_bounds__(kTcThreads, 1) k_gnn_layer_grid(const GridLayerArgs ga) {
  const LayerArgs& a = ga.a;
  extern __shared__ unsigned char tc_smem_raw[];
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) &
                                                       ~static_cast<uintptr_t>(1023));
  const unsigned sb = tc::smem_u32(sm);
  float* s_bias = reinterpret_cast<float*>(sm + kTcBias);
  float* s_wd = s_bias + kH;
  // mbarriers, two of each: A written; A released by the tensor core; accumulator
  // complete; accumulator read; then one a stage: inputs landed; inputs read
  const unsigned bar_afull = sb + kTcBar, bar_aempty = bar_afull + 16;
  const unsigned bar_accf = bar_afull + 32, bar_acce = bar_afull + 48, bar_full = bar_afull + 64;
  const unsigned bar_read = bar_full + 8 * kTcStages;
  volatile unsigned* s_tmem = reinterpret_cast<volatile unsigned*>(sm + kTcBar + 112);
  volatile int* s_abort = reinterpret_cast<volatile int*>(sm + kTcBar + 116);
  const unsigned kFull = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = a.n;
  const int ntiles = (n + kTcTile - 1) / kTcTile;
  const int count = blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  auto tile_base = [&](int c) { return (long long)((int)blockIdx.x + c * (int)gridDim.x) * kTcTile; };
  auto give_up = [&]() {
    *s_abort = 1;
    atomicOr(ga.err, 1);
  };

  // W as the B operand (row o = output feature, K-major, 128-byte swizzle)
  for (int t = tid; t < kH * kIn / 8; t += kTcThreads) {
    const int o = t >> 4, reg = (t >> 3) & 1, c = t & 7;
    *reinterpret_cast<uint4*>(sm + kTcW + reg * (kH * kTcRowB) + o * kTcRowB + ((c ^ (o & 7)) << 4)) =
        reinterpret_cast<const uint4*>(a.W)[t];
  }
  for (int t = tid; t < kH; t += kTcThreads) {
    s_bias[t] = a.P[kOffB + a.layer * kH + t];
    s_wd[t] = a.P[kOffWd + t];
  }
  if (tid == 0) {
    for (int k = 0; k < 2; ++k) {
      tc::mbar_init(bar_afull + 8 * k, kTcAggWarps);
      tc::mbar_init(bar_aempty + 8 * k, 1);
      tc::mbar_init(bar_accf + 8 * k, 1);
      tc::mbar_init(bar_acce + 8 * k, kTcEpiWarps);
    }
    for (int k = 0; k < kTcStages; ++k) {
      tc::mbar_init(bar_full + 8 * k, 1);
      tc::mbar_init(bar_read + 8 * k, kTcAggWarps);
    }
    *s_abort = 0;
    tc::fence_mbar_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(sb + kTcBar + 112, kTcCols);
    tc::tmem_relinquish();
  }
  tc::fence_proxy_async_smem();  // W (generic stores) is read by the tensor core
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const unsigned tmem = *s_tmem;

  if (warp < kTcAggWarps) {
    // ================================================================ aggregation
    const float u = a.P[kOffU + a.layer], cg = a.P[kOffC + a.layer];
    const int ch = lane & 7, group = lane & 24;       // this lane's chunk; the first lane of its node
    const int ln0 = warp * 4 + (lane >> 3);           // its node in a tile's first half
    // chunk ch of row ln0 of A's first region, and of a stage's rows
    unsigned char* const dst0 = sm + kTcA + ln0 * kTcRowB + ((ch ^ (ln0 & 7)) << 4);
    const unsigned src0 = sb + kTcStage + ln0 * kTcRowB + ch * 16;
    int stage = 0;
    unsigned phase = 0;
    bool ok = true;
    // One step: h and m of its nodes into A (beyond the last node whatever the stage
    // holds: a row of A reaches its own row of the result only, which is not stored).
    auto step = [&](int i, unsigned char* dst, bool wait_a, unsigned a_phase) {
      ok = tc::mbar_try_wait(bar_full + 8 * stage, phase) ||
           tc::mbar_wait(bar_full + 8 * stage, phase, kWaitCycles, s_abort);
      if (__any_sync(kFull, !ok)) return false;
      const unsigned st = src0 + stage * kTcStageB;
      const float e = ch < 6 ? lds_f32(sb + kTcStage + stage * kTcStageB + kTcEfOff + ln0 * 24 + ch * 4)
                             : __int_as_float(0x7fc00000);
      const unsigned all = __ballot_sync(kFull, e == e);
      uint4 w[6];
      const uint4 own = lds128(st + kTcXOff + kTcRowB);
      if (all == 0x3f3f3f3fu) {  // four nodes with all six neighbours
        w[0] = lds128(st + kTcZmOff);
        w[1] = lds128(st + kTcYmOff);
        w[2] = lds128(st + kTcXOff);
        w[3] = lds128(st + kTcXOff + 2 * kTcRowB);
        w[4] = lds128(st + kTcYpOff);
        w[5] = lds128(st + kTcZpOff);
      } else {
        const unsigned there = all >> group;
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        w[0] = there & 1 ? lds128(st + kTcZmOff) : zero;
        w[1] = there & 2 ? lds128(st + kTcYmOff) : zero;
        w[2] = there & 4 ? lds128(st + kTcXOff) : zero;
        w[3] = there & 8 ? lds128(st + kTcXOff + 2 * kTcRowB) : zero;
        w[4] = there & 16 ? lds128(st + kTcYpOff) : zero;
        w[5] = there & 32 ? lds128(st + kTcZpOff) : zero;
      }
      const float gate = e == e ? bf16r(sigmoidf(fmaf(u, e, cg))) : 0.f;
      f32x2 acc[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
      for (int d = 0; d < 6; ++d) {
        const float g = __shfl_sync(kFull, gate, group + d);
        const f32x2 g2 = make_f32x2(g, g);
        fma_f32x2(acc[0], g2, unpack_f32x2(w[d].x));
        fma_f32x2(acc[1], g2, unpack_f32x2(w[d].y));
        fma_f32x2(acc[2], g2, unpack_f32x2(w[d].z));
        fma_f32x2(acc[3], g2, unpack_f32x2(w[d].w));
      }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar_read + 8 * stage);
      if (++stage == kTcStages) {
        stage = 0;
        phase ^= 1u;
      }
      const uint4 m = make_uint4(pack_f32x2(acc[0]), pack_f32x2(acc[1]), pack_f32x2(acc[2]), pack_f32x2(acc[3]));
      if (wait_a) {  // this A buffer is free once the tensor core has read the tile before the last
        const unsigned bar = bar_aempty + 8 * ((i >> 1) & 1);
        ok = tc::mbar_try_wait(bar, a_phase) || tc::mbar_wait(bar, a_phase, kWaitCycles, s_abort);
        if (__any_sync(kFull, !ok)) return false;
      }
      *reinterpret_cast<uint4*>(dst) = own;
      *reinterpret_cast<uint4*>(dst + kTcARegion) = m;
      if (a.m_out) {
        const long long node = tile_base(i >> 1) + (i & 1) * kTcHalf + ln0;
        if (node < n) reinterpret_cast<uint4*>(a.m_out + node * kH)[ch] = m;
      }
      return true;
    };
    for (int c = 0; c < count; ++c) {
      unsigned char* const dst = dst0 + (c & 1) * kTcABuf;
      if (!step(2 * c, dst, c >= 2, (unsigned)((c >> 1) - 1) & 1u) ||
          !step(2 * c + 1, dst + kTcHalf * kTcRowB, false, 0u)) {
        give_up();
        break;
      }
      tc::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar_afull + 8 * (c & 1));
    }
  } else if (warp < kTcAggWarps + kTcEpiWarps) {
    // ================================================================ epilogue
    const int q = warp & 3;  // the tensor-memory lane quarter this warp may read
    unsigned char* out = sm + kTcOut + q * kTcOutB;
    for (int c = 0; c < count; ++c) {
      const int bsel = c & 1;
      const long long base = tile_base(c) + 32 * q, gi = base + lane;
      const bool ok = tc::mbar_wait(bar_accf + 8 * bsel, (unsigned)(c >> 1) & 1u, kWaitCycles, s_abort);
      if (__any_sync(kFull, !ok)) {
        give_up();
        break;
      }
      tc::fence_after_sync();
      const unsigned ta = tmem + ((unsigned)(32 * q) << 16) + bsel * kH;
      float y = 0.f;
#pragma unroll
      for (int h = 0; h < 2; ++h) {  // 32 columns at a time
        float v[32];
        tc::tmem_ld32(ta + 32 * h, v);
        if (h == 1) {
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(bar_acce + 8 * bsel);  // the accumulator is read
        }
        // bias, BF16, relu (after the rounding: the same values)
        unsigned o[16];
#pragma unroll
        for (int j4 = 0; j4 < 8; ++j4) {
          const ulonglong2 bb = reinterpret_cast<const ulonglong2*>(s_bias)[8 * h + j4];
          o[2 * j4] = relu_bf16x2(pack_f32x2(add_f32x2(make_f32x2(v[4 * j4], v[4 * j4 + 1]), bb.x)));
          o[2 * j4 + 1] = relu_bf16x2(pack_f32x2(add_f32x2(make_f32x2(v[4 * j4 + 2], v[4 * j4 + 3]), bb.y)));
          if constexpr (LAST) {
            const float4 ww = reinterpret_cast<const float4*>(s_wd)[8 * h + j4];
            const float2 x = unpack_bf16(o[2 * j4]), z = unpack_bf16(o[2 * j4 + 1]);
            y = fmaf(ww.x, x.x, y);
            y = fmaf(ww.y, x.y, y);
            y = fmaf(ww.z, z.x, y);
            y = fmaf(ww.w, z.y, y);
          }
        }
        if (a.h_out) {  // half rows: chunk c8 of row r at c8 ^ (r / 2 & 3)
#pragma unroll
          for (int c8 = 0; c8 < 4; ++c8)
            *reinterpret_cast<uint4*>(out + lane * (kTcRowB / 2) + ((c8 ^ (lane >> 1 & 3)) << 4)) =
                make_uint4(o[4 * c8], o[4 * c8 + 1], o[4 * c8 + 2], o[4 * c8 + 3]);
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 4; ++k) {  // eight half rows at a time
            const int r = 8 * k + (lane >> 2), c8 = lane & 3;
            const uint4 t = *reinterpret_cast<const uint4*>(out + r * (kTcRowB / 2) + ((c8 ^ (r >> 1 & 3)) << 4));
            if (base + r < n) reinterpret_cast<uint4*>(a.h_out + (base + r) * kH)[4 * h + c8] = t;
          }
          __syncwarp();  // the staging is refilled
        }
      }
      if constexpr (LAST) {
        if (gi < n) {
          const double s2 = a.s2[0], is = a.s2[1];
          const float bd = a.P[kOffBd], ws = a.P[kOffWs];
          a.z[gi] = s2 * (double)(y + bd + ws * (float)(a.xr[gi] * is)) * (double)a.isd[gi];
        }
      }
    }
  } else if (warp == kTcAggWarps + kTcEpiWarps) {
    // ================================================================ MMA
    if (lane == 0) {
      int last = -1;  // the last tile whose MMA was issued, for the drain after a failure
      bool ok = true;
      for (int c = 0; c < count; ++c) {
        const int bsel = c & 1;
        const unsigned phase = (unsigned)(c >> 1) & 1u;
        // A of tile c written; the epilogue has read this accumulator's previous tile
        ok = tc::mbar_wait(bar_afull + 8 * bsel, phase, kWaitCycles, s_abort) &&
             (c < 2 || tc::mbar_wait(bar_acce + 8 * bsel, phase ^ 1u, kWaitCycles, s_abort));
        if (!ok) {
          give_up();
          break;
        }
        tc::fence_after_sync();
        constexpr uint32_t idesc = tc::idesc_bf16_f32(kTcTile, kH);
        const unsigned abuf = sb + kTcA + bsel * kTcABuf;
#pragma unroll
        for (int k = 0; k < kIn / 16; ++k) {
          const unsigned aoff = (k >> 2) * kTcARegion + (k & 3) * 32, boff = (k >> 2) * (kH * kTcRowB) + (k & 3) * 32;
          tc::mma_bf16_ss(tmem + bsel * kH, tc::sdesc_sw128(abuf + aoff), tc::sdesc_sw128(sb + kTcW + boff), idesc,
                          k > 0);
        }
        tc::mma_commit(bar_aempty + 8 * bsel);
        tc::mma_commit(bar_accf + 8 * bsel);
        last = c;
      }
      if (!ok && last >= 0)  // drain: no MMA of this CTA's may still run at exit
        tc::mbar_wait(bar_aempty + 8 * (last & 1), (unsigned)(last >> 1) & 1u, kWaitCycles, nullptr);
    }
  } else if (lane == 0) {
    // ================================================================ input copies
    const long long sy = (long long)ga.nx * kH, sz = (long long)ga.sxy * kH;
    // the inputs of step i (half i & 1 of tile i / 2) into its stage
    auto issue = [&](int i, int stage) {
      const long long b = tile_base(i >> 1) + (i & 1) * kTcHalf;
      const unsigned st = sb + kTcStage + stage * kTcStageB, bar = bar_full + 8 * stage;
      if (b >= ga.sxy && b + ga.sxy + kTcHalf <= n) {  // every row of every block exists (sxy >= nx >= 1)
        tc::mbar_expect_tx(bar, kTcStageB);
        const bf16* h = a.h_in + b * kH;
        tc::bulk_g2s(st + kTcZmOff, h - sz, kTcBlockB, bar);
        tc::bulk_g2s(st + kTcYmOff, h - sy, kTcBlockB, bar);
        tc::bulk_g2s(st + kTcXOff, h - kH, kTcBlockB + 2 * kTcRowB, bar);
        tc::bulk_g2s(st + kTcYpOff, h + sy, kTcBlockB, bar);
        tc::bulk_g2s(st + kTcZpOff, h + sz, kTcBlockB, bar);
      } else {
        const long long first[5] = {b - 1, b - ga.nx, b + ga.nx, b - ga.sxy, b + ga.sxy};
        const unsigned dst[5] = {kTcXOff, kTcYmOff, kTcYpOff, kTcZmOff, kTcZpOff};
        long long lo[5];
        int rows[5];
        unsigned bytes = kTcEfBytes;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
          const long long end = first[k] + (k == 0 ? kTcHalf + 2 : kTcHalf);
          lo[k] = first[k] < 0 ? 0 : first[k];
          rows[k] = (int)((end > n ? n : end) - lo[k]);
          if (rows[k] > 0) bytes += (unsigned)rows[k] * kTcRowB;
        }
        tc::mbar_expect_tx(bar, bytes);
#pragma unroll
        for (int k = 0; k < 5; ++k)
          if (rows[k] > 0)
            tc::bulk_g2s(st + dst[k] + (unsigned)(lo[k] - first[k]) * kTcRowB, a.h_in + lo[k] * kH,
                         (unsigned)rows[k] * kTcRowB, bar);
      }
      tc::bulk_g2s(st + kTcEfOff, ga.dir_ef + b * 6, kTcEfBytes, bar);
    };
    int i = 0, stage = 0;
    unsigned phase = 0;
    for (; i < 2 * count; ++i) {
      if (i >= kTcStages && !tc::mbar_wait(bar_read + 8 * stage, phase ^ 1u, kWaitCycles, s_abort)) {
        give_up();
        break;
      }
      issue(i, stage);
      if (++stage == kTcStages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    // the last copies have landed, whether or not a failure left them unread
    for (int k = i - 1; k >= 0 && k >= i - kTcStages; --k)
      tc::mbar_wait(bar_full + 8 * (k % kTcStages), (unsigned)(k / kTcStages) & 1u, kWaitCycles, nullptr);
  }
  __syncwarp();
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, kTcCols);
  }
}

// h1 = relu(W0 x0 + b0), x0 = [xr / s, log(a_ii)/10]: 8 lanes per node, 8 features a lane.
__global__ void __launch_bounds__(kThreads) k_gnn_encode(int n, const float* __restrict__ xr,
                                                         const float* __restrict__ logd10, const double* __restrict__ s2,
                                                         const float* __restrict__ P, bf16* __restrict__ h1) {
  const int sub = threadIdx.x & 7;
  const float inv_s = (float)s2[1];
  float w0a[8], w0b[8], b0v[8];
#pragma unroll
  for (int f = 0; f < 8; ++f) {
    w0a[f] = P[kOffW0 + 2 * (8 * sub + f)];
    w0b[f] = P[kOffW0 + 2 * (8 * sub + f) + 1];
    b0v[f] = P[kOffB0 + 8 * sub + f];
  }
  for (long long v = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 3; v < n;
       v += ((long long)gridDim.x * blockDim.x) >> 3) {
    const float x = xr[v] * inv_s, l = logd10[v];
    float f8[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) f8[q] = fmaxf(fmaf(w0a[q], x, fmaf(w0b[q], l, b0v[q])), 0.f);
    reinterpret_cast<uint4*>(h1 + (size_t)v * kH)[sub] = pack8(f8);
  }
}

// FP32 master weights -> BF16 copies of the dense layers' W.
__global__ void k_gnn_wcopy(const float* __restrict__ P, bf16* __restrict__ Wb) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < kLayers * kH * kIn; t += gridDim.x * blockDim.x)
    Wb[t] = __float2bfloat16_rn(P[kOffW + t]);
}

// ------------------------------------------------------------------ backward
// Warp-per-node kernels leave per-block partial sums in part[block][width];
// k_gnn_reduce_partials adds them in block order (deterministic).
constexpr int kWarpsPerBlock = 8;

// dy_i = dz_i s / sqrt(a_ii) ; dh5_i = dy_i wd ; partials of grad wd (64), bd and ws.
__global__ void __launch_bounds__(256) k_gnn_decode_bwd(int n, const double* __restrict__ dz, const double* __restrict__ s2,
                                                        const float* __restrict__ isd, const float* __restrict__ xr,
                                                        const bf16* __restrict__ h5, const float* __restrict__ P,
                                                        float* __restrict__ dh, float* __restrict__ part) {
  __shared__ float s_acc[kWarpsPerBlock][kH + 2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double s = s2[0];
  const float is = (float)s2[1];
  const unsigned* hv = reinterpret_cast<const unsigned*>(h5);
  const float w0 = P[kOffWd + 2 * lane], w1 = P[kOffWd + 2 * lane + 1];
  float g0 = 0.f, g1 = 0.f, gb = 0.f, gs = 0.f;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
    const float dy = (float)(dz[i] * s * (double)isd[i]);
    const float2 x = unpack_bf16(hv[(size_t)i * (kH / 2) + lane]);
    g0 = fmaf(dy, x.x, g0);
    g1 = fmaf(dy, x.y, g1);
    gb += dy;
    gs = fmaf(dy, xr[i] * is, gs);
    reinterpret_cast<float2*>(dh)[(size_t)i * (kH / 2) + lane] = make_float2(dy * w0, dy * w1);
  }
  s_acc[warp][2 * lane] = g0;
  s_acc[warp][2 * lane + 1] = g1;
  if (lane == 0) {
    s_acc[warp][kH] = gb;
    s_acc[warp][kH + 1] = gs;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < kH + 2; k += blockDim.x) {
    float v = 0.f;
    for (int w = 0; w < kWarpsPerBlock; ++w) v += s_acc[w][k];
    part[(size_t)blockIdx.x * (kH + 2) + k] = v;
  }
}

// [dh_in ; dm] = dpre W on tensor cores, dpre = dh (.) (h_out > 0) rounded to
// BF16; W^T (128 x 64) staged in shared memory with padded rows.
constexpr int kWTStride = kH + 8;
__global__ void __launch_bounds__(256) k_gnn_dense_bwd(int n, const float* __restrict__ dh, const bf16* __restrict__ hout,
                                                       const bf16* __restrict__ W, float* __restrict__ dh_in,
                                                       float* __restrict__ dm) {
  __shared__ __align__(16) bf16 WT[kIn * kWTStride];
  for (int t = threadIdx.x; t < kH * kIn; t += blockDim.x) {
    const int o = t / kIn, k = t % kIn;
    WT[k * kWTStride + o] = W[t];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const unsigned* hv = reinterpret_cast<const unsigned*>(hout);
  auto dpre2 = [&](int row, int col) -> unsigned {  // BF16 pair of dpre[row][col], [col+1]
    const float2 d = reinterpret_cast<const float2*>(dh)[((size_t)row * kH + col) >> 1];
    const float2 hv2 = unpack_bf16(hv[((size_t)row * kH + col) >> 1]);
    return pack_bf16(hv2.x > 0.f ? d.x : 0.f, hv2.y > 0.f ? d.y : 0.f);
  };
  for (int tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; tile * 16 < n; tile += warps) {
    const int r0 = tile * 16 + g, r1 = r0 + 8;
    const bool ok0 = r0 < n, ok1 = r1 < n;
    float acc[16][4];
#pragma unroll
    for (int nb = 0; nb < 16; ++nb) acc[nb][0] = acc[nb][1] = acc[nb][2] = acc[nb][3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const int col = ks * 16 + 2 * t;
      unsigned a[4];
      a[0] = ok0 ? dpre2(r0, col) : 0u;
      a[1] = ok1 ? dpre2(r1, col) : 0u;
      a[2] = ok0 ? dpre2(r0, col + 8) : 0u;
      a[3] = ok1 ? dpre2(r1, col + 8) : 0u;
#pragma unroll
      for (int nb = 0; nb < 16; ++nb) {
        const bf16* wrow = WT + (nb * 8 + g) * kWTStride;
        const unsigned b0 = *reinterpret_cast<const unsigned*>(wrow + col);
        const unsigned b1 = *reinterpret_cast<const unsigned*>(wrow + col + 8);
        mma_bf16(acc[nb], a, b0, b1);
      }
    }
#pragma unroll
    for (int nb = 0; nb < 16; ++nb) {
      const int c = nb * 8 + 2 * t;
      float* dst = c < kH ? dh_in : dm;
      const int cc = c & (kH - 1);
      if (ok0) reinterpret_cast<float2*>(dst)[((size_t)r0 * kH + cc) >> 1] = make_float2(acc[nb][0], acc[nb][1]);
      if (ok1) reinterpret_cast<float2*>(dst)[((size_t)r1 * kH + cc) >> 1] = make_float2(acc[nb][2], acc[nb][3]);
    }
  }
}

// dh_j += sum_{i neighbour of j} g_ij dm_i (in place on dh_in) and the gate
// gradients of row j's edges: dg = dm_j . h_i, ds = dg g (1-g), du += ds e, dc += ds.
__global__ void __launch_bounds__(256) k_gnn_agg_bwd(int n, const int* __restrict__ rp, const int* __restrict__ ci,
                                                     const float* __restrict__ efeat, const int* __restrict__ tidx,
                                                     const float* __restrict__ P, int layer, const bf16* __restrict__ h,
                                                     const float* __restrict__ dm, float* dh, float* __restrict__ part) {
  __shared__ float s_acc[kWarpsPerBlock][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float u = P[kOffU + layer], c = P[kOffC + layer];
  const unsigned* hv = reinterpret_cast<const unsigned*>(h);
  const float2* dm2 = reinterpret_cast<const float2*>(dm);
  float du = 0.f, dc = 0.f;
  for (int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; j < n; j += (gridDim.x * blockDim.x) >> 5) {
    float2 acc = reinterpret_cast<float2*>(dh)[(size_t)j * (kH / 2) + lane];
    const float2 dmj = dm2[(size_t)j * (kH / 2) + lane];
    for (int k = rp[j]; k < rp[j + 1]; ++k) {
      const int i = ci[k];
      if (i == j) continue;
      const float gt = sigmoidf(fmaf(u, efeat[tidx[k]], c));  // g of entry (i, j)
      const float2 dmi = dm2[(size_t)i * (kH / 2) + lane];
      acc.x = fmaf(gt, dmi.x, acc.x);
      acc.y = fmaf(gt, dmi.y, acc.y);
      const float2 hi = unpack_bf16(hv[(size_t)i * (kH / 2) + lane]);
      float dg = fmaf(dmj.x, hi.x, dmj.y * hi.y);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) dg += __shfl_xor_sync(0xffffffffu, dg, off);
      const float e = efeat[k];
      const float gk = sigmoidf(fmaf(u, e, c));
      const float ds = dg * gk * (1.f - gk);
      du = fmaf(ds, e, du);
      dc += ds;
    }
    reinterpret_cast<float2*>(dh)[(size_t)j * (kH / 2) + lane] = acc;
  }
  if (lane == 0) {
    s_acc[warp][0] = du;
    s_acc[warp][1] = dc;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    float s = 0.f;
    for (int w = 0; w < kWarpsPerBlock; ++w) s += s_acc[w][threadIdx.x];
    part[(size_t)blockIdx.x * 2 + threadIdx.x] = s;
  }
}

// Partials of grad W (64 x 128) and grad b (64): sum_i dpre_i [h_i ; m_i]^T in
// FP32, node by node in order (a block's nodes are consecutive).  32 nodes at a
// time are staged in shared memory as floats, the next 32 already on their way
// into registers (five 16-byte loads a thread); a thread owns 4 outputs x 8
// inputs, so a node costs it three 16-byte shared loads and 32 multiply-adds.
// Bound by the FP32 multiply-adds (60 us of them at 64^3 nodes).  Measured at 64^3
// on B200: 1627 us with 1 x 32 tiles a thread, single-word shared loads and a
// four-way bank conflict on each; 120 us now, the same sums in the same order.
__global__ void __launch_bounds__(256) k_gnn_wgrad(int n, const float* __restrict__ dh, const bf16* __restrict__ hout,
                                                   const bf16* __restrict__ h, const bf16* __restrict__ m,
                                                   float* __restrict__ part) {
  constexpr int kRows = 32;
  __shared__ __align__(16) float s_dp[kRows][kH];
  __shared__ __align__(16) float s_in[kRows][kIn];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;  // inputs 4 tx.. and 64 + 4 tx.., outputs 4 ty..
  const int lr = threadIdx.x >> 3, lc = (threadIdx.x & 7) * 8;  // staged: row, first of 8 columns
  float acc[4][8], accb[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    accb[p] = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[p][q] = 0.f;
  }
  const int per = (n + gridDim.x - 1) / gridDim.x;
  const int lo = blockIdx.x * per, hi = min(n, lo + per);
  float4 d0, d1;
  uint4 vo, vh, vm;
  auto load = [&](int base) {
    const int i = base + lr;
    d0 = d1 = make_float4(0.f, 0.f, 0.f, 0.f);
    vo = vh = vm = make_uint4(0u, 0u, 0u, 0u);
    if (i < hi) {
      const size_t at = (size_t)i * kH + lc;
      d0 = __ldg(reinterpret_cast<const float4*>(dh + at));
      d1 = __ldg(reinterpret_cast<const float4*>(dh + at + 4));
      vo = __ldg(reinterpret_cast<const uint4*>(hout + at));
      vh = __ldg(reinterpret_cast<const uint4*>(h + at));
      vm = __ldg(reinterpret_cast<const uint4*>(m + at));
    }
  };
  auto put = [](float* to, const uint4& v) {
    const float2 a = unpack_bf16(v.x), b = unpack_bf16(v.y), c = unpack_bf16(v.z), d = unpack_bf16(v.w);
    *reinterpret_cast<float4*>(to) = make_float4(a.x, a.y, b.x, b.y);
    *reinterpret_cast<float4*>(to + 4) = make_float4(c.x, c.y, d.x, d.y);
  };
  if (lo < hi) load(lo);
  for (int base = lo; base < hi; base += kRows) {
    __syncthreads();
    {
      const float2 a = unpack_bf16(vo.x), b = unpack_bf16(vo.y), c = unpack_bf16(vo.z), d = unpack_bf16(vo.w);
      *reinterpret_cast<float4*>(&s_dp[lr][lc]) = make_float4(a.x > 0.f ? d0.x : 0.f, a.y > 0.f ? d0.y : 0.f,
                                                             b.x > 0.f ? d0.z : 0.f, b.y > 0.f ? d0.w : 0.f);
      *reinterpret_cast<float4*>(&s_dp[lr][lc + 4]) = make_float4(c.x > 0.f ? d1.x : 0.f, c.y > 0.f ? d1.y : 0.f,
                                                                 d.x > 0.f ? d1.z : 0.f, d.y > 0.f ? d1.w : 0.f);
      put(&s_in[lr][lc], vh);
      put(&s_in[lr][kH + lc], vm);
    }
    __syncthreads();
    if (base + kRows < hi) load(base + kRows);
    const int rows = min(kRows, hi - base);
#pragma unroll 4
    for (int r = 0; r < rows; ++r) {
      const float4 dv = *reinterpret_cast<const float4*>(&s_dp[r][4 * ty]);
      const float4 x0 = *reinterpret_cast<const float4*>(&s_in[r][4 * tx]);
      const float4 x1 = *reinterpret_cast<const float4*>(&s_in[r][kH + 4 * tx]);
      const float d[4] = {dv.x, dv.y, dv.z, dv.w};
      const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
      for (int p = 0; p < 4; ++p) {
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[p][q] = fmaf(d[p], x[q], acc[p][q]);
        if (tx == 0) accb[p] += d[p];
      }
    }
  }
  float* out = part + (size_t)blockIdx.x * (kH * kIn + kH);
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    float* row = out + (4 * ty + p) * kIn;
    *reinterpret_cast<float4*>(row + 4 * tx) = make_float4(acc[p][0], acc[p][1], acc[p][2], acc[p][3]);
    *reinterpret_cast<float4*>(row + kH + 4 * tx) = make_float4(acc[p][4], acc[p][5], acc[p][6], acc[p][7]);
    if (tx == 0) out[kH * kIn + 4 * ty + p] = accb[p];
  }
}

// Partials of grad W0 (64 x 2) and b0: dpre0 = dh1 (.) (h1 > 0), x0 recomputed.
__global__ void __launch_bounds__(256) k_gnn_encode_bwd(int n, const float* __restrict__ xr, const double* __restrict__ s2,
                                                        const float* __restrict__ logd10, const bf16* __restrict__ h1,
                                                        const float* __restrict__ dh, float* __restrict__ part) {
  __shared__ float s_acc[kWarpsPerBlock][3 * kH];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float inv_s = (float)s2[1];
  const unsigned* hv = reinterpret_cast<const unsigned*>(h1);
  float a[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // (W0[o][0], W0[o][1], b0[o]) for o = 2 lane, 2 lane + 1
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
    const float x0 = xr[i] * inv_s, x1 = logd10[i];
    const float2 hh = unpack_bf16(hv[(size_t)i * (kH / 2) + lane]);
    const float2 d = reinterpret_cast<const float2*>(dh)[(size_t)i * (kH / 2) + lane];
    const float d0 = hh.x > 0.f ? d.x : 0.f, d1 = hh.y > 0.f ? d.y : 0.f;
    a[0] = fmaf(d0, x0, a[0]);
    a[1] = fmaf(d0, x1, a[1]);
    a[2] += d0;
    a[3] = fmaf(d1, x0, a[3]);
    a[4] = fmaf(d1, x1, a[4]);
    a[5] += d1;
  }
  // layout: W0 (o, 0..1) at 2o, 2o+1 ; b0 at 128 + o
  s_acc[warp][4 * lane + 0] = a[0];
  s_acc[warp][4 * lane + 1] = a[1];
  s_acc[warp][4 * lane + 2] = a[3];
  s_acc[warp][4 * lane + 3] = a[4];
  s_acc[warp][2 * kH + 2 * lane] = a[2];
  s_acc[warp][2 * kH + 2 * lane + 1] = a[5];
  __syncthreads();
  for (int k = threadIdx.x; k < 3 * kH; k += blockDim.x) {
    float s = 0.f;
    for (int w = 0; w < kWarpsPerBlock; ++w) s += s_acc[w][k];
    part[(size_t)blockIdx.x * (3 * kH) + k] = s;
  }
}

// out[k] = sum_b part[b][k], block order.  A block sums 32 outputs: all its
// threads stage 128 blocks' partials at a time in shared memory, one warp adds them in
// order.  (One thread an output fetching for itself waited on L2 for every few
// of its up to ~1,200 partials: 47 us a call against 9 us, the same sums.)
__global__ void __launch_bounds__(256) k_gnn_reduce_partials(int nb, int width, const float* __restrict__ part,
                                                             float* __restrict__ out) {
  constexpr int kStage = 128;
  __shared__ float s_part[2][kStage][32];
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + lane;
  float v[kStage / 8];
  auto load = [&](int base) {
#pragma unroll
    for (int u = 0; u < kStage / 8; ++u) {
      const int b = base + row + 8 * u;
      v[u] = b < nb && k < width ? __ldg(part + (size_t)b * width + k) : 0.f;
    }
  };
  float s = 0.f;
  load(0);
  for (int base = 0, buf = 0; base < nb; base += kStage, buf ^= 1) {
#pragma unroll
    for (int u = 0; u < kStage / 8; ++u) s_part[buf][row + 8 * u][lane] = v[u];
    __syncthreads();
    if (base + kStage < nb) load(base + kStage);
    if (row == 0) {
      const int m = min(kStage, nb - base);
#pragma unroll 16
      for (int b = 0; b < m; ++b) s += s_part[buf][b][lane];
    }
  }
  if (row == 0 && k < width) out[k] = s;
}

// Adam on the FP32 master weights.
__global__ void k_gnn_adam(int np, float* __restrict__ P, const float* __restrict__ g, float* __restrict__ m,
                           float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < np; k += gridDim.x * blockDim.x) {
    const float gk = g[k];
    const float mk = fmaf(b1, m[k], (1.f - b1) * gk);
    const float vk = fmaf(b2, v[k], (1.f - b2) * gk * gk);
    m[k] = mk;
    v[k] = vk;
    P[k] -= lr * (mk / c1) / (sqrtf(vk / c2) + eps);
  }
}

// ------------------------------------------------------------------ flexible CG
// Notay's FCG(m): p_k = z_k - sum_i (z_k . q_i / d_i) p_i over the last m
// directions (q_i = A p_i, d_i = p_i . q_i), alpha_k = p_k . r_k / d_k.  The
// scalars stay on the device; one iteration needs a single host read (of rr,
// for the stop and fallback decisions).
constexpr int kMaxTrunc = 16;
struct FcgScalars {
  double rr;                // r . r after the update
  double alpha;
  double d[kMaxTrunc];      // p_i . A p_i, by window slot
  double coef[kMaxTrunc];   // z . A p_i / d_i of the current step
  int breakdown;            // p . A p == 0
};
struct Window {
  const double* v[kMaxTrunc];
};

// coef_k = z . q_k / d_k for the window's slots 0..count-1 <= C.  A thread's next
// element is loaded beside the current one (its sums take them in order).  With C
// the window's size rounded up to 4, 8 or 16: sixteen sums whatever the window took
// 80 us at 1.7 million rows and a window of 8, 30 now (and k_fcg_dir 36, 21).
template <int C>
__global__ void __launch_bounds__(kThreads) k_fcg_zq(int n, const double* __restrict__ z, const Window q, int count,
                                                     FcgScalars* sc, double* partials, unsigned* counter,
                                                     double* red_out) {
  double acc[C];
#pragma unroll
  for (int k = 0; k < C; ++k) acc[k] = 0.0;
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += 2 * stride) {
    const bool two = i < n - stride;
    const int j = two ? i + stride : i;
    const double zi = z[i], zj = z[j];
    double a[C], b[C];
#pragma unroll
    for (int k = 0; k < C; ++k) {
      a[k] = k < count ? q.v[k][i] : 0.0;
      b[k] = k < count ? q.v[k][j] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < C; ++k) {
      if (k < count) acc[k] = fma(zi, a[k], acc[k]);
      if (k < count && two) acc[k] = fma(zj, b[k], acc[k]);
    }
  }
  if (grid_reduce<C>(acc, partials, counter, red_out)) {
    for (int k = 0; k < count; ++k) sc->coef[k] = sc->d[k] != 0.0 ? red_out[k] / sc->d[k] : 0.0;
  }
}

// p = z - sum_k coef_k p_k (p may be one of the window's vectors: element-wise in
// place; two elements a thread with 16-byte accesses, every window vector starts on
// a 16-byte boundary when n is even).
template <int C>
__global__ void k_fcg_dir(int n, const double* __restrict__ z, const Window pw, int count, const FcgScalars* sc,
                          double* p) {
  double coef[C];
#pragma unroll
  for (int k = 0; k < C; ++k) coef[k] = k < count ? sc->coef[k] : 0.0;
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  const int pairs = n % 2 == 0 ? n / 2 : 0;
  for (int i = t0; i < pairs; i += stride) {
    double2 v = reinterpret_cast<const double2*>(z)[i];
    double2 w[C];
#pragma unroll
    for (int k = 0; k < C; ++k)
      if (k < count) w[k] = reinterpret_cast<const double2*>(pw.v[k])[i];
#pragma unroll
    for (int k = 0; k < C; ++k)
      if (k < count) {
        v.x = fma(-coef[k], w[k].x, v.x);
        v.y = fma(-coef[k], w[k].y, v.y);
      }
    reinterpret_cast<double2*>(p)[i] = v;
  }
  for (int i = 2 * pairs + t0; i < n; i += stride) {
    double v = z[i];
#pragma unroll
    for (int k = 0; k < C; ++k)
      if (k < count) v = fma(-coef[k], pw.v[k][i], v);
    p[i] = v;
  }
}

// d_slot = p . q, alpha = p . r / d_slot (breakdown if d_slot == 0)
__global__ void __launch_bounds__(kThreads) k_fcg_pq(int n, const double* __restrict__ p, const double* __restrict__ q,
                                                     const double* __restrict__ r, int slot, FcgScalars* sc,
                                                     double* partials, unsigned* counter, double* red_out) {
  double acc[2] = {0.0, 0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double pi = p[i];
    acc[0] = fma(pi, q[i], acc[0]);
    acc[1] = fma(pi, r[i], acc[1]);
  }
  if (grid_reduce<2>(acc, partials, counter, red_out)) {
    const double d = red_out[0];
    sc->d[slot] = d;
    sc->alpha = d != 0.0 ? red_out[1] / d : 0.0;
    if (d == 0.0) sc->breakdown = 1;
  }
}

// x += alpha p; r -= alpha q; rr = r . r
__global__ void __launch_bounds__(kThreads) k_fcg_update(int n, const double* __restrict__ p, const double* __restrict__ q,
                                                         double* __restrict__ x, double* __restrict__ r, FcgScalars* sc,
                                                         double* partials, unsigned* counter, double* red_out) {
  const double alpha = sc->alpha;
  double acc[1] = {0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    x[i] = fma(alpha, p[i], x[i]);
    const double rv = fma(-alpha, q[i], r[i]);
    r[i] = rv;
    acc[0] = fma(rv, rv, acc[0]);
  }
  if (grid_reduce<1>(acc, partials, counter, red_out)) sc->rr = red_out[0];
}

}  // namespace
}  // namespace ab2

using namespace ab2;

struct ab2_gnn {
  ab2_context* ctx = nullptr;
  float* d_P = nullptr;      // FP32 master parameters (flat)
  float* d_grad = nullptr;
  float* d_am = nullptr;     // Adam moments
  float* d_av = nullptr;
  bf16* d_Wb = nullptr;      // BF16 copies of the dense layers' W
  int step = 0;
  // binding to a matrix
  const ab2_matrix* A = nullptr;
  int n = 0;
  float *d_isd = nullptr, *d_logd10 = nullptr, *d_efeat = nullptr;
  int* d_tidx = nullptr;
  int nbw = 0;               // neighbour table: slots per node
  int* d_nb_idx = nullptr;
  float* d_nb_ef = nullptr;
  bf16* d_h = nullptr;       // h1..h5, n x 64 each
  bf16* d_m = nullptr;       // m1..m4
  float* d_xr = nullptr;     // r_i / sqrt(a_ii) of the last forward
  double* d_s2 = nullptr;    // its scale s and 1/s
  float *d_dh = nullptr, *d_dh2 = nullptr, *d_dm = nullptr;
  double *d_z = nullptr, *d_d = nullptr, *d_Ad = nullptr, *d_Ae = nullptr;
  float* d_part = nullptr;
  float* d_red = nullptr;    // reduced partials scratch (64 x 128 + 64)
  long long part_cap = 0;
  // the layer kernel: AB2_GNN_LAYER_* requested, and whether the bound
  // matrix's graph is a 3-D 7-point grid (then the grid layer's inputs)
  int layout = AB2_GNN_LAYER_AUTO;
  bool grid = false;
  int gnx = 0, gny = 0, gnz = 0;
  float* d_dir_ef = nullptr;  // [ceil(n/128) 128][6] edge features by direction
  int* d_err = nullptr;       // set by the grid layer when a bounded wait gives up
};

namespace ab2 {
namespace {

int warp_grid(ab2_context* ctx, int n) {
  return std::max(1, std::min((n + kWarpsPerBlock - 1) / kWarpsPerBlock, ctx->num_sms * 8));
}
int tile_grid(ab2_context* ctx, int n) { return std::max(1, std::min((n + 127) / 128, ctx->num_sms * 4)); }
// Two blocks an SM from ~150,000 nodes on (64^3 nodes: 120 us a layer, 157 us with one an SM).
int wgrad_grid(ab2_context* ctx, int n) { return std::max(1, std::min((n + 511) / 512, ctx->num_sms * 2)); }

bf16* hbuf(ab2_gnn* G, int l) { return G->d_h + (size_t)l * G->n * kH; }
bf16* mbuf(ab2_gnn* G, int l) { return G->d_m + (size_t)l * G->n * kH; }

void release_binding(ab2_gnn* G) {
  ab2_context* ctx = G->ctx;
  for (void* p : {(void*)G->d_isd, (void*)G->d_logd10, (void*)G->d_efeat, (void*)G->d_tidx, (void*)G->d_h,
                  (void*)G->d_m, (void*)G->d_xr, (void*)G->d_s2, (void*)G->d_dh, (void*)G->d_dh2, (void*)G->d_dm,
                  (void*)G->d_z, (void*)G->d_d, (void*)G->d_Ad, (void*)G->d_Ae, (void*)G->d_part, (void*)G->d_red,
                  (void*)G->d_nb_idx, (void*)G->d_nb_ef, (void*)G->d_dir_ef, (void*)G->d_err})
    dev_free(ctx, p);
  G->d_dir_ef = nullptr;
  G->d_err = nullptr;
  G->grid = false;
  G->gnx = G->gny = G->gnz = 0;
  G->d_nb_idx = nullptr;
  G->d_nb_ef = nullptr;
  G->nbw = 0;
  G->d_isd = G->d_logd10 = G->d_efeat = G->d_xr = nullptr;
  G->d_tidx = nullptr;
  G->d_h = G->d_m = nullptr;
  G->d_s2 = nullptr;
  G->d_dh = G->d_dh2 = G->d_dm = nullptr;
  G->d_z = G->d_d = G->d_Ad = G->d_Ae = nullptr;
  G->d_part = G->d_red = nullptr;
  G->A = nullptr;
  G->n = 0;
}

template <bool LAST>
void launch_layer(ab2_context* ctx, const LayerArgs& la) {
  static thread_local int configured_device = -1, per_sm = 0, per_sm_nbw = -1;  // per device and table width
  if (configured_device != ctx->device) {
    AB2_CUDA(cudaFuncSetAttribute(k_gnn_layer<LAST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)layer_smem_bytes(kMaxNbw)));
    configured_device = ctx->device;
    per_sm_nbw = -1;
  }
  if (per_sm_nbw != la.nbw) {
    AB2_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gnn_layer<LAST>, kLayerWarps * 32,
                                                           layer_smem_bytes(la.nbw)));
    per_sm = std::max(per_sm, 1);
    per_sm_nbw = la.nbw;
  }
  const int ntiles = (la.n + 15) / 16;
  const int grid = std::max(1, std::min((ntiles + kLayerWarps - 1) / kLayerWarps, per_sm * ctx->num_sms));
  k_gnn_layer<LAST><<<grid, kLayerWarps * 32, layer_smem_bytes(la.nbw), ctx->stream>>>(la);
  check_launch(ctx, "gnn_layer");
}

template <bool LAST>
void launch_layer_grid(ab2_context* ctx, const GridLayerArgs& ga) {
  static thread_local int configured_device = -1;
  if (configured_device != ctx->device) {
    AB2_CUDA(cudaFuncSetAttribute(k_gnn_layer_grid<LAST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem));
    configured_device = ctx->device;
  }
  const int ntiles = (ga.a.n + kTcTile - 1) / kTcTile;
  const int grid = std::max(1, std::min(ntiles, ctx->num_sms));
  k_gnn_layer_grid<LAST><<<grid, kTcThreads, kTcSmem, ctx->stream>>>(ga);
  check_launch(ctx, "gnn_layer_grid");
}

bool use_grid_layer(const ab2_gnn* G) { return G->grid && G->layout != AB2_GNN_LAYER_GATHER; }

// A bounded wait of the grid layer gave up (its outputs are then garbage):
// AB2_ERR_TIMEOUT, the flag cleared for the next call.  Synchronises.
void check_grid_wait(ab2_gnn* G) {
  if (!G->d_err) return;
  ab2_context* ctx = G->ctx;
  int e = 0;
  AB2_CUDA(cudaMemcpyAsync(&e, G->d_err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  AB2_CUDA(cudaStreamSynchronize(ctx->stream));
  if (e) {
    AB2_CUDA(cudaMemsetAsync(G->d_err, 0, sizeof(int), ctx->stream));
    throw Error{AB2_ERR_TIMEOUT, "learned preconditioner: a bounded wait of the grid layer gave up"};
  }
}

// z = network(r) (FP64 in and out).  training: keep m1..m4 and h5 for the
// backward pass (h1..h4 are always written).
void gnn_forward(ab2_gnn* G, const double* r, double* z, bool training = false) {
  ab2_context* ctx = G->ctx;
  const int n = G->n;
  RedSlot red = red_slot(ctx, 5);
  k_gnn_scale<<<red_grid(ctx, n), kThreads, 0, ctx->stream>>>(n, r, G->d_isd, G->d_xr, red.partials, red.counter,
                                                             red.result, G->d_s2);
  check_launch(ctx, "gnn_scale");
  k_gnn_encode<<<grid_for((long long)n * 8), kThreads, 0, ctx->stream>>>(n, G->d_xr, G->d_logd10, G->d_s2, G->d_P,
                                                                         hbuf(G, 0));
  check_launch(ctx, "gnn_encode");
  for (int l = 0; l < kLayers; ++l) {
    LayerArgs la{};
    la.n = n;
    la.nbw = G->nbw;
    la.nb_idx = G->d_nb_idx;
    la.nb_ef = G->d_nb_ef;
    la.P = G->d_P;
    la.W = G->d_Wb + (size_t)l * kH * kIn;
    la.layer = l;
    la.h_in = hbuf(G, l);
    la.xr = G->d_xr;
    la.isd = G->d_isd;
    la.s2 = G->d_s2;
    la.m_out = training ? mbuf(G, l) : nullptr;
    la.h_out = (training || l + 1 < kLayers) ? hbuf(G, l + 1) : nullptr;
    la.z = l + 1 == kLayers ? z : nullptr;
    if (use_grid_layer(G)) {
      const GridLayerArgs ga{la, G->gnx, G->gnx * G->gny, G->d_dir_ef, G->d_err};
      if (l + 1 < kLayers) launch_layer_grid<false>(ctx, ga);
      else launch_layer_grid<true>(ctx, ga);
    } else if (l + 1 < kLayers) {
      launch_layer<false>(ctx, la);
    } else {
      launch_layer<true>(ctx, la);
    }
  }
}

void reduce_into(ab2_gnn* G, int nb, int width, float* out) {
  k_gnn_reduce_partials<<<(width + 31) / 32, 256, 0, G->ctx->stream>>>(nb, width, G->d_part, out);
  check_launch(G->ctx, "gnn_reduce");
}

// Loss (z-e)^T A (z-e) / e^T A e and its gradient into d_grad.
double gnn_loss_grad(ab2_gnn* G, const double* r, const double* e) {
  ab2_context* ctx = G->ctx;
  const ab2_matrix* A = G->A;
  const int n = G->n;
  gnn_forward(G, r, G->d_z, true);
  op_copy(ctx, n, G->d_z, G->d_d);
  op_axpy(ctx, n, -1.0, e, G->d_d);
  op_spmv(ctx, A, G->d_d, G->d_Ad, AB2_SPMV_AUTO);
  op_spmv(ctx, A, e, G->d_Ae, AB2_SPMV_AUTO);
  const double eAe = dot_value(ctx, n, e, G->d_Ae);
  const double dAd = dot_value(ctx, n, G->d_d, G->d_Ad);
  require(eAe > 0, "gnn training pair: e^T A e must be positive");
  op_scal(ctx, n, 2.0 / eAe, G->d_Ad);  // dz
  const int wg = warp_grid(ctx, n);
  k_gnn_decode_bwd<<<wg, 256, 0, ctx->stream>>>(n, G->d_Ad, G->d_s2, G->d_isd, G->d_xr, hbuf(G, kLayers), G->d_P,
                                                G->d_dh, G->d_part);
  check_launch(ctx, "gnn_decode_bwd");
  reduce_into(G, wg, kH + 2, G->d_grad + kOffWd);
  float* dh = G->d_dh;
  float* dh2 = G->d_dh2;
  for (int l = kLayers - 1; l >= 0; --l) {
    const int gg = wgrad_grid(ctx, n);
    k_gnn_wgrad<<<gg, 256, 0, ctx->stream>>>(n, dh, hbuf(G, l + 1), hbuf(G, l), mbuf(G, l), G->d_part);
    check_launch(ctx, "gnn_wgrad");
    reduce_into(G, gg, kH * kIn + kH, G->d_red);
    AB2_CUDA(cudaMemcpyAsync(G->d_grad + kOffW + (size_t)l * kH * kIn, G->d_red, sizeof(float) * kH * kIn,
                             cudaMemcpyDeviceToDevice, ctx->stream));
    AB2_CUDA(cudaMemcpyAsync(G->d_grad + kOffB + l * kH, G->d_red + kH * kIn, sizeof(float) * kH,
                             cudaMemcpyDeviceToDevice, ctx->stream));
    k_gnn_dense_bwd<<<tile_grid(ctx, n), 256, 0, ctx->stream>>>(n, dh, hbuf(G, l + 1), G->d_Wb + (size_t)l * kH * kIn,
                                                                dh2, G->d_dm);
    check_launch(ctx, "gnn_dense_bwd");
    k_gnn_agg_bwd<<<wg, 256, 0, ctx->stream>>>(n, A->d_rp, A->d_ci, G->d_efeat, G->d_tidx, G->d_P, l, hbuf(G, l),
                                               G->d_dm, dh2, G->d_part);
    check_launch(ctx, "gnn_agg_bwd");
    reduce_into(G, wg, 2, G->d_red);
    AB2_CUDA(cudaMemcpyAsync(G->d_grad + kOffU + l, G->d_red, sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
    AB2_CUDA(cudaMemcpyAsync(G->d_grad + kOffC + l, G->d_red + 1, sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
    std::swap(dh, dh2);
  }
  k_gnn_encode_bwd<<<wg, 256, 0, ctx->stream>>>(n, G->d_xr, G->d_s2, G->d_logd10, hbuf(G, 0), dh, G->d_part);
  check_launch(ctx, "gnn_encode_bwd");
  reduce_into(G, wg, 3 * kH, G->d_grad + kOffW0);
  check_grid_wait(G);
  return dAd / eAe;
}

}  // namespace
}  // namespace ab2

extern "C" {

int ab2_gnn_param_count(void) { return kParams; }

int ab2_gnn_create(ab2_context* ctx, const float* params, unsigned long long seed, ab2_gnn** out) {
  if (!ctx || !out) return AB2_ERR_BAD_ARG;
  *out = nullptr;
  ab2_gnn* G = new (std::nothrow) ab2_gnn();
  if (!G) return AB2_ERR_OOM;
  G->ctx = ctx_retain(ctx);
  int rc = guard(ctx, [&] {
    std::vector<float> h(kParams, 0.f);
    if (params) {
      std::copy(params, params + kParams, h.begin());
    } else {  // He-style normal initialisation
      std::mt19937_64 gen(seed);
      std::normal_distribution<float> w0(0.f, 1.f), wl(0.f, std::sqrt(2.f / kIn)),
          wd(0.f, 0.1f * std::sqrt(1.f / kH));  // small: the network starts close to its Jacobi skip
      for (int k = 0; k < 2 * kH; ++k) h[kOffW0 + k] = w0(gen);
      for (int k = 0; k < kLayers * kH * kIn; ++k) h[kOffW + k] = wl(gen);
      for (int k = 0; k < kLayers * kH; ++k) h[kOffB + k] = 0.01f;
      for (int l = 0; l < kLayers; ++l) h[kOffU + l] = 0.5f;
      for (int k = 0; k < kH; ++k) h[kOffWd + k] = wd(gen);
      h[kOffWs] = 1.f;
    }
    G->d_P = dev_alloc<float>(ctx, kParams);
    G->d_grad = dev_alloc<float>(ctx, kParams);
    G->d_am = dev_alloc<float>(ctx, kParams);
    G->d_av = dev_alloc<float>(ctx, kParams);
    G->d_Wb = dev_alloc<bf16>(ctx, (size_t)kLayers * kH * kIn);
    AB2_CUDA(cudaMemcpyAsync(G->d_P, h.data(), sizeof(float) * kParams, cudaMemcpyHostToDevice, ctx->stream));
    AB2_CUDA(cudaMemsetAsync(G->d_grad, 0, sizeof(float) * kParams, ctx->stream));
    AB2_CUDA(cudaMemsetAsync(G->d_am, 0, sizeof(float) * kParams, ctx->stream));
    AB2_CUDA(cudaMemsetAsync(G->d_av, 0, sizeof(float) * kParams, ctx->stream));
    k_gnn_wcopy<<<64, 256, 0, ctx->stream>>>(G->d_P, G->d_Wb);
    check_launch(ctx, "gnn_wcopy");
    AB2_CUDA(cudaStreamSynchronize(ctx->stream));
  });
  if (rc != AB2_OK) {
    ab2_gnn_destroy(G);
    return rc;
  }
  *out = G;
  return AB2_OK;
}

int ab2_gnn_get_params(const ab2_gnn* G, float* params) {
  if (!G || !params) return AB2_ERR_BAD_ARG;
  return guard(G->ctx, [&] {
    AB2_CUDA(cudaMemcpyAsync(params, G->d_P, sizeof(float) * kParams, cudaMemcpyDeviceToHost, G->ctx->stream));
    AB2_CUDA(cudaStreamSynchronize(G->ctx->stream));
  });
}

int ab2_gnn_set_params(ab2_gnn* G, const float* params) {
  if (!G || !params) return AB2_ERR_BAD_ARG;
  return guard(G->ctx, [&] {
    AB2_CUDA(cudaMemcpyAsync(G->d_P, params, sizeof(float) * kParams, cudaMemcpyHostToDevice, G->ctx->stream));
    k_gnn_wcopy<<<64, 256, 0, G->ctx->stream>>>(G->d_P, G->d_Wb);
    check_launch(G->ctx, "gnn_wcopy");
    AB2_CUDA(cudaStreamSynchronize(G->ctx->stream));
  });
}

int ab2_gnn_bind(ab2_gnn* G, const ab2_matrix* A) {
  if (!G || !A || A->n <= 0) return AB2_ERR_BAD_ARG;
  ab2_context* ctx = G->ctx;
  return guard(ctx, [&] {
    ctx_quiesce(ctx);
    release_binding(G);
    const int n = A->n;
    G->A = A;
    G->n = n;
    G->d_isd = dev_alloc<float>(ctx, (size_t)n);
    G->d_logd10 = dev_alloc<float>(ctx, (size_t)n);
    G->d_efeat = dev_alloc<float>(ctx, (size_t)A->nnz);
    G->d_tidx = dev_alloc<int>(ctx, (size_t)A->nnz);
    G->d_h = dev_alloc<bf16>(ctx, (size_t)(kLayers + 1) * n * kH);
    G->d_m = dev_alloc<bf16>(ctx, (size_t)kLayers * n * kH);
    G->d_xr = dev_alloc<float>(ctx, (size_t)n);
    G->d_s2 = dev_alloc<double>(ctx, 2);
    G->d_dh = dev_alloc<float>(ctx, (size_t)n * kH);
    G->d_dh2 = dev_alloc<float>(ctx, (size_t)n * kH);
    G->d_dm = dev_alloc<float>(ctx, (size_t)n * kH);
    G->d_z = dev_alloc<double>(ctx, (size_t)n);
    G->d_d = dev_alloc<double>(ctx, (size_t)n);
    G->d_Ad = dev_alloc<double>(ctx, (size_t)n);
    G->d_Ae = dev_alloc<double>(ctx, (size_t)n);
    G->part_cap = std::max((long long)wgrad_grid(ctx, n) * (kH * kIn + kH), (long long)warp_grid(ctx, n) * 3 * kH);
    G->d_part = dev_alloc<float>(ctx, (size_t)G->part_cap);
    G->d_red = dev_alloc<float>(ctx, (size_t)(kH * kIn + kH));
    int* d_bad = dev_alloc<int>(ctx, 1);
    AB2_CUDA(cudaMemsetAsync(d_bad, 0, sizeof(int), ctx->stream));
    k_gnn_prep<<<grid_for(n), kThreads, 0, ctx->stream>>>(n, A->d_rp, A->d_ci, A->d_v, A->d_dcol, G->d_isd,
                                                          G->d_logd10, G->d_efeat, G->d_tidx, d_bad);
    check_launch(ctx, "gnn_prep");
    int bad = 0;
    AB2_CUDA(cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    AB2_CUDA(cudaStreamSynchronize(ctx->stream));
    dev_free(ctx, d_bad);
    if (!bad) {
      int maxlen = 0;  // off-diagonal entries of the longest row (every row has its diagonal)
      host_profile(A);
      for (int i = 0; i < n; ++i) maxlen = std::max(maxlen, A->h_rp[i + 1] - A->h_rp[i] - 1);
      G->nbw = std::max(2, (maxlen + 1) / 2 * 2);
      if (G->nbw > kMaxNbw) {
        release_binding(G);
        throw Error{AB2_ERR_UNSUPPORTED, "learned preconditioner: at most 16 off-diagonal entries a row"};
      }
      G->d_nb_idx = dev_alloc<int>(ctx, (size_t)n * G->nbw);
      G->d_nb_ef = dev_alloc<float>(ctx, (size_t)n * G->nbw);
      k_gnn_nbr<<<grid_for(n), kThreads, 0, ctx->stream>>>(n, A->d_rp, A->d_ci, G->d_efeat, G->nbw, G->d_nb_idx,
                                                           G->d_nb_ef);
      check_launch(ctx, "gnn_nbr");
      int nx = 0, ny = 0, nz = 0;
      G->grid = stencil_geometry(ctx, A, &nx, &ny, &nz);
      if (G->grid) {
        G->gnx = nx;
        G->gny = ny;
        G->gnz = nz;
        const long long rows = ((long long)n + kTcTile - 1) / kTcTile * kTcTile;
        G->d_dir_ef = dev_alloc<float>(ctx, (size_t)rows * 6);
        G->d_err = dev_alloc<int>(ctx, 1);
        AB2_CUDA(cudaMemsetAsync(G->d_err, 0, sizeof(int), ctx->stream));
        k_gnn_dir_table<<<grid_for(rows), kThreads, 0, ctx->stream>>>(n, rows, nx, nx * ny, A->d_rp, A->d_ci,
                                                                      G->d_efeat, G->d_dir_ef);
        check_launch(ctx, "gnn_dir_table");
      } else if (G->layout == AB2_GNN_LAYER_GRID) {
        release_binding(G);
        throw Error{AB2_ERR_UNSUPPORTED, "learned preconditioner: the grid layer needs a 3-D 7-point matrix"};
      }
    }
    if (bad) {
      release_binding(G);
      throw Error{AB2_ERR_BAD_ARG, bad & 1 ? "learned preconditioner needs a positive diagonal in every row"
                                           : "learned preconditioner needs a structurally symmetric matrix"};
    }
  });
}

int ab2_gnn_set_layer(ab2_gnn* G, int layer) {
  if (!G || layer < AB2_GNN_LAYER_AUTO || layer > AB2_GNN_LAYER_GRID) return AB2_ERR_BAD_ARG;
  G->layout = layer;
  return AB2_OK;
}

int ab2_gnn_get_layer(const ab2_gnn* G, int* layer) {
  if (!G || !layer) return AB2_ERR_BAD_ARG;
  *layer = !G->A ? AB2_GNN_LAYER_AUTO : use_grid_layer(G) ? AB2_GNN_LAYER_GRID : AB2_GNN_LAYER_GATHER;
  return AB2_OK;
}

int ab2_gnn_apply(ab2_gnn* G, const ab2_vector* r, ab2_vector* z) {
  if (!G || !r || !z || !G->A || r->n != G->n || z->n != G->n || r->d == z->d) return AB2_ERR_BAD_ARG;
  PhaseScope phase_scope(G->ctx, "GNN-APPLY");
  return guard(G->ctx, [&] {
    gnn_forward(G, r->d, z->d);
    check_grid_wait(G);
  });
}

int ab2_gnn_loss_grad(ab2_gnn* G, const ab2_vector* r, const ab2_vector* e, double* loss, float* grad) {
  if (!G || !r || !e || !G->A || r->n != G->n || e->n != G->n) return AB2_ERR_BAD_ARG;
  return guard(G->ctx, [&] {
    const double L = gnn_loss_grad(G, r->d, e->d);
    if (loss) *loss = L;
    if (grad) {
      AB2_CUDA(cudaMemcpyAsync(grad, G->d_grad, sizeof(float) * kParams, cudaMemcpyDeviceToHost, G->ctx->stream));
      AB2_CUDA(cudaStreamSynchronize(G->ctx->stream));
    }
  });
}

int ab2_gnn_train_step(ab2_gnn* G, const ab2_vector* r, const ab2_vector* e, double lr, double* loss) {
  if (!G || !r || !e || !G->A || r->n != G->n || e->n != G->n || !(lr >= 0)) return AB2_ERR_BAD_ARG;
  ab2_context* ctx = G->ctx;
  return guard(ctx, [&] {
    const double L = gnn_loss_grad(G, r->d, e->d);
    if (loss) *loss = L;
    G->step += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)G->step), c2 = 1.f - std::pow(b2, (float)G->step);
    k_gnn_adam<<<(kParams + 255) / 256, 256, 0, ctx->stream>>>(kParams, G->d_P, G->d_grad, G->d_am, G->d_av, (float)lr,
                                                               b1, b2, 1e-8f, c1, c2);
    check_launch(ctx, "gnn_adam");
    k_gnn_wcopy<<<64, 256, 0, ctx->stream>>>(G->d_P, G->d_Wb);
    check_launch(ctx, "gnn_wcopy");
  });
}

int ab2_gnn_destroy(ab2_gnn* G) {
  if (!G) return AB2_ERR_BAD_ARG;
  if (G->ctx) {
    ctx_quiesce(G->ctx);
    release_binding(G);
    for (void* p : {(void*)G->d_P, (void*)G->d_grad, (void*)G->d_am, (void*)G->d_av, (void*)G->d_Wb})
      dev_free(G->ctx, p);
    ctx_release(G->ctx);
  }
  delete G;
  return AB2_OK;
}

void ab2_fcg_options_default(ab2_fcg_options* o) {
  if (!o) return;
  std::memset(o, 0, sizeof(*o));
  o->tol = 1e-8;
  o->max_iter = 5000;
  o->fallback_ratio = 1.0;
  o->truncation = 8;
  o->fallback_mode = AB2_FCG_FALLBACK_STEP;
}

// Flexible CG, FCG(m) (truncated A-orthogonalisation of the directions, so
// that a preconditioner which is not a fixed linear operator keeps them
// conjugate): z = network(r) while the network's steps reduce ||r|| by at
// least the factor fallback_ratio, the fallback preconditioner from the first
// step that does not (for the rest of the solve, the direction window
// cleared).  No network: the fallback only.
int ab2_fcg_solve(ab2_context* ctx, const ab2_matrix* A, ab2_gnn* G, const ab2_precond* fallback,
                  const ab2_vector* b, ab2_vector* x, const ab2_fcg_options* o, ab2_fcg_status* st) {
  if (!ctx || !A || !b || !x || !o || !st || b->n != A->n || x->n != A->n) return AB2_ERR_BAD_ARG;
  if (!G && !fallback) return AB2_ERR_BAD_ARG;
  PhaseScope phase_scope(ctx, "FCG-SOLVE");
  if (G && (G->A != A)) return AB2_ERR_BAD_ARG;
  if (fallback && fallback->A != A) return AB2_ERR_BAD_ARG;
  std::memset(st, 0, sizeof(*st));
  st->switched_at = -1;
  if (!(o->truncation >= 1 && o->truncation <= kMaxTrunc)) return AB2_ERR_BAD_ARG;
  if (o->fallback_mode != AB2_FCG_FALLBACK_STICKY && o->fallback_mode != AB2_FCG_FALLBACK_STEP) return AB2_ERR_BAD_ARG;
  return guard(ctx, [&] {
    const int n = A->n;
    const int m = o->truncation;
    cudaEvent_t e0, e1;
    AB2_CUDA(cudaEventCreate(&e0));
    AB2_CUDA(cudaEventCreate(&e1));
    double* r = dev_alloc<double>(ctx, (size_t)n);
    double* z = dev_alloc<double>(ctx, (size_t)n);
    double* pv = dev_alloc<double>(ctx, (size_t)m * n);  // window of directions
    double* qv = dev_alloc<double>(ctx, (size_t)m * n);  // and their products with A
    FcgScalars* sc = dev_alloc<FcgScalars>(ctx, 1);
    double* zq_part = dev_alloc<double>(ctx, (size_t)kMaxTrunc * kMaxRedBlocks);
    double* zq_out = dev_alloc<double>(ctx, kMaxTrunc);
    unsigned* zq_counter = dev_alloc<unsigned>(ctx, 1);
    AB2_CUDA(cudaMemsetAsync(sc, 0, sizeof(FcgScalars), ctx->stream));
    AB2_CUDA(cudaMemsetAsync(zq_counter, 0, sizeof(unsigned), ctx->stream));
    AB2_CUDA(cudaEventRecord(e0, ctx->stream));
    RedSlot red = red_slot(ctx, 7);
    const int rg = red_grid(ctx, n);
    auto dot = [&](const double* u, const double* v) {
      return dot_value(ctx, n, u, v);
    };
    bool use_gnn = G != nullptr;      // the network preconditions the next step
    bool gnn_retired = G == nullptr;  // STICKY fallback has taken over
    auto precond = [&](const double* in, double* out) {
      if (use_gnn) {
        gnn_forward(G, in, out);
        st->gnn_steps += 1;
      } else {
        pc_apply(ctx, fallback, in, out);
        if (pc_error(ctx, fallback)) {
          pc_reset(ctx, fallback);
          throw Error{AB2_ERR_TIMEOUT, "fallback preconditioner: a bounded wait gave up"};
        }
        st->fallback_steps += 1;
      }
    };
    const double nb = std::sqrt(dot(b->d, b->d));
    op_spmv(ctx, A, x->d, z, AB2_SPMV_AUTO);
    op_copy(ctx, n, b->d, r);
    op_axpy(ctx, n, -1.0, z, r);
    double rn = std::sqrt(dot(r, r));
    int it = 0, count = 0, next = 0;
    bool ok = nb == 0.0 || rn / nb < o->tol;
    while (!ok && it < o->max_iter) {
      precond(r, z);
      double* p = pv + (size_t)next * n;
      double* q = qv + (size_t)next * n;
      if (count > 0) {
        Window wq{}, wp{};
        for (int k = 0; k < count; ++k) {
          wq.v[k] = qv + (size_t)k * n;
          wp.v[k] = pv + (size_t)k * n;
        }
        auto ortho = [&](auto c) {
          constexpr int C = decltype(c)::value;
          k_fcg_zq<C><<<rg, kThreads, 0, ctx->stream>>>(n, z, wq, count, sc, zq_part, zq_counter, zq_out);
          check_launch(ctx, "fcg_zq");
          k_fcg_dir<C><<<grid_for(n), kThreads, 0, ctx->stream>>>(n, z, wp, count, sc, p);
          check_launch(ctx, "fcg_dir");
        };
        if (count <= 4) ortho(std::integral_constant<int, 4>());
        else if (count <= 8) ortho(std::integral_constant<int, 8>());
        else ortho(std::integral_constant<int, kMaxTrunc>());
      } else {
        op_copy(ctx, n, z, p);
      }
      op_spmv(ctx, A, p, q, AB2_SPMV_AUTO);
      k_fcg_pq<<<rg, kThreads, 0, ctx->stream>>>(n, p, q, r, next, sc, red.partials, red.counter, red.result);
      check_launch(ctx, "fcg_pq");
      k_fcg_update<<<rg, kThreads, 0, ctx->stream>>>(n, p, q, x->d, r, sc, red.partials, red.counter, red.result);
      check_launch(ctx, "fcg_update");
      FcgScalars h;
      AB2_CUDA(cudaMemcpyAsync(ctx->h_pinned, sc, sizeof(FcgScalars), cudaMemcpyDeviceToHost, ctx->stream));
      AB2_CUDA(cudaStreamSynchronize(ctx->stream));
      std::memcpy(&h, ctx->h_pinned, sizeof(FcgScalars));
      if (h.breakdown) {
        st->error = AB2_ERR_BREAKDOWN;
        break;
      }
      ++it;
      const double rn_new = std::sqrt(h.rr);
      if (rn_new / nb < o->tol) {
        ok = true;
        rn = rn_new;
        break;
      }
      const bool failed = use_gnn && fallback && rn_new > o->fallback_ratio * rn;
      if (failed && st->switched_at < 0) st->switched_at = it;
      if (failed && o->fallback_mode == AB2_FCG_FALLBACK_STICKY) {
        use_gnn = false;  // ILU(0) takes over from here, with the window cleared
        gnn_retired = true;
        count = 0;
        next = 0;
      } else {
        count = std::min(count + 1, m);
        next = (next + 1) % m;
        use_gnn = !gnn_retired && !failed;  // STEP: the fallback for one step after a failed network step
      }
      rn = rn_new;
    }
    AB2_CUDA(cudaEventRecord(e1, ctx->stream));
    AB2_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    AB2_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    op_spmv(ctx, A, x->d, z, AB2_SPMV_AUTO);
    op_copy(ctx, n, b->d, r);
    op_axpy(ctx, n, -1.0, z, r);
    st->true_residual = nb > 0 ? std::sqrt(dot(r, r)) / nb : 0.0;
    st->succeeded = ok ? 1 : 0;
    st->iterations = it;
    st->solve_ms = ms;
    if (!ok && st->error == AB2_OK) st->error = AB2_ERR_NOT_CONVERGED;
    for (double* v : {r, z, pv, qv, zq_part, zq_out}) dev_free(ctx, v);
    dev_free(ctx, sc);
    dev_free(ctx, zq_counter);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (G) check_grid_wait(G);
  });
}

}  // extern "C"
