// ilu_stencil.cu -- ILU(0) factorisation and sweeps scheduled for 7-point
// matrices in lexicographic order.
//
// The arithmetic is exactly the general path's (ILU0Preconditioner.h:156-231:
// same per-row operations, same column order, product and difference rounded
// apart, an IEEE division by the pivot), so factor and applications are bit
// for bit those of the wavefront kernels in precond.cu and of the sequential
// reference.  Only the schedule differs.
//
// Schedule.  In a 3-D 7-point matrix numbered i + nx (j + ny k), row (i,j,k)
// of the forward sweep depends on (i,j,k-1), (i,j-1,k) and (i-1,j,k).  A CTA
// owns a 16 x 16 tile of z-lines, in two strips of 16 x 8 lines; one warp computes
// a strip, 2 x 2 lines a lane, and walks its diagonals: at step s lane (ti, tj)
// computes its four cells of plane k = s - ti - tj.  Its k-1 inputs are its own
// previous values, the i-1 and j-1 inputs the neighbouring lanes' values of step
// s-1 (warp shuffles): nothing in a strip waits on a barrier.  Between strips and
// tiles values are handed over word by word, the word being its own flag (the
// sentinel of sentinel.cuh): from strip to strip through a ring in shared memory,
// from tile to tile through global memory, where polling warps of the next tile
// fetch them into such a ring.  Tiles are claimed from an atomic ticket in
// row-major order (a tile waits only on tiles with a smaller ticket), so no
// co-residency is needed.  Every wait is bounded.
//
// The backward sweep is the same walk in mirrored coordinates (i' = nx - 1 - i
// and so on), its own coefficients packed in that order.
//
// Everything else is kept away from the compute warps: loading warps bring the
// coefficients (packed by strip and step at set-up, one bulk copy for two steps)
// and the right-hand side (natural order, placed by the step that uses it) into
// rings in shared memory, storing warps take the results out of a ring into
// natural order.  So an application is two kernels and moves every band, the
// input, the vector between the sweeps and the output once.
//
// What bounds it: the dependency chain, nx + ny + nz - 2 cells long.  A warp that
// waits for its own results issues one instruction in three to four cycles, so a
// step costs what its instructions cost: 165 ns forward, 272 ns backward (a lone
// tile, 1.9 GHz; FP64 operations 8 cycles apart), and a hand-over to the next tile
// 8 steps + 1.5 us (store, poll and read back through L2).  Four cells a lane and
// step because the cost of a step is mostly not the cells: counting steps on the
// critical path, nx/2 + ny/2 + nz instead of nx + ny + nz.  The division by the
// pivot is three dependent FMAs longer than the subtraction chain instead of ~140
// cycles, off a reciprocal stored at set-up (below).
//
// Measured on B200, one application (both sweeps, FP64): 192^3 541 -> 360 us,
// 128^3 350 -> 200 us, 70 x 90 x 50 204 -> 101 us, against one line a thread, 16 x 16
// threads and a barrier a step, tiles in 2 x 2 clusters, with separate passes that
// brought the vectors into walk order and back.
//
// The factorisation runs once per set-up on the natural-order bands, one line a
// thread (pivots propagate; in a 7-point matrix ILU(0) changes only the diagonal
// and the L values).
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "ab2_internal.cuh"
#include "precond.cuh"
#include "recip.cuh"
#include "sentinel.cuh"

namespace ab2 {

namespace {

constexpr int kTile = 16;  // the factorisation walk: one line a thread
constexpr int kTileThreads = kTile * kTile;
// AB2_ILU_STENCIL and AB2_ILU_STENCIL_CLUSTER name one walk now; callers still
// get (and are refused) the second by the number of planes along z.
constexpr int kClusterPlanes = 346;

struct Geom {
  int nx, ny, nz, ntx, nty;
  long long nxny;
};

struct Bands {
  double *Lk, *Lj, *Li, *Ui, *Uj, *Uk, *P, *D;
};

__global__ void k_stencil_extract(int n, Geom g, const int* __restrict__ rp, const double* __restrict__ v, Bands b) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const int i = r % g.nx, j = (r / g.nx) % g.ny, k = (int)(r / g.nxny);
    int e = rp[r];
    b.Lk[r] = k > 0 ? v[e++] : 0.0;
    b.Lj[r] = j > 0 ? v[e++] : 0.0;
    b.Li[r] = i > 0 ? v[e++] : 0.0;
    b.D[r] = v[e++];
    b.Ui[r] = i < g.nx - 1 ? v[e++] : 0.0;
    b.Uj[r] = j < g.ny - 1 ? v[e++] : 0.0;
    b.Uk[r] = k < g.nz - 1 ? v[e++] : 0.0;
  }
}

__global__ void k_stencil_pack(int n, Geom g, const int* __restrict__ rp, Bands b, double* __restrict__ lu) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const int i = r % g.nx, j = (r / g.nx) % g.ny, k = (int)(r / g.nxny);
    int e = rp[r];
    if (k > 0) lu[e++] = b.Lk[r];
    if (j > 0) lu[e++] = b.Lj[r];
    if (i > 0) lu[e++] = b.Li[r];
    lu[e++] = b.P[r];
    if (i < g.nx - 1) lu[e++] = b.Ui[r];
    if (j < g.ny - 1) lu[e++] = b.Uj[r];
    if (k < g.nz - 1) lu[e++] = b.Uk[r];
  }
}

// The factorisation walk (set-up only, natural-order bands): row (i,j,k)
// divides its L entries by the pivots of its -k, -j, -i neighbours and
// subtracts l * u (the neighbour's U entry towards this row) from its diagonal,
// columns ascending; the resulting pivot propagates.
struct PreF {
  double d, lk, lj, li, uk, uj, ui, bi, bj;
};

__global__ void __launch_bounds__(kTileThreads) k_stencil_factor(Geom g, Bands b, unsigned int* tickets, int* err) {
  constexpr int kPrefetch = 4;
  __shared__ double s_val[2][kTile][kTile + 1];
  __shared__ int s_tile;
  const int li = threadIdx.x % kTile, lj = threadIdx.x / kTile;
  const int ntiles = g.ntx * g.nty;
  const int nsteps = g.nz + 2 * (kTile - 1);
  double* wave = b.P;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_tile = (int)atomicAdd(tickets, 1u);
    __syncthreads();
    const int tile = s_tile;
    if (tile >= ntiles) break;
    const int ai = (tile % g.ntx) * kTile + li;
    const int aj = (tile / g.ntx) * kTile + lj;
    const bool active = ai < g.nx && aj < g.ny;
    const long long line = active ? ai + (long long)g.nx * aj : 0;
    auto cell = [&](int s, long long& r) {
      const int ak = s - li - lj;
      if (!active || ak < 0 || ak >= g.nz) return -1;
      r = line + g.nxny * ak;
      return ak;
    };
    auto load = [&](int s, PreF& p) {
      long long r = 0;
      if (cell(s, r) < 0) return;
      if (lj == 0 && aj > 0) p.bj = ld_relaxed(wave + r - g.nx);
      if (li == 0 && ai > 0) p.bi = ld_relaxed(wave + r - 1);
      p.d = b.D[r];
      p.lk = b.Lk[r];
      p.lj = b.Lj[r];
      p.li = b.Li[r];
      p.uk = r >= g.nxny ? b.Uk[r - g.nxny] : 0.0;
      p.uj = r >= g.nx ? b.Uj[r - g.nx] : 0.0;
      p.ui = r >= 1 ? b.Ui[r - 1] : 0.0;
    };
    PreF pre[kPrefetch];
#pragma unroll
    for (int u = 0; u < kPrefetch; ++u) {
      pre[u] = PreF{0, 0, 0, 0, 0, 0, 0, 0, 0};
      load(u, pre[u]);
    }
    double own = 0.0;
    for (int s0 = 0; s0 < nsteps; s0 += kPrefetch) {
#pragma unroll
      for (int u = 0; u < kPrefetch; ++u) {
        const int s = s0 + u;
        if (s < nsteps) {
          const PreF c = pre[u];
          load(s + kPrefetch, pre[u]);
          long long r = 0;
          const int ak = cell(s, r);
          double val = 0.0;
          if (ak >= 0) {
            const double* prev = &s_val[(s + 1) & 1][0][0];
            double vi = 0.0, vj = 0.0;
            if (aj > 0)
              vj = lj > 0 ? prev[(lj - 1) * (kTile + 1) + li]
                          : (is_sentinel(c.bj) ? wait_value(wave + r - g.nx, err) : c.bj);
            if (ai > 0)
              vi = li > 0 ? prev[lj * (kTile + 1) + li - 1] : (is_sentinel(c.bi) ? wait_value(wave + r - 1, err) : c.bi);
            double d = c.d;  // a_ik /= pivot_k, then a_ii -= a_ik a_ki, columns ascending (-k, -j, -i)
            if (ak > 0) {
              const double l = c.lk / own;
              d = mul_sub_rn(l, c.uk, d);
              b.Lk[r] = l;
            }
            if (aj > 0) {
              const double l = c.lj / vj;
              d = mul_sub_rn(l, c.uj, d);
              b.Lj[r] = l;
            }
            if (ai > 0) {
              const double l = c.li / vi;
              d = mul_sub_rn(l, c.ui, d);
              b.Li[r] = l;
            }
            val = d;
            st_relaxed(wave + r, not_sentinel(val));
            own = val;
          }
          s_val[s & 1][lj][li] = val;
          __syncthreads();
        }
      }
    }
  }
}

// ------------------------------------------------------------------ walk shape
constexpr int kTileI = 16, kTileJ = 16;          // lines of a tile (one CTA)
constexpr int kStrips = 2;                       // strips of a tile, one compute warp each
constexpr int kStripJ = kTileJ / kStrips;        // a strip: 16 x 8 lines, 2 x 2 a lane
constexpr int kLanesI = kTileI / 2, kLanesJ = kStripJ / 2;
constexpr int kSkew = kLanesI - 1 + kLanesJ - 1;  // steps between a strip's first and last lane
constexpr int kStripCells = kTileI * kStripJ;    // cells a strip computes in one step
constexpr int kDepth = 12;                       // steps of inputs in flight or waiting, two on an mbarrier
constexpr int kInRing = 24;                      // ring of input cells by step: kDepth + kSkew and a margin (even)
constexpr int kOutRing = 22;                     // ring of output cells by step (even)
constexpr int kSlots = 32;                       // ring of hand-over slots by step (a power of two)
constexpr int kPollDepth = 2;                    // words a polling lane loads at once
static_assert(kLanesI * kLanesJ == 32 && kInRing > kDepth + kSkew && kOutRing >= kSkew + 12, "walk shape");
// Warps by role.  Warps w, w + 4 and w + 8 share an SM sub-partition: each
// compute warp (0 and 1) shares its own with two polling warps, which mostly wait
// on L2; the helpers -- two loading warps a strip (every other pair of steps) and
// a storing warp a strip -- share the other two.  A helper's loop is a chain of
// dependent instructions, several cycles each: what keeps it out of the compute
// warp's way is having few of them per step.
constexpr int kWalkWarps = 12;
enum class Role { Compute, Load, Store, Poll };
struct WarpRole {
  Role role;
  int strip, part;
};
__device__ __forceinline__ WarpRole warp_role(int warp) {
  if (warp < 2) return {Role::Compute, warp, 0};
  const int turn = warp >> 2;
  if ((warp & 3) < 2) return {Role::Poll, 0, (turn - 1) * 2 + (warp & 1)};
  const int strip = (warp & 3) - 2;
  return turn < 2 ? WarpRole{Role::Load, strip, turn} : WarpRole{Role::Store, strip, 0};
}
static_assert(kStrips == 2, "warp roles");

struct Walk {
  int nx, ny, nz, ntx, nty;
  int nsteps;  // of a strip (even)
  int halo;    // planes of a tile's hand-over words, kSkew unused ones either side
  long long nxny, n;
};

// ------------------------------------------------------------------ strip walk
// Shared-memory words by 32-bit address.  asm volatile keeps these accesses
// in program order among themselves, which is the order one warp's shared
// memory accesses are performed in; no "memory" clobber, so arithmetic and
// prefetched loads may be scheduled around them.
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// By predicate (on: 0 or 1), so that a lane's share of a step is not a
// branch: a divergent branch and its reconvergence cost the compute warp more
// than the access itself.
__device__ __forceinline__ void lds2_if(int on, unsigned a, double& x, double& y) {
  asm volatile("{.reg .pred p; setp.ne.s32 p, %2, 0; @p ld.volatile.shared.v2.f64 {%0, %1}, [%3];}"
               : "+d"(x), "+d"(y) : "r"(on), "r"(a));
}
__device__ __forceinline__ void lds2_if(int on, unsigned a, float& x, float& y) {
  asm volatile("{.reg .pred p; setp.ne.s32 p, %2, 0; @p ld.volatile.shared.v2.f32 {%0, %1}, [%3];}"
               : "+f"(x), "+f"(y) : "r"(on), "r"(a));
}
__device__ __forceinline__ void sts2_if(int on, unsigned a, double x, double y) {
  asm volatile("{.reg .pred p; setp.ne.s32 p, %0, 0; @p st.volatile.shared.v2.f64 [%1], {%2, %3};}" ::"r"(on), "r"(a),
               "d"(x), "d"(y));
}
__device__ __forceinline__ void sts2_if(int on, unsigned a, float x, float y) {
  asm volatile("{.reg .pred p; setp.ne.s32 p, %0, 0; @p st.volatile.shared.v2.f32 [%1], {%2, %3};}" ::"r"(on), "r"(a),
               "f"(x), "f"(y));
}
__device__ __forceinline__ void sts_int_if(int on, unsigned a, int v) {
  asm volatile("{.reg .pred p; setp.ne.s32 p, %0, 0; @p st.volatile.shared.s32 [%1], %2;}" ::"r"(on), "r"(a), "r"(v));
}
// Weak forms for words handed over by an mbarrier or a counter.
__device__ __forceinline__ void ldw2(unsigned a, double& x, double& y) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "r"(a));
}
__device__ __forceinline__ void ldw2(unsigned a, float& x, float& y) {
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x), "=f"(y) : "r"(a));
}
__device__ __forceinline__ void stw2(unsigned a, double x, double y) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(x), "d"(y));
}
__device__ __forceinline__ void stw2(unsigned a, float x, float y) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(x), "f"(y));
}
__device__ __forceinline__ void sts1(unsigned a, double x) {
  asm volatile("st.volatile.shared.f64 [%0], %1;" ::"r"(a), "d"(x));
}
__device__ __forceinline__ void sts1(unsigned a, float x) {
  asm volatile("st.volatile.shared.f32 [%0], %1;" ::"r"(a), "f"(x));
}
__device__ __forceinline__ void lds1(unsigned a, double& x) {
  asm volatile("ld.volatile.shared.f64 %0, [%1];" : "=d"(x) : "r"(a));
}
__device__ __forceinline__ void lds1(unsigned a, float& x) {
  asm volatile("ld.volatile.shared.f32 %0, [%1];" : "=f"(x) : "r"(a));
}
__device__ __forceinline__ int lds_int(unsigned a) {
  int v;
  asm volatile("ld.volatile.shared.s32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts_int(unsigned a, int v) {
  asm volatile("st.volatile.shared.s32 [%0], %1;" ::"r"(a), "r"(v));
}

__device__ __forceinline__ void mbar_init(unsigned a, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned a, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned a, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(a), "r"(parity)
      : "memory");
  return done != 0;
}
// The same without the wait (try_wait may suspend the warp for a while).
__device__ __forceinline__ bool mbar_test(unsigned a, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(a), "r"(parity)
      : "memory");
  return done != 0;
}
// Global -> this CTA's shared memory, completing on the mbarrier.
__device__ __forceinline__ void bulk_load(unsigned dst, const void* src, unsigned bytes, unsigned mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(mbar)
               : "memory");
}
template <int BYTES>
__device__ __forceinline__ void copy_word(unsigned dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}
// This thread's copies so far, one arrival of the mbarrier's count.
__device__ __forceinline__ void copy_arrive(unsigned mbar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void copy_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// Two hand-over words in global memory, each its own flag (no "memory"
// clobber: no other access needs ordering against them).
__device__ __forceinline__ void st_flag2_if(int on, double* p, double x, double y) {
  asm volatile(
      "{.reg .pred p; setp.ne.s32 p, %0, 0; @p st.relaxed.gpu.global.f64 [%1], %2; @p st.relaxed.gpu.global.f64 "
      "[%1+8], %3;}" ::"r"(on), "l"(p), "d"(x), "d"(y));
}
__device__ __forceinline__ void st_flag2_if(int on, float* p, float x, float y) {
  asm volatile(
      "{.reg .pred p; setp.ne.s32 p, %0, 0; @p st.relaxed.gpu.global.f32 [%1], %2; @p st.relaxed.gpu.global.f32 "
      "[%1+4], %3;}" ::"r"(on), "l"(p), "f"(x), "f"(y));
}

template <class T>
__device__ __forceinline__ T quiet_nan();
template <>
__device__ __forceinline__ double quiet_nan<double>() {
  return __longlong_as_double(0x7FF8000000000000LL);
}
template <>
__device__ __forceinline__ float quiet_nan<float>() {
  return __uint_as_float(0x7FC00000u);
}

// Whether a hand-over word has not arrived: the sentinel by its upper half
// alone (a signalling NaN, which no arithmetic result is).
__device__ __forceinline__ bool waiting(double v) { return __double2hiint(v) == (int)(kSentinel >> 32); }
__device__ __forceinline__ bool waiting(float v) { return is_sentinel(v); }

__device__ __forceinline__ bool sign_bit(double v) { return __double2hiint(v) < 0; }
__device__ __forceinline__ bool sign_bit(float v) { return __float_as_int(v) < 0; }

// A bounded wait's give-up test, asked every 256 polls.
__device__ __forceinline__ bool give_up(unsigned it, long long t0, int* err) {
  if ((it & 255) != 0) return false;
  if (clock64() - t0 <= kWaitCycles && *(volatile int*)err == 0) return false;
  atomicOr(err, 1);
  return true;
}

__device__ __noinline__ bool mbar_wait(unsigned a, unsigned parity, int* err) {
  const long long t0 = clock64();
  for (unsigned it = 16;; it += 16) {
    if (mbar_try_wait(a, parity)) return true;
    if (give_up(it, t0, err)) return false;
  }
}
// Waits within the time bound only (copies in flight at the kernel's end).
__device__ __noinline__ bool mbar_drain(unsigned a, unsigned parity) {
  const long long t0 = clock64();
  while (!mbar_try_wait(a, parity))
    if (clock64() - t0 > kWaitCycles) return false;
  return true;
}
// Waits until the counter at `a` is at least `v`.
__device__ __noinline__ bool wait_count(unsigned a, int v, int* err) {
  const long long t0 = clock64();
  for (unsigned it = 1;; ++it) {
    if (lds_int(a) >= v) return true;
    if (give_up(it, t0, err)) return false;
  }
}

// Bytes of one strip step's coefficients: the three bands, and in the
// backward sweep the reciprocal of the pivot (and the pivot, FP64).
template <bool UP, class T>
constexpr int coef_bytes() {
  return kStripCells * (3 * (int)sizeof(T) +
                        (UP ? (int)sizeof(typename Recip<T>::type) + (Recip<T>::keep_pivot ? (int)sizeof(T) : 0) : 0));
}

// Where the two sweeps of one precision keep their arrays (byte offsets from
// one allocation).
struct WalkMem {
  long long coef_l, coef_u, tmp, halo_l, halo_u, total;
  long long halo_words;  // words of one sweep's hand-over buffers
};
template <class T>
WalkMem walk_mem(const Walk& w) {
  const long long steps = (long long)w.ntx * w.nty * kStrips * w.nsteps;
  WalkMem m;
  m.halo_words = (long long)w.ntx * w.nty * w.halo * (kTileI + kTileJ);
  m.coef_l = 0;
  m.coef_u = m.coef_l + steps * coef_bytes<false, T>();
  m.tmp = m.coef_u + steps * coef_bytes<true, T>();
  m.halo_l = m.tmp + (w.n * (long long)sizeof(T) + 255) / 256 * 256;
  m.halo_u = m.halo_l + m.halo_words * (long long)sizeof(T);
  m.total = m.halo_u + m.halo_words * (long long)sizeof(T);
  return m;
}

// The natural row of walk cell (i, j, k), or -1 outside the grid.
template <bool UP>
__device__ __forceinline__ long long walk_row(const Walk& g, int i, int j, int k) {
  if (i >= g.nx || j >= g.ny || (unsigned)k >= (unsigned)g.nz) return -1;
  const long long w = i + (long long)g.nx * j + g.nxny * k;
  return UP ? g.n - 1 - w : w;
}

// The coefficients of every strip step, from the natural-order bands: bands
// 0 and pivots 1 outside the grid.  One thread per pair of cells along i.
template <bool UP>
__global__ void k_walk_pack(Walk g, Bands b, unsigned char* __restrict__ dst) {
  const long long pairs = (long long)g.ntx * g.nty * kStrips * g.nsteps * (kStripCells / 2);
  const double* band[3] = {UP ? b.Ui : b.Lk, UP ? b.Uj : b.Lj, UP ? b.Uk : b.Li};
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < pairs; q += (long long)gridDim.x * blockDim.x) {
    const int pr = (int)(q % (kStripCells / 2));
    const long long st = q / (kStripCells / 2);
    const int lane = pr & 31, row = pr >> 5;
    const int s = (int)(st % g.nsteps);
    const int strip = (int)(st / g.nsteps) % kStrips, tile = (int)(st / g.nsteps) / kStrips;
    const int ti = lane % kLanesI, tj = lane / kLanesI;
    const int i = (tile % g.ntx) * kTileI + 2 * ti, j = (tile / g.ntx) * kTileJ + strip * kStripJ + 2 * tj + row;
    double2* out = reinterpret_cast<double2*>(dst + st * coef_bytes<UP, double>()) + pr;
    const long long r0 = walk_row<UP>(g, i, j, s - ti - tj), r1 = walk_row<UP>(g, i + 1, j, s - ti - tj);
#pragma unroll
    for (int a = 0; a < 3; ++a)
      out[a * (kStripCells / 2)] = make_double2(r0 >= 0 ? band[a][r0] : 0.0, r1 >= 0 ? band[a][r1] : 0.0);
    if (UP) {
      const double p0 = r0 >= 0 ? b.P[r0] : 1.0, p1 = r1 >= 0 ? b.P[r1] : 1.0;
      out[3 * (kStripCells / 2)] = make_double2(Recip<double>::of(p0), Recip<double>::of(p1));
      out[4 * (kStripCells / 2)] = make_double2(p0, p1);
    }
  }
}

// FP32 coefficients: the FP64 ones rounded (bands, pivots), the reciprocal
// in FP64 from the rounded pivot.
template <bool UP>
__global__ void k_walk_pack32(long long steps, const unsigned char* __restrict__ src, unsigned char* __restrict__ dst) {
  constexpr int kP = kStripCells / 2;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < steps * kP; q += (long long)gridDim.x * blockDim.x) {
    const int pr = (int)(q % kP);
    const long long st = q / kP;
    const double2* in = reinterpret_cast<const double2*>(src + st * coef_bytes<UP, double>()) + pr;
    unsigned char* o = dst + st * coef_bytes<UP, float>();
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double2 v = in[a * kP];
      reinterpret_cast<float2*>(o)[a * kP + pr] = make_float2((float)v.x, (float)v.y);
    }
    if (UP) {
      const double2 p = in[4 * kP];
      reinterpret_cast<double2*>(o + 3 * kP * sizeof(float2))[pr] =
          make_double2(Recip<float>::of((float)p.x), Recip<float>::of((float)p.y));
    }
  }
}

// Shared memory of one sweep's CTA (byte offsets).
template <bool UP, class T>
struct WalkSmem {
  static constexpr int kCellBytes = kStripCells * (int)sizeof(T);                 // one step's cells of a strip
  static constexpr int coef = 0;                                                  // [strip][kDepth][coef_bytes]
  static constexpr int in = coef + kStrips * kDepth * coef_bytes<UP, T>();        // [strip][kInRing][cells]
  static constexpr int out = in + kStrips * kInRing * kCellBytes;                 // [strip][kOutRing][cells]
  static constexpr int jslot = out + kStrips * kOutRing * kCellBytes;             // [strip][kSlots][16]
  static constexpr int islot = jslot + kStrips * kSlots * kTileI * (int)sizeof(T);  // [kSlots][16]
  static constexpr int mbar = islot + kSlots * kTileJ * (int)sizeof(T);           // [strip][kDepth / 2]
  static constexpr int done = mbar + kStrips * kDepth / 2 * 8;                        // [strip] last finished step
  static constexpr int outdone = done + kStrips * 4;                              // [strip] last plane written out
  static constexpr int tile = outdone + kStrips * 4;
  static constexpr int always = tile + 4;                                         // a counter that is never behind
  static constexpr int total = tile + 16;
};
// Where a cell of a strip (column c, row r) lives among a step's cells: pairs
// along i, lane by lane, the lanes' lower rows first.
__device__ __forceinline__ int cell_word(int c, int r) { return (((r & 1) * 32 + (r >> 1) * kLanesI + (c >> 1)) << 1) + (c & 1); }

// One triangular sweep.  UP = false: forward sweep x_i = y_i - sum_{k<dcol}
// l_ik x_k (solveL, ILU0Preconditioner.h:181-198).  UP = true: backward sweep
// x_i = (y_i - sum_{k>dcol} u_ik x_k) / u_ii (solveU, :200-231), in mirrored
// coordinates.  src and dst in natural order (different vectors); hi / hj: the
// hand-over words of every tile's last column / last row, [tile][plane][16], at
// the sentinel before and after.
template <bool UP, class T>
__global__ void __launch_bounds__(kWalkWarps * 32, 1)
    k_walk_sweep(Walk g, const unsigned char* __restrict__ coef, const T* __restrict__ src, T* __restrict__ dst,
                 T* __restrict__ hi, T* __restrict__ hj, unsigned int* tickets, int* err) {
  using S = WalkSmem<UP, T>;
  using R = typename Recip<T>::type;
  constexpr int kCoef = coef_bytes<UP, T>();
  constexpr int kT = (int)sizeof(T);
  extern __shared__ __align__(128) unsigned char walk_smem[];
  const unsigned sm = smem_addr(walk_smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    sts_int(sm + S::tile, (int)atomicAdd(tickets + (UP ? 2 : 1), 1u));
    sts_int(sm + S::always, 0x7FFFFFFF);
    for (int w = 0; w < kStrips; ++w) {
      sts_int(sm + S::done + 4 * w, -1);
      sts_int(sm + S::outdone + 4 * w, -1);
      for (int q = 0; q < kDepth / 2; ++q) mbar_init(sm + S::mbar + (w * kDepth / 2 + q) * 8, 33);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int q = threadIdx.x; q < kStrips * kInRing * kStripCells; q += blockDim.x) sts1(sm + S::in + q * kT, T(1));
  for (int q = threadIdx.x; q < (kStrips * kTileI + kTileJ) * kSlots; q += blockDim.x)
    sts1(sm + S::jslot + q * kT, sentinel_of<T>());
  __syncthreads();
  const int tile = lds_int(sm + S::tile);
  const int tx = tile % g.ntx, ty = tile / g.ntx;
  const int nsteps = g.nsteps, nz = g.nz;
  // A strip without any line in the grid has nothing to do (and feeds none).
  const int strips = min(kStrips, (g.ny - ty * kTileJ + kStripJ - 1) / kStripJ);
  // Hand the other sweep its ticket back (it does not run concurrently).
  if (blockIdx.x == 0 && threadIdx.x == 0) tickets[UP ? 1 : 2] = 0u;

  const WarpRole me = warp_role(warp);
  if (me.role == Role::Compute) {
    // ---------------------------------------------------------------- compute
    const int w = me.strip;
    if (w >= strips) return;
    const int ti = lane % kLanesI, tj = lane / kLanesI, d = ti + tj;
    const int slot_i = ti == 0 && tx > 0;              // left values from islot
    const int slot_j = tj == 0 && (w > 0 || ty > 0);   // lower values from jslot
    const int feed_i = ti == kLanesI - 1 && tx + 1 < g.ntx;
    const int feed_w = tj == kLanesJ - 1 && w + 1 < strips;
    const int feed_j = tj == kLanesJ - 1 && w == kStrips - 1 && ty + 1 < g.nty;
    // Shared addresses.  All rings are indexed by this strip's step, the same for
    // every lane: a lane's share of plane k is at step k + d.
    const unsigned a_coef = sm + S::coef + w * kDepth * kCoef + lane * 2 * kT;
    const unsigned a_recip = sm + S::coef + w * kDepth * kCoef + 6 * 64 * kT + lane * 2 * (int)sizeof(R);
    const unsigned a_mbar = sm + S::mbar + w * (kDepth / 2) * 8;
    const unsigned a_in = sm + S::in + w * kInRing * S::kCellBytes + lane * 2 * kT;
    const unsigned a_out = sm + S::out + w * kOutRing * S::kCellBytes + lane * 2 * kT;
    const unsigned a_i = sm + S::islot + (w * kStripJ + 2 * tj) * kT;
    const unsigned a_j = sm + S::jslot + (w * kSlots * kTileI + 2 * ti) * kT;
    const unsigned a_next = a_j + kSlots * kTileI * kT;
    const unsigned a_done = sm + S::done + 4 * w, a_outdone = sm + S::outdone + 4 * w;
    const unsigned a_room = sm + (w + 1 < strips ? S::done + 4 * (w + 1) : S::always);
    T* p_hi = hi + ((long long)tile * g.halo + kSkew - d) * kTileJ + w * kStripJ + 2 * tj;
    T* p_hj = hj + ((long long)tile * g.halo + kSkew - d) * kTileI + 2 * ti;

    struct In {
      T y[4], a[3][4], p[4];
      R r[4];
    };
    // Ring positions of the current pair of steps; odd steps are an immediate
    // offset further (the rings have even sizes).
    unsigned f_coef = 0, f_in = 0, o_out = 0;
    auto fetch = [&](In& c, unsigned off_coef, unsigned off_in) {
      const unsigned a = a_coef + f_coef + off_coef, y = a_in + f_in + off_in;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        ldw2(y + h * 64 * kT, c.y[2 * h], c.y[2 * h + 1]);
#pragma unroll
        for (int b = 0; b < 3; ++b) ldw2(a + (b * 2 + h) * 64 * kT, c.a[b][2 * h], c.a[b][2 * h + 1]);
        if constexpr (UP) {
          ldw2(a_recip + f_coef + off_coef + h * 64 * (int)sizeof(R), c.r[2 * h], c.r[2 * h + 1]);
          if constexpr (Recip<T>::keep_pivot) ldw2(a + (8 + h) * 64 * kT, c.p[2 * h], c.p[2 * h + 1]);
        }
      }
    };

    // What a step waits for -- its hand-over words and, in an odd step, the
    // inputs of the pair after it -- is read and voted on during the step before
    // it, so that in the steady state no load, vote or branch stands between a
    // step's arithmetic and the previous one's.
    T v[4] = {T(0), T(0), T(0), T(0)};             // the previous step's cells
    T l0 = T(0), l1 = T(0), b0 = T(0), b1 = T(0);  // the next step's hand-over words
    unsigned m_next = a_mbar, m_par = 0;           // the next pair's mbarrier
    bool ok = true, go = false;
    auto look = [&](int s, auto odd) {  // the state of what step s waits for
      const unsigned so = (unsigned)(s & (kSlots - 1)) * kTileI * kT;
      lds2_if(slot_i, a_i + so, l0, l1);
      lds2_if(slot_j, a_j + so, b0, b1);
      if constexpr (decltype(odd)::value) ok = mbar_test(m_next, m_par) || s + 1 >= nsteps;
    };
    auto ready = [&]() { return ok && !(waiting(l0) | waiting(l1) | waiting(b0) | waiting(b1)); };
    auto step = [&](int s, In& c, In& nxt, auto odd) {
      constexpr bool kOdd = decltype(odd)::value;
      using Odd = std::bool_constant<kOdd>;
      using NotOdd = std::bool_constant<!kOdd>;
      const unsigned so = (unsigned)(s & (kSlots - 1)) * kTileI * kT;
      const T sl0 = __shfl_up_sync(0xffffffffu, v[1], 1), sl1 = __shfl_up_sync(0xffffffffu, v[3], 1);
      const T sb0 = __shfl_up_sync(0xffffffffu, v[2], kLanesI), sb1 = __shfl_up_sync(0xffffffffu, v[3], kLanesI);
      if (!go) {
        const long long t0 = clock64();
        for (unsigned it = 1;; ++it) {
          look(s, Odd());
          if (__all_sync(0xffffffffu, ready())) break;
          if (__any_sync(0xffffffffu, give_up(it, t0, err))) {  // quiet NaNs from here on
            l0 = l1 = b0 = b1 = quiet_nan<T>();
            break;
          }
        }
      }
      const T xl0 = ti > 0 ? sl0 : l0, xl1 = ti > 0 ? sl1 : l1, xb0 = tj > 0 ? sb0 : b0, xb1 = tj > 0 ? sb1 : b1;
      if constexpr (!kOdd) {
        fetch(nxt, kCoef, S::kCellBytes);
      } else {  // on to the next pair
        f_coef += 2 * kCoef;
        f_in += 2 * S::kCellBytes;
        const bool wrap = f_coef == kDepth * kCoef;
        f_coef = wrap ? 0u : f_coef;
        m_next = wrap ? a_mbar + 8 : m_next + 8;
        f_in = f_in == kInRing * S::kCellBytes ? 0u : f_in;
        fetch(nxt, 0, 0);
        if (m_next == a_mbar + kDepth / 2 * 8) {
          m_next = a_mbar;
          m_par ^= 1u;
        }
      }
      sts2_if(slot_i, a_i + so, sentinel_of<T>(), sentinel_of<T>());
      sts2_if(slot_j, a_j + so, sentinel_of<T>(), sentinel_of<T>());
      look(s + 1, NotOdd());
      if constexpr (!UP) {  // columns ascending: -k, -j, -i
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = mul_sub_rn(c.a[0][q], v[q], c.y[q]);
        v[0] = mul_sub_rn(c.a[2][0], xl0, mul_sub_rn(c.a[1][0], xb0, v[0]));
        v[1] = mul_sub_rn(c.a[2][1], v[0], mul_sub_rn(c.a[1][1], xb1, v[1]));
        v[2] = mul_sub_rn(c.a[2][2], xl1, mul_sub_rn(c.a[1][2], v[0], v[2]));
        v[3] = mul_sub_rn(c.a[2][3], v[2], mul_sub_rn(c.a[1][3], v[1], v[3]));
      } else {  // columns ascending: +i, +j, +k
        T m[4], n[4];
        bool bad[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) m[q] = mul_rn(c.a[2][q], v[q]);
        auto num = [&](int q, T xi, T xj) {
          return sub_rn(mul_sub_rn(c.a[1][q], xj, mul_sub_rn(c.a[0][q], xi, c.y[q])), m[q]);
        };
        n[0] = Recip<T>::div(num(0, xl0, xb0), c.p[0], c.r[0], bad[0]);
        n[1] = Recip<T>::div(num(1, n[0], xb1), c.p[1], c.r[1], bad[1]);
        n[2] = Recip<T>::div(num(2, xl1, n[0]), c.p[2], c.r[2], bad[2]);
        n[3] = Recip<T>::div(num(3, n[2], n[1]), c.p[3], c.r[3], bad[3]);
        if (__any_sync(0xffffffffu, bad[0] | bad[1] | bad[2] | bad[3])) {
          // A dividend of +0 over a positive pivot in range has come out as the division's
          // +0 (empty regions of a right-hand side are full of them); with anything else
          // among the bad ones, the step again with plain divisions.
          auto zero = [&](int q, T x) { return x == T(0) && !sign_bit(x) && c.r[q] > R(0); };
          const bool hard = (bad[0] && !zero(0, num(0, xl0, xb0))) | (bad[1] && !zero(1, num(1, n[0], xb1))) |
                            (bad[2] && !zero(2, num(2, xl1, n[0]))) | (bad[3] && !zero(3, num(3, n[2], n[1])));
          if (__any_sync(0xffffffffu, hard)) {
            n[0] = Recip<T>::slow(num(0, xl0, xb0), c.p[0], c.r[0]);
            n[1] = Recip<T>::slow(num(1, n[0], xb1), c.p[1], c.r[1]);
            n[2] = Recip<T>::slow(num(2, xl1, n[0]), c.p[2], c.r[2]);
            n[3] = Recip<T>::slow(num(3, n[2], n[1]), c.p[3], c.r[3]);
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = n[q];
      }
      // (results of arithmetic are never the sentinel, a signalling NaN)
      st_flag2_if(feed_i, p_hi + (kOdd ? kTileJ : 0), v[1], v[3]);
      st_flag2_if(feed_j, p_hj + (kOdd ? kTileI : 0), v[2], v[3]);
      // the next strip's step: this one less the lanes between (before its first step there is none)
      const int fs = s - (kLanesJ - 1);
      sts2_if(fs >= 0 ? feed_w : 0, a_next + (unsigned)(fs & (kSlots - 1)) * kTileI * kT, v[2], v[3]);
      stw2(a_out + o_out + (kOdd ? S::kCellBytes : 0), v[0], v[1]);
      stw2(a_out + o_out + (kOdd ? S::kCellBytes : 0) + 64 * kT, v[2], v[3]);
      go = __all_sync(0xffffffffu, ready());
      if constexpr (kOdd) {
        p_hi += 2 * kTileJ;
        p_hj += 2 * kTileI;
        o_out = o_out + 2 * S::kCellBytes == kOutRing * S::kCellBytes ? 0u : o_out + 2 * S::kCellBytes;
        sts_int_if(lane == 0, a_done, s);
      }
    };
    In c0, c1;
    if (!mbar_test(m_next, 0)) mbar_wait(m_next, 0, err);
    m_next += 8;
    fetch(c0, 0, 0);
    for (int s = 0; s < nsteps; s += 2) {  // two buffers of inputs, no moves between them
      if ((s & 7) == 0) {
        // room for the next eight steps: in the ring of output cells (step s + 7
        // overwrites step s + 7 - kOutRing, whose cells are of planes up to that
        // number) and in the next strip's slots (step s + 4 at most)
        if (lds_int(a_outdone) < s + 7 - kOutRing) wait_count(a_outdone, min(s + 7 - kOutRing, nz - 1), err);
        if (lds_int(a_room) < s + 4 - kSlots) wait_count(a_room, s + 4 - kSlots, err);
        __syncwarp();
      }
      step(s, c0, c1, std::false_type());
      step(s + 1, c1, c0, std::true_type());
    }
    // the next strip's last steps have no values to wait for
    if (w + 1 < strips) {
      wait_count(a_room, nsteps - 1 - kSlots, err);
      for (int t = nsteps - (kLanesJ - 1); t < nsteps; ++t)
        sts2_if(feed_w, a_next + (unsigned)(t & (kSlots - 1)) * kTileI * kT, T(1), T(1));
    }
  } else if (me.role == Role::Poll) {
    // ---------------------------------------------------------------- hand-overs from other tiles
    // Warps 0 and 2: the columns of the tile's first row; 1 and 3: the rows of its
    // first column.  A side's four half-warps take the steps in turn, a word a
    // lane, kPollDepth of them at once; a step whose plane is outside the grid
    // gets a 1 (its coefficients are 0).  Several warps with little to do in a
    // round, because a round is a trip to L2 and every instruction in it is
    // latency on the next tile's critical path.
    const bool jside = (me.part & 1) == 0;
    const int q = lane & 15;  // column, resp. row
    const int w = jside ? 0 : q / kStripJ;
    const bool need = jside ? ty > 0 : tx > 0 && w < strips;
    const int d = jside ? q / 2 : q % kStripJ / 2;  // the using lane's skew: plane k is its step k + d
    T* p = (jside ? hj + (long long)(tile - g.ntx) * g.halo * kTileI : hi + (long long)(tile - 1) * g.halo * kTileJ) + q +
           (kSkew - d) * 16;
    const unsigned slot = sm + (jside ? S::jslot : S::islot) + q * kT;
    const unsigned a_done = sm + S::done + 4 * w;
    const int phase = (me.part >> 1) * 2 + (lane >> 4);
    int x[kPollDepth];  // the steps this lane waits for, each on its own
#pragma unroll
    for (int u = 0; u < kPollDepth; ++u) x[u] = need ? phase + 4 * u : nsteps;
    unsigned it = 0;
    long long t0 = clock64();
    for (;;) {
      const int lim = min(nsteps, lds_int(a_done) + kSlots + 1);  // a slot is free once its previous step is done
      T v[kPollDepth];
#pragma unroll
      for (int u = 0; u < kPollDepth; ++u) {
        v[u] = T(1);
        if (x[u] < lim && (unsigned)(x[u] - d) < (unsigned)nz) v[u] = ld_relaxed(p + (long long)x[u] * 16);
      }
      bool some = false, left = false;
#pragma unroll
      for (int u = 0; u < kPollDepth; ++u) {
        if (x[u] < lim && !waiting(v[u])) {
          sts1(slot + (unsigned)(x[u] & (kSlots - 1)) * 16 * kT, v[u]);
          p[(long long)x[u] * 16] = sentinel_of<T>();  // ready for the next application
          x[u] += 4 * kPollDepth;
          some = true;
        }
        left |= x[u] < nsteps;
      }
      if (!__any_sync(0xffffffffu, left)) break;
      if (__any_sync(0xffffffffu, some)) {
        it = 0;
      } else if ((++it & 15) == 0) {  // (the same count in every lane)
        if (it == 16) t0 = clock64();
        if (__any_sync(0xffffffffu, give_up(0, t0, err))) break;  // the compute warps' own waits end the same way
      }
    }
  } else if (me.role == Role::Load) {
    // ---------------------------------------------------------------- inputs
    // Two steps' coefficients (one bulk copy) and two planes of src, up to kDepth
    // steps ahead of the compute warp, on one mbarrier; every other pair of
    // steps.  A lane copies column lane & 15 of rows (lane >> 4) + 2 q, each
    // word to its step's cells.  Words outside the grid are left at 1.
    const int w = me.strip, first = me.part;
    if (w >= strips) return;
    const unsigned char* cf = coef + (((long long)tile * kStrips + w) * nsteps + 2 * first) * kCoef;
    const unsigned a_done = sm + S::done + 4 * w, a_mbar = sm + S::mbar + w * (kDepth / 2) * 8;
    const unsigned a_cf = sm + S::coef + w * kDepth * kCoef;
    const unsigned ring = sm + S::in + w * kInRing * S::kCellBytes, ring_end = ring + kInRing * S::kCellBytes;
    const int col = lane & 15, row0 = lane >> 4;
    const long long dz = UP ? -g.nxny : g.nxny;
    const T* from[4];
    unsigned to[4];
    bool in[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const long long r = walk_row<UP>(g, tx * kTileI + col, ty * kTileJ + w * kStripJ + row0 + 2 * q, 0);
      in[q] = r >= 0;
      from[q] = src + (in[q] ? r + 2 * first * dz : 0);
      to[q] = ring + (unsigned)(2 * first + (col >> 1) + q) * S::kCellBytes + cell_word(col, row0 + 2 * q) * kT;
    }
    int s = 2 * first, seen = -1;
    unsigned slot = first;
    for (; s < nsteps; s += 4) {
      if (seen < s + 1 - kDepth) {
        seen = lds_int(a_done);
        if (seen < s + 1 - kDepth) {
          if (!wait_count(a_done, s + 1 - kDepth, err)) break;
          seen = s + 1 - kDepth;
        }
        __syncwarp();
      }
      const unsigned mb = a_mbar + slot * 8;
      if (lane == 0) {
        mbar_expect_tx(mb, 2 * kCoef);
        bulk_load(a_cf + slot * 2 * kCoef, cf, 2 * kCoef, mb);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (s + u < nz) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (in[q]) copy_word<kT>(to[q], from[q] + u * dz);
            to[q] += S::kCellBytes;
            to[q] -= to[q] >= ring_end ? kInRing * S::kCellBytes : 0;
          }
        }
      }
      copy_arrive(mb);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        from[q] += 4 * dz;
        to[q] += 2 * S::kCellBytes;
        to[q] -= to[q] >= ring_end ? kInRing * S::kCellBytes : 0;
      }
      cf += 4 * kCoef;
      slot = slot + 2 >= kDepth / 2 ? first : slot + 2;
    }
    // Copies in flight land before the CTA may leave (also after a failure).
    copy_wait_all();
    __syncwarp();
    if (lane == 0)
      for (int x = s - kDepth; x < s; x += 4)
        if (x >= 0 && !mbar_drain(a_mbar + (x % kDepth) / 2 * 8, (x / kDepth) & 1)) break;
  } else if (me.role == Role::Store) {
    // ---------------------------------------------------------------- outputs
    // Two planes at a time, once the second one's last lane's step is done.
    const int w = me.strip;
    if (w >= strips) return;
    const int col = lane & 15, row0 = lane >> 4;
    const unsigned ring = sm + S::out + w * kOutRing * S::kCellBytes, ring_end = ring + kOutRing * S::kCellBytes;
    const unsigned a_done = sm + S::done + 4 * w, a_outdone = sm + S::outdone + 4 * w;
    const long long dz = UP ? -g.nxny : g.nxny;
    T* to[4];
    unsigned from[4];
    bool in[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const long long r = walk_row<UP>(g, tx * kTileI + col, ty * kTileJ + w * kStripJ + row0 + 2 * q, 0);
      in[q] = r >= 0;
      to[q] = dst + (in[q] ? r : 0);
      from[q] = ring + (unsigned)((col >> 1) + q) * S::kCellBytes + cell_word(col, row0 + 2 * q) * kT;
    }
    int seen = -1;
    for (int k = 0; k < nz; k += 2) {
      const int last = min(k + 1 + kSkew, nsteps - 1);
      if (seen < last) {
        seen = lds_int(a_done);
        if (seen < last) {
          if (!wait_count(a_done, last, err)) return;
          seen = last;
        }
        __syncwarp();
      }
      T v[2][4];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          lds1(from[q], v[u][q]);
          from[q] += S::kCellBytes;
          from[q] -= from[q] >= ring_end ? kOutRing * S::kCellBytes : 0;
        }
      sts_int_if(lane == 0, a_outdone, k + 1);  // (read: the slots may be written again)
      const bool two = k + 1 < nz;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (in[q]) *to[q] = v[0][q];
        if (in[q] && two) *(to[q] + dz) = v[1][q];
        to[q] += 2 * dz;
      }
    }
  }
}

Geom geom_of(const Ilu0Data& d) {
  Geom g;
  g.nx = d.st_nx;
  g.ny = d.st_ny;
  g.nz = d.st_nz;
  g.ntx = (g.nx + kTile - 1) / kTile;
  g.nty = (g.ny + kTile - 1) / kTile;
  g.nxny = (long long)g.nx * g.ny;
  return g;
}

Walk walk_of(const Ilu0Data& d) {
  const Geom g = geom_of(d);
  Walk w;
  w.nx = g.nx;
  w.ny = g.ny;
  w.nz = g.nz;
  w.ntx = (g.nx + kTileI - 1) / kTileI;
  w.nty = (g.ny + kTileJ - 1) / kTileJ;
  w.nsteps = (g.nz + kSkew + 1) / 2 * 2;
  w.halo = w.nsteps + kSkew;
  w.nxny = g.nxny;
  w.n = g.nxny * g.nz;
  return w;
}

Bands bands_of(double* p, int n) {
  const size_t m = (size_t)n;
  return Bands{p, p + m, p + 2 * m, p + 3 * m, p + 4 * m, p + 5 * m, p + 6 * m, p + 7 * m};
}

int wave_grid(ab2_context* ctx, int ntiles) { return std::max(1, std::min(ntiles, ctx->num_sms * 2)); }

int bulk_grid(ab2_context* ctx, long long n) {
  return (int)std::max(1LL, std::min((n + kThreads - 1) / kThreads, (long long)ctx->num_sms * 16));
}

template <class T>
void set_walk_smem() {
  AB2_CUDA(cudaFuncSetAttribute(k_walk_sweep<false, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                WalkSmem<false, T>::total));
  AB2_CUDA(cudaFuncSetAttribute(k_walk_sweep<true, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                WalkSmem<true, T>::total));
}

// One sweep (UP: the backward one); base: the precision's arrays.
template <bool UP, class T>
void walk_sweep(ab2_context* ctx, const Ilu0Data& d, const Walk& w, unsigned char* base, const T* src, T* dst) {
  const WalkMem m = walk_mem<T>(w);
  T* hi = reinterpret_cast<T*>(base + (UP ? m.halo_u : m.halo_l));
  T* hj = hi + (long long)w.ntx * w.nty * w.halo * kTileJ;
  k_walk_sweep<UP, T><<<w.ntx * w.nty, kWalkWarps * 32, WalkSmem<UP, T>::total, ctx->stream>>>(
      w, base + (UP ? m.coef_u : m.coef_l), src, dst, hi, hj, d.d_tile_tickets, d.d_err);
  check_launch(ctx, UP ? "walk_usweep" : "walk_lsweep");
}

// The hand-over words of both sweeps at the sentinel.
void fill_halo(ab2_context* ctx, const Walk& w, double* base) {
  const WalkMem m = walk_mem<double>(w);
  k_fill_bits<<<bulk_grid(ctx, 2 * m.halo_words), kThreads, 0, ctx->stream>>>(2 * m.halo_words, kSentinel,
                                                                              base + m.halo_l / 8);
  check_launch(ctx, "walk_fill");
}
void fill_halo(ab2_context* ctx, const Walk& w, float* base) {
  const WalkMem m = walk_mem<float>(w);
  k_fill_bits32<<<bulk_grid(ctx, 2 * m.halo_words), kThreads, 0, ctx->stream>>>(2 * m.halo_words, kSentinel32,
                                                                                base + m.halo_l / 4);
  check_launch(ctx, "walk_fill32");
}

}  // namespace

bool ilu_stencil_setup(ab2_context* ctx, const ab2_matrix* A, Ilu0Data& d, bool factored, int schedule) {
  const int n = A->n;
  if (n == 0) return false;
  // The 7-point geometry: kept by the matrix (AB2_FMT_STENCIL) or checked here.
  int nx = A->st_nx, ny = A->st_ny, nz = A->st_nz;
  if (nx == 0 && !stencil_geometry(ctx, A, &nx, &ny, &nz)) return false;
  d.walk_cluster = schedule != AB2_ILU_STENCIL && nz <= kClusterPlanes;
  require(schedule != AB2_ILU_STENCIL_CLUSTER || d.walk_cluster,
          "ILU0 cluster schedule requested with more planes along z than it is offered for");
  d.st_nx = nx;
  d.st_ny = ny;
  d.st_nz = nz;
  const Geom g = geom_of(d);

  // Factorisation on natural-order bands.
  d.d_bands = dev_alloc<double>(ctx, (size_t)n * 8);
  d.d_tile_tickets = dev_alloc<unsigned int>(ctx, 3);
  AB2_CUDA(cudaMemsetAsync(d.d_tile_tickets, 0, 3 * sizeof(unsigned int), ctx->stream));
  const Bands b = bands_of(d.d_bands, n);
  if (factored) {
    // d_lu holds the factor: its diagonal is the pivot band.
    k_stencil_extract<<<grid_for(n), kThreads, 0, ctx->stream>>>(n, g, A->d_rp, d.d_lu, b);
    check_launch(ctx, "stencil_extract");
    AB2_CUDA(cudaMemcpyAsync(b.P, b.D, sizeof(double) * (size_t)n, cudaMemcpyDeviceToDevice, ctx->stream));
  } else {
    k_stencil_extract<<<grid_for(n), kThreads, 0, ctx->stream>>>(n, g, A->d_rp, A->d_v, b);
    check_launch(ctx, "stencil_extract");
    k_fill_bits<<<grid_for(n), kThreads, 0, ctx->stream>>>(n, kSentinel, b.P);
    check_launch(ctx, "stencil_fill");
    k_stencil_factor<<<wave_grid(ctx, g.ntx * g.nty), kTileThreads, 0, ctx->stream>>>(g, b, d.d_tile_tickets,
                                                                                         d.d_err);
    check_launch(ctx, "stencil_factor");
    k_stencil_pack<<<grid_for(n), kThreads, 0, ctx->stream>>>(n, g, A->d_rp, b, d.d_lu);
    check_launch(ctx, "stencil_pack");
  }

  // The sweeps' arrays.
  const Walk w = walk_of(d);
  const WalkMem m = walk_mem<double>(w);
  d.d_walk = dev_alloc<double>(ctx, (size_t)(m.total + 7) / 8);
  unsigned char* base = reinterpret_cast<unsigned char*>(d.d_walk);
  const long long pairs = (long long)w.ntx * w.nty * kStrips * w.nsteps * (kStripCells / 2);
  k_walk_pack<false><<<bulk_grid(ctx, pairs), kThreads, 0, ctx->stream>>>(w, b, base + m.coef_l);
  check_launch(ctx, "walk_pack");
  k_walk_pack<true><<<bulk_grid(ctx, pairs), kThreads, 0, ctx->stream>>>(w, b, base + m.coef_u);
  check_launch(ctx, "walk_pack");
  fill_halo(ctx, w, d.d_walk);
  AB2_CUDA(cudaStreamSynchronize(ctx->stream));
  dev_free(ctx, d.d_bands);
  d.d_bands = nullptr;
  set_walk_smem<double>();
  d.stencil = true;
  d.levels_l = d.levels_u = (int)(nx + ny + nz - 2);
  return true;
}

namespace {

template <class T>
void walk_apply(ab2_context* ctx, const Ilu0Data& d, T* base, const T* y, T* z) {
  const Walk w = walk_of(d);
  unsigned char* mem = reinterpret_cast<unsigned char*>(base);
  T* tmp = reinterpret_cast<T*>(mem + walk_mem<T>(w).tmp);
  walk_sweep<false, T>(ctx, d, w, mem, y, tmp);
  walk_sweep<true, T>(ctx, d, w, mem, tmp, z);
}

}  // namespace

// y -> forward walk -> backward walk -> z (y and z may be the same vector).
void ilu_stencil_apply(ab2_context* ctx, const ab2_matrix* A, const Ilu0Data& d, const double* y, double* z) {
  (void)A;
  walk_apply(ctx, d, d.d_walk, y, z);
}

// FP32 walk arrays: the FP64 factor rounded to float.
void ilu_stencil_enable_f32(ab2_context* ctx, Ilu0Data& d) {
  if (d.d_walk32) return;
  const Walk w = walk_of(d);
  const WalkMem m = walk_mem<float>(w), m64 = walk_mem<double>(w);
  d.d_walk32 = dev_alloc<float>(ctx, (size_t)(m.total + 3) / 4);
  const unsigned char* from = reinterpret_cast<const unsigned char*>(d.d_walk);
  unsigned char* to = reinterpret_cast<unsigned char*>(d.d_walk32);
  const long long steps = (long long)w.ntx * w.nty * kStrips * w.nsteps;
  k_walk_pack32<false><<<bulk_grid(ctx, steps * 64), kThreads, 0, ctx->stream>>>(steps, from + m64.coef_l, to + m.coef_l);
  check_launch(ctx, "walk_pack32");
  k_walk_pack32<true><<<bulk_grid(ctx, steps * 64), kThreads, 0, ctx->stream>>>(steps, from + m64.coef_u, to + m.coef_u);
  check_launch(ctx, "walk_pack32");
  fill_halo(ctx, w, d.d_walk32);
  set_walk_smem<float>();
}

void ilu_stencil_apply_f32(ab2_context* ctx, const Ilu0Data& d, const float* y, float* z) {
  require(d.d_walk32 != nullptr, "FP32 ILU0 arrays not built");
  walk_apply(ctx, d, d.d_walk32, y, z);
}

// After a failed application: the hand-over words back to the sentinel (the
// tickets are reset by pc_reset).
void ilu_stencil_reset(ab2_context* ctx, const Ilu0Data& d) {
  const Walk w = walk_of(d);
  if (d.d_walk) fill_halo(ctx, w, d.d_walk);
  if (d.d_walk32) fill_halo(ctx, w, d.d_walk32);
}

}  // namespace ab2
