// Batched solver engine: BSR SpMV, block ILU(k) factorization, block
// triangular sweeps and restarted GMRES / iterative refinement over a batch
// of independent problems (a single problem is a batch of one).
//
// Reference: cusparseDbsrmv, cusparseDbsrilu02 and cusparseDbsrsv2_solve as
// called by examples/iterative/gmres.cu:374-771, and the GMRES loop there
// (left-preconditioned GMRES(m), MGS, host Givens; bugs fixed: dot length
// nvars, m+1 basis vectors, restarts).
//
// Batch layout: every problem keeps its own pattern / values / factor
// buffers; a device table of ProbDev descriptors gives each kernel the
// problem of a global block row (row_prob), its offset in the batch vector
// space and its triangular level structure.
//  * SpMV and the GMRES vector work run over all rows / chunks of the batch.
//  * A triangular sweep runs one CTA, or the CTAs of one cluster, per problem:
//    they walk the problem's levels, so a dependency costs a barrier between
//    warps (or an exchange within the cluster) instead of a device-wide round
//    trip; the problems of a batch run on different SMs at once.
//  * The factorization shares the SMs out over the problems; its rows wait for
//    one another through flags in global memory.
//
// GMRES reductions are segmented per problem over fixed 4096-entry chunks
// aligned to each problem's own vector, with per-problem Arnoldi states, so
// a problem's iterates are bitwise identical alone and inside any batch.
#include <algorithm>
#include <atomic>
#include <array>
#include <chrono>
#include <cmath>
#include <cstring>
#include <mutex>
#include <numeric>
#include <thread>
#include <type_traits>

#include "gf_internal.h"

namespace gf {

enum { ST_TIMEOUT = 1, ST_ZERO_PIVOT = 2, ST_NAN = 4 };
constexpr int kChunk = 4096;
constexpr int kRedThreads = 256;

struct SweepCtl {
  int status;
  int pivot;
  int gave_up, quiet;  // CTAs of split ring sweeps whose wait ran out; those of them that left
                       // with no store in flight to them
};

// ------------------------------------------------ barriers and bulk copies
constexpr unsigned long long kWaitNs = 2000000000ull;  // default bound of every device-side wait
constexpr int kSweepCta = 2;  // CTAs (one thread-block cluster) per problem for triangular work

// Bound (ns) of the waits that end when a bulk copy lands or when the
// partner CTA of a cluster arrives (gf_test_set_waits changes it). The waits
// that drain a CTA's own copies in flight before it leaves always use kWaitNs.
__device__ unsigned long long g_wait_ns = kWaitNs;
// Failure-injection knob for tests (gf_test_set_waits): when non-zero, CTA
// rank 1 of a split problem never arrives on its partner's meeting barriers,
// so the partner's bounded wait runs out and the launch reports ST_TIMEOUT.
// Every wait stays bounded and both CTAs still meet on the final cluster
// barrier, so nothing hangs.
__device__ int g_skip_meet = 0;

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// as mbar_try_wait, but the thread may be suspended (not spinning on issue
// slots) until the phase completes or about hint_ns have passed
__device__ __forceinline__ bool mbar_try_wait_sleep(uint64_t* bar, unsigned parity,
                                                    unsigned hint_ns) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}
// bounded wait; returns false if limit_ns passed first
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity,
                                          unsigned long long limit_ns) {
  // the timer is read only once the first test fails (reading it is slow)
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = gtimer();
  unsigned n = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++n & 255u) == 0u && gtimer() - t0 > limit_ns) return false;
  }
  return true;
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes,
                                         uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ unsigned cluster_map(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_store(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
// arrive on an mbarrier of another CTA of the cluster (releases this CTA's
// earlier writes at cluster scope)
__device__ __forceinline__ void mbar_arrive_remote(unsigned addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait with acquire at cluster scope; false if limit_ns passed first
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, unsigned parity,
                                                  unsigned long long limit_ns) {
  unsigned long long t0 = 0;
  unsigned n = 0;
  while (true) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    if (n == 0) t0 = gtimer();  // read only once the first test fails (reading it is slow)
    if ((++n & 255u) == 0u && gtimer() - t0 > limit_ns) return false;
  }
}
// all threads of all CTAs of the cluster
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" :::
                   "memory");
}


// ------------------------------------------------------------------ SpMV
// y = alpha A x + beta y over all rows of live problems; one warp per block
// row, 4 groups of 6 lanes (group g takes blocks g, g+4, ...), lane r of a
// group row r of a block. Bound by the latency of column -> x and by L1
// requests: a row of a block is read as three 16-byte pieces (FP32: 8-byte)
// instead of six values. 400x200 plate: 57 -> 49 us, 69 % of measured HBM
// (three blocks a lane in flight take 116 registers: 92 us).
__device__ __forceinline__ void row6(const double* a, double (&v)[6]) {
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const double2 t = __ldg(reinterpret_cast<const double2*>(a) + c);
    v[2 * c] = t.x, v[2 * c + 1] = t.y;
  }
}
__device__ __forceinline__ void row6(const float* a, double (&v)[6]) {
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const float2 t = __ldg(reinterpret_cast<const float2*>(a) + c);
    v[2 * c] = t.x, v[2 * c + 1] = t.y;
  }
}
template <class VT>
__global__ void __launch_bounds__(256)
    bspmv_kernel(int nrows, const int32_t* __restrict__ row_prob, const ProbDev* __restrict__ P,
                 const int* __restrict__ live, const double* __restrict__ x, double alpha,
                 double beta, double* __restrict__ y) {
  const int lane = threadIdx.x & 31;
  const int grow = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (grow >= nrows) return;
  const int p = row_prob[grow];
  if (live && !live[p]) return;
  const ProbDev& d = P[p];
  const int i = grow - d.off;
  const VT* A = sizeof(VT) == 8 ? (const VT*)d.A64 : (const VT*)d.A32;
  const double* xb = x + 6 * (size_t)d.off;
  const int g = lane / 6, r = lane % 6;
  double acc = 0.0;
  if (g < 4) {
    const int b0 = d.rowp[i], b1 = d.rowp[i + 1];
    const int32_t* cols = d.cols;
#pragma unroll 2
    for (int blk = b0 + g; blk < b1; blk += 4) {
      double a[6];
      const double* xx = xb + 6 * (size_t)__ldg(cols + blk);
      row6(A + 36 * (size_t)blk + 6 * r, a);
#pragma unroll
      for (int c = 0; c < 6; c++) acc = fma(a[c], __ldg(xx + c), acc);
    }
  }
  acc += __shfl_down_sync(0xffffffffu, acc, 12);
  acc += __shfl_down_sync(0xffffffffu, acc, 6);
  if (lane < 6) {
    double* yy = y + 6 * (size_t)grow + lane;
    *yy = (beta == 0.0) ? alpha * acc : alpha * acc + beta * (*yy);
  }
}

// ----------------------------------------------------- block ILU factorization
// Inverse of a 6x6 block by Gauss-Jordan elimination with row pivoting, in
// registers: lane j < 6 holds column j of the block, lane 6 + j column j of
// the identity (and of the inverse on return); the other lanes repeat them.
// Column c is broadcast once a step, every lane picks the pivot for itself.
__device__ __forceinline__ bool inv6_cols(double (&m)[6]) {
  bool ok = true;
#pragma unroll
  for (int c = 0; c < 6; c++) {
    double f[6];
#pragma unroll
    for (int r = 0; r < 6; r++) f[r] = __shfl_sync(0xffffffffu, m[r], c);
    // the reciprocal of the usual pivot, while the search runs
    double inv = 1.0 / f[c];
    int p = c;
    double best = fabs(f[c]);
#pragma unroll
    for (int r = c + 1; r < 6; r++) {
      const double v = fabs(f[r]);
      if (v > best) {
        best = v;
        p = r;
      }
    }
    ok = ok && best > 0.0 && isfinite(best);
    if (p != c) {  // the same for every lane, and rare
#pragma unroll
      for (int r = c + 1; r < 6; r++)
        if (p == r) {
          double t = m[c];
          m[c] = m[r];
          m[r] = t;
          t = f[c];
          f[c] = f[r];
          f[r] = t;
        }
      inv = 1.0 / f[c];
    }
    m[c] *= inv;
#pragma unroll
    for (int r = 0; r < 6; r++)
      if (r != c) m[r] = fma(-f[r], m[c], m[r]);
  }
  return ok;
}

// IKJ block ILU on each problem's ILU pattern (FP64, in place): lower blocks
// become L_ik = A_ik U_kk^{-1}, the diagonal block is replaced by U_ii^{-1}.
// One warp factors one row. The row's values are staged in the warp's slice
// of shared memory (rows up to kFacVals blocks; longer rows are updated in
// global memory), so the read-modify-writes of the sequential steps cost a
// shared-memory latency. Within a row the steps k (its lower blocks) are
// sequential; a step is L_ik = A_ik U_kk^{-1} and the updates A_ij -= L_ik U_kj
// over the blocks j of U(k) that the row has, on the FP64 tensor instruction
// m8n8k4: the 6x6 blocks are padded to 8 rows and 8 inner columns, four
// blocks fill three tiles of 8 columns, L_ik goes from one product to the
// next through shuffles and U(k) from L2 straight into the operands, all of
// its first 32 blocks in flight together. (As scalar multiply-adds a step
// took 920 instructions, which bounds batches, where every SM has rows to
// factor all the time. Eight warps with all registers beat twelve or sixteen
// whose loads come in two rounds or spill: an acquire drops the SM's L1.)
//
// Scheduling is dataflow, not level-synchronous: the warps of the CTAs a
// problem is given take its rows in factorization order (ascending lower
// level) from a per-problem counter, and step k of row i waits only until
// row k is final (its flag done[k] equals the launch's epoch, stored with
// release after row k's upper part). Rows of later levels therefore run
// while the rows they do not read are still being factored, and a row's
// early steps overlap the end of the rows it reads last. Every row that a
// warp waits for has a lower level, so it was taken earlier by a warp that
// is running; the waits end whatever the CTAs' residency. Each wait is still
// bounded: the first that runs out sets ST_TIMEOUT, which ends the others.
//
// The factorization lasts levels x the chain from one row's flag to the next
// row's: the flag becomes visible, U(k) and U_kk^{-1} arrive, one step, the
// inverse, the stores. Everything else is kept off that chain: the extents
// and columns of U(k) and the slots they update come from the pattern alone
// and are looked up a step ahead, before the wait; the wait polls one
// acquiring load (the limit is checked every 64th time); the inverse stays in
// registers; and the flag follows the upper part of the row at once (nobody
// reads the lower part in this launch), released by one lane. Clocks of that
// chain on a 256x128 plate, ILU(6): operands 1,150, updates 1,300, inverse
// 2,300, stores 640, release 970, the rest is the flag's way to the waiting
// warp. Alone, before -> now (B200): 256x128, ILU(6) 11.7 -> 6.2 ms; 61x37,
// ILU(8) 3.6 -> 2.0 ms; 256x256, ILU(12) 22.6 ms; the 64-plate batch 38 -> 30 ms.
constexpr int kFacWarps = 8;      // warps of a CTA
constexpr int kFacVals = 80;      // row blocks whose values are staged at most
constexpr int kFacSteps = 64;     // steps of a row that are staged
constexpr int kFacMap = 1024;     // column span of a row whose column -> slot map is kept
constexpr uint16_t kFacNone = 0xffff;  // map entry of a column that the row does not have
constexpr size_t kFacSmemMax = 226 * 1024;
// per warp: values of `vals` blocks and one more that padding reads, the
// steps, two lists of updates and the column map
__host__ __device__ constexpr size_t fac_warp_smem(int vals) {
  return sizeof(double) * 36 * ((size_t)vals + 1) + sizeof(int4) * kFacSteps + sizeof(int2) * 64 +
         sizeof(uint16_t) * kFacMap;
}
static_assert(kFacWarps * fac_warp_smem(kFacVals) <= kFacSmemMax, "the warps' rows fit a CTA");
// Whether the column -> slot map of a row from column c0 to column c1 is kept
// (otherwise every block of U(k) is searched for in the row's columns in global
// memory: 130x128 plate, complete factor, rows of 263 blocks, 390 ms searched,
// 271 ms mapped).
__host__ __device__ inline bool fac_mapped(int c0, int c1) { return c1 - c0 < kFacMap; }

__device__ __forceinline__ int find_col(const int32_t* c, int lo, int hi, int j) {
  const int end = hi;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (c[mid] < j)
      lo = mid + 1;
    else
      hi = mid;
  }
  return (lo < end && c[lo] == j) ? lo : -1;
}

__device__ __forceinline__ int ld_relaxed_gpu(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_gpu(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Waits (bounded) until *flag == want and acquires what its writer released.
// False when the bound ran out (ST_TIMEOUT set here) or another wait already
// ran out.
__device__ __forceinline__ bool wait_flag(const int* flag, int want, unsigned long long limit,
                                          SweepCtl* ctl) {
  unsigned long long t0 = 0;
  for (unsigned n = 0;; n++) {
    if (ld_acquire_gpu(flag) == want) return true;
    if ((n & 63u) == 63u) {
      if (t0 == 0) t0 = gtimer();
      if (ld_relaxed_gpu(&ctl->status) & ST_TIMEOUT) return false;
      if (gtimer() - t0 > limit) {
        atomicOr(&ctl->status, ST_TIMEOUT);
        return false;
      }
    }
  }
}

// c += A B, lane = 4 row + k of A (8x4), 4 column + k of B (4x8), 4 row +
// column / 2 of c (8x8): exact FP64 multiply-adds
__device__ __forceinline__ void mma_f64(double2& c, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c.x), "+d"(c.y)
      : "d"(a), "d"(b));
}

// A row's block values (STAGED: in the warp's shared memory, else in the
// factor itself).
template <bool STAGED>
struct RowValues {
  unsigned char* base;
  __device__ __forceinline__ double* at(int slot) const {
    return reinterpret_cast<double*>(base + 288u * (unsigned)slot);
  }
};

// The lower steps of one row (r0 its first block, nlow steps). False when a
// wait ran out.
template <bool STAGED>
__device__ __forceinline__ bool factor_row(const RowValues<STAGED> R, const int4* __restrict__ steps,
                                           int nlow, int len, const int4* sS, int2* sT,
                                           const uint16_t* sMap, int cbase, int span, bool mapped,
                                           const int32_t* __restrict__ cols,
                                           const int32_t* __restrict__ rcols, const double* LU,
                                           const int* done, int epoch, unsigned long long wlim,
                                           SweepCtl* ctl, int lane) {
  const int row = lane >> 2, q = lane & 3;  // tile row (column of B) and inner index
  // column 8 t + row of four blocks side by side is column co[t] of block
  // bo[t]; columns 8 t + 2 q and the next one belong to block bc[t]
  int bo[3], bc[3], cc[3];
  const double* LUt[3];
#pragma unroll
  for (int t = 0; t < 3; t++) {
    bo[t] = (8 * t + row) / 6;
    LUt[t] = LU + 6 * q + (8 * t + row) % 6;
    bc[t] = (8 * t + 2 * q) / 6;
    cc[t] = 6 * row + (8 * t + 2 * q) % 6;
  }
  const bool inner = q < 2, rows6 = row < 6;  // lanes with a second inner index / a block row
  // step t: {slot, k, first and end block of U(k)}
  auto step = [&](int t) { return t < kFacSteps ? sS[t] : __ldg(steps + t); };
  // Lists the updates of 32 blocks of U(k) from block jp0 on (the lane's
  // block has column j, -1: none), padded to a multiple of four; their number.
  auto list_updates = [&](int2* list, int j, int jp0, int slot_k) {
    int slot = -1;
    if (j >= 0) {
      if (mapped) {
        const int o = j - cbase;
        const uint16_t m = o < span ? sMap[o] : kFacNone;
        slot = m != kFacNone ? m : -1;
      } else {
        slot = find_col(rcols, slot_k + 1, len, j);
      }
    }
    const unsigned hit = __ballot_sync(0xffffffffu, slot >= 0);
    const int n = __popc(hit);
    if (slot >= 0) list[__popc(hit & ((1u << lane) - 1u))] = make_int2(9 * (jp0 + lane), slot);
    if (lane < ((4 - n) & 3)) list[n + lane] = make_int2(9 * (jp0 - 1), STAGED ? len : 0);
    return n;
  };
  double b0[24], b1[24];  // U(k) operands of eight groups of four blocks
#pragma unroll
  for (int t = 0; t < 24; t++) b0[t] = b1[t] = 0.0;
  auto load_groups = [&](const int2* list, int n) {
#pragma unroll
    for (int g = 0; g < 8; g++)
      if (4 * g < n)
#pragma unroll
        for (int t = 0; t < 3; t++) {
          const double* src = LUt[t] + 4 * (size_t)(unsigned)list[4 * g + bo[t]].x;
          b0[3 * g + t] = __ldcg(src);
          if (inner) b1[3 * g + t] = __ldcg(src + 24);
        }
  };
  auto update_groups = [&](const int2* list, int n, double l0, double l1) {
#pragma unroll
    for (int h = 0; h < 8; h += 2) {  // two groups at a time
      if (4 * h >= n) break;
      const bool two = 4 * (h + 1) < n;
      // the products of a block are summed by themselves and subtracted once:
      // one rounding a step at the size of A_ij
      double2 c[6], s[6];
      unsigned at[6];
#pragma unroll
      for (int t = 0; t < 6; t++) {
        c[t] = s[t] = make_double2(0.0, 0.0);
        if (t < 3 || two) {
          at[t] = 288u * (unsigned)list[4 * (h + t / 3) + bc[t % 3]].y + 8u * (unsigned)cc[t % 3];
          if (rows6) c[t] = *reinterpret_cast<double2*>(R.base + at[t]);
        }
      }
#pragma unroll
      for (int t = 0; t < 6; t++)
        if (t < 3 || two) mma_f64(s[t], l0, b0[3 * h + t]);
#pragma unroll
      for (int t = 0; t < 6; t++)
        if (t < 3 || two) mma_f64(s[t], l1, b1[3 * h + t]);
#pragma unroll
      for (int t = 0; t < 6; t++)
        if ((t < 3 || two) && rows6 && 4 * (h + t / 3) + bc[t % 3] < n)
          *reinterpret_cast<double2*>(R.base + at[t]) =
              make_double2(c[t].x - s[t].x, c[t].y - s[t].y);
    }
  };
  // this step and the updates of its first 32 blocks
  int nt = 0, cur = 0;
  int4 s0 = make_int4(0, 0, 0, 0);
  if (nlow > 0) {
    s0 = step(0);
    nt = list_updates(sT, s0.z + lane < s0.w ? __ldg(cols + s0.z + lane) : -1, s0.z, s0.x);
  }
  __syncwarp();
  unsigned ready = 0;  // bit z: the row of step (window start + z) is final
  for (int st = 0; st < nlow; st++) {
    if ((st & 31) == 0) {
      // the flags of the next 32 steps, one per lane; a lane that sees its
      // row final acquires it for the warp (the warp barrier below orders
      // that acquire before every lane's later loads)
      const int f = st + lane < nlow ? (ld_acquire_gpu(done + step(st + lane).y) == epoch) : 1;
      ready = __ballot_sync(0xffffffffu, f);
      __syncwarp();
    }
    // the next step's columns, in flight during this one
    int jn = -1;
    int4 s1 = s0;
    if (st + 1 < nlow) {
      s1 = step(st + 1);
      if (s1.z + lane < s1.w) jn = __ldg(cols + s1.z + lane);
    }
    double* Aik = R.at(s0.x);
    const double a0 = rows6 ? Aik[6 * row + q] : 0.0;
    const double a1 = rows6 && inner ? Aik[6 * row + 4 + q] : 0.0;
    if (!((ready >> (st & 31)) & 1u)) {
      int ok = lane == 0 ? (int)wait_flag(done + s0.y, epoch, wlim, ctl) : 0;
      ok = __shfl_sync(0xffffffffu, ok, 0);
      __syncwarp();
      if (!ok) return false;
    }
    // U_kk^{-1} and up to 32 blocks of U(k), all in flight
    const double* Ukk = LU + 36 * (size_t)(s0.z - 1) + 6 * q + row;
    const double k0 = rows6 ? __ldcg(Ukk) : 0.0;
    const double k1 = rows6 && inner ? __ldcg(Ukk + 24) : 0.0;
    const int2* list = sT + 32 * cur;
    load_groups(list, nt);
    double2 l = make_double2(0.0, 0.0);
    mma_f64(l, a0, k0);
    mma_f64(l, a1, k1);
    if (rows6 && q < 3) *reinterpret_cast<double2*>(Aik + 6 * row + 2 * q) = l;
    // column q (and 4 + q) of L_ik for the updates
    const int quad = lane & ~3;
    const double x0 = __shfl_sync(0xffffffffu, l.x, quad + (q >> 1));
    const double y0 = __shfl_sync(0xffffffffu, l.y, quad + (q >> 1));
    const double x1 = __shfl_sync(0xffffffffu, l.x, quad + 2);
    const double y1 = __shfl_sync(0xffffffffu, l.y, quad + 2);
    const double l0 = (q & 1) ? y0 : x0, l1 = !inner ? 0.0 : (q & 1) ? y1 : x1;
    update_groups(list, nt, l0, l1);
    // the rest of U(k), beyond its first 32 blocks
    for (int jb = s0.z + 32; jb < s0.w; jb += 32) {
      __syncwarp();
      const int n = list_updates(sT + 32 * cur, jb + lane < s0.w ? __ldg(cols + jb + lane) : -1, jb, s0.x);
      __syncwarp();
      load_groups(list, n);
      update_groups(list, n, l0, l1);
    }
    cur ^= 1;
    nt = list_updates(sT + 32 * cur, jn, s1.z, s1.x);
    s0 = s1;
    __syncwarp();
  }
  return true;
}

// cta_prob[blockIdx.x]: the problem a CTA works on; grab[p]: problem p's row
// counter (zero at launch). vals: blocks of a row that are staged.
__global__ void __launch_bounds__(kFacWarps * 32)
    bfactor_df(const ProbDev* __restrict__ P, const int32_t* __restrict__ cta_prob,
               int* __restrict__ grab, int epoch, int vals, SweepCtl* ctl) {
  extern __shared__ __align__(16) unsigned char fsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* ws = fsm + (unsigned)warp * (unsigned)fac_warp_smem(vals);
  double2* sR = reinterpret_cast<double2*>(ws);  // staged row values
  int4* sS = reinterpret_cast<int4*>(ws + 288 * (vals + 1));
  int2* sT = reinterpret_cast<int2*>(sS + kFacSteps);  // updates of this and the next step
  uint16_t* sMap = reinterpret_cast<uint16_t*>(sT + 64);  // column - base -> slot, or kFacNone
  for (int t = lane; t < kFacMap; t += 32) sMap[t] = kFacNone;
  if (lane < 18) sR[18 * vals + lane] = make_double2(0.0, 0.0);
  __syncwarp();
  const int prob = cta_prob[blockIdx.x];
  const ProbDev& d = P[prob];
  int* counter = grab + prob;
  int* done = d.done;
  const unsigned long long wlim = g_wait_ns;
  const bool skip_first = g_skip_meet != 0;  // failure injection: row 0 of the order never published
  const int32_t* rowp = d.prowp;
  const int32_t* cols = d.pcols;
  const int32_t* diag = d.pdiag;
  const int4* steps = d.psteps;
  const int32_t* rows = d.levLrows;
  const int n = d.n, off = d.off;
  double* LU = d.LU64;
  int idx = lane == 0 ? atomicAdd(counter, 1) : 0;
  idx = __shfl_sync(0xffffffffu, idx, 0);
  int i = idx < n ? rows[idx] : 0;
  int r0 = rowp[i], r1 = rowp[i + 1], di = diag[i];
  while (idx < n) {
    int nidx = lane == 0 ? atomicAdd(counter, 1) : 0;  // the next row, in flight meanwhile
    const int len = r1 - r0, nlow = di - r0;
    const bool vstaged = len <= vals;
    for (int t = lane; t < min(nlow, kFacSteps); t += 32) sS[t] = __ldg(steps + r0 + t);
    // column -> slot map of the row when its column span fits (binary
    // searches otherwise)
    const int cbase = cols[r0], span = cols[r1 - 1] - cbase + 1;
    const bool mapped = fac_mapped(cbase, cbase + span - 1);
    if (mapped)
      for (int t = lane; t < len; t += 32) sMap[cols[r0 + t] - cbase] = (uint16_t)t;
    double2* dst = reinterpret_cast<double2*>(LU + 36 * (size_t)r0);
    if (vstaged) {
      // eight 16-byte loads in flight per lane
      const int nv = 18 * len;
      for (int t0 = lane; t0 < nv; t0 += 256) {
        double2 v[8];
#pragma unroll
        for (int z = 0; z < 8; z++)
          if (t0 + 32 * z < nv) v[z] = __ldcg(dst + t0 + 32 * z);
#pragma unroll
        for (int z = 0; z < 8; z++)
          if (t0 + 32 * z < nv) sR[t0 + 32 * z] = v[z];
      }
    }
    __syncwarp();
    bool live;
    if (vstaged)
      live = factor_row<true>(RowValues<true>{ws}, steps + r0, nlow, len, sS, sT, sMap,
                              cbase, span, mapped, cols, cols + r0, LU, done, epoch, wlim, ctl, lane);
    else
      live = factor_row<false>(RowValues<false>{reinterpret_cast<unsigned char*>(LU + 36 * (size_t)r0)}, steps + r0, nlow,
                               len, sS, sT, sMap, cbase, span, mapped, cols, cols + r0, LU, done,
                               epoch, wlim, ctl, lane);
    if (!live) break;
    // the next row's extent, in flight during the end of this one
    nidx = __shfl_sync(0xffffffffu, nidx, 0);
    const int ni = nidx < n ? rows[nidx] : 0;
    double* Dii = vstaged ? reinterpret_cast<double*>(ws + 288 * nlow) : LU + 36 * (size_t)di;
    const int j12 = lane % 12;
    double m[6];
#pragma unroll
    for (int e = 0; e < 6; e++) m[e] = j12 < 6 ? Dii[6 * e + j12] : (e == j12 - 6 ? 1.0 : 0.0);
    bool ok = inv6_cols(m);
#pragma unroll
    for (int e = 0; e < 6; e++) ok = ok && isfinite(m[e]);
    if (!ok && lane < 12) {
      atomicOr(&ctl->status, ST_ZERO_PIVOT);
      atomicCAS(&ctl->pivot, 0, off + i + 1);
    }
    __syncwarp();
    if (lane >= 6 && lane < 12)
#pragma unroll
      for (int e = 0; e < 6; e++) Dii[6 * e + lane - 6] = m[e];
    __syncwarp();
    // the upper part, then its flag: the lane's release covers the other
    // lanes' stores, which the warp barrier orders before it
    if (vstaged) {
#pragma unroll 4
      for (int t = 18 * nlow + lane; t < 18 * len; t += 32) dst[t] = sR[t];
    }
    __syncwarp();
    if (lane == 0 && !(skip_first && idx == 0)) st_release_gpu(done + i, epoch);
    const int nr0 = rowp[ni], nr1 = rowp[ni + 1], ndi = diag[ni];
    if (vstaged) {
#pragma unroll 4
      for (int t = lane; t < 18 * nlow; t += 32) dst[t] = sR[t];
    }
    if (mapped)
      for (int t = lane; t < len; t += 32) sMap[cols[r0 + t] - cbase] = kFacNone;
    __syncwarp();
    idx = nidx;
    i = ni;
    r0 = nr0;
    r1 = nr1;
    di = ndi;
  }
}

// Steps of every row for the factorization: {slot of the row, row k, first
// block and end of U(k)} in step order.
__global__ void step_table_kernel(int n, const int32_t* __restrict__ rowp,
                                  const int32_t* __restrict__ cols,
                                  const int32_t* __restrict__ diag,
                                  const int32_t* __restrict__ ord, int4* __restrict__ steps) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= n) return;
  const int r0 = rowp[i];
  for (int t = r0 + lane; t < diag[i]; t += 32) {
    const int kp = ord[t], k = cols[kp];
    steps[t] = make_int4(kp - r0, k, diag[k] + 1, rowp[k + 1]);
  }
}

__global__ void scatter_values_kernel(int nA, const int32_t* __restrict__ map,
                                      const double* __restrict__ A, double* __restrict__ LU) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (size_t)nA * 36) return;
  LU[36 * (size_t)map[t / 36] + t % 36] = A[t];
}
template <class T2>
__global__ void convert_kernel(size_t n, const double* __restrict__ in, T2* __restrict__ out) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) out[t] = (T2)in[t];
}


// ------------------------------------------- prefetched level-major sweeps
// A thread-block cluster of kSweepCta CTAs per problem walks the chunks of
// one triangle in level-major order (a chunk holds rows of one level); each
// CTA solves its half of every chunk's rows from its own stream, and the
// CTAs meet once per chunk on a pair of mbarriers (bounded waits, release /
// acquire at cluster scope). A ring of kStages shared-memory stages
// is filled by 1D bulk copies (cp.async.bulk, completion counted on an
// mbarrier) kStages-1 chunks ahead of the chunk being solved. The x
// entries a chunk multiplies come from two places:
//  - near: rows solved by the previous chunk, kept in a shared-memory ring
//    that both CTAs write (their own and, through distributed shared
//    memory, the partner's);
//  - far: rows solved two or more chunks earlier, loaded from global memory
//    one chunk ahead (issued right after the barrier that ends chunk c-1,
//    consumed by chunk c+1), together with chunk c+1's right-hand sides;
// so a chunk's critical path is two block barriers, shared-memory copies and
// its rows' 6x6 products. x / y live in global memory, written and re-read
// by the problem's cluster only.
constexpr int kSweepThreads = 512;
constexpr int kStages = 2;
constexpr size_t kSweepSmemMax = 220 * 1024;  // dynamic; the static part is < 1 KB

// Dynamic shared memory of one sweep: kStages staging buffers of `stage`
// bytes; two buffers (this chunk, next chunk) of gathered x (capb x 6
// doubles) and right-hand sides (capr x 6); the ring of the two latest
// chunks' results (2 slots x kSweepCta capr rows x 6).
__host__ __device__ inline size_t sweep_smem_bytes(int stage, int capb, int capr) {
  return kStages * (size_t)stage + 96 * ((size_t)capb + capr) + 96 * (size_t)kSweepCta * capr;
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Row r of a 6x6 block (6 consecutive values) times 6 x entries, with
// vector shared-memory loads and two partial sums.
__device__ __forceinline__ double dot6(const double* a, const double* x) {
  const double2 a0 = reinterpret_cast<const double2*>(a)[0], a1 = reinterpret_cast<const double2*>(a)[1],
                a2 = reinterpret_cast<const double2*>(a)[2];
  const double2 x0 = reinterpret_cast<const double2*>(x)[0], x1 = reinterpret_cast<const double2*>(x)[1],
                x2 = reinterpret_cast<const double2*>(x)[2];
  double s0 = a0.x * x0.x, s1 = a0.y * x0.y;
  s0 = fma(a1.x, x1.x, s0);
  s1 = fma(a1.y, x1.y, s1);
  s0 = fma(a2.x, x2.x, s0);
  s1 = fma(a2.y, x2.y, s1);
  return s0 + s1;
}
__device__ __forceinline__ double dot6(const float* a, const double* x) {
  const float2 a0 = reinterpret_cast<const float2*>(a)[0], a1 = reinterpret_cast<const float2*>(a)[1],
               a2 = reinterpret_cast<const float2*>(a)[2];
  const double2 x0 = reinterpret_cast<const double2*>(x)[0], x1 = reinterpret_cast<const double2*>(x)[1],
                x2 = reinterpret_cast<const double2*>(x)[2];
  double s0 = (double)a0.x * x0.x, s1 = (double)a0.y * x0.y;
  s0 = fma((double)a1.x, x1.x, s0);
  s1 = fma((double)a1.y, x1.y, s1);
  s0 = fma((double)a2.x, x2.x, s0);
  s1 = fma((double)a2.y, x2.y, s1);
  return s0 + s1;
}

template <class VT, bool UPPER>
__global__ void __launch_bounds__(kSweepThreads) bsweep_tma(const ProbDev* __restrict__ P,
                                                           const int* __restrict__ live,
                                                           const double* __restrict__ rhs,
                                                           double* out, SweepCtl* ctl,
                                                           unsigned long long* bytes_ctr) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t bar[kStages];
  __shared__ uint64_t xbar[2];  // the partner's "chunk done" arrivals, alternating
  __shared__ int abort_flag;
  const int p = blockIdx.x / kSweepCta;
  const unsigned rank = cluster_rank(), partner = rank ^ 1u;
  if (live && !live[p]) return;  // the same for every CTA of the cluster
  if ((UPPER ? P[p].U.kind : P[p].L.kind) != TRI_LEVEL) return;  // solved by bsweep_df
  const bool split = (UPPER ? P[p].U.nsplit : P[p].L.nsplit) > 1;
  if (!split && rank != 0) return;  // one CTA solves the whole chunk; no cluster traffic
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
  const int g = lane / 6, r = lane % 6;
  const ProbDev& d = P[p];
  const TriDesc T = UPPER ? d.U : d.L;
  // xbuf[h]: gathered x (capb x 6) then right-hand sides (capr x 6) of the
  // chunks with parity h
  double* xbuf = reinterpret_cast<double*>(smem + (size_t)kStages * T.stage);
  const size_t xstride = 6 * ((size_t)T.capb + T.capr);
  const int ringrows = kSweepCta * T.capr;
  double* ring = xbuf + 2 * xstride;  // 2 x ringrows x 6
  const unsigned pring = cluster_map(smem_u32(ring), partner);
  const unsigned pxbar = cluster_map(smem_u32(xbar), partner);
  const int64_t* offs = T.off + (size_t)rank * (T.nch + 1);  // this CTA's half chunks
  const unsigned long long wlim = g_wait_ns;
  const bool arrive = !(g_skip_meet && rank == 1);
  const double* rb = rhs + 6 * (size_t)d.off;
  double* ob = out + 6 * (size_t)d.off;
  if (tid == 0) {
    for (int s = 0; s < kStages; s++) mbar_init(&bar[s], 1);
    mbar_init(&xbar[0], 1);
    mbar_init(&xbar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_flag = 0;
  }
  if (split)
    cluster_barrier();  // both CTAs' barriers exist before any remote arrival
  else
    __syncthreads();
  // chunk byte ranges are read one issue ahead so tid 0 never waits on them
  long long lo = 0, hi = 0;
  const int producer = kSweepThreads - 32;  // lane 0 of the last warp issues every copy
  if (tid == producer) {
    lo = offs[0];
    hi = offs[1];
  }
  auto issue = [&](int c) {  // producer only; lo/hi hold chunk c's range
    uint64_t* b = &bar[c % kStages];
    mbar_expect_tx(b, (unsigned)(hi - lo));
    bulk_g2s(smem + (size_t)(c % kStages) * T.stage, T.stream + lo, (unsigned)(hi - lo), b);
    lo = hi;
    if (c + 2 <= T.nch) hi = offs[c + 2];
  };
  if (tid == producer)
    for (int c = 0; c < kStages - 1 && c < T.nch; c++) issue(c);
  int issued = min(kStages - 1, T.nch);
  // chunk 0 has no earlier rows: only its right-hand sides
  if (!mbar_wait(&bar[0], 0u, wlim)) abort_flag = 1;
  __syncthreads();
  // 6-double rows of x and of the right-hand side move as three 16-byte
  // pieces when both vectors are 16-byte aligned, else as six 8-byte ones
  const bool a16 = ((reinterpret_cast<uintptr_t>(rb) | reinterpret_cast<uintptr_t>(ob)) & 15) == 0;
  // pieces per row as a compile-time constant (3 or 6): the index splits
  // below then compile to multiplications instead of divisions
  auto with_pw = [&](auto fn) {
    if (a16)
      fn(std::integral_constant<int, 3>{});
    else
      fn(std::integral_constant<int, 6>{});
  };
  auto copy_piece = [](auto pwc, double* dst, const double* src, int piece) {
    if (decltype(pwc)::value == 3)
      cp_async16(dst + 2 * piece, src + 2 * piece);
    else
      cp_async8(dst + piece, src + piece);
  };
  if (!abort_flag) {
    const int nr0 = reinterpret_cast<const int4*>(smem)->x;
    const int4* ri0 = reinterpret_cast<const int4*>(smem + 32);
    with_pw([&](auto pwc) {
      constexpr int pw = decltype(pwc)::value;
      for (int t = tid; t < pw * nr0; t += kSweepThreads)
        copy_piece(pwc, xbuf + 6 * T.capb + 6 * (t / pw), rb + 6 * (size_t)ri0[t / pw].x, t % pw);
    });
    cp_async_commit();
  }
  int c = 0;
  for (; c < T.nch; c++) {
    const int s = c % kStages;
    if (c > 0 && !mbar_wait(&bar[s], (unsigned)((c / kStages) & 1), wlim)) abort_flag = 1;
    cp_async_wait_all();  // this thread's copies for chunk c have landed
    __syncthreads();      // this CTA's half of chunk c-1 solved; its stage and xbuf[(c+1)&1] are free
    if (c > 0 && split) {
      // meet the partner: its half of chunk c-1 (global x, ring rows in
      // this CTA) is complete and visible once its arrival is seen
      if (tid == 0) {
        const unsigned slot = (unsigned)((c - 1) & 1);
        if (arrive) mbar_arrive_remote(pxbar + 8u * slot);
        if (!mbar_wait_cluster(&xbar[slot], (unsigned)(((c - 1) >> 1) & 1), wlim)) abort_flag = 1;
      }
      __syncthreads();
    }
    if (abort_flag) break;
    const unsigned char* st = smem + (size_t)s * T.stage;
    const int4 h0 = reinterpret_cast<const int4*>(st)[0];
    const int4 h1 = reinterpret_cast<const int4*>(st)[1];
    const int nr = h0.x, nb = h0.y, nn = h0.z, nf1 = h1.x, nr1 = h1.y;
    const int4* ri = reinterpret_cast<const int4*>(st + 32);
    const int2* nearl = reinterpret_cast<const int2*>(ri + nr);
    const int2* far1 = nearl + nn;
    const int32_t* rows1 = reinterpret_cast<const int32_t*>(far1 + nf1);
    const size_t voff = (32 + 16 * (size_t)nr + 8 * (size_t)(nn + nf1) + 4 * (size_t)nr1 + 15) &
                        ~(size_t)15;
    const VT* sv = reinterpret_cast<const VT*>(st + voff);
    double* xs = xbuf + xstride * (c & 1);
    double* rs = xs + 6 * (size_t)T.capb;
    // asynchronous copies for chunk c+1 (waited for one chunk later): far x
    // entries (rows solved by chunks <= c-1, complete at the barrier above)
    // and right-hand sides, into the gather area chunk c-1 used. When the
    // chunk has fewer rows than the CTA has warps, the warps without a row
    // issue them while the others solve theirs; otherwise every thread
    // issues them first.
    auto issue_next = [&](int t0, int stride) {
      double* xn = xbuf + xstride * ((c + 1) & 1);
      with_pw([&](auto pwc) {
        constexpr int pw = decltype(pwc)::value;
        for (int t = t0; t < pw * (nf1 + nr1); t += stride) {
          if (t < pw * nf1) {
            const int2 f = far1[t / pw];
            copy_piece(pwc, xn + 6 * f.x, ob + 6 * (size_t)f.y, t % pw);
          } else {
            const int t2 = t - pw * nf1;
            copy_piece(pwc, xn + 6 * T.capb + 6 * (t2 / pw), rb + 6 * (size_t)rows1[t2 / pw],
                       t2 % pw);
          }
        }
      });
    };
    const bool idle_issue = nr < nw;
    if (!idle_issue) issue_next(tid, kSweepThreads);
    // near entries: results of chunk c-1 from the ring
    {
      const double2* rp =
          reinterpret_cast<const double2*>(ring + 6 * (size_t)ringrows * ((c + 1) & 1));
      double2* xs2 = reinterpret_cast<double2*>(xs);
      for (int t = tid; t < 3 * nn; t += kSweepThreads) {
        const int2 q = nearl[t / 3];
        xs2[3 * q.x + t % 3] = rp[3 * q.y + t % 3];
      }
    }
    __syncthreads();
    // the producer warp (the last) refills the stage chunk c-1 used, then
    // solves rows like the others (it is given a row only when a chunk has
    // as many rows as the CTA has warps)
    if (issued < T.nch) {
      if (tid == producer) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        issue(issued);
      }
      issued++;
    }
    if (idle_issue && warp >= nr) issue_next(tid - 32 * nr, 32 * (nw - nr));
    cp_async_commit();
    double* wp = ring + 6 * (size_t)ringrows * (c & 1);
    const unsigned pwp = pring + 8u * 6u * (unsigned)ringrows * (unsigned)(c & 1);
    for (int k = warp; k < nr; k += nw) {
      const int4 row = ri[k];
      const int i = row.x, rbeg = row.y, rcnt = row.z, gk = row.w;
      const int first = UPPER ? 1 : 0;  // U rows start with U_ii^{-1}
      // row `lane` of U_ii^{-1} (lanes 0..5), loaded while the products run
      double di[6];
      if (UPPER) {
        const VT* Di = sv + (size_t)rbeg * 36 + 6 * (lane < 6 ? lane : 0);
#pragma unroll
        for (int cc = 0; cc < 6; cc++) di[cc] = (double)Di[cc];
      }
      double acc = 0.0;
      if (g < 4) {
        double acc1 = 0.0;
        int j = first + g;
        for (; j + 4 < rcnt; j += 8) {
          acc += dot6(sv + (size_t)(rbeg + j) * 36 + 6 * r, xs + 6 * (rbeg + j));
          acc1 += dot6(sv + (size_t)(rbeg + j + 4) * 36 + 6 * r, xs + 6 * (rbeg + j + 4));
        }
        if (j < rcnt) acc += dot6(sv + (size_t)(rbeg + j) * 36 + 6 * r, xs + 6 * (rbeg + j));
        acc += acc1;
      }
      acc += __shfl_down_sync(0xffffffffu, acc, 12);
      acc += __shfl_down_sync(0xffffffffu, acc, 6);
      const double t = (lane < 6 ? rs[6 * k + lane] : 0.0) - acc;
      double v = t;
      if (UPPER) {
        double tc[6];
#pragma unroll
        for (int cc = 0; cc < 6; cc++) tc[cc] = __shfl_sync(0xffffffffu, t, cc);
        v = fma(di[4], tc[4], fma(di[2], tc[2], di[0] * tc[0])) +
            fma(di[5], tc[5], fma(di[3], tc[3], di[1] * tc[1]));
      }
      if (lane < 6) {
        ob[6 * (size_t)i + lane] = v;
        wp[6 * gk + lane] = v;
        if (split) cluster_store(pwp + 8u * (unsigned)(6 * gk + lane), v);
      }
    }
  }
  cp_async_wait_all();  // no copy may land after the kernel ends
  if (!abort_flag && tid == 0 && rank == 0 && bytes_ctr)
    atomicAdd(bytes_ctr, (unsigned long long)T.abytes);
  if (abort_flag && tid == producer) {
    atomicOr(&ctl->status, ST_TIMEOUT);
    // chunks c .. issued-1 may still be in flight: let them land (bounded)
    for (int q = c; q < issued; q++)
      mbar_wait(&bar[q % kStages], (unsigned)((q / kStages) & 1), kWaitNs);
  }
  // neither CTA leaves while the other may still write into its shared
  // memory; every path of both CTAs of a split problem reaches this point
  if (split) cluster_barrier();
}

// --------------------------------------------- register-fed level sweeps
// The default sweep. What bounds a level is the latency of its chain (x
// entries -> products -> reduction -> U_ii^{-1} -> result -> barrier), so the
// chain holds nothing else:
//  - every x entry a triangle still needs sits in a shared-memory ring of
//    the latest results (48 bytes a row; the ring covers the triangle's
//    dependency reach), read straight into the products;
//  - the warps form groups that take the levels in turn: while one group
//    runs the chain of its level, the others load and convert the values of
//    theirs. A level waits only for the level before it (bar.sync of its
//    group against bar.arrive of the one before);
//  - a warp takes a row 16 blocks a pass; lane (j, h) multiplies rows
//    3h..3h+2 of block j. The values are read once, so they go from L2
//    straight to registers while the other groups' levels run, and every pass
//    prefetches from HBM into L2, kRingAhead bytes ahead of itself, a line of
//    128 bytes for each lane that has values: all that a pass of the same
//    length takes in FP32, 8/9 of it in FP64, and not U_ii^{-1};
//  - the 16 partial sums of a row meet in a reduce-scatter of five 64-bit
//    shuffles (a butterfly over three sums takes twelve);
//  - rows of more than 16 blocks are shared by several warps.
// In a triangle split over the CTAs of a cluster every result also goes to
// the others' rings with st.async, whose bytes their mbarriers count per
// level (bounded waits; no release of other stores is waited for). A warp
// whose wait runs out solves, arms and sends nothing from that level on, nor
// does any warp of its CTA from the next level on (ring_leave), so no barrier
// ever counts the bytes of more than two levels (below the 2^20 - 1 that it
// can); the CTA ends once the bytes that were sent to it have landed
// (ring_drain). Microseconds a level, chunked sweep -> this one (B200): 17x16
// plate, ILU(8), FP32 1.19 -> 0.45; 256x128, ILU(6), FP32 2.22 -> 0.76, FP64
// 3.54 -> 0.79; 250x220, ILU(12), FP32 2.15 -> 0.83; 40x20, complete factor,
// FP64 1.50 -> 0.47. Still latency-bound: ~120 dependent instructions a level,
// so what the compiler knows to be uniform and what spills shows at once (with
// one body for split and unsplit triangles 0.47, 0.79, 0.83, 0.82, 0.47; then
// with 24 warps of 80 registers 0.51, 0.88, 0.94, 0.91, 0.50; without the broadcast
// of the warp's number 0.56, 0.85, 0.89, 0.92, 0.58).
constexpr int kRingThreads = 32 * kRingWarps;
constexpr size_t kRingSmemMax = 218 * 1024;  // dynamic; the static part is < 2 KB
// Cost model of a level in clocks (it only chooses CTAs and groups): least
// squares over 300 applies on B200 (22 plates from 17x16 to 256x128, ILU(6) to
// ILU(12) and complete factors, FP32 and FP64, each with 1, 2, 4 CTAs and 2, 3,
// 4 groups). Terms: the chain, the exchange of a split, the issue slots of the
// passes of the busiest CTA, every further round of its busiest warp (a second
// pass finds its values not there yet), and what the other groups' levels do
// not hide. Of these layouts it takes the fastest on all plates but one (4 %
// off). us a level where groups or CTAs decide: 28x28 ILU(12) on one CTA, 2 / 3
// / 4 groups 0.50 / 0.49 / 0.47; 85x60 ILU(8) on four 0.73 / 0.71 / 0.69;
// 148x122 ILU(12) on four 0.75 / 0.71 / 1.03 (a second round).
constexpr double kRingChain = 695.0, kRingSplit = 316.0, kRingSplit4 = 72.0, kRingIssue = 33.0,
                 kRingRound = 864.0, kRingRoundG = 313.0, kRingLate = 408.0;
constexpr int kRingAhead = 96 * 1024;  // bytes of values prefetched into L2 ahead of their use
// rows up to which the chunked level sweep (bsweep_tma) always has a stage:
// its chunk bound is then the base size of either precision
constexpr int kRingRowAlways = 136;

// position (in values, from the first value of the row's group of nb <= 16
// blocks) of entry e = 6 r + c of block jj of the group; nb = 0: U_ii^{-1},
// stored row-major. Lane 2 jj + r / 3 loads its 18 values as 16-byte pieces
// (and one of 8 bytes in FP32), piece k of all lanes together.
template <class VT>
__host__ __device__ __forceinline__ int ring_value_pos(int nb, int jj, int e) {
  if (nb == 0) return e;
  constexpr int pv = 16 / (int)sizeof(VT);  // values of a 16-byte piece
  constexpr int full = 18 / pv;             // whole pieces of a lane
  const int r = e / 6, lane = 2 * jj + r / 3, v = 6 * (r % 3) + e % 6;
  if (v < full * pv) return (v / pv * 2 * nb + lane) * pv + v % pv;
  return full * 2 * nb * pv + lane * (18 - full * pv) + (v - full * pv);
}

__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p) : "memory");
}
// 8 bytes into another CTA's shared memory, counted on its mbarrier
__device__ __forceinline__ void st_async(unsigned addr, double v, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(
                   addr),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void named_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void named_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void ring_load(const float* p, int lane, int n2, float (&v)[18]) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(p) + k * n2 + lane);
    v[4 * k] = q.x, v[4 * k + 1] = q.y, v[4 * k + 2] = q.z, v[4 * k + 3] = q.w;
  }
  const float2 q = __ldg(reinterpret_cast<const float2*>(p + 16 * n2) + lane);
  v[16] = q.x, v[17] = q.y;
}
__device__ __forceinline__ void ring_load(const double* p, int lane, int n2, double (&v)[18]) {
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const double2 q = __ldg(reinterpret_cast<const double2*>(p) + k * n2 + lane);
    v[2 * k] = q.x, v[2 * k + 1] = q.y;
  }
}
// volatile: the conversions stay ahead of the barrier that follows them
__device__ __forceinline__ void ring_take(const float (&v)[18], double (&d)[18]) {
#pragma unroll
  for (int k = 0; k < 18; k++) asm volatile("cvt.f64.f32 %0, %1;" : "=d"(d[k]) : "f"(v[k]));
}
__device__ __forceinline__ void ring_take(const double (&v)[18], double (&d)[18]) {
#pragma unroll
  for (int k = 0; k < 18; k++) d[k] = v[k];
}

// Waits (bounded) until a phase of bar is complete, as one warp: false when
// the bound ran out (abort_flag set here) or another warp's did. That comes
// first: past a level in which a warp gave up, a barrier may be a phase behind,
// and its parity then reads as complete.
__device__ __noinline__ bool ring_wait(uint64_t* bar, unsigned parity,
                                       volatile int* abort_flag) {
  const unsigned long long t0 = gtimer();
  while (true) {
    if (__any_sync(0xffffffffu, *abort_flag)) return false;
    if (__all_sync(0xffffffffu, mbar_try_wait_cluster(bar, parity))) return true;
    if (__any_sync(0xffffffffu, gtimer() - t0 > g_wait_ns)) {
      *abort_flag = 1;
      return false;
    }
  }
}

// The rest of a warp's levels after it has given up in level lev (pass t, whose
// barrier it has met): it only meets the barriers that other warps wait at.
__device__ __noinline__ void ring_leave(const int4* t, int lev, int nlev, int groups, int warp) {
  const int wpg = kRingWarps / groups, gi = warp / wpg, bar_threads = 64 * wpg;
  const int bar_in = 1 + (gi ? gi - 1 : groups - 1), bar_out = 1 + gi;
  for (bool met = true; lev < nlev; met = false) {
    const int4 k = __ldg(t++);
    if ((k.y & kRingBegin) && !met) named_sync(bar_in, bar_threads);
    const int helpers = (k.y >> 5) & 31;
    if (k.y & kRingLast) {
      if (k.x == -2)
        named_arrive((1 + groups + k.w / 2) & 15, 32 * (helpers + 1));
      else if (helpers)
        named_sync((1 + groups + warp / 2) & 15, 32 * (helpers + 1));
    }
    if (k.y & kRingEnd) {
      if (lev + 1 < nlev) named_arrive(bar_out, bar_threads);
      lev += groups;
    }
  }
}

// A CTA that gave up waits here (bounded) for the stores that are still on
// their way into it; nothing is sent to it any more. gone[q][w] is the level
// in which warp w of CTA q gave up: it armed and sent nothing from there on.
// The bytes sent to this CTA and the bytes its barriers were armed for follow
// from the task lists; where they differ the last phase's count is set right,
// so that it completes with the last byte.
__device__ __noinline__ void ring_drain(const TriDesc& T, unsigned rank,
                                        const int (*gone)[kRingWarps], uint64_t* xbar,
                                        SweepCtl* ctl) {
  __shared__ int armed[2], sent[2], arms[2];  // bytes, bytes, phases of even / odd levels
  const int tid = threadIdx.x;
  if (tid < 2) armed[tid] = sent[tid] = arms[tid] = 0;
  __syncthreads();
  if (tid < T.nsplit * kRingWarps) {
    const int q = tid / kRingWarps, w = tid % kRingWarps, wpg = kRingWarps / T.groups;
    const bool lead = w % wpg == 0, mine = q == (int)rank;
    const int end = min(T.nlev, gone[q][w]);
    const int4* t = T.tasks + T.lists[q * kRingWarps + w];
    int lev = w / wpg < T.groups ? w / wpg : T.nlev;
    for (; lev < end; t++) {
      const int4 k = *t;
      if (mine) {
        if (lead && (k.y & kRingBegin)) {
          atomicAdd(&armed[lev & 1], 8 * (int)((unsigned)k.y >> 16));
          atomicAdd(&arms[lev & 1], 1);
        }
      } else if (k.x >= 0 ? (k.y & kRingLast) : (k.x == -1 && lead && (k.y & kRingBegin))) {
        atomicAdd(&sent[lev & 1], k.x >= 0 ? 48 : 8);
      }
      if (k.y & kRingEnd) lev += T.groups;
    }
  }
  __syncthreads();
  if (tid != 0) return;
  bool quiet = true;
  for (int z = 0; z < 2; z++) {
    const int more = sent[z] - armed[z];
    if (more < 0)
      asm volatile("mbarrier.complete_tx.relaxed.cluster.shared::cta.b64 [%0], %1;" ::"r"(
                       smem_u32(&xbar[z])),
                   "r"(-more)
                   : "memory");
    if (arms[z] > 0)
      quiet &= mbar_wait_cluster(&xbar[z], (unsigned)((arms[z] - 1) & 1), kWaitNs);
    if (more > 0 && quiet) {
      mbar_expect_tx(&xbar[z], (unsigned)more);
      quiet &= mbar_wait_cluster(&xbar[z], (unsigned)(arms[z] & 1), kWaitNs);
    }
  }
  atomicOr(&ctl->status, ST_TIMEOUT);
  atomicAdd(&ctl->gave_up, 1);
  if (quiet) atomicAdd(&ctl->quiet, 1);
}

struct RingShared {
  uint64_t xbar[2];            // the other CTAs' results of even / odd levels
  double part[kRingWarps][6];  // a helper's sums for the row's warp
  int gone[kRingCta][kRingWarps];  // per CTA and warp: level in which it gave up (ring_drain)
  volatile int abort_flag;         // a warp of this CTA has
};

// The sweep of one triangle; SPLIT: shared by the CTAs of a cluster. (In one
// body for both, what a split needs costs an unsplit level too: 33x21 plate,
// ILU(8), FP64 0.55 us instead of 0.52.)
template <class VT, bool UPPER, bool SPLIT>
__device__ __forceinline__ void ring_sweep(unsigned char* ring, RingShared& sh, const TriDesc& T,
                                           int nsplit, unsigned rank, const double* rb, double* ob,
                                           SweepCtl* ctl, unsigned long long* bytes_ctr) {
  uint64_t* xbar = sh.xbar;
  auto part = sh.part;
  auto gone = sh.gone;
  volatile int& abort_flag = sh.abort_flag;
  // the broadcast tells the compiler that a warp's passes are the same for all
  // its lanes: no reconvergence around the shuffles of the chain
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31, h = lane & 1;
  if (tid == 0) {
    mbar_init(&xbar[0], 1);
    mbar_init(&xbar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_flag = 0;
  }
  if (tid < 6) reinterpret_cast<double*>(ring)[tid] = 0.0;
  if (tid < kRingCta * kRingWarps) gone[0][tid] = 0x7fffffff;
  if (SPLIT)
    cluster_barrier();  // every CTA's barriers exist before any remote store
  else
    __syncthreads();
  const bool mute = g_skip_meet && rank == 1;  // failure injection
  const int peers = SPLIT && !mute ? nsplit : 0;
  const unsigned char* stream = T.stream;
  const VT* vals = reinterpret_cast<const VT*>(stream);
  const int32_t* slots = T.slots;
  const int groups = T.groups, wpg = kRingWarps / groups, nlev = T.nlev;
  const int gi = warp / wpg;  // the warp's group
  const bool lead = warp == gi * wpg && lane == 0;
  // barriers of the level before (of this group) and of this group's
  // levels; the others serve rows that several warps share
  const int bar_in = 1 + (gi ? gi - 1 : groups - 1), bar_out = 1 + gi;
  const int bar_threads = 64 * wpg;
  const size_t vbytes = (size_t)T.nblocks * 36 * sizeof(VT);
  for (size_t a = 128 * (size_t)tid; a < min(vbytes, (size_t)kRingAhead); a += 128 * kRingThreads)
    prefetch_l2(stream + a);
  // the row (of the block's six) whose sum ends in this lane, and whether
  // the lane writes it
  const int rr = 3 * h + ((lane & 16) ? 2 : (lane & 8) ? 1 : 0);
  const bool writer = (lane & 6) == 0 && (lane & 24) != 24;
  const bool b4 = lane & 16, b3 = lane & 8;
  const int4* tasks = T.tasks + T.lists[rank * kRingWarps + warp];
  VT v[18];  // values of this pass
  VT di[6];  // row rr of U_ii^{-1}
  double acc[3] = {0.0, 0.0, 0.0}, rv = 0.0;
  int slot = 0;  // ring offset of this lane's x entries
#pragma unroll
  for (int k = 0; k < 6; k++) di[k] = (VT)0;
  auto load = [&](const int4& t) {
    const int nb = t.y & 31;
    slot = 0;
#pragma unroll
    for (int k = 0; k < 18; k++) v[k] = (VT)0;
    if (lane < 2 * nb) {
      slot = __ldg(slots + t.z + (lane >> 1));
      ring_load(vals + 36 * (size_t)t.z, lane, 2 * nb, v);
      const size_t a = 36 * sizeof(VT) * (size_t)t.z + kRingAhead + 128 * (size_t)lane;
      if (lane * 128 < 36 * (int)sizeof(VT) * nb + 127 && a < vbytes) prefetch_l2(stream + a);
    }
    if (t.x >= 0 && (t.y & kRingFirst)) {
      rv = rb[6 * (size_t)t.x + rr];
      if (UPPER) {
        using V2 = typename std::conditional<sizeof(VT) == 8, double2, float2>::type;
        // U_ii^{-1} precedes the row's first block
        const V2* q = reinterpret_cast<const V2*>(vals + 36 * (size_t)(t.z - 1) + 6 * rr);
#pragma unroll
        for (int k = 0; k < 3; k++) {
          const V2 u = __ldg(q + k);
          di[2 * k] = u.x, di[2 * k + 1] = u.y;
        }
      }
    }
  };
  int4 t0 = __ldg(tasks), t1 = __ldg(tasks + 1);
  tasks += 2;
  load(t0);
  int lev = gi < groups ? gi : nlev;  // this group's level (a warp beyond the groups has none)
  while (lev < nlev) {
    const int4 t2 = __ldg(tasks++);
    double d[18];
    ring_take(v, d);
    if (t0.y & kRingFirst) acc[0] = acc[1] = acc[2] = 0.0;
    if (t0.y & kRingBegin) {
      if (lev > 0) {
        named_sync(bar_in, bar_threads);
        if (SPLIT) {  // the results of the other CTAs, as one warp
          uint64_t* b = &xbar[(lev - 1) & 1];
          const unsigned par = (unsigned)(((lev - 1) >> 1) & 1);
          const int quit = abort_flag;  // a warp has given up, here or in a level before
          if (!__all_sync(0xffffffffu, mbar_try_wait_cluster(b, par) && !quit) &&
              !__all_sync(0xffffffffu, ring_wait(b, par, &abort_flag))) {
            if (lane == 0) gone[rank][warp] = lev;
            ring_leave(tasks - 3, lev, nlev, groups, warp);
            break;
          }
        }
      }
    }
    if (t0.x != -1) {
      {
        // lanes without a block multiply zeros
        const double2* x = reinterpret_cast<const double2*>(ring + slot);
        const double2 x0 = x[0], x1 = x[1], x2 = x[2];
#pragma unroll
        for (int r = 0; r < 3; r++) {
          acc[r] = fma(d[6 * r], x0.x, acc[r]);
          acc[r] = fma(d[6 * r + 1], x0.y, acc[r]);
          acc[r] = fma(d[6 * r + 2], x1.x, acc[r]);
          acc[r] = fma(d[6 * r + 3], x1.y, acc[r]);
          acc[r] = fma(d[6 * r + 4], x2.x, acc[r]);
          acc[r] = fma(d[6 * r + 5], x2.y, acc[r]);
        }
      }
      if (t0.y & kRingLast) {
        // lanes with bit 4 keep row 2, the others rows 0 and 1; those split
        // on bit 3
        const double y0 = __shfl_xor_sync(0xffffffffu, b4 ? acc[0] : acc[2], 16);
        const double y1 = __shfl_xor_sync(0xffffffffu, acc[1], 16);
        const double k0 = (b4 ? acc[2] : acc[0]) + y0, k1 = acc[1] + y1;
        const double y2 = __shfl_xor_sync(0xffffffffu, b4 || b3 ? k0 : k1, 8);
        double a = (b4 || !b3 ? k0 : k1) + y2;
        a += __shfl_xor_sync(0xffffffffu, a, 4);
        a += __shfl_xor_sync(0xffffffffu, a, 2);
        const int helpers = (t0.y >> 5) & 31;
        if (t0.x == -2) {  // this warp helps warp t0.w with its row
          if (writer) part[warp][rr] = a;
          named_arrive((1 + groups + t0.w / 2) & 15, 32 * (helpers + 1));
        } else {
          if (helpers) {
            named_sync((1 + groups + warp / 2) & 15, 32 * (helpers + 1));
            for (int k = 1; k <= helpers; k++) a += part[warp + k][rr];
          }
          double z = rv - a;
          if (UPPER) {
            double tc[6];
#pragma unroll
            for (int c = 0; c < 6; c++)
              tc[c] = __shfl_sync(0xffffffffu, z, c / 3 + (c % 3 == 2 ? 16 : 8 * (c % 3)));
            z = fma((double)di[4], tc[4], fma((double)di[2], tc[2], (double)di[0] * tc[0])) +
                fma((double)di[5], tc[5], fma((double)di[3], tc[3], (double)di[1] * tc[1]));
          }
          if (writer) {
            const unsigned o = (unsigned)t0.w + 8u * (unsigned)rr;
            *reinterpret_cast<double*>(ring + o) = z;
            if (SPLIT)
#pragma unroll
              for (int q = 1; q < kRingCta; q++) {
                if (q >= peers) break;
                const unsigned c = rank ^ q;
                st_async(cluster_map(smem_u32(ring + o), c), z,
                         cluster_map(smem_u32(&xbar[lev & 1]), c));
              }
            ob[6 * (size_t)t0.x + rr] = z;
          }
        }
      }
    } else if (SPLIT && lead && (t0.y & kRingBegin)) {
      // a CTA without rows in this level says that it has got here (a zero
      // into slot 0, where a zero is): no CTA solves level l + 1 before every
      // other one has the results of level l - 1, so bytes of at most two
      // levels are on their way to a barrier pair, and no ring is written
      // further ahead than its margin
      for (int q = 1; q < peers; q++) {
        const unsigned c = rank ^ q;
        st_async(cluster_map(smem_u32(ring), c), 0.0,
                 cluster_map(smem_u32(&xbar[lev & 1]), c));
      }
    }
    // bytes of this level may have landed before; arming after the pass keeps
    // it off the chain (85x60, ILU(8), FP32 0.65 -> 0.63 us a level)
    if (SPLIT && lead && (t0.y & kRingBegin))
      mbar_expect_tx(&xbar[lev & 1], 8u * ((unsigned)t0.y >> 16));
    if (t0.y & kRingEnd) {
      if (lev + 1 < nlev) named_arrive(bar_out, bar_threads);
      lev += groups;
    }
    t0 = t1;
    t1 = t2;
    load(t0);
  }
  if (SPLIT) {
    // the other CTAs' results of the last level have landed
    __syncthreads();
    if (tid == 0 && !abort_flag &&
        !mbar_wait_cluster(&xbar[(nlev - 1) & 1], (unsigned)(((nlev - 1) >> 1) & 1), g_wait_ns))
      abort_flag = 1;
    __syncthreads();
    if ((abort_flag || mute) && tid < kRingWarps)
      for (int q = 1; q < nsplit; q++)
        asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(cluster_map(
                         smem_u32(&gone[rank][tid]), rank ^ q)),
                     "r"(mute ? 0 : gone[rank][tid])
                     : "memory");
  }
  if (tid == 0 && rank == 0 && bytes_ctr && !abort_flag)
    atomicAdd(bytes_ctr, (unsigned long long)T.abytes);
  if (SPLIT) {
    // From here on nobody sends. A CTA that has not given up has waited for
    // every byte of every level; one that has waits for what it was sent.
    __syncwarp();  // the barrier is one instruction of a whole warp
    cluster_barrier();
    if (abort_flag) ring_drain(T, rank, gone, xbar, ctl);
  }
}

template <class VT, bool UPPER>
__global__ void __launch_bounds__(kRingThreads, 1)
    bsweep_ring(const ProbDev* __restrict__ P, const int* __restrict__ live,
                const double* __restrict__ rhs, double* out, SweepCtl* ctl,
                unsigned long long* bytes_ctr) {
  extern __shared__ __align__(128) unsigned char ring[];
  __shared__ RingShared sh;
  unsigned ncta;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ncta));
  const int p = blockIdx.x / ncta;
  const unsigned rank = cluster_rank();
  if (live && !live[p]) return;  // the same for every CTA of the cluster
  const TriDesc& T = UPPER ? P[p].U : P[p].L;
  if (T.kind != TRI_RING) return;
  const int nsplit = T.nsplit;
  // CTAs without rows leave at once (a cluster barrier counts only threads
  // that have not exited, and no other CTA writes here)
  if ((int)rank >= nsplit) return;
  const double* rb = rhs + 6 * (size_t)P[p].off;
  double* ob = out + 6 * (size_t)P[p].off;
  if (nsplit > 1)
    ring_sweep<VT, UPPER, true>(ring, sh, T, nsplit, rank, rb, ob, ctl, bytes_ctr);
  else
    ring_sweep<VT, UPPER, false>(ring, sh, T, 1, 0, rb, ob, ctl, bytes_ctr);
}

// Factor values into a ring sweep's stream: block q of the triangle takes
// the 6x6 block src[map[q]]; code[q] = (blocks of its group << 8) + its
// number in the group (0 for U_ii^{-1}).
template <class VT>
__global__ void repack_ring_kernel(size_t nblocks, const int32_t* __restrict__ map,
                                   const uint16_t* __restrict__ code,
                                   const double* __restrict__ src, VT* __restrict__ dst) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nblocks * 36) return;
  const size_t q = t / 36;
  const int e = (int)(t % 36), nb = code[q] >> 8, jj = code[q] & 255;
  dst[36 * (q - jj) + ring_value_pos<VT>(nb, jj, e)] = (VT)src[36 * (size_t)map[q] + e];
}

// One sweep of a batch: a cluster of `ctas` CTAs per problem.
typedef void (*SweepKernel)(const ProbDev*, const int*, const double*, double*, SweepCtl*,
                            unsigned long long*);
static cudaError_t launch_sweep(SweepKernel kernel, int ctas, int threads, int np, size_t smem,
                                cudaStream_t st, const ProbDev* desc, const int* live,
                                const double* rhs, double* out, SweepCtl* ctl,
                                unsigned long long* ctr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(np * ctas));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ::gf::count_launch();
  return cudaLaunchKernelEx(&cfg, kernel, desc, live, rhs, out, ctl, ctr);
}

// ------------------------------------------------------ dataflow sweeps
// One CTA per problem walks one triangle row by row in level order without
// block barriers: compute warp w solves the rows of every chunk whose
// chunk-local index is w mod kDfWarps, and a row waits only for the rows it
// multiplies. A solved row's x entries go to global memory (the result) and
// to a shared-memory ring of the latest `ring` positions; every ring slot
// has an mbarrier whose phase k completes when position slot + k ring is
// written, so a consumer waits (bounded, suspended in hardware rather than
// spinning) on the phase of exactly the position it reads, with release /
// acquire ordering at CTA scope. A row's blocks are ordered by the position
// they depend on, so the lane groups multiply the long-solved rows while the
// latest ones finish.
// Flow control keeps the phases unambiguous: before overwriting a slot with
// position p a warp waits until every warp has moved past p - ring + maxdist
// (so all readers of the slot's previous position are done), using the
// positions the warps publish in wpos[]. Every position below min(wpos) is
// solved, so the warp holding that minimum can always proceed: nothing
// waits in a cycle.
// The factor stream arrives through kDfStages shared-memory stages filled by
// 1D bulk copies, which a producer warp issues as the compute warps release
// stages (full / empty mbarriers), and a gather warp copies each chunk's
// right-hand sides into the chunk's stage with cp.async (completion counted
// on a third mbarrier), so no row waits on a global load. The compute warps
// store nothing to global memory: a writer warp copies every solved row from
// the ring to the result vector in position order (it waits on the same
// slot barriers and takes part in the flow control), so the release
// operations of the compute warps order shared-memory writes only and never
// wait for global stores to complete. All waits are bounded; on a timeout
// the CTA records ST_TIMEOUT and ends after its copies in flight have landed.
constexpr int kDfThreads = 576;
constexpr int kDfWarps = kDfThreads / 32 - 3;  // compute warps
constexpr int kDfProducer = kDfWarps;          // issues the stage copies
constexpr int kDfGather = kDfWarps + 1;        // gathers the right-hand sides
constexpr int kDfWriter = kDfWarps + 2;        // writes results to global memory
constexpr int kDfStages = 4;
constexpr int kDfRows = 64;                    // rows per chunk at most
constexpr int kDfWriteBatch = 64;              // positions the writer reports at once

// dynamic shared memory of a dataflow sweep: the stages, their right-hand
// sides, the ring's x entries (6 doubles), row indices and mbarriers
__host__ __device__ inline size_t df_smem_bytes(int stage, int ring) {
  return kDfStages * ((size_t)stage + 48 * (size_t)kDfRows) + (size_t)ring * (48 + 8 + 4);
}
__device__ __forceinline__ void mbar_arrive_local(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ int ld_acquire_s32(const int* p) {
  int v;
  asm volatile("ld.acquire.cta.shared.b32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_s32(int* p, int v) {
  asm volatile("st.release.cta.shared.b32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
// arrive on `bar` once all of this thread's earlier cp.async copies have
// landed (the arrival is not counted in advance)
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void cp_async8_df(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src)
               : "memory");
}

template <class VT, bool UPPER>
__global__ void __launch_bounds__(kDfThreads) bsweep_df(const ProbDev* __restrict__ P,
                                                       const int* __restrict__ live,
                                                       const double* __restrict__ rhs,
                                                       double* out, SweepCtl* ctl,
                                                       unsigned long long* bytes_ctr) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t full[kDfStages], empty[kDfStages], rhsb[kDfStages];
  // every position below wpos[w] that compute warp w owns is solved; every
  // position below wpos[kDfWarps] has been written out by the writer warp
  __shared__ int wpos[kDfWarps + 1];
  __shared__ volatile int abort_flag;
  const int p = blockIdx.x;
  if (live && !live[p]) return;
  const ProbDev& d = P[p];
  const TriDesc T = UPPER ? d.U : d.L;
  if (T.kind != TRI_DATAFLOW) return;  // solved by bsweep_tma
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rmask = T.ring - 1, rlog = __ffs(T.ring) - 1;
  // layout: stages | right-hand sides of the stages | ring x | ring mbarriers
  double* srhs = reinterpret_cast<double*>(smem + (size_t)kDfStages * T.stage);
  double* rx = srhs + (size_t)kDfStages * 6 * kDfRows;
  uint64_t* rbar = reinterpret_cast<uint64_t*>(rx + 6 * (size_t)T.ring);
  int* ridx = reinterpret_cast<int*>(rbar + T.ring);  // row index of each slot's position
  for (int t = tid; t < T.ring; t += kDfThreads) mbar_init(&rbar[t], 1);
  if (tid <= kDfWarps) wpos[tid] = 0;
  if (tid == 0) {
    for (int s = 0; s < kDfStages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kDfWarps);
      mbar_init(&rhsb[s], 32);
    }
    abort_flag = 0;
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  const unsigned long long wlim = g_wait_ns;
  // bounded wait that also gives up once another warp has aborted
  // Waiting warps sleep in the barrier test instead of spinning, so the warps
  // that have work get the issue slots; the timer is read only once the
  // first test fails.
  auto wait_bar = [&](uint64_t* bar, unsigned par) {
    if (mbar_try_wait(bar, par)) return true;
    const unsigned long long t0 = gtimer();
    unsigned n = 0;
    while (!mbar_try_wait_sleep(bar, par, 2000u))
      if ((++n & 15u) == 0u && (abort_flag || gtimer() - t0 > wlim)) return false;
    return true;
  };
  auto fail = [&]() {
    if (!abort_flag) {
      abort_flag = 1;
      atomicOr(&ctl->status, ST_TIMEOUT);
    }
  };
  if (warp == kDfProducer) {
    if (lane == 0) {
      int issued = 0;
      for (int c = 0; c < T.nch; c++) {
        const int s = c % kDfStages;
        // the compute warps have released chunk c - kDfStages
        if (c >= kDfStages && !wait_bar(&empty[s], (unsigned)(((c / kDfStages) - 1) & 1))) {
          fail();
          break;
        }
        const long long lo = T.off[c], hi = T.off[c + 1];
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&full[s], (unsigned)(hi - lo));
        bulk_g2s(smem + (size_t)s * T.stage, T.stream + lo, (unsigned)(hi - lo), &full[s]);
        issued = c + 1;
      }
      // no copy may land after the CTA ends: the last stages' copies (all
      // earlier ones were consumed before their stages were reused)
      for (int q = max(0, issued - kDfStages); q < issued; q++)
        mbar_wait(&full[q % kDfStages], (unsigned)((q / kDfStages) & 1), kWaitNs);
    }
    return;
  }
  if (warp == kDfGather) {
    // the right-hand sides of each chunk's rows into the chunk's stage, as
    // soon as the chunk's records have landed
    const double* rb = rhs + 6 * (size_t)d.off;
    for (int c = 0; c < T.nch; c++) {
      const int s = c % kDfStages;
      if (!wait_bar(&full[s], (unsigned)((c / kDfStages) & 1))) {
        if (lane == 0) fail();
        break;
      }
      const unsigned char* st = smem + (size_t)s * T.stage;
      const int nr = reinterpret_cast<const int4*>(st)->x;
      const int4* rec = reinterpret_cast<const int4*>(st + 16);
      double* dst = srhs + (size_t)s * 6 * kDfRows;
      for (int t = lane; t < 6 * nr; t += 32)
        cp_async8_df(dst + t, rb + 6 * (size_t)rec[t / 6].x + t % 6);
      cp_async_arrive(&rhsb[s]);
    }
    cp_async_wait_all();  // no copy may land after the CTA ends
    return;
  }
  double* ob = out + 6 * (size_t)d.off;
  const int n = d.n;
  if (warp == kDfWriter) {
    // lane group g5 (5 groups of 6 lanes) writes position q0 + g5
    const int g5 = lane / 6, r6 = lane % 6;
    bool okw = true;
    for (int q0 = 0; q0 < n && okw; q0 += 5) {
      const int q = q0 + g5;
      if (lane < 30 && q < n) {
        if (!wait_bar(&rbar[q & rmask], (unsigned)((q >> rlog) & 1))) {
          fail();
          okw = false;
        } else {
          const int slot = q & rmask;
          ob[6 * (size_t)ridx[slot] + r6] = rx[6 * slot + r6];
        }
      }
      if (__any_sync(0xffffffffu, !okw)) break;
      const int next = q0 + 5;
      // report progress every kDfWriteBatch positions (the ring has room for
      // no longer lag than that: build_df); the release makes the slot reads
      // above complete before any warp may overwrite the slots
      if (next / kDfWriteBatch != q0 / kDfWriteBatch || next >= n) {
        __syncwarp();
        if (lane == 0) st_release_s32(&wpos[kDfWarps], next >= n ? 0x7fffffff : next);
      }
    }
    return;
  }
  const int g = lane / 6, r = lane % 6;
  // failure-injection knob for tests: warp 0 never publishes its rows
  const bool publish = !(g_skip_meet && warp == 0);
  int seen_min = 0;  // a lower bound of min(wpos)
  bool ok = true;
  for (int c = 0; c < T.nch && ok; c++) {
    const int s = c % kDfStages;
    const unsigned par = (unsigned)((c / kDfStages) & 1);
    if (!wait_bar(&full[s], par) || !wait_bar(&rhsb[s], par)) {
      fail();
      ok = false;
    }
    if (__any_sync(0xffffffffu, !ok)) break;
    const unsigned char* st = smem + (size_t)s * T.stage;
    const int4 h = *reinterpret_cast<const int4*>(st);
    const int nr = h.x, nb = h.y, p0 = h.z;
    const int4* rec = reinterpret_cast<const int4*>(st + 16);
    const int* dep = reinterpret_cast<const int*>(rec + nr);
    const VT* val = reinterpret_cast<const VT*>(
        st + ((16 + 16 * (size_t)nr + 4 * (size_t)nb + 15) & ~(size_t)15));
    const double* crhs = srhs + (size_t)s * 6 * kDfRows;
    for (int k = warp; k < nr; k += kDfWarps) {
      const int pos = p0 + k;
      if (lane == 0) st_release_s32(&wpos[warp], pos);
      const int4 row = rec[k];
      const int i = row.x, b0 = row.y, cnt = row.z;
      const double rv = lane < 6 ? crhs[6 * k + lane] : 0.0;
      double acc = 0.0;
      if (g < 4) {
        for (int j = (UPPER ? 1 : 0) + g; j < cnt; j += 4) {
          const int q = dep[b0 + j];
          if (!wait_bar(&rbar[q & rmask], (unsigned)((q >> rlog) & 1))) {
            fail();
            ok = false;
            break;
          }
          acc += dot6(val + (size_t)(b0 + j) * 36 + 6 * r, rx + 6 * (size_t)(q & rmask));
        }
      }
      if (__any_sync(0xffffffffu, !ok)) {
        ok = false;
        break;
      }
      acc += __shfl_down_sync(0xffffffffu, acc, 12);
      acc += __shfl_down_sync(0xffffffffu, acc, 6);
      const double t = rv - acc;
      double v = t;
      if (UPPER) {
        const VT* Di = val + (size_t)b0 * 36;
        v = 0.0;
#pragma unroll
        for (int cc = 0; cc < 6; cc++) {
          const double tc = __shfl_sync(0xffffffffu, t, cc);
          if (lane < 6) v = fma((double)Di[6 * lane + cc], tc, v);
        }
      }
      // flow control: the slot's previous position (pos - ring) is read
      // only by rows at positions <= pos - ring + maxdist
      const int slot = pos & rmask;
      const int lim = pos - T.ring + T.maxdist;
      if (lim >= seen_min) {
        unsigned long long t0 = 0;
        for (int it = 0;; it++) {
          int m = lane <= kDfWarps ? ld_acquire_s32(&wpos[lane]) : 0x7fffffff;
          m = __reduce_min_sync(0xffffffffu, m);
          seen_min = m;
          if (m > lim) break;
          if (it == 0) t0 = gtimer();
          const int stop =
              __shfl_sync(0xffffffffu, lane == 0 && (abort_flag || gtimer() - t0 > wlim), 0);
          if (stop) {
            if (lane == 0) fail();
            ok = false;
            break;
          }
        }
        if (!ok) break;
      }
      if (lane < 6) rx[6 * slot + lane] = v;
      if (lane == 0) ridx[slot] = i;
      __syncwarp();
      if (lane == 0 && publish) mbar_arrive_local(&rbar[slot]);
    }
    if (!ok) break;
    __syncwarp();
    if (lane == 0) {
      mbar_arrive_local(&empty[s]);
      st_release_s32(&wpos[warp], p0 + nr + warp);  // its first position in the next chunk
    }
  }
  if (lane == 0) st_release_s32(&wpos[warp], 0x7fffffff);
  if (ok && tid == 0 && bytes_ctr) atomicAdd(bytes_ctr, (unsigned long long)T.abytes);
}

// Factor values into a chunk stream: block slot q of the triangle takes
// the 6x6 block src[map[q]] (zero for padding, map < 0) at element offset
// vpos[q] of the stream viewed as VT.
template <class VT>
__global__ void repack_kernel(size_t nslots, const int32_t* __restrict__ map,
                              const int64_t* __restrict__ vpos, const double* __restrict__ src,
                              VT* __restrict__ dst) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nslots * 36) return;
  const size_t q = t / 36, e = t % 36;
  const int m = map[q];
  dst[vpos[q] + e] = m >= 0 ? (VT)src[36 * (size_t)m + e] : (VT)0;
}

// ------------------------------------------------- segmented vector kernels
struct Chunks {
  int n;                   // number of chunks
  const int32_t* prob;     // chunk -> problem
  const int64_t* lo;       // chunk start (doubles, batch space)
  const int64_t* hi;       // chunk end
  const int32_t* pstart;   // problem -> first chunk, [np + 1]
};

__device__ __forceinline__ double block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) s += sh[k];
  __syncthreads();
  return s;
}

// partial[i * C.n + c] = V_i . w over chunk c, i = 0..jj, for running problems.
// w stays in registers; eight basis vectors at a time are read with all
// their loads in flight and reduced together (the same summation order as
// one vector at a time: per thread in element order, then the warp tree,
// then the warps in order).
constexpr int kDotGroup = 8;
__global__ void __launch_bounds__(kRedThreads) seg_dots(const double* __restrict__ V,
                                                        const double* __restrict__ w, size_t N,
                                                        int jj, Chunks C,
                                                        const int* __restrict__ run,
                                                        double* partial) {
  constexpr int E = kChunk / kRedThreads;  // elements per thread
  __shared__ double sh[kDotGroup][kRedThreads / 32];
  const int c = blockIdx.x;
  if (!run[C.prob[c]]) return;
  const int64_t lo = C.lo[c], hi = C.hi[c];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double wr[E];
#pragma unroll
  for (int e = 0; e < E; e++) {
    const int64_t t = lo + threadIdx.x + (int64_t)e * kRedThreads;
    wr[e] = t < hi ? w[t] : 0.0;
  }
  for (int i0 = 0; i0 <= jj; i0 += kDotGroup) {
    double acc[kDotGroup];
#pragma unroll
    for (int q = 0; q < kDotGroup; q++) {
      acc[q] = 0.0;
      if (i0 + q <= jj) {
        const double* v = V + (size_t)(i0 + q) * N;
#pragma unroll
        for (int e = 0; e < E; e++) {
          const int64_t t = lo + threadIdx.x + (int64_t)e * kRedThreads;
          if (t < hi) acc[q] = fma(v[t], wr[e], acc[q]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < kDotGroup; q++)
      for (int o = 16; o > 0; o >>= 1) acc[q] += __shfl_down_sync(0xffffffffu, acc[q], o);
    if (lane == 0)
#pragma unroll
      for (int q = 0; q < kDotGroup; q++) sh[q][warp] = acc[q];
    __syncthreads();
    if (threadIdx.x < kDotGroup && i0 + (int)threadIdx.x <= jj) {
      double s = 0.0;
      for (int k = 0; k < kRedThreads / 32; k++) s += sh[threadIdx.x][k];
      partial[(size_t)(i0 + threadIdx.x) * C.n + c] = s;
    }
    __syncthreads();
  }
}

struct GmArrays {
  double* H;       // np * (m+1) * m
  double* g;       // np * (m+1)
  double* cs;      // np * m
  double* ss;      // np * m
  double* y;       // np * m
  double* hn;      // np
  double* target;  // np
  int* jcnt;       // np
  int* run;        // np
  int* live;       // np
};

// Sum of v[c] over the chunks c0 .. c1 - 1 of a problem by one warp (every
// lane returns it; the order depends on the problem's own chunks alone).
__device__ __forceinline__ double chunk_sum(const double* v, int c0, int c1, int lane) {
  double s = 0.0;
  for (int c = c0 + lane; c < c1; c += 32) s += v[c];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}
// h_p[i] = sum of the dots' partials over p's chunks, by every chunk for
// itself (no launch of its own: a step of a small problem is a row of
// launches); the problem's first chunk also keeps H_p[i][jj] (+)= h_p[i].
// Then w -= sum_{i<=jj} h_p[i] V_i over chunk c; optional per-chunk |w|^2.
__global__ void __launch_bounds__(kRedThreads)
    seg_update(const double* __restrict__ V, double* __restrict__ w, size_t N, int jj, int m,
               Chunks C, GmArrays G, const double* __restrict__ partial, int acc_h, double* pnorm) {
  __shared__ double sh[32];
  __shared__ double hs[1024];
  const int c = blockIdx.x;
  const int p = C.prob[c];
  if (!G.run[p]) return;
  const int c0 = C.pstart[p], c1 = C.pstart[p + 1], lane = threadIdx.x & 31;
  for (int i = threadIdx.x >> 5; i <= jj; i += kRedThreads / 32) {
    const double s = chunk_sum(partial + (size_t)i * C.n, c0, c1, lane);
    if (lane == 0) {
      hs[i] = s;
      if (c == c0) {
        double* Hij = &G.H[(size_t)p * (m + 1) * m + (size_t)i * m + jj];
        *Hij = acc_h ? *Hij + s : s;
      }
    }
  }
  __syncthreads();
  const int64_t lo = C.lo[c], hi = C.hi[c];
  double acc = 0.0;
  for (int64_t t = lo + threadIdx.x; t < hi; t += blockDim.x) {
    double s = w[t];
#pragma unroll 8
    for (int i = 0; i <= jj; i++) s = fma(-hs[i], V[(size_t)i * N + t], s);
    w[t] = s;
    acc = fma(s, s, acc);
  }
  if (pnorm) {
    const double b = block_sum(acc, sh);
    if (threadIdx.x == 0) pnorm[c] = b;
  }
}
// per-chunk sum of squares over problems with mask[p] (all when mask is null)
__global__ void seg_sumsq(const double* __restrict__ v, Chunks C, const int* __restrict__ mask,
                          double* pnorm) {
  __shared__ double sh[32];
  const int c = blockIdx.x;
  if (mask && !mask[C.prob[c]]) return;
  double acc = 0.0;
  for (int64_t t = C.lo[c] + threadIdx.x; t < C.hi[c]; t += blockDim.x)
    acc = fma(v[t], v[t], acc);
  const double b = block_sum(acc, sh);
  if (threadIdx.x == 0) pnorm[c] = b;
}
__global__ void seg_norm_out(const double* pnorm, Chunks C, int np, const int* mask,
                             double* out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  if (mask && !mask[p]) return;
  double s = 0.0;
  for (int c = C.pstart[p]; c < C.pstart[p + 1]; c++) s += pnorm[c];
  out[p] = sqrt(s);
}
// dst = src / |w|: the norm from the update's per-chunk sums, by every chunk
// for itself
__global__ void __launch_bounds__(kRedThreads)
    seg_normalize(const double* __restrict__ src, double* __restrict__ dst, Chunks C,
                  const int* __restrict__ run, const double* __restrict__ pnorm) {
  const int c = blockIdx.x;
  const int p = C.prob[c];
  if (!run[p]) return;
  const double hn = sqrt(chunk_sum(pnorm, C.pstart[p], C.pstart[p + 1], threadIdx.x & 31));
  const double inv = hn > 0.0 ? 1.0 / hn : 0.0;
  for (int64_t t = C.lo[c] + threadIdx.x; t < C.hi[c]; t += blockDim.x) dst[t] = src[t] * inv;
}
__global__ void seg_scale(const double* __restrict__ src, double* __restrict__ dst, Chunks C,
                          const int* __restrict__ run, const double* __restrict__ hn) {
  const int c = blockIdx.x;
  const int p = C.prob[c];
  if (!run[p]) return;
  const double inv = hn[p] > 0.0 ? 1.0 / hn[p] : 0.0;
  for (int64_t t = C.lo[c] + threadIdx.x; t < C.hi[c]; t += blockDim.x) dst[t] = src[t] * inv;
}
// Givens update of column jj (examples/iterative/gmres.cu:672-699), one warp
// per problem. The column's running entry stays in a register, so the loads of
// the rotations do not wait for one another. seen (host memory): the problem's
// run flag and, behind the flags, the sweeps' status, for the host's poll.
__global__ void bgivens(int np, int jj, int m, int step_limit, GmArrays G,
                        const double* __restrict__ pnorm, Chunks C, const SweepCtl* ctl,
                        volatile int* seen) {
  const int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (p >= np) return;
  if (p == 0 && lane == 0) seen[np] = ctl->status;
  if (!G.run[p]) {
    if (lane == 0) seen[p] = 0;
    return;
  }
  const double hn = sqrt(chunk_sum(pnorm, C.pstart[p], C.pstart[p + 1], lane));
  if (lane != 0) return;
  double* H = G.H + (size_t)p * (m + 1) * m;
  double* g = G.g + (size_t)p * (m + 1);
  double* cs = G.cs + (size_t)p * m;
  double* ss = G.ss + (size_t)p * m;
  double a = H[jj];
#pragma unroll 4
  for (int i = 0; i < jj; i++) {
    const double c = H[(size_t)(i + 1) * m + jj], ci = cs[i], si = ss[i];
    H[(size_t)i * m + jj] = ci * a + si * c;
    a = -si * a + ci * c;
  }
  const double c = hn;
  const double hyp = sqrt(a * a + c * c);
  const double cj = hyp > 0.0 ? a / hyp : 1.0, sj = hyp > 0.0 ? c / hyp : 0.0;
  cs[jj] = cj;
  ss[jj] = sj;
  H[(size_t)jj * m + jj] = cj * a + sj * c;
  H[(size_t)(jj + 1) * m + jj] = 0.0;
  const double gj = g[jj], gn = -sj * gj;
  g[jj + 1] = gn;
  g[jj] = cj * gj;
  G.hn[p] = hn;
  G.jcnt[p] = jj + 1;
  const int run =
      !(fabs(gn) <= G.target[p] || hn == 0.0 || !isfinite(gn) || jj + 1 >= step_limit);
  G.run[p] = run;
  seen[p] = run;
}
__global__ void bbacksolve(int np, int m, GmArrays G) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np || !G.live[p]) return;
  const int j = G.jcnt[p];
  const double* H = G.H + (size_t)p * (m + 1) * m;
  const double* g = G.g + (size_t)p * (m + 1);
  double* y = G.y + (size_t)p * m;
  for (int i = j - 1; i >= 0; i--) {
    double s = g[i];
    for (int k = i + 1; k < j; k++) s -= H[(size_t)i * m + k] * y[k];
    y[i] = s / H[(size_t)i * m + i];
  }
}
// out = sum_{i < jcnt_p} y_p[i] V_i over live problems (zero otherwise)
__global__ void seg_combine(const double* __restrict__ V, size_t N, int m, Chunks C, GmArrays G,
                            double* __restrict__ out) {
  __shared__ double ys[1024];
  const int c = blockIdx.x;
  const int p = C.prob[c];
  const int j = G.live[p] ? G.jcnt[p] : 0;
  for (int i = threadIdx.x; i < j; i += blockDim.x) ys[i] = G.y[(size_t)p * m + i];
  __syncthreads();
  for (int64_t t = C.lo[c] + threadIdx.x; t < C.hi[c]; t += blockDim.x) {
    double s = 0.0;
    for (int i = 0; i < j; i++) s = fma(ys[i], V[(size_t)i * N + t], s);
    out[t] = s;
  }
}
// cycle start: beta_p = ||src_p||, g_p = (beta, 0, ...), run_p = live_p
// tfac (may be null): target = tfac[p] * beta, the Arnoldi residual
// reduction this cycle must reach.
__global__ void bcycle_init(const double* pnorm, Chunks C, int np, int m, GmArrays G,
                            const double* tfac) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  double s = 0.0;
  if (G.live[p])
    for (int c = C.pstart[p]; c < C.pstart[p + 1]; c++) s += pnorm[c];
  const double beta = sqrt(s);
  G.hn[p] = beta;
  if (tfac && G.live[p]) G.target[p] = tfac[p] * beta;
  G.jcnt[p] = 0;
  G.run[p] = (G.live[p] && beta > 0.0) ? 1 : 0;
  double* g = G.g + (size_t)p * (m + 1);
  g[0] = beta;
  for (int i = 1; i <= m; i++) g[i] = 0.0;
}
// y += a * x over problems with mask[p] (all when mask is null)
__global__ void seg_axpy(double a, const double* __restrict__ x, double* __restrict__ y,
                         Chunks C, const int* __restrict__ mask) {
  const int c = blockIdx.x;
  if (mask && !mask[C.prob[c]]) return;
  for (int64_t t = C.lo[c] + threadIdx.x; t < C.hi[c]; t += blockDim.x) y[t] += a * x[t];
}
__global__ void seg_copy(const double* __restrict__ x, double* __restrict__ y, Chunks C,
                         const int* __restrict__ mask) {
  const int c = blockIdx.x;
  if (mask && !mask[C.prob[c]]) return;
  for (int64_t t = C.lo[c] + threadIdx.x; t < C.hi[c]; t += blockDim.x) y[t] = x[t];
}
__global__ void set_target(int np, const double* norms, double rtol, GmArrays G) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < np) G.target[p] = rtol * norms[p];
}
// natural <-> batch-space permutation, one problem per blockIdx.y
struct PermEntry {
  const int32_t* perm;
  int n, off;
  const double* in;
  double* out;
};
__global__ void bpermute(const PermEntry* E, int dir) {
  const PermEntry e = E[blockIdx.y];
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 6 * e.n; t += gridDim.x * blockDim.x) {
    const int i = t / 6, k = t % 6;
    if (dir == 0)
      e.out[6 * ((size_t)e.off + e.perm[i]) + k] = e.in[t];
    else
      e.out[t] = e.in[6 * ((size_t)e.off + e.perm[i]) + k];
  }
}

}  // namespace gf

using namespace gf;

// ---------------------------------------------------------------- handles
struct gf_precond {
  gf_assembler* a = nullptr;
  int fill = 0, prec = GF_PREC_FP64;
  Pattern pat;
  int nlevL = 0, nlevU = 0;
  std::vector<int32_t> lvL, lvU;
  DevBuf<int32_t> d_rowp, d_cols, d_diag, d_amap;
  DevBuf<int32_t> d_levLptr, d_levLrows;  // factorization order
  DevBuf<int32_t> d_done;                  // per row: epoch of the factorization that finished it
  DevBuf<int4> d_steps;                    // per row: its factorization steps in order
  long long fwork = 0;                     // block updates of one factorization
  int maxrow = 0;                          // blocks of the longest row
  int sym_gpu = 0;                         // ILU(k) pattern computed on the GPU
  double sym_ms = 0.0, setup_ms = 0.0;     // host wall time of the pattern / of the whole setup
  DevBuf<double> d_lu;
  struct Tri {
    int nch = 0, stage = 0, capb = 0, capr = 0, nsplit = 1;
    int kind = TRI_LEVEL, ring = 0, maxdist = 0;
    size_t nslots = 0;
    long long abytes = 0;
    DevBuf<int64_t> off, vpos;
    DevBuf<int32_t> map;
    DevBuf<unsigned char> stream;
    int nlev = 0, groups = 0;     // ring sweep
    DevBuf<int4> tasks;
    DevBuf<int32_t> slots, lists;
    DevBuf<uint16_t> code;
  } tri[2];  // 0 = L, 1 = U
  gf_batch* self = nullptr;  // batch of one, built on first use
};

namespace gf {
// The chunks of one triangle (layout described at TriDesc): their rows, split
// over the CTAs.
struct TriPlan {
  int nsplit, capb, capr, nch;
  long long real = 0;                        // stored blocks
  std::vector<int32_t> chunk_of, grow;       // of a row: its chunk and its number in it
  std::vector<std::vector<int32_t>> hrows;   // rows of half chunk h * nch + c
  // bytes of a half chunk ahead of its values: two int4 headers, row records
  // {row, first block, blocks, row index in the chunk}, the near list, the far
  // list and rows of the next half chunk, then (16-byte aligned) values
  static int64_t head_bytes(int64_t rows, int64_t near, int64_t far1, int64_t rows1) {
    return (32 + 16 * rows + 8 * near + 8 * far1 + 4 * rows1 + 15) & ~(int64_t)15;
  }
};
static cudaError_t plan_tri(const gf_precond* p, const std::vector<int32_t>& diag, bool upper,
                            TriPlan& t) {
  const Pattern& P = p->pat;
  const int n = P.n;
  const std::vector<int32_t>& lv = upper ? p->lvU : p->lvL;
  const int nlev = upper ? p->nlevU : p->nlevL;
  auto cnt = [&](int i) { return upper ? P.rowp[i + 1] - diag[i] : diag[i] - P.rowp[i]; };
  std::vector<int32_t> ptr(nlev + 1, 0), rows(n);
  for (int i = 0; i < n; i++) ptr[lv[i] + 1]++;
  for (int l = 0; l < nlev; l++) ptr[l + 1] += ptr[l];
  {
    std::vector<int32_t> f(ptr.begin(), ptr.end() - 1);
    for (int i = 0; i < n; i++) rows[f[lv[i]]++] = i;
  }
  int maxc = 0;
  long long real = 0;
  for (int i = 0; i < n; i++) {
    maxc = std::max(maxc, cnt(i));
    real += cnt(i);
  }
  const int mc4 = (maxc + 3) & ~3;
  const int base = p->prec == GF_PREC_FP32 ? 416 : 208;
  const int capr = 128;
  // One CTA or the two CTAs of the problem's cluster per chunk, whichever
  // the chunk model of B200 clock64 traces makes cheaper: a chunk costs
  // ~1,000 cycles of copies and barriers plus ~1,900 cycles per round of
  // rows over the 16 warps of a CTA (a row's latency), and splitting it
  // adds ~1,450 cycles for the two CTAs' meeting. Splitting pays when levels
  // have more rows than one CTA's warps or more blocks than its stage.
  auto model = [&](int ns) {
    const int cb = ns > 1 ? ns * (std::max(base, ((3 * mc4 + 1) / 2 + 3) & ~3) - mc4)
                          : std::max(base, mc4);
    const int cr = ns * capr, warps = kSweepThreads / 32;
    double cyc = 0.0;
    int cur = 0, nr = 0;
    auto close = [&]() {
      const int per_cta = (nr + ns - 1) / ns;
      cyc += 1000.0 + (ns > 1 ? 1450.0 : 0.0) + 1900.0 * ((per_cta + warps - 1) / warps);
      cur = nr = 0;
    };
    for (int l = 0; l < nlev; l++) {
      for (int k = ptr[l]; k < ptr[l + 1]; k++) {
        const int c = cnt(rows[k]);
        if (nr > 0 && (cur + c > cb || nr == cr)) close();
        cur += c;
        nr++;
      }
      if (nr > 0) close();
    }
    return cyc;
  };
  const int nsplit = model(kSweepCta) < model(1) ? kSweepCta : 1;
  // per CTA: blocks of one half chunk. Split chunks are bounded so that
  // giving each row to the lighter half leaves every half within capb (a
  // half exceeds the mean by at most half a row) and a longest row fits.
  const int capb = nsplit > 1 ? std::max(base, ((3 * mc4 + 1) / 2 + 3) & ~3) : std::max(base, mc4);
  const int gcapb = nsplit > 1 ? nsplit * (capb - mc4) : capb, gcapr = nsplit * capr;
  // pass 1: chunk boundaries (row ranges of `rows`); a chunk never spans two levels
  std::vector<int32_t> ck{0};
  {
    int cur = 0, nr = 0;
    for (int l = 0; l < nlev; l++) {
      for (int k = ptr[l]; k < ptr[l + 1]; k++) {
        const int c = cnt(rows[k]);
        if (nr > 0 && (cur + c > gcapb || nr == gcapr)) {
          ck.push_back(k);
          cur = nr = 0;
        }
        cur += c;
        nr++;
      }
      if (nr > 0) {
        ck.push_back(ptr[l + 1]);
        cur = nr = 0;
      }
    }
  }
  const int nch = (int)ck.size() - 1;
  // split every chunk's rows over the CTAs: each row goes to the half with
  // fewer blocks so far (ties: fewer rows), within capr rows a half
  std::vector<int32_t> chunk_of(n), grow(n);
  std::vector<std::vector<int32_t>> hrows((size_t)kSweepCta * nch);  // [h * nch + c]
  for (int c = 0; c < nch; c++) {
    int hb[kSweepCta] = {0}, hr[kSweepCta] = {0};
    for (int k = ck[c]; k < ck[c + 1]; k++) {
      const int i = rows[k];
      int h = 0;
      for (int q = 1; q < nsplit; q++)
        if (hr[h] == capr || (hr[q] < capr && (hb[q] < hb[h] || (hb[q] == hb[h] && hr[q] < hr[h]))))
          h = q;
      chunk_of[i] = c;
      grow[i] = k - ck[c];
      hb[h] += cnt(i);
      hr[h]++;
      hrows[(size_t)h * nch + c].push_back(i);
    }
    for (int h = 0; h < kSweepCta; h++)
      if (hb[h] > capb || hr[h] > capr) return cudaErrorInvalidValue;
  }
  t.nsplit = nsplit;
  t.capb = capb;
  t.capr = capr;
  t.nch = nch;
  t.real = real;
  t.chunk_of.swap(chunk_of);
  t.grow.swap(grow);
  t.hrows.swap(hrows);
  return cudaSuccess;
}
// Bytes of a plan's largest half chunk, from counts alone.
static int tri_stage(const gf_precond* p, const std::vector<int32_t>& diag, bool upper,
                     const TriPlan& t) {
  const Pattern& P = p->pat;
  const int nch = t.nch;
  const int64_t vs = p->prec == GF_PREC_FP32 ? 4 : 8;
  int64_t stage = 0;
  for (int h = 0; h < kSweepCta; h++) {
    // of the half chunk behind this one: rows, blocks solved before the chunk ahead
    int64_t rows1 = 0, far1 = 0;
    for (int c = nch - 1; c >= 0; c--) {
      const auto& rows = t.hrows[(size_t)h * nch + c];
      int64_t near = 0, far = 0;
      for (int i : rows)
        for (int jp = upper ? diag[i] + 1 : P.rowp[i]; jp < (upper ? P.rowp[i + 1] : diag[i]); jp++)
          (t.chunk_of[P.cols[jp]] == c - 1 ? near : far)++;
      const int64_t b = near + far + (upper ? (int64_t)rows.size() : 0);
      stage = std::max(stage, TriPlan::head_bytes((int64_t)rows.size(), near, far1, rows1) +
                                  36 * vs * std::max<int64_t>(4, (b + 3) & ~(int64_t)3));
      rows1 = (int64_t)rows.size();
      far1 = far;
    }
  }
  return (int)stage;
}
// Chunk stream of one triangle.
static cudaError_t build_tri(gf_precond* p, const std::vector<int32_t>& diag, bool upper) {
  const Pattern& P = p->pat;
  const int n = P.n;
  const size_t vs = p->prec == GF_PREC_FP32 ? 4 : 8;
  TriPlan plan;
  if (const cudaError_t bad = plan_tri(p, diag, upper, plan)) return bad;
  const int nch = plan.nch;
  const auto &chunk_of = plan.chunk_of, &grow = plan.grow;
  const auto& hrows = plan.hrows;
  auto cnt = [&](int i) { return upper ? P.rowp[i + 1] - diag[i] : diag[i] - P.rowp[i]; };
  // per half chunk: stored blocks (padded), and where each block's x comes
  // from. Near: row solved by the previous chunk (either CTA; ring position
  // = its row index within that chunk); far: solved earlier (global row).
  // U's diagonal block U_ii^{-1} multiplies no x; padding is unused.
  const size_t HC = (size_t)kSweepCta * nch;
  std::vector<int32_t> nbp(HC);
  std::vector<std::vector<int32_t>> nearl(HC), farl(HC);  // pairs (slot, source)
  for (int h = 0; h < kSweepCta; h++)
    for (int c = 0; c < nch; c++) {
      const size_t hc = (size_t)h * nch + c;
      int b = 0;
      auto src = [&](int slot, int j) {
        if (chunk_of[j] == c - 1) {
          nearl[hc].push_back(slot);
          nearl[hc].push_back(grow[j]);
        } else {
          farl[hc].push_back(slot);
          farl[hc].push_back(j);
        }
      };
      for (int i : hrows[hc]) {
        if (upper) {
          b++;  // U_ii^{-1}
          for (int jp = diag[i] + 1; jp < P.rowp[i + 1]; jp++) src(b++, P.cols[jp]);
        } else {
          for (int jp = P.rowp[i]; jp < diag[i]; jp++) src(b++, P.cols[jp]);
        }
      }
      nbp[hc] = std::max(4, (b + 3) & ~3);
    }
  for (int h = 0; h < kSweepCta; h++)
    if (!farl[(size_t)h * nch].empty() || !nearl[(size_t)h * nch].empty())
      return cudaErrorInvalidValue;  // level 0 depends on nothing
  // half h's chunks are contiguous; off[h * (nch + 1) + c] is the start of half chunk (h, c)
  auto pre = [&](int h, int c) {
    const size_t hc = (size_t)h * nch + c;
    const bool more = c + 1 < nch;
    return TriPlan::head_bytes((int64_t)hrows[hc].size(), (int64_t)nearl[hc].size() / 2,
                               more ? (int64_t)farl[hc + 1].size() / 2 : 0,
                               more ? (int64_t)hrows[hc + 1].size() : 0);
  };
  std::vector<int64_t> off((size_t)kSweepCta * (nch + 1), 0);
  size_t nslots = 0;
  int stage = 0;
  int64_t pos = 0;
  for (int h = 0; h < kSweepCta; h++)
    for (int c = 0; c <= nch; c++) {
      off[(size_t)h * (nch + 1) + c] = pos;
      if (c == nch) break;
      const int64_t bytes = pre(h, c) + 36 * (int64_t)vs * nbp[(size_t)h * nch + c];
      pos += bytes;
      stage = (int)std::max<int64_t>(stage, bytes);
      nslots += nbp[(size_t)h * nch + c];
    }
  std::vector<unsigned char> bytes(pos, 0);
  std::vector<int32_t> map(nslots, -1);
  std::vector<int64_t> vpos(nslots);
  size_t q = 0;
  for (int h = 0; h < kSweepCta; h++)
    for (int c = 0; c < nch; c++) {
      const size_t hc = (size_t)h * nch + c;
      const int64_t o = off[(size_t)h * (nch + 1) + c];
      int32_t* w = reinterpret_cast<int32_t*>(bytes.data() + o);
      const int nr = (int)hrows[hc].size(), nb = nbp[hc];
      const int nn = (int)nearl[hc].size() / 2;
      const int nf1 = c + 1 < nch ? (int)farl[hc + 1].size() / 2 : 0;
      const int nr1 = c + 1 < nch ? (int)hrows[hc + 1].size() : 0;
      w[0] = nr;
      w[1] = nb;
      w[2] = nn;
      w[4] = nf1;
      w[5] = nr1;
      int32_t* rec = w + 8;
      int b = 0;
      for (int k = 0; k < nr; k++) {
        const int i = hrows[hc][k];
        rec[4 * k + 0] = i;
        rec[4 * k + 1] = b;
        rec[4 * k + 2] = cnt(i);
        rec[4 * k + 3] = grow[i];
        if (upper) {
          map[q + b++] = diag[i];
          for (int jp = diag[i] + 1; jp < P.rowp[i + 1]; jp++) map[q + b++] = jp;
        } else {
          for (int jp = P.rowp[i]; jp < diag[i]; jp++) map[q + b++] = jp;
        }
      }
      int32_t* lists = rec + 4 * nr;
      std::copy(nearl[hc].begin(), nearl[hc].end(), lists);
      lists += nearl[hc].size();
      if (c + 1 < nch) {
        std::copy(farl[hc + 1].begin(), farl[hc + 1].end(), lists);
        lists += farl[hc + 1].size();
        for (int i : hrows[hc + 1]) *lists++ = i;
      }
      const int64_t v0 = (o + pre(h, c)) / (int64_t)vs;
      for (int k = 0; k < nb; k++) vpos[q + k] = v0 + 36 * (int64_t)k;
      q += nb;
    }
  // algorithmic bytes of one sweep (compulsory unique traffic): per stored
  // block its values and column index; per row a row pointer, its
  // right-hand side and its result (each x entry is read once, however many
  // blocks multiply it)
  gf_precond::Tri& t = p->tri[upper ? 1 : 0];
  t.nsplit = plan.nsplit;
  t.abytes = plan.real * (36 * (long long)vs + 4) + (long long)n * (4 + 48 + 48) + 4;
  t.nch = nch;
  t.stage = stage;
  t.capb = plan.capb;
  t.capr = plan.capr;
  t.nslots = nslots;
  cudaError_t e = cudaSuccess;
  auto up = [&](cudaError_t x) {
    if (e == cudaSuccess) e = x;
  };
  up(t.off.upload(off));
  up(t.vpos.upload(vpos));
  up(t.map.upload(map));
  up(t.stream.upload(bytes));
  return e;
}
// Stream of one triangle for the dataflow sweep (layout described at
// TriDesc). Returns cudaSuccess with *used = false, building nothing, when
// the triangle's ring and stages do not fit one CTA's shared memory.
static cudaError_t build_df(gf_precond* p, const std::vector<int32_t>& diag, bool upper,
                            bool* used) {
  const Pattern& P = p->pat;
  const int n = P.n;
  const std::vector<int32_t>& lv = upper ? p->lvU : p->lvL;
  const int nlev = upper ? p->nlevU : p->nlevL;
  const size_t vs = p->prec == GF_PREC_FP32 ? 4 : 8;
  *used = false;
  // positions: rows by level, ties by row index
  std::vector<int32_t> ptr(nlev + 1, 0), order(n), pos(n);
  for (int i = 0; i < n; i++) ptr[lv[i] + 1]++;
  for (int l = 0; l < nlev; l++) ptr[l + 1] += ptr[l];
  {
    std::vector<int32_t> f(ptr.begin(), ptr.end() - 1);
    for (int i = 0; i < n; i++) order[f[lv[i]]++] = i;
  }
  for (int k = 0; k < n; k++) pos[order[k]] = k;
  // a row's blocks: (position multiplied, factor block), U_ii^{-1} first in U
  auto blocks = [&](int i, std::vector<std::pair<int32_t, int32_t>>& out) {
    out.clear();
    if (upper) {
      for (int jp = diag[i] + 1; jp < P.rowp[i + 1]; jp++) out.emplace_back(pos[P.cols[jp]], jp);
    } else {
      for (int jp = P.rowp[i]; jp < diag[i]; jp++) out.emplace_back(pos[P.cols[jp]], jp);
    }
    std::sort(out.begin(), out.end());
    if (upper) out.insert(out.begin(), std::make_pair(-1, diag[i]));
  };
  std::vector<std::pair<int32_t, int32_t>> bl;
  int maxdist = 1, maxcnt = 0;
  long long real = 0;
  for (int i = 0; i < n; i++) {
    blocks(i, bl);
    maxcnt = std::max(maxcnt, (int)bl.size());
    real += (long long)bl.size();
    for (auto& b : bl)
      if (b.first >= 0) maxdist = std::max(maxdist, pos[i] - b.first);
  }
  // the ring holds every position a row may still need (maxdist back) plus
  // the lag of the progress the warps report (a chunk's rows for the compute
  // warps, a report batch for the writer), so flow control never waits on a
  // warp that is itself waiting
  int ring = 64;
  while (ring < 2 * (maxdist + 1) || ring < maxdist + 2 * kDfRows + kDfWriteBatch + 8) ring *= 2;
  const int capb = std::max(vs == 4 ? 224 : 112, maxcnt), capr = kDfRows;
  // chunks: consecutive positions, at most capb blocks and capr rows
  std::vector<int32_t> ck{0};
  {
    int cb = 0, cr = 0;
    for (int k = 0; k < n; k++) {
      const int cnt = upper ? P.rowp[order[k] + 1] - diag[order[k]] : diag[order[k]] - P.rowp[order[k]];
      if (cr > 0 && (cb + cnt > capb || cr == capr)) {
        ck.push_back(k);
        cb = cr = 0;
      }
      cb += cnt;
      cr++;
    }
    ck.push_back(n);
  }
  const int nch = (int)ck.size() - 1;
  std::vector<int64_t> off(nch + 1, 0);
  auto head = [&](int c, int nb) {
    return (16 + 16 * (int64_t)(ck[c + 1] - ck[c]) + 4 * (int64_t)nb + 15) & ~(int64_t)15;
  };
  std::vector<int32_t> nbc(nch, 0);
  int stage = 0;
  for (int c = 0; c < nch; c++) {
    for (int k = ck[c]; k < ck[c + 1]; k++) {
      const int i = order[k];
      nbc[c] += upper ? P.rowp[i + 1] - diag[i] : diag[i] - P.rowp[i];
    }
    const int64_t bytes = head(c, nbc[c]) + 36 * (int64_t)vs * nbc[c];
    off[c + 1] = off[c] + bytes;
    stage = (int)std::max<int64_t>(stage, bytes);
  }
  if (df_smem_bytes(stage, ring) > kSweepSmemMax) return cudaSuccess;
  std::vector<unsigned char> bytes(off[nch], 0);
  const size_t nslots = (size_t)real;
  std::vector<int32_t> map(nslots);
  std::vector<int64_t> vpos(nslots);
  size_t q = 0;
  for (int c = 0; c < nch; c++) {
    int32_t* w = reinterpret_cast<int32_t*>(bytes.data() + off[c]);
    const int nr = ck[c + 1] - ck[c];
    w[0] = nr;
    w[1] = nbc[c];
    w[2] = ck[c];
    int32_t* rec = w + 4;
    int32_t* dep = rec + 4 * nr;
    const int64_t v0 = (off[c] + head(c, nbc[c])) / (int64_t)vs;
    int b = 0;
    for (int k = 0; k < nr; k++) {
      const int i = order[ck[c] + k];
      blocks(i, bl);
      rec[4 * k + 0] = i;
      rec[4 * k + 1] = b;
      rec[4 * k + 2] = (int)bl.size();
      for (auto& e : bl) {
        dep[b] = e.first;
        map[q] = e.second;
        vpos[q] = v0 + 36 * (int64_t)b;
        q++;
        b++;
      }
    }
  }
  gf_precond::Tri& t = p->tri[upper ? 1 : 0];
  t.kind = TRI_DATAFLOW;
  t.nsplit = 1;
  t.ring = ring;
  t.maxdist = maxdist;
  t.nch = nch;
  t.stage = stage;
  t.capb = capb;
  t.capr = capr;
  t.nslots = nslots;
  t.abytes = real * (36 * (long long)vs + 4) + (long long)n * (4 + 48 + 48) + 4;
  cudaError_t e = cudaSuccess;
  auto up = [&](cudaError_t x) {
    if (e == cudaSuccess) e = x;
  };
  up(t.off.upload(off));
  up(t.vpos.upload(vpos));
  up(t.map.upload(map));
  up(t.stream.upload(bytes));
  if (e == cudaSuccess) *used = true;
  return e;
}
// Streams of one triangle for the register-fed level sweep (layout described
// at TriDesc). Returns cudaSuccess with *used = false, building nothing, when
// the ring would not fit one CTA's shared memory.
static cudaError_t build_ring(gf_precond* p, const std::vector<int32_t>& diag, bool upper,
                              bool* used) {
  const Pattern& P = p->pat;
  const int n = P.n;
  const std::vector<int32_t>& lv = upper ? p->lvU : p->lvL;
  const int nlev = upper ? p->nlevU : p->nlevL;
  const size_t vs = p->prec == GF_PREC_FP32 ? 4 : 8;
  const int first = upper ? 1 : 0;
  *used = false;
  auto beg = [&](int i) { return upper ? diag[i] + 1 : P.rowp[i]; };
  auto end = [&](int i) { return upper ? P.rowp[i + 1] : diag[i]; };
  std::vector<int32_t> ptr(nlev + 1, 0), rows(n), pos(n);
  for (int i = 0; i < n; i++) ptr[lv[i] + 1]++;
  int maxlev = 0;
  for (int l = 0; l < nlev; l++) {
    maxlev = std::max(maxlev, ptr[l + 1]);
    ptr[l + 1] += ptr[l];
  }
  {
    std::vector<int32_t> f(ptr.begin(), ptr.end() - 1);
    for (int i = 0; i < n; i++) {
      pos[i] = f[lv[i]]++;
      rows[pos[i]] = i;
    }
  }
  int maxdist = 0;
  for (int i = 0; i < n; i++)
    for (int jp = beg(i); jp < end(i); jp++) maxdist = std::max(maxdist, pos[i] - pos[P.cols[jp]]);
  // while rows of level l are still being solved the partner may already
  // write rows of level l + 1
  const long long ring = (long long)maxdist + 2ll * maxlev + 1;
  if ((ring + 1) * 48 > (long long)kRingSmemMax || maxlev > 10000) return cudaSuccess;
  auto slot = [&](int i) { return (int)(pos[i] % ring + 1) * 48; };  // slot 0 holds zeros
  // a level's rows over the CTAs: each to the one with fewer blocks so far
  // (ties: fewer rows)
  std::vector<int32_t> mine[kRingCta];
  auto deal = [&](int l, int ns) {
    long long hb[kRingCta] = {0};
    for (auto& m : mine) m.clear();
    for (int k = ptr[l]; k < ptr[l + 1]; k++) {
      int h = 0;
      for (int q = 1; q < ns; q++)
        if (hb[q] < hb[h] || (hb[q] == hb[h] && mine[q].size() < mine[h].size())) h = q;
      hb[h] += end(rows[k]) - beg(rows[k]) + first;
      mine[h].push_back(rows[k]);
    }
  };
  auto passes = [&](int i) { return std::max(1, (end(i) - beg(i) + 15) / 16); };
  // warps that share a row of np passes which meets its CTA's warp w with
  // `left` rows to come: rows are shared while every row still finds warps of
  // its own (a barrier of helpers is used once a level; the room is 0 or less
  // once a second round began); the others take their passes one by one
  auto share = [](int np, int wpg, int w, int left) {
    return std::max(1, std::min(np, wpg - w - left));
  };
  // clocks of all levels on ns CTAs with 2, 3 and 4 groups
  auto model = [&](int ns, double (&cyc)[5]) {
    for (int l = 0; l < nlev; l++) {
      deal(l, ns);
      for (int g = 2; g <= 4; g++) {
        const int wpg = kRingWarps / g;
        int rounds = 1, most = 0;
        for (int h = 0; h < ns; h++) {
          int cnt[kRingWarps] = {0}, w = 0, left = (int)mine[h].size(), all = 0;
          for (int i : mine[h]) {
            const int np = passes(i), segs = share(np, wpg, w, --left);
            for (int q = 0; q < segs; q++) {
              int& c = cnt[w % wpg + q];
              rounds = std::max(rounds, c += np * (q + 1) / segs - np * q / segs);
            }
            w += segs;
            all += np;
          }
          most = std::max(most, all);
        }
        cyc[g] += kRingChain + (ns > 1 ? kRingSplit : 0.0) + (ns > 2 ? kRingSplit4 : 0.0) +
                  kRingIssue * most + (rounds - 1) * (kRingRound + kRingRoundG / g) + kRingLate / g;
      }
    }
  };
  int nsplit = 1, groups = 2;
  double best = 1e300;
  for (int ns = 1; ns <= kRingCta; ns *= 2) {
    double cyc[5] = {0.0};
    model(ns, cyc);
    for (int g = 2; g <= 4; g++)
      if (cyc[g] < best) {
        best = cyc[g];
        nsplit = ns;
        groups = g;
      }
  }
  const int wpg = kRingWarps / groups;
  size_t nblocks = (size_t)first * n;
  for (int i = 0; i < n; i++) nblocks += end(i) - beg(i);
  std::vector<int32_t> slots(nblocks + 4, 0), map(nblocks);
  std::vector<uint16_t> code(nblocks);
  std::vector<std::vector<int4>> lists((size_t)kRingCta * kRingWarps);
  size_t b = 0;
  long long npass = 0;
  for (int l = 0; l < nlev; l++) {
    deal(l, nsplit);
    for (int h = 0; h < nsplit; h++) {
      // eights of bytes from the other CTAs: six a row, one where there is none
      int others = 0;
      for (int q = 0; q < nsplit; q++)
        if (q != h) others += std::max<int>(1, 6 * (int)mine[q].size());
      const int w0 = h * kRingWarps + (l % groups) * wpg;
      // lists of the group's warps, this level's part
      size_t start[kRingWarps];
      for (int w = 0; w < wpg; w++) start[w] = lists[w0 + w].size();
      int w = 0, left = (int)mine[h].size();
      for (int i : mine[h]) {
        const int nb = end(i) - beg(i), np = passes(i);
        const int segs = share(np, wpg, w, --left);
        int pass = 0;
        for (int q = 0; q < segs; q++) {
          auto& L = lists[w0 + w % wpg + q];
          const int p1 = np * (q + 1) / segs;
          if (upper && q == 0) {
            map[b] = diag[i];
            code[b++] = 0;
          }
          for (int p0 = pass; pass < p1; pass++) {
            const int j0 = 16 * pass, m = std::min(16, nb - j0);
            const int flags = (pass == p0 ? kRingFirst : 0) |
                              (pass + 1 == p1 ? kRingLast | (segs - 1) << 5 : 0);
            L.push_back(make_int4(q ? -2 : i, m | flags, (int)b,
                                  q ? (l % groups) * wpg + w : slot(i)));
            for (int j = 0; j < m; j++) {
              const int jp = beg(i) + j0 + j;
              map[b] = jp;
              slots[b] = slot(P.cols[jp]);
              code[b++] = (uint16_t)(m << 8 | j);
            }
          }
        }
        w += segs;
      }
      for (int q = 0; q < wpg; q++) {
        auto& L = lists[w0 + q];
        if (L.size() == start[q]) L.push_back(make_int4(-1, 0, (int)b, 0));
        L[start[q]].y |= kRingBegin | others << 16;
        L.back().y |= kRingEnd;
        npass = std::max(npass, (long long)L.size());
      }
    }
  }
  std::vector<int4> all;
  std::vector<int32_t> where;
  for (auto& L : lists) {
    where.push_back((int32_t)all.size());
    all.insert(all.end(), L.begin(), L.end());
    all.insert(all.end(), kRingPad, make_int4(-1, 0, 0, 0));
  }
  gf_precond::Tri& t = p->tri[upper ? 1 : 0];
  t.kind = TRI_RING;
  t.nsplit = nsplit;
  t.groups = groups;
  t.ring = (int)ring;
  t.maxdist = maxdist;
  t.nch = (int)npass;
  t.nlev = nlev;
  t.nslots = nblocks;
  t.abytes = (long long)nblocks * (36 * (long long)vs + 4) + (long long)n * (4 + 48 + 48) + 4;
  cudaError_t e = cudaSuccess;
  auto up = [&](cudaError_t x) {
    if (e == cudaSuccess) e = x;
  };
  up(t.tasks.upload(all));
  up(t.slots.upload(slots));
  up(t.lists.upload(where));
  up(t.map.upload(map));
  up(t.code.upload(code));
  up(t.stream.alloc(nblocks * 36 * vs));
  if (e == cudaSuccess) *used = true;
  return e;
}
static TriDesc tri_desc(const gf_precond* p, int which) {
  const gf_precond::Tri& t = p->tri[which];
  return TriDesc{t.nch,    t.stage,  t.capb,    t.capr,    t.off.p,   t.stream.p, t.abytes,
                 t.nsplit, t.kind,   t.ring,    t.maxdist, t.tasks.p, t.slots.p,  t.lists.p,
                 t.nlev,   (int)t.nslots, t.groups};
}
static size_t sweep_smem(const gf_precond* p, int which) {
  const gf_precond::Tri& t = p->tri[which];
  if (t.kind == TRI_RING) return 48 * ((size_t)t.ring + 1);
  return t.kind == TRI_DATAFLOW ? df_smem_bytes(t.stage, t.ring)
                                : sweep_smem_bytes(t.stage, t.capb, t.capr);
}
}  // namespace gf

// Host memory and events through which a solve follows its problems: norms and
// step counts, and the run flags (and the sweeps' status) of the latest two
// GMRES steps, which bgivens writes straight to the host. Pinned memory takes
// milliseconds to get and to free, so a batch hands its block on: blocks for
// up to kPollProblems problems go to a list that keeps at most kPollKept of
// them (4 KB each) and frees the others. A block belongs to one batch at a
// time, and a batch's solves have ended when it is destroyed. With the last
// assembler the list is given back but for one block: a program that makes
// and destroys all its objects for every solve would pay for a new one each
// time (33x21 plate, FP64: 4.2-5.1 instead of 2.8 ms). A block is handed out
// only while it is what it was: a device reset frees it behind the list's
// back, so its memory has to be pinned still and to bear its mark.
constexpr int kPollProblems = 64, kPollKept = 8;
struct PollBlock {
  void* mem = nullptr;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  int device = -1, cap = 0;
  static size_t bytes(int cap) {
    return ((sizeof(double) * 2 * cap + sizeof(int) * (3 * (size_t)cap + 2) + 7) & ~(size_t)7) +
           sizeof(uint64_t);
  }
  uint64_t* mark() const {
    return reinterpret_cast<uint64_t*>(static_cast<char*>(mem) + bytes(cap)) - 1;
  }
  uint64_t sign() const {
    return 0x9e3779b97f4a7c15ull * (uint64_t)reinterpret_cast<uintptr_t>(mem) ^
           (uint64_t)reinterpret_cast<uintptr_t>(ev[0]);
  }
  bool intact() const {
    cudaPointerAttributes at;
    const cudaError_t e = cudaPointerGetAttributes(&at, mem);
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess && at.type == cudaMemoryTypeHost && *mark() == sign();
  }
};
static std::mutex g_poll_mu;
static std::vector<PollBlock> g_poll_kept;
static int g_poll_users = 0;  // assemblers alive

struct SolvePoll {
  PollBlock blk;
  double* norms = nullptr;  // 2 np
  int* counts = nullptr;    // np
  int* flags = nullptr;     // 2 (np + 1)
  cudaEvent_t* ev = blk.ev;
  SolvePoll() = default;
  SolvePoll(const SolvePoll&) = delete;
  SolvePoll& operator=(const SolvePoll&) = delete;
  int* seen(int step, int np) const { return flags + (size_t)(step & 1) * (np + 1); }
  static void free_block(PollBlock& b) {
    for (auto& x : b.ev)
      if (x) cudaEventDestroy(x);
    if (b.mem) cudaFreeHost(b.mem);
    b = PollBlock();
  }
  cudaError_t create(int np) {
    if (blk.mem) return cudaSuccess;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const int cap = std::max(np, kPollProblems);
    if (cap == kPollProblems) {
      std::lock_guard<std::mutex> lk(g_poll_mu);
      for (size_t k = 0; k < g_poll_kept.size() && !blk.mem;) {
        if (g_poll_kept[k].device != dev) {
          k++;
          continue;
        }
        if (g_poll_kept[k].intact()) blk = g_poll_kept[k];
        g_poll_kept.erase(g_poll_kept.begin() + k);
      }
    }
    if (!blk.mem) {
      blk.device = dev;
      blk.cap = cap;
      e = cudaHostAlloc(&blk.mem, PollBlock::bytes(cap), cudaHostAllocMapped | cudaHostAllocPortable);
      for (auto& x : blk.ev)
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&x, cudaEventDisableTiming);
      if (e != cudaSuccess) {
        free_block(blk);
        return e;
      }
      *blk.mark() = blk.sign();
    }
    norms = static_cast<double*>(blk.mem);
    counts = reinterpret_cast<int*>(norms + 2 * np);
    flags = counts + np;
    return cudaSuccess;
  }
  ~SolvePoll() {
    for (auto& x : blk.ev)
      if (x) cudaEventSynchronize(x);  // no step of an aborted solve writes here any more
    if (blk.mem && blk.cap == kPollProblems) {
      std::lock_guard<std::mutex> lk(g_poll_mu);
      if (g_poll_kept.size() < (size_t)(g_poll_users > 0 ? kPollKept : 1)) {
        g_poll_kept.push_back(blk);
        return;
      }
    }
    free_block(blk);
  }
};

namespace gf {
void count_assemblers(int more) {
  std::vector<PollBlock> gone;
  {
    std::lock_guard<std::mutex> lk(g_poll_mu);
    g_poll_users += more;
    while (g_poll_users == 0 && g_poll_kept.size() > 1) {
      gone.push_back(g_poll_kept.back());
      g_poll_kept.pop_back();
    }
  }
  for (auto& b : gone)
    if (b.intact()) SolvePoll::free_block(b);
}
}  // namespace gf

struct gf_batch {
  int np = 0, nrows = 0, maxlevL = 0, maxlevU = 0;
  size_t smemL = 0, smemU = 0;  // dynamic shared memory of the level-synchronous sweeps
  size_t dfL = 0, dfU = 0;      // ... of the dataflow sweeps
  size_t ringL = 0, ringU = 0;  // ... and of the register-fed level sweeps
  // problems solved by each kind
  int nlevelL = 0, nlevelU = 0, ndfL = 0, ndfU = 0, nringL = 0, nringU = 0;
  int ctasL = 1, ctasU = 1;      // cluster size of the register-fed sweeps
  int pprec = GF_PREC_FP64;      // factor precision shared by the batch's preconditioners
  size_t N = 0;  // doubles in batch space
  std::vector<gf_assembler*> asms;
  std::vector<gf_bsr*> mats;
  std::vector<gf_precond*> pcs;
  std::vector<int> offs;
  DevBuf<ProbDev> d_desc;
  DevBuf<int32_t> d_row_prob;
  DevBuf<SweepCtl> d_ctl;
  int gave_up = 0, quiet = 0;        // SweepCtl's, when it was last read
  DevBuf<double> d_tmp, d_b, d_x;
  int nchunks = 0;
  DevBuf<int32_t> d_cprob, d_pstart;
  int fac_grid = 0;                  // CTAs of the dataflow factorization
  int fac_vals = 0;                  // row blocks staged per warp
  DevBuf<int32_t> d_fcta, d_fgrab;   // problem of each CTA; per-problem row counters
  DevBuf<int64_t> d_clo, d_chi;
  DevBuf<PermEntry> d_perm_b, d_perm_x, d_perm_out;
  int m = 0;
  DevBuf<double> V, H, g, cs, ss, y, hn, target, partial, pnorm, w, t, r, d, e, norms, bnorm;
  DevBuf<double> tfac;
  DevBuf<int> jcnt, run, live, live2;
  SolvePoll poll;
  gf::BatchAsm* basm = nullptr;  // launch data of the batched assembly
  int scatter = 0;               // 0: coloured, GF_ASSEMBLE_ATOMIC: atomic
  Chunks chunks() const { return Chunks{nchunks, d_cprob.p, d_clo.p, d_chi.p, d_pstart.p}; }
  ~gf_batch() { gf::batch_asm_free(basm); }
};

namespace gf {

static int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// Order of the factorization steps of every row (ord[r0 .. di) = slots of
// the row's lower blocks in the order they are taken). Step k must follow
// every step k' whose row k' has column k in its upper part (k' updates
// A_ik), and nothing else; among the steps whose predecessors are done the
// one whose row k has the lowest lower level goes first (ties: lower
// column). Rows finish roughly in level order in the dataflow
// factorization, so the steps that wait for the last-finishing rows move to
// the end of the row and the steps after them shrink to those that really
// depend on them. Rows longer than kOrderMax lower blocks keep ascending
// order (complete factors: there every step depends on the previous one).
constexpr int kOrderMax = 128;
static void step_order_rows(const Pattern& P, const std::vector<int32_t>& diag,
                            const std::vector<int32_t>& lv, std::vector<int32_t>& ord, int i0,
                            int i1) {
  std::vector<int32_t> indeg, head, nxt, to, heap;
  for (int i = i0; i < i1; i++) {
    const int r0 = P.rowp[i], di = diag[i], m = di - r0;
    if (m <= 1 || m > kOrderMax) {
      for (int t = r0; t < di; t++) ord[t] = t;
      continue;
    }
    indeg.assign(m, 0);
    head.assign(m, -1);
    nxt.clear();
    to.clear();
    for (int a = 0; a < m; a++) {
      const int k = P.cols[r0 + a];
      // columns of U(k) that are lower columns of row i after a (both ascending)
      int u = diag[k] + 1;
      const int u1 = P.rowp[k + 1];
      int b = a + 1;
      while (u < u1 && b < m) {
        const int cu = P.cols[u], cb = P.cols[r0 + b];
        if (cu < cb) {
          u++;
        } else if (cb < cu) {
          b++;
        } else {
          to.push_back(b);
          nxt.push_back(head[a]);
          head[a] = (int)to.size() - 1;
          indeg[b]++;
          u++;
          b++;
        }
      }
    }
    // Kahn's algorithm with a min-heap on (level, column) = (lv, local index)
    auto key = [&](int a) { return ((long long)lv[P.cols[r0 + a]] << 32) | (unsigned)a; };
    auto cmp = [&](int x, int y) { return key(x) > key(y); };
    heap.clear();
    for (int a = 0; a < m; a++)
      if (indeg[a] == 0) heap.push_back(a);
    std::make_heap(heap.begin(), heap.end(), cmp);
    int t = r0;
    while (!heap.empty()) {
      std::pop_heap(heap.begin(), heap.end(), cmp);
      const int a = heap.back();
      heap.pop_back();
      ord[t++] = r0 + a;
      for (int e = head[a]; e >= 0; e = nxt[e])
        if (--indeg[to[e]] == 0) {
          heap.push_back(to[e]);
          std::push_heap(heap.begin(), heap.end(), cmp);
        }
    }
  }
}
// Length of the factorization's dependency chain in step units when every
// row takes its steps in the order `ord` (null: ascending) and finishing a
// row costs two steps: a row's step k starts once its previous step and
// row k are done.
static double step_chain(const Pattern& P, const std::vector<int32_t>& diag,
                         const std::vector<int32_t>* ord) {
  std::vector<double> done(P.n, 0.0);
  double longest = 0.0;
  for (int i = 0; i < P.n; i++) {
    double t = 0.0;
    for (int s = P.rowp[i]; s < diag[i]; s++) {
      const int k = P.cols[ord ? (*ord)[s] : s];
      t = std::max(t, done[k]) + 1.0;
    }
    done[i] = t + 2.0;
    longest = std::max(longest, done[i]);
  }
  return longest;
}

// Rows are independent: host threads take contiguous row ranges. The order
// is kept only where it shortens the dependency chain by 15 % or more
// (natural-ordered grids, where a row's last-finishing dependency otherwise
// sits before its same-line steps: 18-24 % on plates, a 1.5-3x faster
// factorization); elsewhere (RCM orders: 0-9 %) the steps stay ascending,
// the order of the host and reference factorizations. The summation order
// matters on ill-conditioned shells: on the jittered 100x50 cantilever
// (RCM, ILU(8), factor entries up to 3e8) the two orders give factors with
// the same backward error, 6e-16, but right-preconditioned GMRES needs 59
// steps with the ascending one and 118 with the reordered one.
static void step_order(const Pattern& P, const std::vector<int32_t>& diag,
                       const std::vector<int32_t>& lv, std::vector<int32_t>& ord) {
  const int n = P.n;
  ord.assign(P.nnz(), 0);
  const int nt = (int)std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
  if (nt == 1 || n < 4096) {
    step_order_rows(P, diag, lv, ord, 0, n);
  } else {
    std::vector<std::thread> th;
    for (int t = 0; t < nt; t++) {
      const int i0 = (int)((long long)n * t / nt), i1 = (int)((long long)n * (t + 1) / nt);
      th.emplace_back([&, i0, i1] { step_order_rows(P, diag, lv, ord, i0, i1); });
    }
    for (auto& x : th) x.join();
  }
  if (step_chain(P, diag, &ord) * 1.15 > step_chain(P, diag, nullptr))
    for (int i = 0; i < n; i++)
      for (int t = P.rowp[i]; t < diag[i]; t++) ord[t] = t;
}

// CTAs of the dataflow factorization for one problem given `budget` CTAs for
// it: at least one, at most one per 32 rows (four rows per warp) and 128.
static int fac_ctas_cap(const gf_precond* p, int budget) {
  return std::max(1, std::min({budget, 128, p->pat.n / (4 * kFacWarps)}));
}
// A preconditioner factored alone gets the whole GPU (one CTA per SM).
static int fac_ctas_alone(const gf_precond* p) { return fac_ctas_cap(p, sm_count()); }

// Spreads one CTA per SM over the batch's problems in proportion to their
// block updates to the power 0.7 (largest remainders first), within each
// problem's cap: the small problems' dependency chains need a few CTAs more
// than their share of the updates (64-plate batch on B200, factorization
// ms by exponent: 0.5 43.3, 0.6 40.1, 0.7 38.0, 0.85 39.2, 1 41.4, 1.5 56.6);
// fills cta_prob with the problem of every CTA.
static void fac_plan(const std::vector<gf_precond*>& pcs, std::vector<int>& ctas,
                     std::vector<int32_t>& cta_prob) {
  const int np = (int)pcs.size(), total = std::max(sm_count(), np);
  double W = 0.0;
  for (auto* p : pcs) W += std::pow((double)std::max<long long>(p->fwork, 1), 0.7);
  ctas.assign(np, 1);
  std::vector<std::pair<double, int>> rem;
  int used = 0;
  for (int k = 0; k < np; k++) {
    const double want = total * std::pow((double)std::max<long long>(pcs[k]->fwork, 1), 0.7) / W;
    const int cap = fac_ctas_cap(pcs[k], total);
    ctas[k] = std::max(1, std::min(cap, (int)want));
    used += ctas[k];
    if (ctas[k] < cap) rem.push_back({want - ctas[k], k});
  }
  std::sort(rem.begin(), rem.end(), [](const auto& a, const auto& b) { return a.first > b.first; });
  for (size_t q = 0; q < rem.size() && used < total; q++) {
    ctas[rem[q].second]++;
    used++;
  }
  cta_prob.clear();
  for (int k = 0; k < np; k++)
    for (int c = 0; c < ctas[k]; c++) cta_prob.push_back(k);
}

// Descriptor table (rebuilt when a buffer such as the FP32 matrix copy is
// allocated).
static gf_status upload_desc(gf_batch* B) {
  std::vector<ProbDev> h(B->np);
  for (int k = 0; k < B->np; k++) {
    gf_assembler* a = B->asms[k];
    gf_precond* p = B->pcs[k];
    ProbDev& d = h[k];
    d.n = a->nnodes;
    d.off = B->offs[k];
    d.rowp = a->d_rowp.p;
    d.cols = a->d_cols.p;
    d.A64 = B->mats[k]->vals.p;
    d.A32 = B->mats[k]->vals32.p;
    d.prowp = p->d_rowp.p;
    d.pcols = p->d_cols.p;
    d.pdiag = p->d_diag.p;
    d.LU64 = p->d_lu.p;
    d.nlevL = p->nlevL;
    d.done = p->d_done.p;
    d.psteps = p->d_steps.p;
    d.nlevU = p->nlevU;
    d.levLptr = p->d_levLptr.p;
    d.levLrows = p->d_levLrows.p;
    d.L = tri_desc(p, 0);
    d.U = tri_desc(p, 1);
  }
  GF_CUDA(cudaMemcpy(B->d_desc.p, h.data(), sizeof(ProbDev) * B->np, cudaMemcpyHostToDevice));
  return GF_OK;
}

static gf_status batch_build(gf_batch* B) {
  const int np = B->np;
  B->offs.resize(np + 1);
  B->offs[0] = 0;
  for (int k = 0; k < np; k++) B->offs[k + 1] = B->offs[k] + B->asms[k]->nnodes;
  B->nrows = B->offs[np];
  B->N = (size_t)6 * B->nrows;
  std::vector<int32_t> row_prob(B->nrows);
  B->pprec = B->pcs[0]->prec;
  for (int k = 0; k < np; k++) {
    if (B->pcs[k]->prec != B->pprec) return GF_INVALID_ARG;  // one factor precision per batch
    for (int w = 0; w < 2; w++) {
      const int kind = B->pcs[k]->tri[w].kind;
      size_t& sm = kind == TRI_DATAFLOW ? (w ? B->dfU : B->dfL)
                   : kind == TRI_RING   ? (w ? B->ringU : B->ringL)
                                        : (w ? B->smemU : B->smemL);
      sm = std::max(sm, sweep_smem(B->pcs[k], w));
      if (kind == TRI_RING) {
        int& c = w ? B->ctasU : B->ctasL;
        c = std::max(c, B->pcs[k]->tri[w].nsplit);
      }
      (kind == TRI_DATAFLOW ? (w ? B->ndfU : B->ndfL)
       : kind == TRI_RING   ? (w ? B->nringU : B->nringL)
                            : (w ? B->nlevelU : B->nlevelL))++;
    }
    for (int i = 0; i < B->asms[k]->nnodes; i++) row_prob[B->offs[k] + i] = k;
    B->maxlevL = std::max(B->maxlevL, B->pcs[k]->nlevL);
    B->maxlevU = std::max(B->maxlevU, B->pcs[k]->nlevU);
  }
  // reduction chunks aligned to each problem
  std::vector<int32_t> cprob, pstart(np + 1);
  std::vector<int64_t> clo, chi;
  for (int k = 0; k < np; k++) {
    pstart[k] = (int32_t)cprob.size();
    const int64_t lo = 6ll * B->offs[k], hi = 6ll * B->offs[k + 1];
    for (int64_t s = lo; s < hi; s += kChunk) {
      cprob.push_back(k);
      clo.push_back(s);
      chi.push_back(std::min(hi, s + (int64_t)kChunk));
    }
  }
  pstart[np] = (int32_t)cprob.size();
  B->nchunks = (int)cprob.size();
  cudaError_t e = cudaSuccess;
  auto up = [&](cudaError_t x) {
    if (e == cudaSuccess) e = x;
  };
  up(B->d_desc.alloc(np));
  {
    std::vector<int> ctas;
    std::vector<int32_t> cta_prob;
    fac_plan(B->pcs, ctas, cta_prob);
    B->fac_grid = (int)cta_prob.size();
    // stage the longest row (up to kFacVals blocks)
    int most = 8;
    for (auto* p : B->pcs) most = std::max(most, p->maxrow);
    B->fac_vals = std::min(most, kFacVals);
    up(B->d_fcta.upload(cta_prob));
    up(B->d_fgrab.alloc(np));
  }
  up(B->d_row_prob.upload(row_prob));
  up(B->d_ctl.alloc(1));
  if (e == cudaSuccess) up(cudaMemset(B->d_ctl.p, 0, sizeof(SweepCtl)));
  up(B->d_tmp.alloc(B->N));
  up(B->d_b.alloc(B->N));
  up(B->d_x.alloc(B->N));
  up(B->d_cprob.upload(cprob));
  up(B->d_pstart.upload(pstart));
  up(B->d_clo.upload(clo));
  up(B->d_chi.upload(chi));
  up(B->d_perm_b.alloc(np));
  up(B->d_perm_x.alloc(np));
  up(B->d_perm_out.alloc(np));
  up(B->norms.alloc(np));
  up(B->bnorm.alloc(np));
  up(B->live2.alloc(np));
  if (e != cudaSuccess) {
    set_last_error("batch build", e);
    return e == cudaErrorMemoryAllocation ? GF_OOM : GF_CUDA_ERROR;
  }
  return upload_desc(B);
}

static gf_status ensure_gmres(gf_batch* B, int m) {
  if (B->m == m) return GF_OK;
  const int np = B->np;
  cudaError_t e = cudaSuccess;
  auto al = [&](cudaError_t x) {
    if (e == cudaSuccess) e = x;
  };
  al(B->V.alloc((size_t)(m + 1) * B->N));
  al(B->H.alloc((size_t)np * (m + 1) * m));
  al(B->g.alloc((size_t)np * (m + 1)));
  al(B->cs.alloc((size_t)np * m));
  al(B->ss.alloc((size_t)np * m));
  al(B->y.alloc((size_t)np * m));
  al(B->hn.alloc(np));
  al(B->target.alloc(np));
  al(B->tfac.alloc(np));
  al(B->partial.alloc((size_t)(m + 1) * B->nchunks));
  al(B->pnorm.alloc(B->nchunks));
  al(B->w.alloc(B->N));
  al(B->t.alloc(B->N));
  al(B->r.alloc(B->N));
  al(B->d.alloc(B->N));
  al(B->e.alloc(B->N));
  al(B->jcnt.alloc(np));
  al(B->run.alloc(np));
  al(B->live.alloc(np));
  al(B->poll.create(np));
  if (e != cudaSuccess) {
    set_last_error("gmres workspace", e);
    B->m = 0;
    return e == cudaErrorMemoryAllocation ? GF_OOM : GF_CUDA_ERROR;
  }
  GF_CUDA(cudaMemset(B->H.p, 0, sizeof(double) * B->H.n));
  B->m = m;
  return GF_OK;
}

static GmArrays arrays(gf_batch* B) {
  return GmArrays{B->H.p,      B->g.p,    B->cs.p,  B->ss.p, B->y.p, B->hn.p,
                  B->target.p, B->jcnt.p, B->run.p, B->live.p};
}


// Sweep timing for benchmarks (gf_timing_enable / gf_timing_read): CUDA
// events bracket the two sweep launches of every preconditioner apply on the
// launching stream, and the sweeps add their algorithmic bytes to a device
// counter. Off by default; the events come from a pool that is drained
// (synchronised and summed) when it runs full.
namespace {
struct Timing {
  std::mutex mu;
  bool on = false;
  unsigned long long* d_bytes = nullptr;
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> pool;
  size_t used = 0;
  double ms = 0.0;
  long long launches = 0;
};
Timing g_timing;
constexpr size_t kTimingPool = 8192;
cudaError_t timing_drain_locked() {
  for (size_t k = 0; k < g_timing.used; k++) {
    float t = 0.f;
    cudaError_t e = cudaEventSynchronize(g_timing.pool[k].second);
    if (e == cudaSuccess) e = cudaEventElapsedTime(&t, g_timing.pool[k].first, g_timing.pool[k].second);
    if (e != cudaSuccess) return e;
    g_timing.ms += t;
  }
  g_timing.used = 0;
  return cudaSuccess;
}
}  // namespace
// Records the opening event of one sweep pair when timing is on; *e1 gets
// the closing event to record after the second launch.
static gf_status timing_begin(cudaStream_t st, unsigned long long** ctr, cudaEvent_t* e1) {
  std::lock_guard<std::mutex> lk(g_timing.mu);
  if (!g_timing.on) return GF_OK;
  if (g_timing.used == g_timing.pool.size()) {
    if (g_timing.pool.size() < kTimingPool) {
      cudaEvent_t a, b;
      GF_CUDA(cudaEventCreate(&a));
      GF_CUDA(cudaEventCreate(&b));
      g_timing.pool.emplace_back(a, b);
    } else {
      GF_CUDA(timing_drain_locked());
    }
  }
  auto& pr = g_timing.pool[g_timing.used++];
  GF_CUDA(cudaEventRecord(pr.first, st));
  *e1 = pr.second;
  *ctr = g_timing.d_bytes;
  g_timing.launches += 2;
  return GF_OK;
}

// z = U^{-1} L^{-1} r for problems with live[p] (all when live is null).
// The factor values are in the preconditioners' precision (one per batch),
// independent of the precision of the Krylov loop that calls this.
// One triangle of every problem of the batch: the dataflow kernel for the
// problems whose triangle has a dataflow stream, the level-synchronous
// kernel for the others (each kernel skips the other kind's problems).
template <class VT, bool UPPER>
static cudaError_t launch_tri(gf_batch* B, cudaStream_t st, const int* live, const double* rhs,
                              double* out, unsigned long long* ctr) {
  // the same caps for every batch: threads launching batches with different
  // footprints concurrently must not lower them under each other
  cudaError_t e = cudaSuccess;
  if (UPPER ? B->ndfU : B->ndfL) {
    e = cudaFuncSetAttribute(bsweep_df<VT, UPPER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kSweepSmemMax);
    if (e != cudaSuccess) return e;
    ::gf::count_launch();
    bsweep_df<VT, UPPER><<<B->np, kDfThreads, UPPER ? B->dfU : B->dfL, st>>>(
        B->d_desc.p, live, rhs, out, B->d_ctl.p, ctr);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  if (UPPER ? B->nlevelU : B->nlevelL) {
    e = cudaFuncSetAttribute(bsweep_tma<VT, UPPER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kSweepSmemMax);
    if (e != cudaSuccess) return e;
    e = launch_sweep(bsweep_tma<VT, UPPER>, kSweepCta, kSweepThreads, B->np, UPPER ? B->smemU : B->smemL, st,
                     B->d_desc.p, live, rhs, out, B->d_ctl.p, ctr);
    if (e != cudaSuccess) return e;
  }
  if (UPPER ? B->nringU : B->nringL) {
    e = cudaFuncSetAttribute(bsweep_ring<VT, UPPER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kSweepSmemMax);
    if (e != cudaSuccess) return e;
    e = launch_sweep(bsweep_ring<VT, UPPER>, UPPER ? B->ctasU : B->ctasL, kRingThreads, B->np,
                     UPPER ? B->ringU : B->ringL, st, B->d_desc.p, live, rhs, out, B->d_ctl.p, ctr);
  }
  return e;
}

static bool sweeps_fit(const gf_batch* B) {
  return B->smemL <= kSweepSmemMax && B->smemU <= kSweepSmemMax && B->dfL <= kSweepSmemMax &&
         B->dfU <= kSweepSmemMax;
}

// y = L^{-1} r into tmp, z = U^{-1} y, for the problems with live[p].
template <class VT>
static gf_status bsweeps(gf_batch* B, const int* live, const double* r, double* tmp, double* z,
                         cudaStream_t st, bool timed) {
  unsigned long long* ctr = nullptr;
  cudaEvent_t e1 = nullptr;
  if (timed && timing_begin(st, &ctr, &e1) != GF_OK) return GF_CUDA_ERROR;
  GF_CUDA((launch_tri<VT, false>(B, st, live, r, tmp, ctr)));
  GF_CUDA((launch_tri<VT, true>(B, st, live, tmp, z, ctr)));
  GF_CHECK_LAUNCH();
  if (e1) GF_CUDA(cudaEventRecord(e1, st));
  return GF_OK;
}
template <class VT>
static gf_status bprecond(gf_batch* B, const int* live, const double* r, double* z,
                          cudaStream_t st) {
  if (!sweeps_fit(B)) return GF_INVALID_ARG;
  return B->pprec == GF_PREC_FP32 ? bsweeps<float>(B, live, r, B->d_tmp.p, z, st, true)
                                  : bsweeps<double>(B, live, r, B->d_tmp.p, z, st, true);
}

template <class VT>
static gf_status bspmv(gf_batch* B, const int* live, const double* x, double alpha, double beta,
                       double* y, cudaStream_t st) {
  bspmv_kernel<VT><<<(B->nrows + 7) / 8, 256, 0, st>>>(B->nrows, B->d_row_prob.p, B->d_desc.p,
                                                       live, x, alpha, beta, y); ::gf::count_launch();
  GF_CHECK_LAUNCH();
  return GF_OK;
}

// Reads and clears the status flags that the batch's kernels have recorded
// since the last read (timeouts of bounded waits, zero pivots). Flags are
// cleared only here, after they have been read, so a flag set by a launch
// whose caller did not wait (gf_precond_apply) is reported by the next call
// that reads them.
static gf_status read_ctl(gf_batch* B, cudaStream_t st, SweepCtl* h) {
  GF_CUDA(cudaMemcpyAsync(h, B->d_ctl.p, sizeof(SweepCtl), cudaMemcpyDeviceToHost, st));
  GF_CUDA(cudaMemsetAsync(B->d_ctl.p, 0, sizeof(SweepCtl), st));
  GF_CUDA(cudaStreamSynchronize(st));
  B->gave_up = h->gave_up;
  B->quiet = h->quiet;
  return GF_OK;
}
static gf_status ctl_status(const SweepCtl& h) {
  if (h.status & ST_TIMEOUT) {
    set_last_error_text("a bounded device-side wait ran out (a stalled copy or partner CTA)");
    return GF_TIMEOUT;
  }
  if (h.status & ST_ZERO_PIVOT) {
    set_last_error_text("singular diagonal block in block row " + std::to_string(h.pivot - 1) +
                        " (batch space)");
    return GF_ZERO_PIVOT;
  }
  return GF_OK;
}

static gf_status batch_factor(gf_batch* B, cudaStream_t st) {
  for (int k = 0; k < B->np; k++) {
    gf_precond* p = B->pcs[k];
    const size_t nv = (size_t)36 * p->pat.nnz();
    GF_CUDA(cudaMemsetAsync(p->d_lu.p, 0, sizeof(double) * nv, st));
    const size_t na = (size_t)36 * p->a->pat.nnz();
    scatter_values_kernel<<<(unsigned)((na + 255) / 256), 256, 0, st>>>(
        p->a->pat.nnz(), p->d_amap.p, B->mats[k]->vals.p, p->d_lu.p); ::gf::count_launch();
  }
  GF_CHECK_LAUNCH();
  {
    // a fresh epoch per launch: flags left by earlier factorizations (of any
    // batch holding these preconditioners) never equal it
    static std::atomic<int> epochs{0};
    int epoch = ++epochs;
    if (epoch <= 0) {
      epochs = 1;
      epoch = 1;
    }
    GF_CUDA(cudaMemsetAsync(B->d_fgrab.p, 0, sizeof(int32_t) * B->np, st));
    ::gf::count_launch();
    GF_CUDA(cudaFuncSetAttribute(bfactor_df, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kFacSmemMax));
    bfactor_df<<<(unsigned)B->fac_grid, kFacWarps * 32, kFacWarps * fac_warp_smem(B->fac_vals),
                 st>>>(B->d_desc.p, B->d_fcta.p, B->d_fgrab.p, epoch, B->fac_vals, B->d_ctl.p);
  }
  GF_CHECK_LAUNCH();
  for (int k = 0; k < B->np; k++) {
    gf_precond* p = B->pcs[k];
    for (int w = 0; w < 2; w++) {
      gf_precond::Tri& t = p->tri[w];
      const unsigned nb = (unsigned)((t.nslots * 36 + 255) / 256);
      if (t.nslots == 0) continue;
      if (t.kind == TRI_RING) {
        if (p->prec == GF_PREC_FP32)
          repack_ring_kernel<float><<<nb, 256, 0, st>>>(t.nslots, t.map.p, t.code.p, p->d_lu.p,
                                                        reinterpret_cast<float*>(t.stream.p));
        else
          repack_ring_kernel<double><<<nb, 256, 0, st>>>(t.nslots, t.map.p, t.code.p, p->d_lu.p,
                                                         reinterpret_cast<double*>(t.stream.p));
        ::gf::count_launch();
        continue;
      }
      if (p->prec == GF_PREC_FP32)
        repack_kernel<float><<<nb, 256, 0, st>>>(t.nslots, t.map.p, t.vpos.p, p->d_lu.p,
                                                  reinterpret_cast<float*>(t.stream.p));
      else
        repack_kernel<double><<<nb, 256, 0, st>>>(t.nslots, t.map.p, t.vpos.p, p->d_lu.p,
                                                   reinterpret_cast<double*>(t.stream.p));
      ::gf::count_launch();
    }
  }
  GF_CHECK_LAUNCH();
  SweepCtl h;
  gf_status s = read_ctl(B, st, &h);
  if (s != GF_OK) return s;
  return ctl_status(h);
}

// Batched restarted GMRES on A x = b (batch space) for problems with
// live0[p] != 0. side 1: right preconditioning (Givens residual = true
// residual); side 0: left (the reference's choice). Per-problem outputs:
// iters, restarts, rel (true ||b - A x|| / ||b||).
template <class VT>
static gf_status bgmres(gf_batch* B, const double* b, double* x, int m, int max_it, double rtol,
                        int side, const std::vector<int>& live0,
                        std::vector<int>& iters, std::vector<int>& restarts,
                        std::vector<double>& rel, cudaStream_t st) {
  const int np = B->np;
  gf_status s = ensure_gmres(B, m);
  if (s != GF_OK) return s;
  const Chunks C = B->chunks();
  const GmArrays G = arrays(B);
  const int nc = B->nchunks;
  const int pb = (np + 127) / 128;
  double* const hbn = B->poll.norms;  // host: |b|, then |r| per problem
  double* const rn = hbn + np;
  int* const jc = B->poll.counts;
  std::vector<double> bn(np, 1.0);
  GF_CUDA(cudaMemcpyAsync(B->live.p, live0.data(), sizeof(int) * np, cudaMemcpyHostToDevice, st));
  seg_sumsq<<<nc, kRedThreads, 0, st>>>(b, C, nullptr, B->pnorm.p); ::gf::count_launch();
  seg_norm_out<<<pb, 128, 0, st>>>(B->pnorm.p, C, np, nullptr, B->bnorm.p); ::gf::count_launch();
  GF_CUDA(cudaMemcpyAsync(hbn, B->bnorm.p, sizeof(double) * np, cudaMemcpyDeviceToHost, st));
  if (side != 0) set_target<<<pb, 128, 0, st>>>(np, B->bnorm.p, rtol, G), ::gf::count_launch();
  GF_CHECK_LAUNCH();
  std::vector<int> live = live0;
  std::vector<double> tf(np, 0.0);
  iters.assign(np, 0);
  restarts.assign(np, 0);
  rel.assign(np, 0.0);
  int steps_total = 0;
  bool first = true;
  while (true) {
    // r = b - A x and the true relative residual of every live problem
    seg_copy<<<nc, kRedThreads, 0, st>>>(b, B->r.p, C, B->live.p); ::gf::count_launch();
    s = bspmv<VT>(B, B->live.p, x, -1.0, 1.0, B->r.p, st);
    if (s != GF_OK) return s;
    seg_sumsq<<<nc, kRedThreads, 0, st>>>(B->r.p, C, B->live.p, B->pnorm.p); ::gf::count_launch();
    seg_norm_out<<<pb, 128, 0, st>>>(B->pnorm.p, C, np, B->live.p, B->norms.p); ::gf::count_launch();
    GF_CUDA(cudaMemcpyAsync(rn, B->norms.p, sizeof(double) * np, cudaMemcpyDeviceToHost, st));
    GF_CUDA(cudaStreamSynchronize(st));
    if (first)
      for (int p = 0; p < np; p++)
        if (hbn[p] != 0.0) bn[p] = hbn[p];
    bool any = false, bad = false;
    for (int p = 0; p < np; p++) {
      if (!live[p]) continue;
      rel[p] = rn[p] / bn[p];
      if (!std::isfinite(rel[p])) {
        bad = true;
        live[p] = 0;
      } else if (rel[p] <= rtol) {
        live[p] = 0;
      } else {
        any = true;
        if (!first) restarts[p]++;
      }
    }
    first = false;
    if (bad) return GF_NAN;
    if (!any || steps_total >= max_it) break;
    GF_CUDA(cudaMemcpyAsync(B->live.p, live.data(), sizeof(int) * np, cudaMemcpyHostToDevice,
                            st));
    const double* src = B->r.p;
    if (side == 0) {
      s = bprecond<VT>(B, B->live.p, B->r.p, B->t.p, st);
      if (s != GF_OK) return s;
      src = B->t.p;
      // Left preconditioning minimises ||M^-1 r||, which can sit far from
      // ||r|| when M is ill-conditioned: every cycle asks the preconditioned
      // residual to drop by the factor the true residual still needs (with
      // a margin of 2 after the first cycle).
      for (int p = 0; p < np; p++)
        tf[p] = live[p] ? (restarts[p] ? 0.5 : 1.0) * rtol * bn[p] / rn[p] : 0.0;
      GF_CUDA(cudaMemcpyAsync(B->tfac.p, tf.data(), sizeof(double) * np, cudaMemcpyHostToDevice,
                              st));
    }
    seg_sumsq<<<nc, kRedThreads, 0, st>>>(src, C, B->live.p, B->pnorm.p); ::gf::count_launch();
    bcycle_init<<<pb, 128, 0, st>>>(B->pnorm.p, C, np, m, G, side == 0 ? B->tfac.p : nullptr);
    ::gf::count_launch();
    seg_scale<<<nc, kRedThreads, 0, st>>>(src, B->V.p, C, B->run.p, B->hn.p); ::gf::count_launch();
    GF_CHECK_LAUNCH();
    const int steps = std::min(m, max_it - steps_total);
    for (int jj = 0; jj < steps; jj++) {
      const double* vj = B->V.p + (size_t)jj * B->N;
      if (side == 0) {
        s = bspmv<VT>(B, B->run.p, vj, 1.0, 0.0, B->t.p, st);
        if (s == GF_OK) s = bprecond<VT>(B, B->run.p, B->t.p, B->w.p, st);
      } else {
        s = bprecond<VT>(B, B->run.p, vj, B->t.p, st);
        if (s == GF_OK) s = bspmv<VT>(B, B->run.p, B->t.p, 1.0, 0.0, B->w.p, st);
      }
      if (s != GF_OK) return s;
      for (int pass = 0; pass < 2; pass++) {  // CGS2
        seg_dots<<<nc, kRedThreads, 0, st>>>(B->V.p, B->w.p, B->N, jj, C, B->run.p, B->partial.p);
        ::gf::count_launch();
        seg_update<<<nc, kRedThreads, 0, st>>>(B->V.p, B->w.p, B->N, jj, m, C, G, B->partial.p,
                                               pass, pass ? B->pnorm.p : nullptr);
        ::gf::count_launch();
      }
      seg_normalize<<<nc, kRedThreads, 0, st>>>(B->w.p, B->V.p + (size_t)(jj + 1) * B->N, C,
                                                B->run.p, B->pnorm.p);
      ::gf::count_launch();
      bgivens<<<(np + 3) / 4, 128, 0, st>>>(np, jj, m, steps, G, B->pnorm.p, C, B->d_ctl.p,
                                            B->poll.seen(jj, np));
      ::gf::count_launch();
      GF_CHECK_LAUNCH();
      GF_CUDA(cudaEventRecord(B->poll.ev[jj & 1], st));
      // The step before this one: the GPU keeps a step in hand while the host
      // launches the next, and at most one step runs after the last problem
      // has converged (all its kernels return at once). A poll every 25 steps
      // let a solve of six steps launch 19 such steps: 0.9 ms of 3.3 ms.
      const int look = jj + 1 < steps ? jj - 1 : jj;
      if (look < 0) continue;
      GF_CUDA(cudaEventSynchronize(B->poll.ev[look & 1]));
      const volatile int* was = B->poll.seen(look, np);
      // a sweep whose bounded wait ran out left a partial z: stop (the
      // caller reads and clears the flag)
      if (was[np] & ST_TIMEOUT) {
        GF_CUDA(cudaStreamSynchronize(st));
        return GF_TIMEOUT;
      }
      bool running = false;
      for (int p = 0; p < np && !running; p++) running = was[p] != 0;
      if (!running) break;
    }
    bbacksolve<<<pb, 128, 0, st>>>(np, m, G); ::gf::count_launch();
    seg_combine<<<nc, kRedThreads, 0, st>>>(B->V.p, B->N, m, C, G, B->w.p); ::gf::count_launch();
    GF_CHECK_LAUNCH();
    if (side == 1) {
      s = bprecond<VT>(B, B->live.p, B->w.p, B->t.p, st);
      if (s != GF_OK) return s;
      seg_axpy<<<nc, kRedThreads, 0, st>>>(1.0, B->t.p, x, C, B->live.p); ::gf::count_launch();
    } else {
      seg_axpy<<<nc, kRedThreads, 0, st>>>(1.0, B->w.p, x, C, B->live.p); ::gf::count_launch();
    }
    GF_CHECK_LAUNCH();
    GF_CUDA(cudaMemcpyAsync(jc, B->jcnt.p, sizeof(int) * np, cudaMemcpyDeviceToHost, st));
    GF_CUDA(cudaStreamSynchronize(st));
    int mx = 0;
    for (int p = 0; p < np; p++)
      if (live[p]) {
        iters[p] += jc[p];
        mx = std::max(mx, jc[p]);
      }
    steps_total += mx;
  }
  return GF_OK;
}

// Full solve of the batch (vectors in batch space): FP64 GMRES, or FP64
// iterative refinement around an FP32-valued inner GMRES (FP32 SpMV + FP32
// ILU apply with FP64 vectors and accumulation).
static gf_status batch_solve_space(gf_batch* B, const gf_solve_opts& o,
                                   std::vector<gf_solve_stats>& S, cudaStream_t st) {
  const int np = B->np;
  auto t0 = std::chrono::steady_clock::now();
  std::vector<int> live(np, 1), iters, rest;
  std::vector<double> rel;
  S.assign(np, gf_solve_stats{});
  gf_status result = GF_OK;
  if (!o.mixed) {
    result = bgmres<double>(B, B->d_b.p, B->d_x.p, o.restart, o.max_iters, o.rtol, o.side,
                            live, iters, rest, rel, st);
    for (int p = 0; p < np && !iters.empty(); p++) {
      S[p].iterations = iters[p];
      S[p].restarts = rest[p];
      S[p].rel_residual = rel[p];
    }
  } else {
    for (int k = 0; k < np; k++) {
      gf_bsr* A = B->mats[k];
      const size_t n36 = (size_t)36 * A->a->pat.nnz();
      if (A->vals32.n != n36) {
        GF_CUDA(A->vals32.alloc(n36));
        gf_status s2 = upload_desc(B);
        if (s2 != GF_OK) return s2;
      }
      convert_kernel<float><<<(unsigned)((n36 + 255) / 256), 256, 0, st>>>(n36, A->vals.p,
                                                                           A->vals32.p); ::gf::count_launch();
    }
    GF_CHECK_LAUNCH();
    gf_status s = ensure_gmres(B, o.restart);
    if (s != GF_OK) return s;
    const Chunks C = B->chunks();
    const int nc = B->nchunks, pb = (np + 127) / 128;
    std::vector<double> bn(np), rn(np);
    seg_sumsq<<<nc, kRedThreads, 0, st>>>(B->d_b.p, C, nullptr, B->pnorm.p); ::gf::count_launch();
    seg_norm_out<<<pb, 128, 0, st>>>(B->pnorm.p, C, np, nullptr, B->bnorm.p); ::gf::count_launch();
    GF_CUDA(cudaMemcpyAsync(bn.data(), B->bnorm.p, sizeof(double) * np, cudaMemcpyDeviceToHost,
                            st));
    GF_CUDA(cudaStreamSynchronize(st));
    for (int p = 0; p < np; p++)
      if (bn[p] == 0.0) bn[p] = 1.0;
    std::vector<int> tot_it(np, 0), tot_rs(np, 0), nref(np, 0);
    std::vector<double> relv(np, 1.0);
    int refine = 0;
    while (true) {
      GF_CUDA(cudaMemcpyAsync(B->live2.p, live.data(), sizeof(int) * np, cudaMemcpyHostToDevice,
                              st));
      seg_copy<<<nc, kRedThreads, 0, st>>>(B->d_b.p, B->d.p, C, B->live2.p); ::gf::count_launch();
      s = bspmv<double>(B, B->live2.p, B->d_x.p, -1.0, 1.0, B->d.p, st);
      if (s != GF_OK) return s;
      seg_sumsq<<<nc, kRedThreads, 0, st>>>(B->d.p, C, B->live2.p, B->pnorm.p); ::gf::count_launch();
      seg_norm_out<<<pb, 128, 0, st>>>(B->pnorm.p, C, np, B->live2.p, B->norms.p); ::gf::count_launch();
      GF_CUDA(cudaMemcpyAsync(rn.data(), B->norms.p, sizeof(double) * np,
                              cudaMemcpyDeviceToHost, st));
      GF_CUDA(cudaStreamSynchronize(st));
      bool any = false;
      for (int p = 0; p < np; p++) {
        if (!live[p]) continue;
        relv[p] = rn[p] / bn[p];
        if (!std::isfinite(relv[p])) {
          result = GF_NAN;
          live[p] = 0;
        } else if (relv[p] <= o.rtol) {
          live[p] = 0;
        } else {
          any = true;
        }
      }
      if (!any || refine >= o.max_refine) break;
      int maxit = 0;
      for (int p = 0; p < np; p++)
        if (live[p]) maxit = std::max(maxit, o.max_iters - tot_it[p]);
      if (maxit <= 0) break;
      // inner solve A32 e = r from zero
      GF_CUDA(cudaMemsetAsync(B->e.p, 0, sizeof(double) * B->N, st));
      s = bgmres<float>(B, B->d.p, B->e.p, o.restart, maxit, o.inner_rtol, o.side,
                        live, iters, rest, rel, st);
      if (s != GF_OK) {
        result = s;
        break;
      }
      GF_CUDA(cudaMemcpyAsync(B->live2.p, live.data(), sizeof(int) * np, cudaMemcpyHostToDevice,
                              st));
      seg_axpy<<<nc, kRedThreads, 0, st>>>(1.0, B->e.p, B->d_x.p, C, B->live2.p); ::gf::count_launch();
      GF_CHECK_LAUNCH();
      for (int p = 0; p < np; p++)
        if (live[p]) {
          tot_it[p] += iters[p];
          tot_rs[p] += rest[p];
          nref[p]++;
        }
      refine++;
    }
    for (int p = 0; p < np; p++) {
      S[p].iterations = tot_it[p];
      S[p].restarts = tot_rs[p];
      S[p].refinements = nref[p];
      S[p].rel_residual = relv[p];
    }
  }
  const double ms =
      std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  for (int p = 0; p < np; p++) {
    S[p].time_ms = ms;
    // hard failures (NaN, CUDA, timeout) mark every problem; otherwise each
    // problem's status is its own convergence
    gf_status sp = result;
    if (sp == GF_OK || sp == GF_NOT_CONVERGED)
      sp = (S[p].rel_residual <= o.rtol) ? GF_OK : GF_NOT_CONVERGED;
    S[p].status = sp;
    if (result == GF_OK && sp != GF_OK) result = sp;
  }
  return result;
}

static gf_status batch_create_impl(int n, gf_assembler* const* asms, gf_bsr* const* mats,
                                   gf_precond* const* pcs, gf_batch** out) {
  gf_batch* B = new gf_batch();
  B->np = n;
  B->asms.assign(asms, asms + n);
  B->mats.assign(mats, mats + n);
  B->pcs.assign(pcs, pcs + n);
  gf_status s = batch_build(B);
  if (s != GF_OK) {
    delete B;
    return s;
  }
  *out = B;
  return GF_OK;
}

static gf_status self_batch(gf_precond* p, gf_bsr* A) {
  if (p->self && p->self->mats[0] == A) return GF_OK;
  if (p->self) {
    delete p->self;
    p->self = nullptr;
  }
  gf_assembler* a = p->a;
  return batch_create_impl(1, &a, &A, &p, &p->self);
}

static bool opts_ok(const gf_solve_opts& o) {
  return o.restart >= 1 && o.restart <= 1000 && o.max_iters >= 1 && o.rtol > 0.0 &&
         o.check_every >= 1 && (o.side == 0 || o.side == 1) && o.max_refine >= 0 &&
         (!o.mixed || o.inner_rtol > 0.0);
}

}  // namespace gf

// ------------------------------------------------------------------ C ABI
extern "C" {

gf_status gf_precond_create(gf_assembler* a, int32_t fill_level, int32_t precision,
                            gf_precond** out) {
  return gf_precond_create_ex(a, fill_level, precision, GF_SWEEP_AUTO, out);
}

gf_status gf_precond_create_ex(gf_assembler* a, int32_t fill_level, int32_t precision,
                               int32_t sweep, gf_precond** out) {
  if (!a || !out || fill_level < 0 || (precision != GF_PREC_FP64 && precision != GF_PREC_FP32) ||
      sweep < GF_SWEEP_AUTO || sweep > GF_SWEEP_LEVEL)
    return GF_INVALID_ARG;
  const auto t_setup = std::chrono::steady_clock::now();
  gf_precond* p = new gf_precond();
  p->a = a;
  p->fill = fill_level;
  p->prec = precision;
  {
    const auto t0 = std::chrono::steady_clock::now();
    if (fill_level == 0) {
      p->pat = a->pat;
    } else {
      p->sym_gpu = iluk_pattern_gpu(a->pat, fill_level, p->pat) ? 1 : 0;
      if (!p->sym_gpu) p->pat = iluk_pattern(a->pat, fill_level);
    }
    p->sym_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  }
  const int n = a->nnodes;
  std::vector<int32_t> diag(n), amap(a->pat.nnz());
  for (int i = 0; i < n; i++) {
    const int32_t* b0 = p->pat.cols.data() + p->pat.rowp[i];
    const int32_t* b1 = p->pat.cols.data() + p->pat.rowp[i + 1];
    diag[i] = (int32_t)(std::lower_bound(b0, b1, i) - p->pat.cols.data());
    for (int jp = a->pat.rowp[i]; jp < a->pat.rowp[i + 1]; jp++) {
      const int32_t* f = std::lower_bound(b0, b1, a->pat.cols[jp]);
      amap[jp] = (int32_t)(f - p->pat.cols.data());
    }
  }
  p->nlevL = levels(p->pat, true, p->lvL);
  p->nlevU = levels(p->pat, false, p->lvU);
  auto group = [n](const std::vector<int32_t>& lv, int nl, std::vector<int32_t>& ptr,
                   std::vector<int32_t>& rows) {
    ptr.assign(nl + 1, 0);
    for (int i = 0; i < n; i++) ptr[lv[i] + 1]++;
    for (int l = 0; l < nl; l++) ptr[l + 1] += ptr[l];
    rows.resize(n);
    std::vector<int32_t> fill(ptr.begin(), ptr.end() - 1);
    for (int i = 0; i < n; i++) rows[fill[lv[i]]++] = i;
  };
  std::vector<int32_t> lptr, lrows;
  group(p->lvL, p->nlevL, lptr, lrows);
  cudaError_t e = cudaSuccess;
  auto up = [&](cudaError_t x) {
    if (e == cudaSuccess) e = x;
  };
  up(p->d_rowp.upload(p->pat.rowp));
  up(p->d_cols.upload(p->pat.cols));
  up(p->d_diag.upload(diag));
  up(p->d_amap.upload(amap));
  up(p->d_levLptr.upload(lptr));
  up(p->d_levLrows.upload(lrows));
  up(p->d_lu.alloc((size_t)36 * p->pat.nnz()));
  up(p->d_done.alloc((size_t)n));
  {
    std::vector<int32_t> ord;
    step_order(p->pat, diag, p->lvL, ord);
    DevBuf<int32_t> d_ord;
    up(d_ord.upload(ord));
    up(p->d_steps.alloc((size_t)p->pat.nnz()));
    if (e == cudaSuccess) {
      step_table_kernel<<<(unsigned)((n + 7) / 8), 256>>>(n, p->d_rowp.p, p->d_cols.p, p->d_diag.p,
                                                          d_ord.p, p->d_steps.p);
      ::gf::count_launch();
      up(cudaGetLastError());
      up(cudaStreamSynchronize(nullptr));  // d_ord ends here
    }
  }
  if (e == cudaSuccess) up(cudaMemset(p->d_done.p, 0, sizeof(int32_t) * (size_t)n));
  // block updates of one factorization: per step (i, k) the block L_ik and
  // one update per block of U(k)
  p->fwork = 0;
  for (int i = 0; i < n; i++) p->maxrow = std::max(p->maxrow, p->pat.rowp[i + 1] - p->pat.rowp[i]);
  for (int i = 0; i < n; i++)
    for (int kp = p->pat.rowp[i]; kp < diag[i]; kp++) {
      const int k = p->pat.cols[kp];
      p->fwork += p->pat.rowp[k + 1] - diag[k];
    }
  bool refused = false;
  for (int w = 0; w < 2 && e == cudaSuccess; w++) {
    bool df = false;
    if (sweep == GF_SWEEP_DATAFLOW) e = build_df(p, diag, w == 1, &df);
    // the factors that are refused for their longest row are those that the
    // chunked level sweep cannot stage, whichever sweep solves them: short
    // rows always fit, for others its chunks are counted (150x140 plate,
    // complete factor, FP64: laid out instead, they took 1,000 of 1,090 ms of
    // setup beside the pattern)
    if (sweep == GF_SWEEP_AUTO) {
      int most = 0;
      for (int i = 0; i < n; i++)
        most = std::max(most, w ? p->pat.rowp[i + 1] - diag[i] : diag[i] - p->pat.rowp[i]);
      if (most > kRingRowAlways) {
        TriPlan plan;
        e = plan_tri(p, diag, w == 1, plan);
        if (e != cudaSuccess) break;
        refused = sweep_smem_bytes(tri_stage(p, diag, w == 1, plan), plan.capb, plan.capr) >
                  kSweepSmemMax;
        if (refused) break;
      }
      e = build_ring(p, diag, w == 1, &df);
    }
    if (e == cudaSuccess && !df) {
      if (sweep == GF_SWEEP_DATAFLOW) {
        set_last_error_text("gf_precond_create_ex: the dataflow sweep's ring and stages of this "
                            "factor do not fit one CTA's shared memory");
        delete p;
        return GF_INVALID_ARG;
      }
      e = build_tri(p, diag, w == 1);
    }
  }
  auto fits = [&](int w) {
    return sweep_smem(p, w) <= kSweepSmemMax;
  };
  if (refused || (e == cudaSuccess && !(fits(0) && fits(1)))) {
    set_last_error_text("gf_precond_create: the ILU(" + std::to_string(fill_level) +
                        ") factor has rows too long for the triangular sweep's "
                        "shared-memory stage; use a lower fill level");
    delete p;
    return GF_INVALID_ARG;  // a factor row longer than one staging buffer
  }
  if (e != cudaSuccess) {
    set_last_error("gf_precond_create", e);
    delete p;
    return e == cudaErrorMemoryAllocation ? GF_OOM : GF_CUDA_ERROR;
  }
  p->setup_ms =
      std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_setup).count();
  *out = p;
  return GF_OK;
}

gf_status gf_precond_destroy(gf_precond* p) {
  if (p && p->self) delete p->self;
  delete p;
  return GF_OK;
}

gf_status gf_precond_info(const gf_precond* p, int32_t* nnzb, int32_t* nl, int32_t* nu) {
  if (!p) return GF_INVALID_ARG;
  if (nnzb) *nnzb = p->pat.nnz();
  if (nl) *nl = p->nlevL;
  if (nu) *nu = p->nlevU;
  return GF_OK;
}

gf_status gf_precond_setup_info(const gf_precond* p, int32_t* symbolic_on_gpu, double* symbolic_ms,
                                double* setup_ms) {
  if (!p) return GF_INVALID_ARG;
  if (symbolic_on_gpu) *symbolic_on_gpu = p->sym_gpu;
  if (symbolic_ms) *symbolic_ms = p->sym_ms;
  if (setup_ms) *setup_ms = p->setup_ms;
  return GF_OK;
}

gf_status gf_precond_layout(const gf_precond* p, int32_t* nsplit_L, int32_t* nsplit_U,
                            int32_t* fac_ctas, int32_t* chunks_L, int32_t* chunks_U) {
  if (!p) return GF_INVALID_ARG;
  if (nsplit_L) *nsplit_L = std::min(p->tri[0].nsplit, 2);
  if (nsplit_U) *nsplit_U = std::min(p->tri[1].nsplit, 2);
  if (fac_ctas) *fac_ctas = fac_ctas_alone(p);
  if (chunks_L) *chunks_L = p->tri[0].nch;
  if (chunks_U) *chunks_U = p->tri[1].nch;
  return GF_OK;
}

gf_status gf_precond_factor_layout(const gf_precond* p, int32_t* staged, int32_t* mapped) {
  if (!p) return GF_INVALID_ARG;
  int ns = 0, nm = 0;
  const Pattern& P = p->pat;
  for (int i = 0; i < P.n; i++) {
    const int r0 = P.rowp[i], r1 = P.rowp[i + 1];
    ns += r1 - r0 <= kFacVals;
    nm += fac_mapped(P.cols[r0], P.cols[r1 - 1]);
  }
  if (staged) *staged = ns;
  if (mapped) *mapped = nm;
  return GF_OK;
}

gf_status gf_precond_sweeps(const gf_precond* p, int32_t* kind_L, int32_t* kind_U,
                            int32_t* ring_L, int32_t* ring_U) {
  if (!p) return GF_INVALID_ARG;
  auto kind = [](const gf_precond::Tri& t) {
    return t.kind == TRI_DATAFLOW ? GF_SWEEP_DATAFLOW : GF_SWEEP_LEVEL;
  };
  if (kind_L) *kind_L = kind(p->tri[0]);
  if (kind_U) *kind_U = kind(p->tri[1]);
  auto slots = [](const gf_precond::Tri& t) { return t.kind == TRI_DATAFLOW ? t.ring : 0; };
  if (ring_L) *ring_L = slots(p->tri[0]);
  if (ring_U) *ring_U = slots(p->tri[1]);
  return GF_OK;
}

gf_status gf_precond_sweep_layout(const gf_precond* p, int32_t upper, int32_t* kernel,
                                  int32_t* ctas, int32_t* groups) {
  if (!p || upper < 0 || upper > 1) return GF_INVALID_ARG;
  const gf_precond::Tri& t = p->tri[upper];
  if (kernel)
    *kernel = t.kind == TRI_RING       ? GF_SWEEP_KERNEL_RING
              : t.kind == TRI_DATAFLOW ? GF_SWEEP_KERNEL_DATAFLOW
                                       : GF_SWEEP_KERNEL_CHUNKED;
  if (ctas) *ctas = t.nsplit;
  if (groups) *groups = t.kind == TRI_RING ? t.groups : 1;
  return GF_OK;
}

gf_status gf_precond_status(gf_precond* p, void* stream) {
  if (!p) return GF_INVALID_ARG;
  if (!p->self) return GF_OK;  // nothing has run
  SweepCtl h;
  gf_status s = read_ctl(p->self, as_stream(stream), &h);
  if (s != GF_OK) return s;
  return ctl_status(h);
}

gf_status gf_test_set_waits(unsigned long long wait_ns, int32_t skip_meetings) {
  const unsigned long long w = wait_ns ? wait_ns : kWaitNs;
  const int k = skip_meetings ? 1 : 0;
  GF_CUDA(cudaMemcpyToSymbol(g_wait_ns, &w, sizeof(w)));
  GF_CUDA(cudaMemcpyToSymbol(g_skip_meet, &k, sizeof(k)));
  return GF_OK;
}

int32_t gf_test_kept_blocks(void) {
  std::lock_guard<std::mutex> lk(g_poll_mu);
  return (int32_t)g_poll_kept.size();
}

gf_status gf_test_sweep_exits(const gf_precond* p, int32_t* gave_up, int32_t* quiet) {
  if (!p) return GF_INVALID_ARG;
  if (gave_up) *gave_up = p->self ? p->self->gave_up : 0;
  if (quiet) *quiet = p->self ? p->self->quiet : 0;
  return GF_OK;
}

gf_status gf_precond_get(const gf_precond* p, int32_t* rowPtr, int32_t* colPtr,
                         double* h_values) {
  if (!p) return GF_INVALID_ARG;
  if (rowPtr) std::copy(p->pat.rowp.begin(), p->pat.rowp.end(), rowPtr);
  if (colPtr) std::copy(p->pat.cols.begin(), p->pat.cols.end(), colPtr);
  if (h_values)
    GF_CUDA(cudaMemcpy(h_values, p->d_lu.p, sizeof(double) * 36 * p->pat.nnz(),
                       cudaMemcpyDeviceToHost));
  return GF_OK;
}

gf_status gf_precond_factor(gf_precond* p, gf_bsr* A, void* stream) {
  if (!p || !A || A->a != p->a) return GF_INVALID_ARG;
  gf_status s = self_batch(p, A);
  if (s != GF_OK) return s;
  return batch_factor(p->self, as_stream(stream));
}

gf_status gf_precond_apply(gf_precond* p, const double* d_r, double* d_z, void* stream) {
  if (!p || !d_r || !d_z || !p->self) return GF_INVALID_ARG;
  cudaStream_t st = as_stream(stream);
  gf_batch* B = p->self;
  gf_status s = bprecond<double>(B, nullptr, d_r, B->d_x.p, st);
  if (s != GF_OK) return s;
  GF_CUDA(cudaMemcpyAsync(d_z, B->d_x.p, sizeof(double) * B->N, cudaMemcpyDeviceToDevice, st));
  return GF_OK;
}

// ---- preconditioner apply without allocation --------------------------
// The intermediate vector of gf_precond_apply_noalloc. One array per device
// for the whole process; its address on a device is looked up once, by the
// first call made with that device current.
static __device__ __align__(256) double g_noalloc_y[GF_NOALLOC_MAX_DOUBLES];
static constexpr int kNoAllocDevices = 64;
static std::mutex g_noalloc_mu;
static double* g_noalloc_ptr[kNoAllocDevices] = {};

gf_status gf_precond_apply_noalloc(gf_precond* p, const double* d_r, double* d_z, void* stream) {
  if (!p || !d_r || !d_z || !p->self) return GF_INVALID_ARG;
  gf_batch* B = p->self;
  const size_t need = (size_t)6 * p->pat.n;
  if (need > (size_t)GF_NOALLOC_MAX_DOUBLES) {
    set_last_error_text("gf_precond_apply_noalloc: the problem needs " + std::to_string(need) +
                        " doubles of scratch, more than the fixed " +
                        std::to_string(GF_NOALLOC_MAX_DOUBLES));
    return GF_INVALID_ARG;
  }
  int dev = 0;
  GF_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocDevices) {
    set_last_error_text("gf_precond_apply_noalloc: device index " + std::to_string(dev) +
                        " is above the " + std::to_string(kNoAllocDevices) +
                        " devices this entry point supports");
    return GF_INVALID_ARG;
  }
  double* y = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
      void* a = nullptr;
      GF_CUDA(cudaGetSymbolAddress(&a, g_noalloc_y));
      g_noalloc_ptr[dev] = static_cast<double*>(a);
    }
    y = g_noalloc_ptr[dev];
  }
  if (!sweeps_fit(B)) {
    set_last_error_text("gf_precond_apply_noalloc: the sweeps need more shared memory than a "
                        "CTA has");
    return GF_INVALID_ARG;
  }
  // the same two sweeps as gf_precond_apply; y in the fixed array and z
  // written straight into d_z (a batch of one starts at offset 0)
  const gf_status s = p->prec == GF_PREC_FP32
                          ? bsweeps<float>(B, nullptr, d_r, y, d_z, as_stream(stream), false)
                          : bsweeps<double>(B, nullptr, d_r, y, d_z, as_stream(stream), false);
  return s;
}

gf_status gf_timing_enable(int32_t enable) {
  std::lock_guard<std::mutex> lk(g_timing.mu);
  GF_CUDA(timing_drain_locked());
  g_timing.ms = 0.0;
  g_timing.launches = 0;
  if (enable && !g_timing.d_bytes) {
    void* p = nullptr;
    GF_CUDA(cudaMalloc(&p, sizeof(unsigned long long)));
    g_timing.d_bytes = static_cast<unsigned long long*>(p);
  }
  if (g_timing.d_bytes) GF_CUDA(cudaMemset(g_timing.d_bytes, 0, sizeof(unsigned long long)));
  g_timing.on = enable != 0;
  return GF_OK;
}

gf_status gf_timing_read(double* sweep_ms, long long* sweep_launches, double* sweep_bytes) {
  std::lock_guard<std::mutex> lk(g_timing.mu);
  GF_CUDA(timing_drain_locked());
  unsigned long long b = 0;
  if (g_timing.d_bytes)
    GF_CUDA(cudaMemcpy(&b, g_timing.d_bytes, sizeof(b), cudaMemcpyDeviceToHost));
  if (sweep_ms) *sweep_ms = g_timing.ms;
  if (sweep_launches) *sweep_launches = g_timing.launches;
  if (sweep_bytes) *sweep_bytes = (double)b;
  return GF_OK;
}

void gf_solve_opts_default(gf_solve_opts* o) {
  if (!o) return;
  o->restart = 50;
  o->max_iters = 5000;
  o->rtol = 1e-8;
  o->side = 1;
  o->mixed = 0;
  o->inner_rtol = 1e-4;
  o->max_refine = 30;
  o->check_every = 25;
}

gf_status gf_batch_create(int32_t n, gf_assembler* const* asms, gf_bsr* const* mats,
                          gf_precond* const* pcs, gf_batch** out) {
  if (n <= 0 || !asms || !mats || !pcs || !out) return GF_INVALID_ARG;
  for (int k = 0; k < n; k++)
    if (!asms[k] || !mats[k] || !pcs[k] || mats[k]->a != asms[k] || pcs[k]->a != asms[k])
      return GF_INVALID_ARG;
  return batch_create_impl(n, asms, mats, pcs, out);
}

gf_status gf_batch_destroy(gf_batch* b) {
  delete b;
  return GF_OK;
}

gf_status gf_batch_assemble(gf_batch* B, void* stream) {
  return gf_batch_assemble_ex(B, nullptr, stream);
}

gf_status gf_batch_assemble_ex(gf_batch* B, const double* const* d_thick, void* stream) {
  if (!B) return GF_INVALID_ARG;
  std::vector<double*> values(B->np);
  for (int k = 0; k < B->np; k++) values[k] = B->mats[k]->vals.p;
  return batch_assemble(B->basm, B->asms, values, d_thick, GF_ASSEMBLE_FUSE_BCS | B->scatter,
                        as_stream(stream));
}

gf_status gf_batch_set_scatter(gf_batch* B, int32_t flags) {
  if (!B || (flags != 0 && flags != GF_ASSEMBLE_ATOMIC)) return GF_INVALID_ARG;
  B->scatter = flags;
  return GF_OK;
}

gf_status gf_batch_factor(gf_batch* B, void* stream) {
  if (!B) return GF_INVALID_ARG;
  return batch_factor(B, as_stream(stream));
}

gf_status gf_batch_solve(gf_batch* B, const double* const* d_b, double* const* d_x,
                         const gf_solve_opts* opts, gf_solve_stats* stats, void* stream) {
  if (!B || !d_b || !d_x) return GF_INVALID_ARG;
  gf_solve_opts o;
  gf_solve_opts_default(&o);
  if (opts) o = *opts;
  if (!opts_ok(o)) return GF_INVALID_ARG;
  for (int k = 0; k < B->np; k++)
    if (!d_b[k] || !d_x[k]) return GF_INVALID_ARG;
  cudaStream_t st = as_stream(stream);
  std::vector<PermEntry> eb(B->np), ex(B->np), eo(B->np);
  int maxn = 0;
  for (int k = 0; k < B->np; k++) {
    gf_assembler* a = B->asms[k];
    eb[k] = PermEntry{a->d_perm.p, a->nnodes, B->offs[k], d_b[k], B->d_b.p};
    ex[k] = PermEntry{a->d_perm.p, a->nnodes, B->offs[k], d_x[k], B->d_x.p};
    eo[k] = PermEntry{a->d_perm.p, a->nnodes, B->offs[k], B->d_x.p, d_x[k]};
    maxn = std::max(maxn, a->nnodes);
  }
  GF_CUDA(cudaMemcpyAsync(B->d_perm_b.p, eb.data(), sizeof(PermEntry) * B->np,
                          cudaMemcpyHostToDevice, st));
  GF_CUDA(cudaMemcpyAsync(B->d_perm_x.p, ex.data(), sizeof(PermEntry) * B->np,
                          cudaMemcpyHostToDevice, st));
  GF_CUDA(cudaMemcpyAsync(B->d_perm_out.p, eo.data(), sizeof(PermEntry) * B->np,
                          cudaMemcpyHostToDevice, st));
  const dim3 grid((unsigned)std::max(1, std::min(64, (6 * maxn + 255) / 256)), (unsigned)B->np);
  bpermute<<<grid, 256, 0, st>>>(B->d_perm_b.p, 0); ::gf::count_launch();
  bpermute<<<grid, 256, 0, st>>>(B->d_perm_x.p, 0); ::gf::count_launch();
  GF_CHECK_LAUNCH();
  std::vector<gf_solve_stats> S;
  gf_status s = batch_solve_space(B, o, S, st);
  bpermute<<<grid, 256, 0, st>>>(B->d_perm_out.p, 1); ::gf::count_launch();
  GF_CHECK_LAUNCH();
  // every sweep of the solve has run: read and clear the device status
  SweepCtl h;
  gf_status sc = read_ctl(B, st, &h);
  if (sc == GF_OK) sc = ctl_status(h);
  if (sc != GF_OK) {
    s = sc;
    for (auto& x : S) x.status = sc;
  }
  if (stats)
    for (int k = 0; k < B->np && k < (int)S.size(); k++) stats[k] = S[k];
  return s;
}

gf_status gf_gmres_solve(gf_assembler* a, gf_bsr* A, gf_precond* p, const double* d_b,
                         double* d_x, const gf_solve_opts* opts, gf_solve_stats* stats,
                         void* stream) {
  if (!a || !A || !p || !d_b || !d_x || A->a != a || p->a != a) return GF_INVALID_ARG;
  gf_status s = self_batch(p, A);
  if (s != GF_OK) return s;
  return gf_batch_solve(p->self, &d_b, &d_x, opts, stats, stream);
}

gf_status gf_direct_solve(gf_assembler* a, gf_bsr* A, const double* d_b, double* d_x,
                          gf_solve_stats* stats, void* stream) {
  if (!a || !A || !d_b || !d_x || A->a != a) return GF_INVALID_ARG;
  gf_precond* p = nullptr;
  gf_status s = gf_precond_create(a, GF_FILL_FULL, GF_PREC_FP64, &p);
  if (s != GF_OK) return s;
  s = gf_precond_factor(p, A, stream);
  gf_solve_stats st{};
  if (s == GF_OK) {
    // x = (LU)^{-1} b is the first step of right-preconditioned GMRES from
    // x = 0 with the complete factor; the further steps are FP64 iterative
    // refinement, run until the residual stops falling (at most 4 steps)
    const size_t n = (size_t)6 * a->nnodes;
    cudaError_t e = cudaMemsetAsync(d_x, 0, sizeof(double) * n, as_stream(stream));
    if (e != cudaSuccess) {
      set_last_error("gf_direct_solve", e);
      s = GF_CUDA_ERROR;
    } else {
      gf_solve_opts o;
      gf_solve_opts_default(&o);
      o.restart = 4;
      o.max_iters = 4;
      o.rtol = 1e-15;
      o.side = 1;
      s = gf_gmres_solve(a, A, p, d_b, d_x, &o, &st, stream);
      if (s == GF_NOT_CONVERGED) s = GF_OK;  // a direct solve has no tolerance to miss
      st.status = s;
    }
  }
  if (stats) *stats = st;
  gf_precond_destroy(p);
  return s;
}

gf_status gf_bsr_spmv(gf_bsr* m, double alpha, const double* d_x, double beta, double* d_y,
                      void* stream) {
  if (!m || !d_x || !d_y) return GF_INVALID_ARG;
  gf_assembler* a = m->a;
  cudaStream_t st = as_stream(stream);
  if (!m->desc.p) {
    ProbDev d{};
    d.n = a->nnodes;
    d.off = 0;
    d.rowp = a->d_rowp.p;
    d.cols = a->d_cols.p;
    d.A64 = m->vals.p;
    GF_CUDA(m->desc.upload(&d, 1));
    GF_CUDA(m->rowprob.alloc(a->nnodes));
    GF_CUDA(cudaMemset(m->rowprob.p, 0, sizeof(int32_t) * a->nnodes));
  }
  bspmv_kernel<double><<<(a->nnodes + 7) / 8, 256, 0, st>>>(a->nnodes, m->rowprob.p, m->desc.p,
                                                            nullptr, d_x, alpha, beta, d_y); ::gf::count_launch();
  GF_CHECK_LAUNCH();
  return GF_OK;
}

}  // extern "C"
