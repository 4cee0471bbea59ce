// Shell residual / Jacobian / energy assembly kernels and their C ABI.
//
// Reference: add_residual_gpu / add_jacobian_gpu (include/base/elem_group.cuh:17-211)
// launch one thread per (element, quadrature point[, Jacobian column]) and
// scatter with FP64 atomicAdd (include/linalg/vec.h:278-293,
// include/linalg/bsr_mat.h:229-276).
//
// Here a CTA of four warps owns a chunk of up to eight neighbouring elements:
//   * the chunk's coordinates and DOFs are gathered into shared memory; the
//     node normals, the frames of the four nodes and of the four quadrature
//     points are computed with one lane per (element, point);
//   * a warp tabulates its element's 24 columns (ElemData); lane (i, q) then
//     evaluates the strains of columns i, 8 + i, 16 + i at quadrature point q
//     and K_e = sum_q B_q^T D B_q is accumulated by FP64 tensor instructions
//     (mma.m8n8k4) whose contraction index is the quadrature point, one
//     strain component a step: the operands are the lane's own values, so no
//     strain matrix is ever stored. K_e is symmetric: six of nine 8x8 tiles,
//     the others are mirrored as they go to shared memory;
//   * the chunk's elements are summed block by block from shared memory, in
//     element order, and every block goes to global memory once per chunk;
//   * the scatter follows the coloured schedule built on the host: chunks of
//     one colour share no node and run concurrently, one launch per colour.
//     The launches overlap (programmatic dependent launch): a chunk computes
//     its K_e while the colour before still scatters, and waits only before
//     its own scatter. The first colour that touches a block stores, later
//     ones read-modify-write; there are no atomics and the result is bitwise
//     reproducible;
//   * with GF_ASSEMBLE_ATOMIC the colours are ignored: the outputs are zeroed
//     and one launch over all chunks adds with FP64 atomics (the reference's
//     scatter; sums in arrival order, so not bitwise reproducible);
//   * the residual and the energy need no strain columns: a warp takes a chunk,
//     lane (k, q) evaluates element k's strains at quadrature point q from the
//     displacements and applies the transposed maps;
//   * a batch of problems runs each colour of all its problems in one launch
//     (work items = (problem, chunk) per CTA), or all chunks of all problems
//     in one launch with atomics.
// Measured on B200 (one warp taking a chunk's elements one after another with
// stored strain matrices -> this): Jacobian and residual of a 10x10 plate
// 169 -> 25 us, of a 400x200 plate 738 -> 307 us; residual of a 300x300 plate
// 580 -> 95 us. The Jacobian is bound by instruction latency and shared-memory
// wavefronts (l1tex 62 %, FP64 pipe 20 %, 15 warps an SM), the residual by
// instruction latency (FP64 pipe 28 %).
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstring>

#include "gf_internal.h"

namespace gf {

static double ms_since(std::chrono::steady_clock::time_point t) {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t).count();
}

constexpr int kChunkSize = 8;     // elements per chunk
constexpr int kAsmThreads = 128;  // a warp takes every fourth element

struct ChunkSlot {
  ElemData e[kChunkSize];
  double U[kChunkSize][24];
  double Re[kChunkSize][24];
  double thick[kChunkSize];
  Material mat[kChunkSize];
  int4 brec[16 * kChunkSize];
};

// A block (or node) that a chunk contributes to: x = block (node), y = info,
// (z, w) = up to eight contributions, one byte each: element of the chunk
// * 16 + block 4a + b of the element (* 4 + node a). Info: Dirichlet rows and
// columns (6 bits each), diagonal block, first chunk to touch it, number of
// contributions.
enum { kRecColShift = 6, kRecDiag = 1 << 12, kRecFirst = 1 << 13, kRecCountShift = 16 };
constexpr int kRecMost = 8;  // contributions a record holds, a byte each
// an element has four different nodes, so it adds at most once to a block
static_assert(kChunkSize <= kRecMost, "a chunk's contributions to a block fit its record");

// Records of chunk blockIdx.x, in the order of their first contributions (recs
// null: their numbers only, blocks | nodes << 16 in count). A thread a
// contribution: 16 blocks an element, then 4 nodes. Built on the host (a hash
// table a chunk) the records were half of an assembler's setup: 400x200 plate
// 19 of 37 ms, now 1.7 of 24, most of it the upload of the elemIndMap; 10x10
// 0.06 -> 0.09 ms (two launches and a read-back).
__global__ void __launch_bounds__(16 * kChunkSize)
    chunk_records_kernel(const int32_t* __restrict__ chunk_start, const int32_t* __restrict__ order,
                         const int32_t* __restrict__ sconn, const int32_t* __restrict__ emap,
                         const uint32_t* __restrict__ first_touch,
                         const uint8_t* __restrict__ bcmask, const int32_t* __restrict__ ptr,
                         int32_t* __restrict__ count, int4* __restrict__ recs) {
  constexpr int T = 16 * kChunkSize;
  __shared__ int key[2][T];             // block or node of each contribution
  __shared__ unsigned char touch[2][T];  // first chunk to touch it
  __shared__ int warps[T / 32];
  const int li = blockIdx.x, t = threadIdx.x, lane = t & 31;
  const int s0 = chunk_start[li], cnt = chunk_start[li + 1] - s0;
  for (int z = 0; z < 2; z++) {  // blocks, nodes
    const int per = z ? 4 : 16, k = t / per, x = t % per;
    const bool on = k < cnt;
    const int e = on ? order[s0 + k] : 0;
    key[z][t] = !on ? -1 : z ? sconn[4 * (s0 + k) + x] : emap[16 * (size_t)e + x];
    touch[z][t] = on ? (first_touch[e] >> (16 * z + x)) & 1 : 0;
  }
  __syncthreads();
  for (int z = 0; z < 2; z++) {
    const int n = (z ? 4 : 16) * cnt, mine = key[z][t];
    bool first = t < n;
    for (int j = 0; j < t && j < n; j++) first = first && key[z][j] != mine;
    const unsigned vote = __ballot_sync(0xffffffffu, first);
    if (lane == 0) warps[t >> 5] = __popc(vote);
    __syncthreads();
    int at = __popc(vote & ((1u << lane) - 1u)), all = 0;
    for (int w = 0; w < T / 32; w++) {
      if (w < t >> 5) at += warps[w];
      all += warps[w];
    }
    __syncthreads();
    if (!recs) {
      if (t == 0) count[li] = z ? count[li] | all << 16 : all;
      continue;
    }
    if (!first) continue;
    const int a = z ? mine : sconn[4 * s0 + t / 4], b = z ? a : sconn[4 * (s0 + t / 16) + t % 4];
    int4 r = make_int4(mine, bcmask[a], 0, 0);
    if (!z) r.y |= bcmask[b] << kRecColShift | (a == b ? kRecDiag : 0);
    int m = 0;
    for (int j = t; j < n; j++) {
      if (key[z][j] != mine) continue;
      if (touch[z][j]) r.y |= kRecFirst;
      (m < 4 ? r.z : r.w) |= (int)((unsigned)j << (8 * (m & 3)));
      m++;
    }
    r.y |= m << kRecCountShift;
    recs[ptr[z * (gridDim.x + 1) + li] + at] = r;
  }
}

// The records of all chunks; the schedule's own arrays are on the device already.
static cudaError_t chunk_records(gf_assembler* a, const std::vector<uint8_t>& bcmask) {
  const Schedule& s = a->sched;
  const int nc = s.nchunks;
  // one table: elemIndMap, first touches, constrained DOFs, records per chunk
  const size_t ne = s.first_touch.size(), words = 17 * ne + (bcmask.size() + 3) / 4;
  DevBuf<int32_t> d_table;
  cudaError_t e = cudaSuccess;
  auto up = [&](cudaError_t x) {
    if (e == cudaSuccess) e = x;
  };
  auto launch = [&](const int32_t* ptr, int4* recs) {
    if (e != cudaSuccess) return;
    const int32_t* t = d_table.p;
    chunk_records_kernel<<<nc, 16 * kChunkSize>>>(
        a->d_chunk_start.p, a->d_sorder.p, a->d_sconn.p, t,
        reinterpret_cast<const uint32_t*>(t + 16 * ne),
        reinterpret_cast<const uint8_t*>(t + 17 * ne), ptr, d_table.p + words, recs);
    ::gf::count_launch();
    up(cudaGetLastError());
  };
  up(d_table.alloc(words + nc));
  auto put = [&](size_t at, const void* src, size_t bytes) {
    if (e == cudaSuccess) up(cudaMemcpy(d_table.p + at, src, bytes, cudaMemcpyHostToDevice));
  };
  put(0, a->emap.data(), sizeof(int32_t) * 16 * ne);
  put(16 * ne, s.first_touch.data(), sizeof(uint32_t) * ne);
  put(17 * ne, bcmask.data(), bcmask.size());
  launch(nullptr, nullptr);
  std::vector<int32_t> n(nc), ptr(2 * (size_t)(nc + 1), 0);
  if (e == cudaSuccess)
    up(cudaMemcpy(n.data(), d_table.p + words, sizeof(int32_t) * nc, cudaMemcpyDeviceToHost));
  for (int z = 0, at = 0; z < 2; z++)
    for (int li = 0; li <= nc; li++) {
      ptr[(size_t)z * (nc + 1) + li] = at;
      if (li < nc) at += z ? n[li] >> 16 : n[li] & 0xffff;
    }
  up(a->d_rptr.upload(ptr));
  up(a->d_recs.alloc(ptr.back()));
  launch(a->d_rptr.p, a->d_recs.p);
  if (e == cudaSuccess) up(cudaStreamSynchronize(nullptr));  // the table ends here
  return e;
}

struct AsmParams {
  const double* xpts;
  const double* vars;
  const int32_t* sconn;
  const double* sthick;
  const int32_t* smat;
  const Material* mats;
  const int32_t* chunk_start;
  const double* thick_nat;   // optional per-call thickness (natural element order)
  const int32_t* sorder;     // schedule position -> element
  const int4* brec;          // block records of all chunks, and where a chunk's begin
  const int32_t* bptr;
  const int4* nrec;          // node records
  const int32_t* nptr;
  double* values;
  double* res;
  double* energy_part;
  int chunk_base, chunk_end;
  int flags, pad;
};

enum { MODE_JAC = 0, MODE_RES = 1, MODE_ENERGY = 2 };

// c += A B over k = 4 (A row-major 8x4, B column-major 4x8, lane = 4 row + k
// and 4 column + k); exact FP64 multiply-adds
__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}
// upper 8x8 tiles of a 24x24 product, one strain component of all points
__device__ __forceinline__ void mma_step(double (&acc)[6][2], const double (&E)[3],
                                         const double (&S)[3]) {
  mma_f64(acc[0], E[0], S[0]);
  mma_f64(acc[1], E[0], S[1]);
  mma_f64(acc[2], E[0], S[2]);
  mma_f64(acc[3], E[1], S[1]);
  mma_f64(acc[4], E[1], S[2]);
  mma_f64(acc[5], E[2], S[2]);
}

// K_e of one element by one warp; d holds the element's tables on entry and
// K_e (rows of kKeStride doubles) on exit.
__device__ __forceinline__ void element_stiffness(ElemData& d, const Material& m, double t,
                                                  int lane) {
  const int i = lane >> 2, q = lane & 3;
  const Stiffness D = stiffness(m, t, d.scale[q]);
  double acc[6][2];
#pragma unroll
  for (int k = 0; k < 6; k++) acc[k][0] = acc[k][1] = 0.0;
  ColumnAt c[3];
#pragma unroll
  for (int k = 0; k < 3; k++) c[k] = column_at(d, 8 * k + i, q);
  // Smallest terms first, the membrane's last: fewer roundings at the size of
  // the sum.
  double E0[3], E1[3], E2[3], E[3], S[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    E0[k] = tying_row(d, q, 0, c[k].g);
    E1[k] = tying_row(d, q, 1, c[k].g);
    E2[k] = tying_row(d, q, 2, c[k].g);
  }
#pragma unroll
  for (int k = 0; k < 3; k++)
    E[k] = c[k].e3, S[k] = D.b0 * E0[k] + D.b1 * E1[k] + D.d0 * c[k].e3 + D.d1 * c[k].e4;
  mma_step(acc, E, S);
#pragma unroll
  for (int k = 0; k < 3; k++)
    E[k] = c[k].e4, S[k] = D.b1 * E0[k] + D.b0 * E1[k] + D.d1 * c[k].e3 + D.d0 * c[k].e4;
  mma_step(acc, E, S);
#pragma unroll
  for (int k = 0; k < 3; k++) E[k] = c[k].e5, S[k] = D.b5 * E2[k] + D.d5 * E[k];
  mma_step(acc, E, S);
#pragma unroll
  for (int z = 3; z < 5; z++) {
#pragma unroll
    for (int k = 0; k < 3; k++) E[k] = tying_row(d, q, z, c[k].g), S[k] = D.s * E[k];
    mma_step(acc, E, S);
  }
#pragma unroll
  for (int k = 0; k < 3; k++) E[k] = c[k].e8, S[k] = D.r * E[k];
  mma_step(acc, E, S);
#pragma unroll
  for (int k = 0; k < 3; k++) S[k] = D.a5 * E2[k] + D.b5 * c[k].e5;
  mma_step(acc, E2, S);
#pragma unroll
  for (int k = 0; k < 3; k++)
    S[k] = D.a0 * E0[k] + D.a1 * E1[k] + D.b0 * c[k].e3 + D.b1 * c[k].e4;
  mma_step(acc, E0, S);
#pragma unroll
  for (int k = 0; k < 3; k++)
    S[k] = D.a1 * E0[k] + D.a0 * E1[k] + D.b1 * c[k].e3 + D.b0 * c[k].e4;
  mma_step(acc, E1, S);
  __syncwarp();  // the tables have been read
  double* K = reinterpret_cast<double*>(&d);
  int tile = 0;
#pragma unroll
  for (int mi = 0; mi < 3; mi++)
#pragma unroll
    for (int ni = mi; ni < 3; ni++, tile++) {
      const int r = 8 * mi + i, col = 8 * ni + 2 * q;
      *reinterpret_cast<double2*>(&K[r * kKeStride + col]) = make_double2(acc[tile][0], acc[tile][1]);
      if (ni > mi) {
        K[col * kKeStride + r] = acc[tile][0];
        K[(col + 1) * kKeStride + r] = acc[tile][1];
      }
    }
}

// Node sums of a chunk: contributions in Re (24 per element), summed in
// element order.
__device__ __forceinline__ void scatter_residual(const AsmParams& P, int li, const double (*Re)[24],
                                                 int tid, int threads) {
  const bool fuse = (P.flags & GF_ASSEMBLE_FUSE_BCS) != 0;
  const bool add = (P.flags & GF_ASSEMBLE_ADD) != 0;
  const bool atomic = (P.flags & GF_ASSEMBLE_ATOMIC) != 0;
  const int n0 = P.nptr[li], nn = 6 * (P.nptr[li + 1] - n0);
  for (int t = tid; t < nn; t += threads) {
    const int4 rec = __ldg(P.nrec + n0 + t / 6);
    const int c = t % 6, n = rec.y >> kRecCountShift;
    double v = 0.0;
    for (int k = 0; k < n; k++) {
      const int code = ((k < 4 ? rec.z : rec.w) >> (8 * (k & 3))) & 255;
      v += Re[code >> 2][6 * (code & 3) + c];
    }
    if (fuse && ((rec.y >> c) & 1)) v = 0.0;
    double* dst = P.res + 6 * (size_t)rec.x + c;
    if (atomic)
      atomicAdd(dst, v);
    else
      *dst = (rec.y & kRecFirst) && !add ? v : *dst + v;
  }
}

// K (and R = K_e u_e) of chunk li (in schedule order) by one CTA.
__device__ __forceinline__ void jacobian_chunk(const AsmParams& P, int li, ChunkSlot& w) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int s0 = P.chunk_start[li], cnt = P.chunk_start[li + 1] - s0;
  const int b0 = P.bptr[li], nblk = P.bptr[li + 1] - b0;
  // everything the chunk reads, all loads in flight together
  if (tid < cnt) {
    w.thick[tid] = P.thick_nat ? P.thick_nat[P.sorder[s0 + tid]] : P.sthick[s0 + tid];
    w.mat[tid] = P.mats[P.smat[s0 + tid]];
  }
  if (tid < nblk) w.brec[tid] = __ldg(P.brec + b0 + tid);
  for (int t = tid; t < cnt * 12; t += kAsmThreads) {
    const int k = t / 12, x = t % 12;
    w.e[k].X[x] = P.xpts[3 * (size_t)P.sconn[4 * (s0 + k) + x / 3] + x % 3];
  }
  if (P.res)
    for (int t = tid; t < cnt * 24; t += kAsmThreads) {
      const int k = t / 24, x = t % 24;
      w.U[k][x] = P.vars[6 * (size_t)P.sconn[4 * (s0 + k) + x / 6] + x % 6];
    }
  __syncthreads();
  if (tid < 4 * cnt)
    elem_normal(w.e[tid >> 2].X, tid & 3, &w.e[tid >> 2].fn[3 * (tid & 3)]);
  __syncthreads();
  {
    // nodes on warp 0, quadrature points on warp 1
    const int k = lane >> 2;
    if (warp < 2 && k < cnt) elem_point(w.e[k], w.mat[k], 4 * warp + (lane & 3));
  }
  __syncthreads();
  // tables: 96 translation columns, then 96 rotation columns, then bending
  for (int t = tid; t < 96; t += kAsmThreads)
    if (t / 12 < cnt) elem_column(w.e[t / 12], 6 * (t % 12 / 3) + t % 3);
  for (int t = kAsmThreads - 1 - tid; t < 96; t += kAsmThreads)
    if (t / 12 < cnt) elem_column(w.e[t / 12], 6 * (t % 12 / 3) + t % 3 + 3);
  for (int k = warp; k < cnt; k += kAsmThreads / 32)
    elem_bending(w.e[k], lane >> 3, (lane >> 2) & 1, lane & 3);
  __syncthreads();
  for (int k = warp; k < cnt; k += kAsmThreads / 32)
    element_stiffness(w.e[k], w.mat[k], w.thick[k], lane);
  __syncthreads();
  const bool fuse = (P.flags & GF_ASSEMBLE_FUSE_BCS) != 0;
  const bool add = (P.flags & GF_ASSEMBLE_ADD) != 0;
  const bool atomic = (P.flags & GF_ASSEMBLE_ATOMIC) != 0;
  // the colours before have scattered
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // one row (of six) of a block a thread
  for (int t = tid; t < 6 * nblk; t += kAsmThreads) {
    const int4 rec = w.brec[t / 6];
    const int r = t % 6, info = rec.y, n = info >> kRecCountShift;
    double2* dst = reinterpret_cast<double2*>(P.values + 36 * (size_t)rec.x + 6 * r);
    const bool first = info & kRecFirst;
    double2 o[3];
    if (!atomic && (!first || add))
#pragma unroll
      for (int c = 0; c < 3; c++) o[c] = dst[c];
    else
#pragma unroll
      for (int c = 0; c < 3; c++) o[c] = make_double2(0.0, 0.0);
    double2 v[3] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
    for (int k = 0; k < n; k++) {
      const int code = ((k < 4 ? rec.z : rec.w) >> (8 * (k & 3))) & 255;
      const double2* K = reinterpret_cast<const double2*>(
          reinterpret_cast<const double*>(&w.e[code >> 4]) +
          (6 * ((code >> 2) & 3) + r) * kKeStride + 6 * (code & 3));
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double2 x = K[c];
        v[c].x += x.x;
        v[c].y += x.y;
      }
    }
    if (fuse && (info & (kRecDiag - 1))) {
      const double one = (info & kRecDiag) && first ? 1.0 : 0.0;
      const int masked = ((info >> r) & 1) ? 63 : info >> kRecColShift;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        if ((masked >> (2 * c)) & 1) v[c].x = r == 2 * c ? one : 0.0;
        if ((masked >> (2 * c + 1)) & 1) v[c].y = r == 2 * c + 1 ? one : 0.0;
      }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      if (atomic) {
        atomicAdd(reinterpret_cast<double*>(dst + c), v[c].x);
        atomicAdd(reinterpret_cast<double*>(dst + c) + 1, v[c].y);
      } else {
        dst[c] = make_double2(o[c].x + v[c].x, o[c].y + v[c].y);
      }
    }
  }
  if (!P.res) return;
  for (int t = tid; t < 24 * cnt; t += kAsmThreads) {
    const int k = t / 24, r = t % 24;
    const double* K = reinterpret_cast<const double*>(&w.e[k]) + r * kKeStride;
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < 24; c += 2) {
      const double2 x = *reinterpret_cast<const double2*>(K + c);
      s = fma(x.x, w.U[k][c], s);
      s = fma(x.y, w.U[k][c + 1], s);
    }
    w.Re[k][r] = s;
  }
  __syncthreads();
  scatter_residual(P, li, w.Re, tid, kAsmThreads);
}

__global__ void __launch_bounds__(kAsmThreads, 4) jacobian_kernel(const AsmParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  asm volatile("griddepcontrol.launch_dependents;");
  jacobian_chunk(P, P.chunk_base + blockIdx.x, *reinterpret_cast<ChunkSlot*>(smem_raw));
}

// Batched form: CTA w of the launch works on chunk work[w].y of problem
// work[w].x, whose parameters are copied to shared memory first.
__global__ void __launch_bounds__(kAsmThreads, 4)
    jacobian_batch_kernel(const AsmParams* __restrict__ PP, const int2* __restrict__ work) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ AsmParams sp;
  asm volatile("griddepcontrol.launch_dependents;");
  const int2 it = work[blockIdx.x];
  static_assert(sizeof(AsmParams) % 8 == 0, "copied in 8-byte words");
  if (threadIdx.x < sizeof(AsmParams) / 8)
    reinterpret_cast<unsigned long long*>(&sp)[threadIdx.x] =
        reinterpret_cast<const unsigned long long*>(PP + it.x)[threadIdx.x];
  __syncthreads();
  jacobian_chunk(sp, it.y, *reinterpret_cast<ChunkSlot*>(smem_raw));
}

// Residual (or energy) of a chunk by one warp, without strain columns: lane
// (k, q) evaluates the strains of element k at quadrature point q from the
// displacements themselves and applies the transposed maps; as node n = q of
// the element it does the nodal work. What the four points and nodes of an
// element exchange goes through the element's slot.
struct ResSlot {
  double X[12], U[24], fn[12];
  double d[4][3];       // director displacements theta x fn of the nodes
  double drill[4];      // nodal drill strains
  double V[4][15];      // per point: adjoints of u_xi, u_eta, d_xi, d_eta, d
  double G[4][5];       // ... of the tying strains g11 g22 g12 g23 g13
  double S8[4];         // ... of the drill strain
  double pad;           // slots in different banks
};
constexpr int kResWarps = 4;  // warps (chunks) per CTA

template <int MODE>
__device__ __forceinline__ void residual_chunk(const AsmParams& P, int li, ResSlot* w,
                                               double (*Re)[24], int lane) {
  const int s0 = P.chunk_start[li], cnt = P.chunk_start[li + 1] - s0;
  for (int t = lane; t < cnt * 12; t += 32) {
    const int k = t / 12, x = t % 12;
    w[k].X[x] = P.xpts[3 * (size_t)P.sconn[4 * (s0 + k) + x / 3] + x % 3];
  }
  for (int t = lane; t < cnt * 24; t += 32) {
    const int k = t / 24, x = t % 24;
    w[k].U[x] = P.vars[6 * (size_t)P.sconn[4 * (s0 + k) + x / 6] + x % 6];
  }
  __syncwarp();
  const int k = lane >> 2, q = lane & 3, ia = q & 1, ja = q >> 1;
  const bool on = k < cnt;
  ResSlot& e = w[on ? k : 0];
  if (on) {
    double fn[3];
    elem_normal(e.X, q, fn);
    for (int c = 0; c < 3; c++) e.fn[3 * q + c] = fn[c];
    cross3(&e.U[6 * q + 3], fn, e.d[q]);
  }
  __syncwarp();
  PointFrame f;
  double tc[3], sx[3], sy[3];  // this node's drill strain is sx.u_xi + sy.u_eta - tc.theta
  Material m;
  if (on) {
    m = P.mats[P.smat[s0 + k]];
    point_frame(e.X, e.fn, m, node_xi(q), node_eta(q), f);
    const double t0[3] = {f.T[0], f.T[3], f.T[6]}, t1[3] = {f.T[1], f.T[4], f.T[7]};
    cross3(t0, t1, tc);
    double s = 0.0;
    for (int c = 0; c < 3; c++) {
      sx[c] = 0.5 * (t1[c] * f.A[0] - t0[c] * f.A[1]);
      sy[c] = 0.5 * (t1[c] * f.A[3] - t0[c] * f.A[4]);
      // derivatives at the node: differences along its two edges
      const double ux = 0.5 * (e.U[12 * ja + 6 + c] - e.U[12 * ja + c]);
      const double uy = 0.5 * (e.U[6 * ia + 12 + c] - e.U[6 * ia + c]);
      s += sx[c] * ux + sy[c] * uy - tc[c] * e.U[6 * q + 3 + c];
    }
    e.drill[q] = s;
  }
  __syncwarp();
  double energy = 0.0;
  if (on) {
    double xi, eta;
    quad_point(q, xi, eta);
    point_frame(e.X, e.fn, m, xi, eta, f);
    const double t = P.thick_nat ? P.thick_nat[P.sorder[s0 + k]] : P.sthick[s0 + k];
    const Stiffness D = stiffness(m, t, f.det);
    double M[5][5];
    tying_rows(f.A, M);
    double Az[3][2];
    point_bending(f, Az);
    // tying strains, interpolated to the point (basis.h:314-368)
    const double x[2] = {0.5 * (1.0 - xi), 0.5 * (1.0 + xi)};
    const double y[2] = {0.5 * (1.0 - eta), 0.5 * (1.0 + eta)};
    double g[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    double Xc[3], Yc[3], uc[3], vc[3];
    for (int c = 0; c < 3; c++) {
      uc[c] = vc[c] = 0.0;
      Xc[c] = 0.25 * (((e.X[3 + c] - e.X[c]) - e.X[6 + c]) + e.X[9 + c]);
      Yc[c] = 0.25 * (((-e.X[c] - e.X[3 + c]) + e.X[6 + c]) + e.X[9 + c]);
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {  // edges along xi (eta = -1, 1) and along eta
      double e11 = 0.0, e13 = 0.0, e22 = 0.0, e23 = 0.0;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double X = 0.5 * (e.X[6 * j + 3 + c] - e.X[6 * j + c]);
        const double u = 0.5 * (e.U[12 * j + 6 + c] - e.U[12 * j + c]);
        const double n = 0.5 * (e.fn[6 * j + c] + e.fn[6 * j + 3 + c]);
        const double d = 0.5 * (e.d[2 * j][c] + e.d[2 * j + 1][c]);
        e11 = fma(X, u, e11);
        e13 += n * u + X * d;
        uc[c] += 0.5 * u;
        const double Y = 0.5 * (e.X[3 * j + 6 + c] - e.X[3 * j + c]);
        const double v = 0.5 * (e.U[6 * j + 12 + c] - e.U[6 * j + c]);
        const double n2 = 0.5 * (e.fn[3 * j + c] + e.fn[3 * j + 6 + c]);
        const double d2 = 0.5 * (e.d[j][c] + e.d[j + 2][c]);
        e22 = fma(Y, v, e22);
        e23 += n2 * v + Y * d2;
        vc[c] += 0.5 * v;
      }
      g[0] = fma(y[j], e11, g[0]);
      g[1] = fma(x[j], e22, g[1]);
      g[3] = fma(x[j], 0.5 * e23, g[3]);
      g[4] = fma(y[j], 0.5 * e13, g[4]);
    }
    g[2] = 0.5 * (dot3(Xc, vc) + dot3(Yc, uc));
    double E[9], S[9];
    const int row[5] = {0, 1, 2, 6, 7};
#pragma unroll
    for (int r = 0; r < 5; r++)
      E[row[r]] = M[r][0] * g[0] + M[r][1] * g[1] + M[r][2] * g[2] + M[r][3] * g[3] + M[r][4] * g[4];
    // bending: p_j = u_xi Az_0j + u_eta Az_1j + d_xi A_0j + d_eta A_1j + d Az_2j
    double p[2][3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double u0 = e.U[c], u1 = e.U[6 + c], u2 = e.U[12 + c], u3 = e.U[18 + c];
      const double d0 = e.d[0][c], d1 = e.d[1][c], d2 = e.d[2][c], d3 = e.d[3][c];
      const double ux = 0.5 * (y[0] * (u1 - u0) + y[1] * (u3 - u2));
      const double uy = 0.5 * (x[0] * (u2 - u0) + x[1] * (u3 - u1));
      const double dx = 0.5 * (y[0] * (d1 - d0) + y[1] * (d3 - d2));
      const double dy = 0.5 * (x[0] * (d2 - d0) + x[1] * (d3 - d1));
      const double d = y[0] * (x[0] * d0 + x[1] * d1) + y[1] * (x[0] * d2 + x[1] * d3);
#pragma unroll
      for (int j = 0; j < 2; j++)
        p[j][c] = ux * Az[0][j] + uy * Az[1][j] + dx * f.A[j] + dy * f.A[3 + j] + d * Az[2][j];
    }
    const double* T = f.T;
    E[3] = T[0] * p[0][0] + T[3] * p[0][1] + T[6] * p[0][2];
    E[4] = T[1] * p[1][0] + T[4] * p[1][1] + T[7] * p[1][2];
    E[5] = T[0] * p[1][0] + T[3] * p[1][1] + T[6] * p[1][2] + T[1] * p[0][0] + T[4] * p[0][1] +
           T[7] * p[0][2];
    E[8] = y[0] * (x[0] * e.drill[0] + x[1] * e.drill[1]) +
           y[1] * (x[0] * e.drill[2] + x[1] * e.drill[3]);
    S[0] = D.a0 * E[0] + D.a1 * E[1] + D.b0 * E[3] + D.b1 * E[4];
    S[1] = D.a1 * E[0] + D.a0 * E[1] + D.b1 * E[3] + D.b0 * E[4];
    S[2] = D.a5 * E[2] + D.b5 * E[5];
    S[3] = D.b0 * E[0] + D.b1 * E[1] + D.d0 * E[3] + D.d1 * E[4];
    S[4] = D.b1 * E[0] + D.b0 * E[1] + D.d1 * E[3] + D.d0 * E[4];
    S[5] = D.b5 * E[2] + D.d5 * E[5];
    S[6] = D.s * E[6];
    S[7] = D.s * E[7];
    S[8] = D.r * E[8];
    if (MODE == MODE_ENERGY) {
#pragma unroll
      for (int r = 0; r < 9; r++) energy = fma(0.5 * E[r], S[r], energy);
    } else {
#pragma unroll
      for (int z = 0; z < 5; z++)
        e.G[q][z] = M[0][z] * S[0] + M[1][z] * S[1] + M[2][z] * S[2] + M[3][z] * S[6] + M[4][z] * S[7];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double p0 = T[3 * c] * S[3] + T[3 * c + 1] * S[5];
        const double p1 = T[3 * c + 1] * S[4] + T[3 * c] * S[5];
        e.V[q][c] = Az[0][0] * p0 + Az[0][1] * p1;
        e.V[q][3 + c] = Az[1][0] * p0 + Az[1][1] * p1;
        e.V[q][6 + c] = f.A[0] * p0 + f.A[1] * p1;
        e.V[q][9 + c] = f.A[3] * p0 + f.A[4] * p1;
        e.V[q][12 + c] = Az[2][0] * p0 + Az[2][1] * p1;
      }
      e.S8[q] = S[8];
    }
  }
  if (MODE == MODE_ENERGY) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) energy += __shfl_xor_sync(0xffffffffu, energy, o);
    if (lane == 0) P.energy_part[li] = energy;
    // this launch ends after the colours before it
    asm volatile("griddepcontrol.wait;" ::: "memory");
    return;
  }
  __syncwarp();
  // node q of element k
  double ru[3], rd[3], dn = 0.0;
  if (on) {
    const double sa = node_xi(q), ta = node_eta(q);
    double G[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // adjoints of the node's own tying points
    for (int c = 0; c < 3; c++) ru[c] = rd[c] = 0.0;
#pragma unroll
    for (int z = 0; z < 4; z++) {
      double xi, eta, N, Nx, Ne;
      quad_point(z, xi, eta);
      shape(q, xi, eta, N, Nx, Ne);
      const double wx = 0.5 * (1.0 + sa * xi), wy = 0.5 * (1.0 + ta * eta);
      G[0] = fma(wy, e.G[z][0], G[0]);
      G[1] = fma(wx, e.G[z][1], G[1]);
      G[2] += e.G[z][2];
      G[3] = fma(wx, e.G[z][3], G[3]);
      G[4] = fma(wy, e.G[z][4], G[4]);
      dn = fma(N, e.S8[z], dn);
      const double* V = e.V[z];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        ru[c] += Nx * V[c] + Ne * V[3 + c];
        rd[c] += Nx * V[6 + c] + Ne * V[9 + c] + N * V[12 + c];
      }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double X = 0.5 * (e.X[6 * ja + 3 + c] - e.X[6 * ja + c]);
      const double Y = 0.5 * (e.X[3 * ia + 6 + c] - e.X[3 * ia + c]);
      const double Xc = 0.25 * (((e.X[3 + c] - e.X[c]) - e.X[6 + c]) + e.X[9 + c]);
      const double Yc = 0.25 * (((-e.X[c] - e.X[3 + c]) + e.X[6 + c]) + e.X[9 + c]);
      const double n1 = 0.5 * (e.fn[6 * ja + c] + e.fn[6 * ja + 3 + c]);
      const double n2 = 0.5 * (e.fn[3 * ia + c] + e.fn[3 * ia + 6 + c]);
      ru[c] += 0.5 * sa * (X * G[0] + 0.5 * n1 * G[4]) + 0.5 * ta * (Y * G[1] + 0.5 * n2 * G[3]) +
               0.125 * (sa * Yc + ta * Xc) * G[2];
      rd[c] += 0.25 * (X * G[4] + Y * G[3]);
    }
  }
  // drill adjoints of the three nodes whose strains this node's displacement
  // enters: its own (both edges) and its neighbours along xi and eta
  const int nx = lane ^ 1, ny = lane ^ 2;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const double ax = dn * sx[c], ay = dn * sy[c];
    const double bx = __shfl_sync(0xffffffffu, ax, nx), by = __shfl_sync(0xffffffffu, ay, ny);
    if (on) ru[c] += 0.5 * node_xi(q) * (ax + bx) + 0.5 * node_eta(q) * (ay + by);
  }
  if (on) {
    double th[3];
    cross3(&e.fn[3 * q], rd, th);
    for (int c = 0; c < 3; c++) {
      Re[k][6 * q + c] = ru[c];
      Re[k][6 * q + 3 + c] = th[c] - tc[c] * dn;
    }
  }
  __syncwarp();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  scatter_residual(P, li, Re, lane, 32);
}

template <int MODE>
__global__ void __launch_bounds__(32 * kResWarps, 3) residual_kernel(const AsmParams P) {
  __shared__ ResSlot slots[kResWarps][kChunkSize];
  __shared__ double Re[kResWarps][kChunkSize][24];
  asm volatile("griddepcontrol.launch_dependents;");
  const int warp = threadIdx.x >> 5, li = P.chunk_base + blockIdx.x * kResWarps + warp;
  if (li < P.chunk_end) residual_chunk<MODE>(P, li, slots[warp], Re[warp], threadIdx.x & 31);
}

// One launch of an assembly; `after` lets it start while the launch before it
// (the colour before) still runs.
template <class... Args>
static cudaError_t launch_chunks(void (*kernel)(Args...), int grid, int threads, size_t smem,
                                 bool after, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = after ? 1 : 0;
  ::gf::count_launch();
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

__global__ void sum_kernel(const double* part, int n, double* out) {
  // deterministic single-thread-per-lane tree over a fixed partition
  __shared__ double s[256];
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) acc += part[i];
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = s[0];
}

// Dirichlet rows and columns (apply_mat_bcs_rows_kernel /
// apply_mat_bcs_cols_kernel, include/linalg/bsr_mat.cuh:1-104) in one pass
// over a precomputed entry list: (block, block row, is_column, inner index).
__global__ void bc_mat_kernel(const int32_t* entries, int n, const int32_t* cols,
                              double* values) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int4 e = reinterpret_cast<const int4*>(entries)[t];
  const int blk = e.x, brow = e.y, is_col = e.z, inner = e.w;
  const int bcol = cols[blk];
  double* v = values + 36 * (size_t)blk;
  for (int k = 0; k < 6; k++) {
    const int r = is_col ? k : inner, c = is_col ? inner : k;
    v[6 * r + c] = (6 * brow + r == 6 * bcol + c) ? 1.0 : 0.0;
  }
}

__global__ void gather_thickness(const int32_t* order, int n, const double* in, double* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) out[t] = in[order[t]];
}

__global__ void bc_vec_kernel(const int32_t* bcs, int n, double* vec) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) vec[bcs[t]] = 0.0;
}

__global__ void permute_kernel(const int32_t* perm, int nnodes, const double* in, double* out,
                               int dir) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 6 * nnodes) return;
  const int i = t / 6, k = t % 6;
  if (dir == 0)
    out[6 * (size_t)perm[i] + k] = in[t];
  else
    out[t] = in[6 * (size_t)perm[i] + k];
}

static AsmParams asm_params(gf_assembler* a, double* values, double* res, int flags,
                            const double* thick_nat) {
  AsmParams P;
  std::memset(&P, 0, sizeof(P));
  P.xpts = a->d_xpts.p;
  P.vars = a->d_vars.p;
  P.sconn = a->d_sconn.p;
  P.sthick = a->d_sthick.p;
  P.smat = a->d_smat.p;
  P.mats = a->d_mats.p;
  P.chunk_start = a->d_chunk_start.p;
  P.thick_nat = thick_nat;
  P.sorder = a->d_sorder.p;
  P.brec = P.nrec = a->d_recs.p;
  P.bptr = a->d_rptr.p;
  P.nptr = a->d_rptr.p + a->sched.nchunks + 1;
  P.values = values;
  P.res = res;
  P.energy_part = a->d_energy_part.p;
  P.flags = flags;
  return P;
}

template <int MODE>
static gf_status launch_assembly(gf_assembler* a, double* values, double* res, int flags,
                                 cudaStream_t st, const double* thick_nat = nullptr) {
  AsmParams P = asm_params(a, values, res, flags, thick_nat);
  // per device and constant, so setting it on every call is race-free
  if (MODE == MODE_JAC)
    GF_CUDA(cudaFuncSetAttribute(jacobian_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(ChunkSlot)));
  const Schedule& s = a->sched;
  const bool atomic = (flags & GF_ASSEMBLE_ATOMIC) != 0;
  if (atomic && !(flags & GF_ASSEMBLE_ADD)) {
    if (values) GF_CUDA(cudaMemsetAsync(values, 0, sizeof(double) * 36 * (size_t)a->pat.nnz(), st));
    if (res) GF_CUDA(cudaMemsetAsync(res, 0, sizeof(double) * 6 * (size_t)a->nnodes, st));
  }
  bool after = false;
  for (int cc = 0; cc < (atomic ? 1 : s.ncc); cc++) {
    const int lo = atomic ? 0 : s.cc_start[cc], hi = atomic ? s.nchunks : s.cc_start[cc + 1];
    if (hi == lo) continue;
    P.chunk_base = lo;
    P.chunk_end = hi;
    if (MODE == MODE_JAC)
      GF_CUDA(launch_chunks(jacobian_kernel, hi - lo, kAsmThreads, sizeof(ChunkSlot), after, st,
                            (const AsmParams)P));
    else
      GF_CUDA(launch_chunks(residual_kernel<MODE == MODE_JAC ? MODE_RES : MODE>,
                            (hi - lo + kResWarps - 1) / kResWarps, 32 * kResWarps, 0, after, st,
                            (const AsmParams)P));
    after = true;
  }
  return GF_OK;
}

// Cached launch data of a batch's assembly: per-problem parameters (rebuilt
// when a problem's thickness pointer or the flags change) and the work lists.
struct BatchAsm {
  std::vector<AsmParams> host;
  DevBuf<AsmParams> d_params;
  DevBuf<int2> d_work;
  std::vector<int> off;  // work ranges: per colour (coloured) or one (atomic)
  int flags = -1;
};

void batch_asm_free(BatchAsm* b) { delete b; }

gf_status batch_assemble(BatchAsm*& cache, const std::vector<gf_assembler*>& asms,
                         const std::vector<double*>& values, const double* const* thick,
                         int flags, cudaStream_t st) {
  const int np = (int)asms.size();
  if (!cache) cache = new BatchAsm();
  BatchAsm& B = *cache;
  std::vector<AsmParams> h(np);
  for (int k = 0; k < np; k++) {
    h[k] = asm_params(asms[k], values[k], nullptr, flags, thick ? thick[k] : nullptr);
  }
  const bool atomic = (flags & GF_ASSEMBLE_ATOMIC) != 0;
  if (B.flags != flags || B.host.size() != h.size() ||
      std::memcmp(B.host.data(), h.data(), sizeof(AsmParams) * h.size()) != 0) {
    // work items: (problem, chunk), colour by colour, or all chunks at once
    std::vector<int2> work;
    B.off.assign(1, 0);
    if (atomic) {
      for (int k = 0; k < np; k++)
        for (int c = 0; c < asms[k]->sched.nchunks; c++) work.push_back(make_int2(k, c));
      B.off.push_back((int)work.size());
    } else {
      int ncc = 0;
      for (auto* a : asms) ncc = std::max(ncc, a->sched.ncc);
      for (int cc = 0; cc < ncc; cc++) {
        for (int k = 0; k < np; k++) {
          const Schedule& s = asms[k]->sched;
          if (cc >= s.ncc) continue;
          for (int c = s.cc_start[cc]; c < s.cc_start[cc + 1]; c++) work.push_back(make_int2(k, c));
        }
        B.off.push_back((int)work.size());
      }
    }
    GF_CUDA(B.d_work.alloc(work.size()));
    GF_CUDA(B.d_params.alloc(h.size()));
    GF_CUDA(cudaMemcpyAsync(B.d_work.p, work.data(), sizeof(int2) * work.size(),
                            cudaMemcpyHostToDevice, st));
    GF_CUDA(cudaMemcpyAsync(B.d_params.p, h.data(), sizeof(AsmParams) * h.size(),
                            cudaMemcpyHostToDevice, st));
    GF_CUDA(cudaStreamSynchronize(st));  // the host copies are reused
    B.host = h;
    B.flags = flags;
  }
  if (atomic && !(flags & GF_ASSEMBLE_ADD))
    for (int k = 0; k < np; k++)
      GF_CUDA(cudaMemsetAsync(values[k], 0, sizeof(double) * 36 * (size_t)asms[k]->pat.nnz(), st));
  GF_CUDA(cudaFuncSetAttribute(jacobian_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sizeof(ChunkSlot)));
  bool after = false;
  for (size_t r = 0; r + 1 < B.off.size(); r++) {
    const int nwork = B.off[r + 1] - B.off[r];
    if (nwork == 0) continue;
    GF_CUDA(launch_chunks(jacobian_batch_kernel, nwork, kAsmThreads, sizeof(ChunkSlot), after, st,
                          (const AsmParams*)B.d_params.p, (const int2*)(B.d_work.p + B.off[r])));
    after = true;
  }
  return GF_OK;
}

}  // namespace gf

using namespace gf;

// ------------------------------------------------------------------ C ABI
extern "C" {

gf_status gf_assembler_create(const gf_mesh_desc* d, gf_assembler** out) {
  if (!d || !out || d->num_nodes <= 0 || d->num_elements <= 0 || !d->conn || !d->xpts ||
      !d->data || (d->num_bcs > 0 && !d->bcs))
    return GF_INVALID_ARG;
  *out = nullptr;
  const int nn = d->num_nodes, ne = d->num_elements;
  for (size_t i = 0; i < (size_t)4 * ne; i++)
    if (d->conn[i] < 0 || d->conn[i] >= nn) return GF_INVALID_ARG;
  for (int e = 0; e < ne; e++)
    for (int x = 0; x < 4; x++)
      for (int y = x + 1; y < 4; y++)
        if (d->conn[4 * e + x] == d->conn[4 * e + y]) return GF_INVALID_ARG;
  for (int i = 0; i < d->num_bcs; i++)
    if (d->bcs[i] < 0 || d->bcs[i] >= 6 * nn) return GF_INVALID_ARG;
  int dev_count = 0;
  if (cudaGetDeviceCount(&dev_count) != cudaSuccess || dev_count == 0) return GF_NO_DEVICE;

  const auto t_setup = std::chrono::steady_clock::now();
  gf_assembler* a = new gf_assembler();
  a->nnodes = nn;
  a->nelem = ne;
  a->nbcs = d->num_bcs;
  a->conn.assign(d->conn, d->conn + 4 * (size_t)ne);
  a->bcs.assign(d->bcs, d->bcs + d->num_bcs);
  if (pattern_from_conn_gpu(ne, nn, d->conn, a->pat0))
    a->sym_flags |= 1;
  else
    a->pat0 = pattern_from_conn(ne, nn, d->conn);
  order_nodes(a->pat0, d, a->perm);
  a->iperm.resize(nn);
  for (int i = 0; i < nn; i++) a->iperm[a->perm[i]] = i;
  a->pat = permute_pattern(a->pat0, a->perm);
  if (elem_ind_map_gpu(ne, d->conn, a->pat, a->perm, a->emap))
    a->sym_flags |= 2;
  else
    elem_ind_map(ne, d->conn, a->pat, a->perm, a->emap);
  if (build_schedule(ne, nn, d->conn, a->emap, a->pat.nnz(), kChunkSize, a->sched) != 0) {
    delete a;
    return GF_INVALID_ARG;
  }
  // materials: dedupe (E, nu, tOffset, refAxis) per element; thickness per element
  std::vector<int32_t> emat(ne);
  std::vector<double> thick(ne);
  for (int e = 0; e < ne; e++) {
    const gf_shell_data& sd = d->data[e];
    thick[e] = sd.thick;
    Material m{sd.E, sd.nu, sd.tOffset, {sd.refAxis[0], sd.refAxis[1], sd.refAxis[2]},
               sd.has_ref_axis ? 1 : 0, 0, 0.0, 0.0, 0.0};
    material_constants(m);
    int found = -1;
    for (size_t k = 0; k < a->mats.size(); k++) {
      const Material& o = a->mats[k];
      if (o.E == m.E && o.nu == m.nu && o.tOffset == m.tOffset &&
          o.has_ref_axis == m.has_ref_axis && o.refAxis[0] == m.refAxis[0] &&
          o.refAxis[1] == m.refAxis[1] && o.refAxis[2] == m.refAxis[2]) {
        found = (int)k;
        break;
      }
    }
    if (found < 0) {
      found = (int)a->mats.size();
      a->mats.push_back(m);
    }
    emat[e] = found;
  }
  const Schedule& s = a->sched;
  std::vector<int32_t> sconn((size_t)4 * ne), smat(ne);
  std::vector<double> sthick(ne);
  for (int k = 0; k < ne; k++) {
    const int e = s.order[k];
    for (int x = 0; x < 4; x++) sconn[4 * k + x] = d->conn[4 * e + x];
    sthick[k] = thick[e];
    smat[k] = emat[e];
  }
  std::vector<uint8_t> bcmask(nn, 0);
  for (int i = 0; i < d->num_bcs; i++) bcmask[d->bcs[i] / 6] |= (uint8_t)(1u << (d->bcs[i] % 6));
  // BC entry list (solver order): rows of constrained DOFs and the matching columns
  std::vector<int32_t> ent;
  const Pattern& P = a->pat;
  for (int i = 0; i < d->num_bcs; i++) {
    const int node = a->perm[d->bcs[i] / 6], inner = d->bcs[i] % 6;
    for (int jp = P.rowp[node]; jp < P.rowp[node + 1]; jp++) {
      ent.insert(ent.end(), {jp, node, 0, inner});
      const int j = P.cols[jp];  // symmetric pattern: block (j, node) exists
      const int32_t* b0 = P.cols.data() + P.rowp[j];
      const int32_t* b1 = P.cols.data() + P.rowp[j + 1];
      const int32_t* f = std::lower_bound(b0, b1, node);
      ent.insert(ent.end(), {(int32_t)(f - P.cols.data()), j, 1, inner});
    }
  }
  a->nbc_entries = (int)(ent.size() / 4);
  std::vector<int32_t> diag(nn);
  for (int i = 0; i < nn; i++) {
    const int32_t* b0 = P.cols.data() + P.rowp[i];
    const int32_t* b1 = P.cols.data() + P.rowp[i + 1];
    diag[i] = (int32_t)(std::lower_bound(b0, b1, i) - P.cols.data());
  }
  gf_status st = GF_OK;
  auto up = [&](cudaError_t e) {
    if (e != cudaSuccess && st == GF_OK) {
      set_last_error("gf_assembler_create upload", e);
      st = (e == cudaErrorMemoryAllocation) ? GF_OOM : GF_CUDA_ERROR;
    }
  };
  up(a->d_xpts.upload(d->xpts, (size_t)3 * nn));
  up(a->d_vars.alloc((size_t)6 * nn));
  if (st == GF_OK) up(cudaMemset(a->d_vars.p, 0, sizeof(double) * 6 * nn));
  up(a->d_perm.upload(a->perm));
  up(a->d_bcs.upload(a->bcs));
  up(a->d_sconn.upload(sconn));
  up(a->d_smat.upload(smat));
  up(a->d_sthick.upload(sthick));
  up(a->d_sorder.upload(s.order));
  up(a->d_chunk_start.upload(s.chunk_start));
  up(a->d_mats.upload(a->mats));
  up(a->d_rowp.upload(P.rowp));
  up(a->d_cols.upload(P.cols));
  up(a->d_bc_entries.upload(ent));
  up(a->d_energy_part.alloc(s.nchunks + 1));
  up(a->d_diag.upload(diag));
  if (st == GF_OK) {
    const auto t_rec = std::chrono::steady_clock::now();
    up(chunk_records(a, bcmask));
    a->records_ms = ms_since(t_rec);
  }
  if (st != GF_OK) {
    delete a;
    return st;
  }
  a->setup_ms = ms_since(t_setup);
  count_assemblers(1);
  *out = a;
  return GF_OK;
}

gf_status gf_assembler_destroy(gf_assembler* a) {
  if (a) count_assemblers(-1);
  delete a;
  return GF_OK;
}

int32_t gf_assembler_num_nodes(const gf_assembler* a) { return a ? a->nnodes : 0; }
int32_t gf_assembler_num_elements(const gf_assembler* a) { return a ? a->nelem : 0; }
int32_t gf_assembler_num_vars(const gf_assembler* a) { return a ? 6 * a->nnodes : 0; }
int32_t gf_assembler_nnzb(const gf_assembler* a) { return a ? a->pat.nnz() : 0; }

gf_status gf_assembler_get_pattern(const gf_assembler* a, int32_t* rowPtr, int32_t* colPtr,
                                   int32_t* perm, int32_t* elemIndMap) {
  if (!a) return GF_INVALID_ARG;
  if (rowPtr) std::copy(a->pat.rowp.begin(), a->pat.rowp.end(), rowPtr);
  if (colPtr) std::copy(a->pat.cols.begin(), a->pat.cols.end(), colPtr);
  if (perm) std::copy(a->perm.begin(), a->perm.end(), perm);
  if (elemIndMap) std::copy(a->emap.begin(), a->emap.end(), elemIndMap);
  return GF_OK;
}

gf_status gf_assembler_get_schedule(const gf_assembler* a, int32_t* elem_chunk,
                                    int32_t* chunk_color, int32_t* elem_color,
                                    uint32_t* first_touch, int32_t* num_chunk_colors,
                                    int32_t* num_chunks) {
  if (!a) return GF_INVALID_ARG;
  const Schedule& s = a->sched;
  if (elem_chunk) std::copy(s.elem_chunk.begin(), s.elem_chunk.end(), elem_chunk);
  if (chunk_color) std::copy(s.chunk_color.begin(), s.chunk_color.end(), chunk_color);
  if (elem_color) std::copy(s.elem_color.begin(), s.elem_color.end(), elem_color);
  if (first_touch) std::copy(s.first_touch.begin(), s.first_touch.end(), first_touch);
  if (num_chunk_colors) *num_chunk_colors = s.ncc;
  if (num_chunks) *num_chunks = s.nchunks;
  return GF_OK;
}

gf_status gf_set_variables(gf_assembler* a, const double* d_vars, void* stream) {
  if (!a || !d_vars) return GF_INVALID_ARG;
  GF_CUDA(cudaMemcpyAsync(a->d_vars.p, d_vars, sizeof(double) * 6 * a->nnodes,
                          cudaMemcpyDeviceToDevice, as_stream(stream)));
  return GF_OK;
}

gf_status gf_add_residual(gf_assembler* a, double* d_res, int32_t flags, void* stream) {
  if (!a || !d_res) return GF_INVALID_ARG;
  return launch_assembly<MODE_RES>(a, nullptr, d_res, flags, as_stream(stream));
}

gf_status gf_assembler_setup_info(const gf_assembler* a, int32_t* pattern_on_gpu,
                                  int32_t* elem_map_on_gpu) {
  if (!a) return GF_INVALID_ARG;
  if (pattern_on_gpu) *pattern_on_gpu = (a->sym_flags & 1) ? 1 : 0;
  if (elem_map_on_gpu) *elem_map_on_gpu = (a->sym_flags & 2) ? 1 : 0;
  return GF_OK;
}

gf_status gf_assembler_setup_times(const gf_assembler* a, double* records_ms, double* setup_ms) {
  if (!a) return GF_INVALID_ARG;
  if (records_ms) *records_ms = a->records_ms;
  if (setup_ms) *setup_ms = a->setup_ms;
  return GF_OK;
}

gf_status gf_add_jacobian(gf_assembler* a, double* d_res, gf_bsr* mat, int32_t flags,
                          void* stream) {
  if (!a || !mat || mat->a != a) return GF_INVALID_ARG;
  return launch_assembly<MODE_JAC>(a, mat->vals.p, d_res, flags, as_stream(stream));
}

gf_status gf_add_jacobian_thick(gf_assembler* a, const double* d_thick, double* d_res,
                                gf_bsr* mat, int32_t flags, void* stream) {
  if (!a || !mat || mat->a != a || !d_thick) return GF_INVALID_ARG;
  return launch_assembly<MODE_JAC>(a, mat->vals.p, d_res, flags, as_stream(stream), d_thick);
}

gf_status gf_add_energy(gf_assembler* a, double* h_energy, void* stream) {
  if (!a || !h_energy) return GF_INVALID_ARG;
  cudaStream_t st = as_stream(stream);
  gf_status s = launch_assembly<MODE_ENERGY>(a, nullptr, nullptr, 0, st);
  if (s != GF_OK) return s;
  sum_kernel<<<1, 256, 0, st>>>(a->d_energy_part.p, a->sched.nchunks,
                                a->d_energy_part.p + a->sched.nchunks); ::gf::count_launch();
  GF_CHECK_LAUNCH();
  GF_CUDA(cudaMemcpyAsync(h_energy, a->d_energy_part.p + a->sched.nchunks, sizeof(double),
                          cudaMemcpyDeviceToHost, st));
  GF_CUDA(cudaStreamSynchronize(st));
  return GF_OK;
}

gf_status gf_assembler_set_thickness(gf_assembler* a, const double* d_thick, void* stream) {
  if (!a || !d_thick) return GF_INVALID_ARG;
  gather_thickness<<<(a->nelem + 255) / 256, 256, 0, as_stream(stream)>>>(
      a->d_sorder.p, a->nelem, d_thick, a->d_sthick.p); ::gf::count_launch();
  GF_CHECK_LAUNCH();
  return GF_OK;
}

gf_status gf_apply_bcs_vec(gf_assembler* a, double* d_vec, void* stream) {
  if (!a || !d_vec) return GF_INVALID_ARG;
  if (a->nbcs == 0) return GF_OK;
  bc_vec_kernel<<<(a->nbcs + 255) / 256, 256, 0, as_stream(stream)>>>(a->d_bcs.p, a->nbcs,
                                                                      d_vec); ::gf::count_launch();
  GF_CHECK_LAUNCH();
  return GF_OK;
}

gf_status gf_apply_bcs_mat(gf_assembler* a, gf_bsr* mat, void* stream) {
  if (!a || !mat || mat->a != a) return GF_INVALID_ARG;
  if (a->nbc_entries == 0) return GF_OK;
  bc_mat_kernel<<<(a->nbc_entries + 127) / 128, 128, 0, as_stream(stream)>>>(
      a->d_bc_entries.p, a->nbc_entries, a->d_cols.p, mat->vals.p); ::gf::count_launch();
  GF_CHECK_LAUNCH();
  return GF_OK;
}

gf_status gf_bsr_create(gf_assembler* a, gf_bsr** out) {
  if (!a || !out) return GF_INVALID_ARG;
  gf_bsr* m = new gf_bsr();
  m->a = a;
  cudaError_t e = m->vals.alloc((size_t)36 * a->pat.nnz());
  if (e == cudaSuccess) e = cudaMemset(m->vals.p, 0, sizeof(double) * 36 * a->pat.nnz());
  if (e != cudaSuccess) {
    set_last_error("gf_bsr_create", e);
    delete m;
    return e == cudaErrorMemoryAllocation ? GF_OOM : GF_CUDA_ERROR;
  }
  *out = m;
  return GF_OK;
}

gf_status gf_bsr_destroy(gf_bsr* m) {
  delete m;
  return GF_OK;
}

double* gf_bsr_values(gf_bsr* m) { return m ? m->vals.p : nullptr; }

gf_status gf_bsr_zero(gf_bsr* m, void* stream) {
  if (!m) return GF_INVALID_ARG;
  GF_CUDA(cudaMemsetAsync(m->vals.p, 0, sizeof(double) * m->vals.n, as_stream(stream)));
  return GF_OK;
}

gf_status gf_permute_vec(gf_assembler* a, const double* d_in, double* d_out, int32_t dir,
                         void* stream) {
  if (!a || !d_in || !d_out || d_in == d_out || (dir != 0 && dir != 1)) return GF_INVALID_ARG;
  const int n = 6 * a->nnodes;
  permute_kernel<<<(n + 255) / 256, 256, 0, as_stream(stream)>>>(a->d_perm.p, a->nnodes, d_in,
                                                                  d_out, dir); ::gf::count_launch();
  GF_CHECK_LAUNCH();
  return GF_OK;
}

}  // extern "C"
