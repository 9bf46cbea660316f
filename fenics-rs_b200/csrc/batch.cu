// Batched Jacobi-PCG over many independent systems (no reference
// counterpart; the batch of the scope table's multi-mesh case).
//
// The systems are the diagonal blocks of one block-diagonal matrix: meshes
// of uneven sizes are concatenated into one mesh (vertex ranges disjoint), so
// the library's pattern, assembly, load-vector and Dirichlet kernels build
// the whole batch in one pass each, and block i is rows [off[i], off[i+1]).
//
// Each instance is solved by one thread-block cluster, whose CTAs own contiguous
// shares of its rows and sum their partials through distributed shared memory
// in rank order, so instances converge, stop and report independently and no
// grid-wide synchronisation exists. The arithmetic per instance is that of the
// library's single-system PCG (cg.rs:40-149 for FP64; for mixed, FP32
// difference-form operator with FP64 r, x and dots and FP64 residual
// replacement). Two forms: the resident one holds the instance on chip
// (clusters of 1 to 16 CTAs, one launch per cluster size, the launches side by
// side); the streaming one, for instances that do not fit, reads its data from
// memory each iteration (clusters of 1 to 8 that take instances from a queue in
// order of estimated cost). Several launches are captured in a CUDA graph, which
// later solves replay. The streaming form's lanes per row, threads per CTA and
// CTAs per cluster are picked by timing the candidates on its instances (first
// solve of a matrix and precision), unless FCU_BATCH_VPR / FCU_BATCH_THREADS /
// FCU_BATCH_CLUSTER fix them. A single system (the small-system path of the PCG)
// is taken if all of it fits on chip.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <memory>
#include <string>
#include <vector>

#include <cooperative_groups.h>

#include "internal.cuh"

namespace cg = cooperative_groups;

void build_rowsum32(fcu_matrix m);

namespace {

constexpr unsigned BFULL = 0xffffffffu;

__device__ __forceinline__ double bwarp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(BFULL, v, o);
  return v;
}

// Sum NV doubles over the cluster that owns the instance; every thread of
// every CTA of the cluster gets the totals. Each CTA reduces its threads in a
// fixed order and publishes its sum in a shared-memory slot; after the
// cluster barrier (release/acquire at cluster scope, so it also orders the
// CTAs' global-memory writes) every thread adds the slots in rank order. The
// slots alternate between two buffers: a CTA rewrites a buffer only after the
// next barrier, which every CTA reaches after reading it.
template <int NV, int BT>
__device__ __forceinline__ void cluster_sum(double (&v)[NV], double (*slots)[4], int& parity,
                                            cg::cluster_group& cl) {
  __shared__ double sh[NV][BT / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const double x = bwarp_sum(v[j]);
    if (lane == 0) sh[j][w] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      double t = 0.0;
      for (int q = 0; q < BT / 32; ++q) t += sh[j][q];
      slots[parity][j] = t;
    }
  }
  cl.sync();
  const unsigned nr = cl.num_blocks();
#pragma unroll
  for (int j = 0; j < NV; ++j) v[j] = 0.0;
  for (unsigned k = 0; k < nr; ++k) {
    const double* rs = cl.map_shared_rank(&slots[parity][0], k);
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] += rs[j];
  }
  parity ^= 1;
}

// One CSR row with VPR >= 2 lanes (all lanes of the warp call it). DIFF: the
// mixed operator y_i = sum_{j != i} a_ij (x_j - x_i) + S_i x_i, with S_i in
// the diagonal slot; otherwise y_i = sum_j a_ij x_j.
template <int VPR, bool DIFF, class T, class GV>
__device__ __forceinline__ T batch_row(const int* __restrict__ rp, const int* __restrict__ ci,
                                       const T* __restrict__ val, i64 row, bool valid, int sub, const GV& xv) {
  T s = T(0);
  if (valid) {
    const int b = rp[row], e = rp[row + 1];
    const T xi = DIFF ? xv(row) : T(0);
    for (int q = b + sub; q < e; q += VPR) {
      const int c = ci[q];
      if (DIFF) s += val[q] * (c == (int)row ? xi : xv(c) - xi);
      else s += val[q] * xv(c);
    }
  }
#pragma unroll
  for (int o = VPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(BFULL, s, o);
  return s;
}

// One CSR row per thread (VPR = 1): a block of entries (eight for FP32,
// four for FP64, to stay within the register budget) is loaded, values and
// columns, then all its operand entries, before the arithmetic. Entries are
// summed in CSR order; unused slots read row 0's operand with weight 0.
template <bool DIFF, class T, class GV>
__device__ __forceinline__ T batch_row1(int a0, int a1, const int* __restrict__ ci, const T* __restrict__ val, i64 row,
                                        const GV& xv) {
  constexpr int E = sizeof(T) == 4 ? 8 : 4;
  const T xa = DIFF ? xv(row) : T(0);
  T s = T(0);
  for (int k0 = a0; k0 < a1; k0 += E) {
    const int na = a1 - k0;
    int c[E];
    T wv[E], g[E];
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const bool h = k < na;
      c[k] = h ? ci[k0 + k] : 0;
      wv[k] = h ? val[k0 + k] : T(0);
    }
#pragma unroll
    for (int k = 0; k < E; ++k) g[k] = xv(c[k]);
#pragma unroll
    for (int k = 0; k < E; ++k) {
      if (DIFF) s += wv[k] * (c[k] == (int)row ? xa : g[k] - xa);
      else s += wv[k] * g[k];
    }
  }
  return s;
}

struct BatchArgs {
  const int* rp;
  const int* ci;
  const double* val64;
  const float* val32;
  const i64* off;    // nb + 1 row offsets
  const int* order;  // instances, largest first
  int nb;
  const double* b;
  double* x;
  double* r;
  const double* invd;
  void* z;   // T
  void* p;   // T
  void* ap;  // T
  void* p2;  // T: the second direction buffer (p alternates between p and p2)
  double tol;
  i64 max_iter;
  double delta;
  unsigned* counter;  // queue head (zeroed before every launch)
  i64* iters;
  i64* updates;
  double* relres;
  double* resid;  // absolute residual ||r|| per instance
  int* status;
};

// Operator rows [c0, c1) of this CTA: y = A v; emit(row, y) once per row.
template <int VPR, int BT, bool DIFF, class T, class GV, class Emit>
__device__ __forceinline__ void batch_spmv(const int* __restrict__ rp, const int* __restrict__ ci,
                                           const T* __restrict__ val, i64 c0, i64 c1, const GV& v, Emit emit) {
  const int tid = threadIdx.x;
  if (VPR == 1) {
    // the next row's bounds are fetched while this row is summed
    i64 row = c0 + tid;
    int a0 = 0, a1 = 0;
    if (row < c1) {
      a0 = rp[row];
      a1 = rp[row + 1];
    }
    for (; row < c1; row += BT) {
      const i64 nxt = row + BT;
      int n0 = 0, n1 = 0;
      if (nxt < c1) {
        n0 = rp[nxt];
        n1 = rp[nxt + 1];
      }
      emit(row, batch_row1<DIFF, T>(a0, a1, ci, val, row, v));
      a0 = n0;
      a1 = n1;
    }
  } else {
    constexpr int G = BT / VPR;
    const int g = tid / VPR, sub = tid % VPR;
    for (i64 base = c0; base < c1; base += G) {
      const i64 row = base + g;
      const bool valid = row < c1;
      const T s = batch_row<VPR, DIFF, T>(rp, ci, val, row, valid, sub, v);
      if (valid && sub == 0) emit(row, s);
    }
  }
}

// Operand gathers of the batched SpMV: a plain vector, or the new direction
// p = z + beta p_old formed on the fly from the previous iteration's z and
// p_old (one fused multiply-add, as the direction update rounds it), so no
// cluster barrier is needed between forming p and reading it.
template <class T>
struct BatchPlain {
  const T* v;
  __device__ __forceinline__ T operator()(i64 i) const { return v[i]; }
};
template <class T>
struct BatchDirection {
  const T* z;
  const T* pold;
  T beta;
  __device__ __forceinline__ T operator()(i64 i) const { return fma(beta, pold[i], z[i]); }
};

// A cluster of CTAs (1 to 8; the launch's cluster size) solves one instance
// at a time: CTA rank k owns rows [r0 + k len / CL, r0 + (k + 1) len / CL)
// for every phase, and the phases are separated by cluster barriers.
// FD: the direction p = z + beta p_old is formed where the SpMV reads it,
// with p alternating between two buffers (no direction phase and no cluster
// barrier before the SpMV, at the cost of gathering z and p_old); otherwise
// a direction phase writes p in place and a cluster barrier follows it. Both
// round p with one fused multiply-add, so the iterates are the same.
template <int VPR, int BT, class T, bool FD>
__global__ void __launch_bounds__(BT, 1024 / BT) k_batch_pcg(BatchArgs a) {
  constexpr bool MIXED = sizeof(T) == 4;
  __shared__ int s_q;
  __shared__ double slots[2][4];
  cg::cluster_group cl = cg::this_cluster();
  const unsigned ncl = cl.num_blocks(), rank = cl.block_rank();
  int parity = 0;
  // the parameter block's address is never taken (no local copy of it)
  T* const z = static_cast<T*>(a.z);
  T* const pa = static_cast<T*>(a.p);
  T* const pb = static_cast<T*>(a.p2);
  T* const ap = static_cast<T*>(a.ap);
  const int tid = threadIdx.x;

  for (;;) {
    if (rank == 0 && tid == 0) s_q = (int)atomicAdd(a.counter, 1u);
    cl.sync();
    const int q = *cl.map_shared_rank(&s_q, 0);
    cl.sync();
    if (q >= a.nb) break;
    const int inst = a.order[q];
    const i64 r0 = a.off[inst], r1 = a.off[inst + 1];
    // rank k owns len / ncl rows, one more for the first len % ncl ranks
    // (32-bit arithmetic: rows are int32-indexed)
    const unsigned len = (unsigned)(r1 - r0);
    const unsigned share = len / ncl, extra = len % ncl;
    const i64 c0 = r0 + (i64)(share * rank + min(rank, extra));
    const i64 c1 = c0 + (i64)(share + (rank < extra ? 1u : 0u));

    // x0 = 0: r = b, z = D^-1 r, p = 0; r.z, r.r, b.b (cg.rs:79-90)
    double v3[3] = {0.0, 0.0, 0.0};
    for (i64 i = c0 + tid; i < c1; i += BT) {
      a.x[i] = 0.0;
      const double ri = a.b[i];
      a.r[i] = ri;
      const double zi = ri * a.invd[i];
      z[i] = (T)zi;
      pa[i] = T(0);
      v3[0] += ri * zi;
      v3[1] += ri * ri;
    }
    v3[2] = v3[1];
    cluster_sum<3, BT>(v3, slots, parity, cl);
    double rz = v3[0], rr = v3[1];
    const double bnorm = sqrt(v3[2]);
    double maxr = sqrt(rr);
    double beta = 0.0;
    i64 iter = 0, updates = 0;
    int status = FCU_ERR_NO_CONVERGENCE;
    [[maybe_unused]] int flip = 0;  // FD: p_old is pa when 0, pb when 1
    {
      const double r0n = sqrt(rr);
      if (r0n < a.tol || (bnorm > 0.0 && r0n / bnorm < a.tol)) status = FCU_OK;
    }
    while (status != FCU_OK && iter < a.max_iter) {
      const T* const vals = MIXED ? reinterpret_cast<const T*>(a.val32) : reinterpret_cast<const T*>(a.val64);
      double v1[1] = {0.0};
      T* p;
      if constexpr (FD) {
        // Ap and p.Ap with p = z + beta p_old formed where it is read; each
        // row's p is stored for the update and the next iteration
        const BatchDirection<T> dir{z, flip ? pb : pa, (T)beta};
        p = flip ? pa : pb;
        flip ^= 1;
        batch_spmv<VPR, BT, MIXED, T>(a.rp, a.ci, vals, c0, c1, dir, [&v1, ap, p, &dir](i64 row, T s) {
          const T pr = dir(row);
          p[row] = pr;
          ap[row] = s;
          v1[0] += (double)pr * (double)s;
        });
      } else {
        // direction, then Ap and p.Ap
        p = pa;
        const T bt = (T)beta;
        for (i64 i = c0 + tid; i < c1; i += 4 * BT) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const i64 k = i + u * BT;
            if (k < c1) p[k] = fma(bt, p[k], z[k]);
          }
        }
        cl.sync();
        batch_spmv<VPR, BT, MIXED, T>(a.rp, a.ci, vals, c0, c1, BatchPlain<T>{p}, [&v1, ap, p](i64 row, T s) {
          ap[row] = s;
          v1[0] += (double)p[row] * (double)s;
        });
      }
      cluster_sum<1, BT>(v1, slots, parity, cl);
      if (fabs(v1[0]) < 1e-30) {  // cg.rs:102-107
        iter += 1;
        status = FCU_ERR_BREAKDOWN;
        break;
      }
      const double alpha = rz / v1[0];
      // x += alpha p, r -= alpha Ap, z = D^-1 r
      double v2[2] = {0.0, 0.0};
      for (i64 i = c0 + tid; i < c1; i += 2 * BT) {
        double xi[2], ri[2], di[2];
        T pi[2], api[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const i64 k = i + u * BT;
          if (k < c1) {
            xi[u] = a.x[k];
            ri[u] = a.r[k];
            di[u] = a.invd[k];
            pi[u] = p[k];
            api[u] = ap[k];
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const i64 k = i + u * BT;
          if (k < c1) {
            a.x[k] = xi[u] + alpha * (double)pi[u];
            const double rn = ri[u] - alpha * (double)api[u];
            a.r[k] = rn;
            const double zi = rn * di[u];
            z[k] = (T)zi;
            v2[0] += rn * zi;
            v2[1] += rn * rn;
          }
        }
      }
      cluster_sum<2, BT>(v2, slots, parity, cl);
      iter += 1;
      rr = v2[1];
      const double res = sqrt(v2[1]);
      const double rel = bnorm > 0.0 ? res / bnorm : res;
      if (!MIXED) {
        if (rel < a.tol) {
          status = FCU_OK;
          break;
        }
        beta = v2[0] / rz;
        rz = v2[0];
        continue;
      }
      if (!(rel < a.tol || res < a.delta * maxr)) {
        beta = v2[0] / rz;
        rz = v2[0];
        continue;
      }
      // residual replacement with the FP64 matrix: r = b - A64 x, z = D^-1 r
      // (x of the whole instance is complete since the cluster sum above)
      double v4[2] = {0.0, 0.0};
      batch_spmv<VPR, BT, false, double>(a.rp, a.ci, a.val64, c0, c1, BatchPlain<double>{a.x},
                                         [&v4, z, rv = a.r, bv = a.b, dv = a.invd](i64 row, double s) {
                                           const double rn = bv[row] - s;
                                           rv[row] = rn;
                                           const double zi = rn * dv[row];
                                           z[row] = (T)zi;
                                           v4[0] += rn * zi;
                                           v4[1] += rn * rn;
                                         });
      cluster_sum<2, BT>(v4, slots, parity, cl);
      updates += 1;
      rr = v4[1];
      const double res2 = sqrt(v4[1]);
      const double rel2 = bnorm > 0.0 ? res2 / bnorm : res2;
      if (rel2 < a.tol) {
        status = FCU_OK;
        break;
      }
      maxr = res2;
      beta = v4[0] / rz;
      rz = v4[0];
    }
    if (rank == 0 && tid == 0) {
      a.iters[inst] = iter;
      a.updates[inst] = updates;
      a.relres[inst] = bnorm > 0.0 ? sqrt(rr) / bnorm : sqrt(rr);
      a.resid[inst] = sqrt(rr);
      a.status[inst] = status;
    }
  }
}

// ---------------------------------------------------------------------------
// Resident form: a cluster of 1 to 16 CTAs holds its whole instance on chip for
// the duration of its PCG. Each CTA owns a contiguous share of the rows; the
// share's matrix entries lie in shared memory (ELL: entry e of all rows
// together, two 16-bit columns to a word, relative to the CTA's window of the
// direction), x, r and D^-1 in registers (RM rows per thread), and the window
// of p (own rows plus the band on either side) in shared memory. An iteration
// touches no global memory; it has two cluster barriers:
//   p = z + beta p over the window (z of other CTAs' rows read from their
//   shared memory), Ap from shared memory           -> p.Ap over the cluster
//   x, r updated in registers, z stored             -> r.z and r.r
// What bounds it: instruction issue of the product (29k warp instructions per SM
// and iteration with full shares, 50 % of the issue slots; 5.1k of them shared
// loads) and the two cluster barriers of 1.1 us. A 257^2 instance takes 6.9 us
// per iteration on 16 SMs; the streaming form, bound by chains of L2 loads,
// took 100 us on its two. 256 instances of 32^2 to 256^2 cells, mixed, to 1e-8:
// 108 -> 61 ms (FP64 140 -> 92); one 64^2: 1.67 -> 1.05 ms. One row at a time
// per thread: sums of three rows side by side, and shapes with fewer rows on
// more threads, spilled and took 5 to 30 % longer. The diagonal is entry 0, on
// the row's own operand, so that no entry has to be compared with its row.
// Rows that do not fit (FP64, the largest instances) stay in global memory and
// are read from there.
// ---------------------------------------------------------------------------

constexpr int RNT = 512;        // threads per CTA
constexpr int RM = 9;           // rows per thread, at most
constexpr int RMAXC = 16;       // CTAs per cluster, at most
constexpr int RMAX_WIDTH = 32;  // entries per row, at most

struct ResidentInfo {
  int width;  // entries of the longest row, a diagonal slot included
  int band;   // largest |column - row|
  int cap;    // rows of a CTA's share held in shared memory
  int share;  // rows per CTA
};

// Byte offsets of a CTA's shared memory: the window of p first (the stored
// columns are byte offsets into it), own z, the matrix.
struct ResidentLayout {
  size_t z, val, col, end;
  __host__ __device__ ResidentLayout(int wv, int share, int band, int width, int cap) {
    auto al = [](size_t x) { return (x + 15) & ~(size_t)15; };
    z = al(((size_t)share + 2 * (size_t)band) * wv);
    val = z + al((size_t)share * wv);
    col = val + al((size_t)width * cap * wv);
    end = col + al((size_t)((width + 1) / 2) * cap * 4);
  }
};

// NV sums over the cluster: the CTA's sum goes to every CTA's slots before the
// cluster barrier, after which each warp adds its own copy in rank order (a
// fixed shuffle tree), so every thread of every CTA has the same totals.
template <int NV>
__device__ __forceinline__ void resident_sum(double (&v)[NV], double (*sh)[RNT / 32], double (*slots)[2][RMAXC],
                                             int& parity, cg::cluster_group& cl, unsigned ncl, unsigned rank) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const double x = bwarp_sum(v[j]);
    if (lane == 0) sh[j][w] = x;
  }
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const double x = bwarp_sum(lane < RNT / 32 ? sh[j][lane] : 0.0);
      if (lane < (int)ncl) *cl.map_shared_rank(&slots[parity][j][rank], lane) = x;
    }
  }
  if (ncl > 1) cl.sync();
  else __syncthreads();
#pragma unroll
  for (int j = 0; j < NV; ++j) v[j] = bwarp_sum(lane < (int)ncl ? slots[parity][j][lane] : 0.0);
  parity ^= 1;
}

template <class T>
__global__ void __launch_bounds__(RNT, 1) k_batch_resident(BatchArgs a, const int* __restrict__ list,
                                                          const ResidentInfo* __restrict__ info, int count,
                                                          int* __restrict__ next) {
  constexpr bool MIXED = sizeof(T) == 4;
  extern __shared__ __align__(16) unsigned char res_smem[];
  __shared__ double sh[2][RNT / 32];
  __shared__ double slots[2][2][RMAXC];
  __shared__ int turn;
  cg::cluster_group cl = cg::this_cluster();
  const unsigned ncl = cl.num_blocks(), rank = cl.block_rank();
  int parity = 0;
  const int tid = threadIdx.x;
  // The first sum stores into the other CTAs' shared memory: all of them have to have started.
  if (ncl > 1) cl.sync();
  // instances: as many as clusters at once, the others as clusters come free
  for (int at = (int)(blockIdx.x / ncl); at < count;) {
    const int inst = list[at];
    const ResidentInfo in = info[inst];
    const int r0 = (int)a.off[inst], r1 = (int)a.off[inst + 1];
    const int c0 = min(r0 + (int)rank * in.share, r1), c1 = min(c0 + in.share, r1);
    const int nloc = c1 - c0;
    const int wlo = max(r0, c0 - in.band), whi = min(r1, c1 + in.band);  // window of p
    const int off = c0 - wlo;
    const int lo_halo = nloc > 0 ? off : 0, hi_halo = nloc > 0 ? whi - c1 : 0;
    const ResidentLayout L(sizeof(T), in.share, in.band, in.width, in.cap);
    T* const pw = reinterpret_cast<T*>(res_smem);
    T* const zs = reinterpret_cast<T*>(res_smem + L.z);
    T* const ev = reinterpret_cast<T*>(res_smem + L.val);
    unsigned* const ec = reinterpret_cast<unsigned*>(res_smem + L.col);
    const T* const vals = MIXED ? reinterpret_cast<const T*>(a.val32) : reinterpret_cast<const T*>(a.val64);

    // the matrix: the diagonal slot first (its column is not looked up), then the
    // row's other entries; unused ones have weight 0 on the row's own operand
    for (int i = tid; i < min(nloc, in.cap); i += RNT) {
      const int a1 = a.rp[c0 + i + 1];
      int q = a.rp[c0 + i];
      const unsigned self = (unsigned)(off + i) * (unsigned)sizeof(T);
      T d = T(0);
      auto next = [&](T& v) {  // the next off-diagonal entry: weight, offset of its p
        for (; q < a1; ++q) {
          const int c = a.ci[q] - wlo;
          v = vals[q];
          if (c != off + i) {
            ++q;
            return (unsigned)c * (unsigned)sizeof(T);
          }
          d += v;
        }
        v = T(0);
        return self;
      };
      for (int e = 0; e < in.width; e += 2) {
        T v0, v1;
        const unsigned k0 = e ? next(v0) : self, k1 = next(v1);
        ec[(e >> 1) * in.cap + i] = k0 | (k1 << 16);
        if (e) ev[e * in.cap + i] = v0;
        if (e + 1 < in.width) ev[(e + 1) * in.cap + i] = v1;
      }
      while (q < a1) {  // only the diagonal can be left
        T v;
        next(v);
      }
      ev[i] = d;
    }
    // x0 = 0: r = b, z = D^-1 r, p = 0 (cg.rs:79-90)
    double xv[RM], rv[RM], dv[RM];
    double v2[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < RM; ++k) {
      const int i = tid + k * RNT;
      xv[k] = 0.0;
      rv[k] = i < nloc ? a.b[c0 + i] : 0.0;
      dv[k] = i < nloc ? a.invd[c0 + i] : 0.0;
      if (i < nloc) {
        const double zi = rv[k] * dv[k];
        zs[i] = (T)zi;
        v2[0] += rv[k] * zi;
        v2[1] += rv[k] * rv[k];
      }
    }
    for (int j = tid; j < whi - wlo; j += RNT) pw[j] = T(0);
    resident_sum<2>(v2, sh, slots, parity, cl, ncl, rank);
    double rz = v2[0], rr = v2[1];
    const double bnorm = sqrt(rr);
    double maxr = bnorm, beta = 0.0;
    i64 iter = 0, updates = 0;
    int status = FCU_ERR_NO_CONVERGENCE;
    if (bnorm < a.tol || (bnorm > 0.0 && bnorm / bnorm < a.tol)) status = FCU_OK;
    while (status != FCU_OK && iter < a.max_iter) {
      // p = z + beta p over the window
      const T bt = (T)beta;
      for (int i = tid; i < nloc; i += RNT) pw[off + i] = fma(bt, pw[off + i], zs[i]);
      for (int h = tid; h < lo_halo + hi_halo; h += RNT) {
        const int j = h < lo_halo ? h : h + nloc;
        const int g = wlo + j - r0;
        const int q = g / in.share;
        const T z = *cl.map_shared_rank(zs + (g - q * in.share), q);
        pw[j] = fma(bt, pw[j], z);
      }
      __syncthreads();
      // Ap and p.Ap
      double v1[1] = {0.0};
      T apv[RM];
#pragma unroll
      for (int k = 0; k < RM; ++k) {
        const int i = tid + k * RNT;
        apv[k] = T(0);
        if (i < nloc) {
          // the diagonal slot on its own operand; mixed: the others act on
          // differences
          const T own = pw[off + i];
          T s;
          auto add = [&](T v, unsigned at) {  // at: byte offset of the column's p
            const T y = *reinterpret_cast<const T*>(res_smem + at);
            s += v * (MIXED ? y - own : y);
          };
          if (i < in.cap) {
            const unsigned* pc = ec + i;
            const T* pv = ev + i;
            s = pv[0] * own;
            if (in.width > 1) add(pv[in.cap], *pc >> 16);
            int e = 2;
#pragma unroll 2
            for (; e + 1 < in.width; e += 2) {
              pc += in.cap;
              pv += 2 * in.cap;
              const unsigned cc = *pc;
              add(pv[0], cc & 0xffffu);
              add(pv[in.cap], cc >> 16);
            }
            if (e < in.width) add(pv[2 * in.cap], pc[in.cap] & 0xffffu);
          } else {
            const int a1 = a.rp[c0 + i + 1];
            s = T(0);
            for (int q = a.rp[c0 + i]; q < a1; ++q) {
              const int c = a.ci[q] - wlo;
              s += vals[q] * (MIXED && c != off + i ? pw[c] - own : pw[c]);
            }
          }
          apv[k] = s;
          v1[0] += (double)own * (double)s;
        }
      }
      resident_sum<1>(v1, sh, slots, parity, cl, ncl, rank);
      if (fabs(v1[0]) < 1e-30) {  // cg.rs:102-107
        iter += 1;
        status = FCU_ERR_BREAKDOWN;
        break;
      }
      const double alpha = rz / v1[0];
      // x += alpha p, r -= alpha Ap, z = D^-1 r
      v2[0] = v2[1] = 0.0;
#pragma unroll
      for (int k = 0; k < RM; ++k) {
        const int i = tid + k * RNT;
        if (i < nloc) {
          xv[k] += alpha * (double)pw[off + i];
          rv[k] -= alpha * (double)apv[k];
          const double zi = rv[k] * dv[k];
          zs[i] = (T)zi;
          v2[0] += rv[k] * zi;
          v2[1] += rv[k] * rv[k];
        }
      }
      resident_sum<2>(v2, sh, slots, parity, cl, ncl, rank);
      iter += 1;
      rr = v2[1];
      const double res = sqrt(rr);
      const double rel = bnorm > 0.0 ? res / bnorm : res;
      if (!MIXED) {
        if (rel < a.tol) {
          status = FCU_OK;
          break;
        }
      } else if (rel < a.tol || res < a.delta * maxr) {
        // residual replacement with the FP64 matrix: r = b - A64 x, z = D^-1 r
#pragma unroll
        for (int k = 0; k < RM; ++k)
          if (tid + k * RNT < nloc) a.x[c0 + tid + k * RNT] = xv[k];
        if (ncl > 1) cl.sync();
        else __syncthreads();
        v2[0] = v2[1] = 0.0;
#pragma unroll
        for (int k = 0; k < RM; ++k) {
          const int i = tid + k * RNT;
          if (i < nloc) {
            double s = 0.0;
            const int a1 = a.rp[c0 + i + 1];
            for (int q = a.rp[c0 + i]; q < a1; ++q) s += a.val64[q] * __ldcg(a.x + a.ci[q]);
            rv[k] = a.b[c0 + i] - s;
            const double zi = rv[k] * dv[k];
            zs[i] = (T)zi;
            v2[0] += rv[k] * zi;
            v2[1] += rv[k] * rv[k];
          }
        }
        resident_sum<2>(v2, sh, slots, parity, cl, ncl, rank);
        updates += 1;
        rr = v2[1];
        const double res2 = sqrt(rr);
        const double rel2 = bnorm > 0.0 ? res2 / bnorm : res2;
        if (rel2 < a.tol) {
          status = FCU_OK;
          break;
        }
        maxr = res2;
      }
      beta = v2[0] / rz;
      rz = v2[0];
    }
#pragma unroll
    for (int k = 0; k < RM; ++k)
      if (tid + k * RNT < nloc) a.x[c0 + tid + k * RNT] = xv[k];
    if (rank == 0 && tid == 0) {
      a.iters[inst] = iter;
      a.updates[inst] = updates;
      a.relres[inst] = bnorm > 0.0 ? sqrt(rr) / bnorm : sqrt(rr);
      a.resid[inst] = sqrt(rr);
      a.status[inst] = status;
    }
    if ((int)(gridDim.x / ncl) >= count) break;
    if (rank == 0 && tid < 32) {  // the whole first warp, so that the mask holds lane 0
      int v = 0;
      if (tid == 0) v = (int)(gridDim.x / ncl) + atomicAdd(next, 1);
      v = __shfl_sync(BFULL, v, 0);
      if (tid < (int)ncl) *cl.map_shared_rank(&turn, tid) = v;
    }
    cl.sync();
    at = turn;
  }
}

// D^-1 from the diagonal slots (cg.rs:52-64: 1 when |a_kk| <= 1e-15).
__global__ void k_batch_invd(const int* __restrict__ diag_pos, const double* __restrict__ val, i64 n,
                             double* __restrict__ invd) {
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    const int dp = diag_pos[i];
    const double d = dp >= 0 ? val[dp] : 0.0;
    invd[i] = fabs(d) > 1e-15 ? 1.0 / d : 1.0;
  }
}

// Every row of block i must only reference columns of block i; its entries,
// longest row and bandwidth (info[4 i ..]). Blocks (i, *) share instance i.
__global__ void k_batch_check(const int* __restrict__ rp, const int* __restrict__ ci, const i64* __restrict__ off,
                              int nb, int* __restrict__ bad, int* __restrict__ info) {
  const int inst = blockIdx.x;
  if (inst >= nb) return;
  const i64 r0 = off[inst], r1 = off[inst + 1];
  int nnz = 0, len = 0, band = 0;
  for (i64 row = r0 + blockIdx.y * blockDim.x + threadIdx.x; row < r1; row += (i64)gridDim.y * blockDim.x) {
    const int b = rp[row], e = rp[row + 1];
    nnz += e - b;
    int others = 0;
    for (int q = b; q < e; ++q) {
      const int c = ci[q];
      others += c != (int)row;
      if (c < r0 || c >= r1) atomicExch(bad, 1);
      band = max(band, abs(c - (int)row));
    }
    len = max(len, others + 1);
  }
  nnz = __reduce_add_sync(BFULL, nnz);
  len = __reduce_max_sync(BFULL, len);
  band = __reduce_max_sync(BFULL, band);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&info[4 * inst], nnz);
    atomicMax(&info[4 * inst + 1], len);
    atomicMax(&info[4 * inst + 2], band);
  }
}

// One resident launch: the instances that take clusters of this size.
struct ResidentClass {
  int cluster = 1;
  int first = 0, count = 0;  // in the class list
  int clusters = 0;          // launched; fewer than count: they take instances in turn
  size_t smem = 0;
};

struct BatchConfig {
  int vpr = 1;
  int threads = 1024;
  int cluster = 1;
};

using BatchKernel = void (*)(BatchArgs);

template <class T>
BatchKernel batch_kernel(int vpr, int threads, bool fd) {
#define FCU_BATCH_CASE(V, B) \
  if (vpr == V && threads == B) return fd ? k_batch_pcg<V, B, T, true> : k_batch_pcg<V, B, T, false>;
  FCU_BATCH_CASE(1, 512) FCU_BATCH_CASE(1, 1024)
  FCU_BATCH_CASE(2, 512) FCU_BATCH_CASE(2, 1024)
  FCU_BATCH_CASE(4, 512) FCU_BATCH_CASE(4, 1024)
#undef FCU_BATCH_CASE
  return nullptr;
}

}  // namespace

// Per-matrix state of the batched solver: the instance layout, work buffers,
// the tuned configuration and the instantiated graph, per precision.
struct BatchWorkspace {
  int nb = 0;
  std::vector<i64> off;  // host copy of the offsets
  DBuf<i64> off_d;
  DBuf<double> b, x, r, invd;
  DBuf<double> z64, p64, q64, ap64;  // q: the second direction buffer
  DBuf<float> z32, p32, q32, ap32;
  DBuf<unsigned> counter;
  DBuf<i64> results;  // nb each: iterations, replacements, relative and absolute residual, status
  std::vector<int> nnz, width, band;  // per instance: entries, longest row, bandwidth
  std::vector<ResidentClass> classes[2];  // resident launches (FP64, FP32), then the instances left to the queue
  DBuf<ResidentInfo> info[2];
  DBuf<int> lists[2];                 // instances by class, the queue's last
  DBuf<int> turns;                    // by cluster size: instances taken so far beyond the first ones
  int nqueue[2] = {0, 0};
  std::vector<cudaStream_t> side;     // branches of the captured launch
  std::vector<cudaEvent_t> joins;
  BatchConfig cfg[2];
  bool planned[2] = {false, false}, tuned[2] = {false, false};
  bool on_chip[2] = {false, false};   // every instance is resident, with all of its rows
  cudaGraphExec_t graph[2] = {nullptr, nullptr};
  double tol_g[2] = {0.0, 0.0};
  i64 iters_g[2] = {0, 0};
  ~BatchWorkspace() {
    for (auto& g : graph)
      if (g) cudaGraphExecDestroy(g);
    for (auto& e : joins) cudaEventDestroy(e);
    for (auto& t : side) cudaStreamDestroy(t);
  }
};

void destroy_batch_ws(BatchWorkspace* w) { delete w; }

namespace {

int env_int(const char* name, int dflt) {
  const char* e = getenv(name);
  return e ? atoi(e) : dflt;
}

BatchArgs make_args(fcu_matrix m, BatchWorkspace* w, bool mixed, double tol, i64 max_iter) {
  BatchArgs a;
  a.rp = m->row_ptr;
  a.ci = m->col_idx;
  a.val64 = m->val64.p;
  a.val32 = m->val32.p;
  a.off = w->off_d.p;
  a.order = w->lists[mixed ? 1 : 0].p + (w->nb - w->nqueue[mixed ? 1 : 0]);
  a.nb = w->nqueue[mixed ? 1 : 0];
  a.b = w->b.p;
  a.x = w->x.p;
  a.r = w->r.p;
  a.invd = w->invd.p;
  a.z = mixed ? (void*)w->z32.p : (void*)w->z64.p;
  a.p = mixed ? (void*)w->p32.p : (void*)w->p64.p;
  a.p2 = mixed ? (void*)w->q32.p : (void*)w->q64.p;
  a.ap = mixed ? (void*)w->ap32.p : (void*)w->ap64.p;
  a.tol = tol;
  a.max_iter = max_iter;
  a.delta = 0.1;
  a.counter = w->counter.p;
  a.iters = w->results.p;
  a.updates = w->results.p + w->nb;
  a.relres = reinterpret_cast<double*>(w->results.p + 2 * (i64)w->nb);
  a.resid = reinterpret_cast<double*>(w->results.p + 3 * (i64)w->nb);
  a.status = reinterpret_cast<int*>(w->results.p + 4 * (i64)w->nb);
  return a;
}

// The streaming form makes directions in the SpMV (FD) for FP64 and for a queue
// of one instance, where the saved cluster barrier pays; mixed queues keep the
// direction phase. Measured with every instance streamed, as all were before
// most moved on chip: 256 problems mixed 108.9 (FD) against 106.7 ms, FP64 138.6
// against 144.7; single systems of 4k-16k rows gained 9-14 %.
bool fused_direction(bool mixed, int nb) { return !mixed || nb == 1; }

BatchKernel pick_kernel(bool mixed, const BatchConfig& c, int nb) {
  const bool fd = fused_direction(mixed, nb);
  return mixed ? batch_kernel<float>(c.vpr, c.threads, fd) : batch_kernel<double>(c.vpr, c.threads, fd);
}

// Persistent grid: as many clusters as fit on the device at once (at most
// one per instance). 0 when the configuration cannot be placed.
int batch_grid(fcu_ctx ctx, BatchKernel k, const BatchConfig& c, int nb) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(c.cluster * std::max(1, std::min(nb, ctx->num_sms))));
  cfg.blockDim = dim3((unsigned)c.threads);
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)c.cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int nclusters = 0;
  if (cudaOccupancyMaxActiveClusters(&nclusters, k, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return c.cluster * std::min(nb, nclusters);
}

void launch_batch(cudaStream_t stream, BatchWorkspace* w, BatchKernel k, const BatchConfig& c, int grid,
                  const BatchArgs& a) {
  CUDA_CHECK(cudaMemsetAsync(w->counter.p, 0, sizeof(unsigned), stream));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)c.threads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)c.cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  CUDA_CHECK(cudaLaunchKernelEx(&cfg, k, a));
}

// Time each candidate (lanes per row x threads per CTA x CTAs per cluster) on
// the batch itself with a short iteration cap and keep the fastest.
BatchConfig autotune(fcu_matrix m, BatchWorkspace* w, bool mixed, double tol) {
  BatchConfig fixed;
  fixed.vpr = env_int("FCU_BATCH_VPR", 0);
  fixed.threads = env_int("FCU_BATCH_THREADS", 0);
  fixed.cluster = env_int("FCU_BATCH_CLUSTER", 0);
  if (fixed.vpr && fixed.threads && fixed.cluster && pick_kernel(mixed, fixed, w->nqueue[mixed ? 1 : 0]) &&
      batch_grid(m->ctx, pick_kernel(mixed, fixed, w->nqueue[mixed ? 1 : 0]), fixed, w->nqueue[mixed ? 1 : 0]) > 0)
    return fixed;
  fcu_ctx ctx = m->ctx;
  const int vprs[3] = {1, 2, 4};
  const int thr[2] = {512, 1024};
  const int cls[4] = {1, 2, 4, 8};
  BatchConfig best;
  float best_ms = 1e30f;
  cudaEvent_t e0, e1;
  CUDA_CHECK(cudaEventCreate(&e0));
  CUDA_CHECK(cudaEventCreate(&e1));
  const BatchArgs a = make_args(m, w, mixed, tol, 24);
  for (int v : vprs)
    for (int t : thr)
      for (int cs : cls) {
        BatchConfig c;
        c.vpr = v;
        c.threads = t;
        c.cluster = cs;
        BatchKernel k = pick_kernel(mixed, c, w->nqueue[mixed ? 1 : 0]);
        if (!k) continue;
        const int grid = batch_grid(ctx, k, c, w->nqueue[mixed ? 1 : 0]);
        if (grid <= 0) continue;
        launch_batch(ctx->stream, w, k, c, grid, a);  // warm
        CUDA_CHECK(cudaEventRecord(e0, ctx->stream));
        launch_batch(ctx->stream, w, k, c, grid, a);
        CUDA_CHECK(cudaEventRecord(e1, ctx->stream));
        CUDA_CHECK(cudaEventSynchronize(e1));
        float ms = 0.f;
        CUDA_CHECK(cudaEventElapsedTime(&ms, e0, e1));
        if (ms < best_ms) {
          best_ms = ms;
          best = c;
        }
      }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (best_ms >= 1e30f) fail(FCU_ERR_UNSUPPORTED, "no batched PCG configuration fits this device");
  return best;
}

// Dynamic shared memory a resident CTA may use; allows it, and clusters of 16,
// to the kernel.
template <class T>
size_t resident_limit(fcu_ctx ctx) {
  int optin = 0;
  CUDA_CHECK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
  const size_t limit = (size_t)optin - 2048;  // its static arrays
  CUDA_CHECK(cudaFuncSetAttribute(k_batch_resident<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
  CUDA_CHECK(cudaFuncSetAttribute(k_batch_resident<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  return limit;
}

template <class T>
cudaLaunchConfig_t resident_config(fcu_ctx ctx, cudaLaunchAttribute* attr, int cluster, int count, size_t smem,
                                   cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(cluster * count));
  cfg.blockDim = dim3(RNT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = (unsigned)cluster;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// Sorts the instances into resident launches by cluster size, largest cost
// first within each, and the rest (rows long or of very different lengths, or
// an instance larger than a cluster holds) to the queue of the streaming
// kernel. An instance takes the smallest cluster that holds all of it on chip,
// so that a CTA always has about as many rows to work on between barriers;
// where none does (FP64 above about 40k rows of seven entries), the largest
// cluster, with the rows that do not fit read from global memory. A batch that
// would leave most SMs idle takes larger clusters.
template <class T>
void plan_resident(fcu_matrix m, BatchWorkspace* w, const std::vector<int>& by_cost) {
  fcu_ctx ctx = m->ctx;
  const int k = sizeof(T) == 4 ? 1 : 0, wv = (int)sizeof(T);
  const size_t limit = resident_limit<T>(ctx);
  // clusters of each size that the device runs at a time with full shared memory
  std::array<int, RMAXC + 1>& active = ctx->batch_clusters[k];
  if (!active[1])
    for (int c = RMAXC; c > 0; --c) {
      cudaLaunchAttribute attr;
      const cudaLaunchConfig_t cfg = resident_config<T>(ctx, &attr, c, 1, limit, ctx->stream);
      if (cudaOccupancyMaxActiveClusters(&active[c], k_batch_resident<T>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        active[c] = 0;
      }
    }
  int cmax = RMAXC;
  while (cmax > 0 && !active[cmax]) --cmax;
  const int nb = w->nb;
  std::vector<int> cl(nb, 0);
  std::vector<ResidentInfo> info(nb);
  auto fit = [&](int i, int c, bool whole) {
    const i64 rows = w->off[i + 1] - w->off[i];
    const i64 share = std::max<i64>(1, (rows + c - 1) / c);
    const int width = std::max(1, w->width[i]), band = w->band[i];
    if (share > RNT * RM || (share + 2 * (i64)band) * wv > 65535) return false;
    const ResidentLayout L0(wv, (int)share, band, width, 0);
    if (L0.end + 64 > limit) return false;
    const i64 per = (i64)width * wv + (width + 1) / 2 * 4;
    const i64 cap = std::min<i64>(share, (i64)(limit - L0.end - 64) / per);
    if (whole ? cap < share : 4 * cap < share) return false;
    cl[i] = c;
    info[i] = ResidentInfo{width, band, (int)cap, (int)share};
    return true;
  };
  i64 ctas = 0;
  for (int i = 0; i < nb; ++i) {
    const double rows = (double)(w->off[i + 1] - w->off[i]);
    if (w->width[i] > RMAX_WIDTH || w->width[i] > 2.0 * w->nnz[i] / std::max(rows, 1.0) + 4.0) continue;
    for (int c = 1; c <= cmax && !cl[i]; ++c) fit(i, c, true);
    if (cl[i]) {  // a larger cluster of which as many run (67 -> 62 ms for the 256)
      int c = cl[i];
      while (c < cmax && active[c + 1] == active[cl[i]]) ++c;
      fit(i, c, true);
    } else if (cmax > 0) {
      fit(i, cmax, false);
    }
    ctas += cl[i];
  }
  // A few instances leave SMs idle: spread them over larger clusters while a
  // thread keeps a row (one 64^2 instance, FP64: 3.6 us per iteration on 8 SMs,
  // 4.9 on one).
  for (bool grown = true; grown && 2 * ctas <= ctx->num_sms;) {
    grown = false;
    for (int i = 0; i < nb; ++i) {
      const int c = cl[i], to = std::min(2 * c, cmax);
      if (to > c && w->off[i + 1] - w->off[i] >= (i64)to * RNT && fit(i, to, true)) {
        ctas += to - c;
        grown = true;
      }
    }
  }
  std::vector<int> lists;
  auto& classes = w->classes[k];
  classes.clear();
  for (int c = RMAXC; c > 0; --c) {
    ResidentClass rc;
    rc.cluster = c;
    rc.first = (int)lists.size();
    for (int i : by_cost)
      if (cl[i] == c) {
        const ResidentInfo& in = info[i];
        rc.smem = std::max(rc.smem, ResidentLayout(wv, in.share, in.band, in.width, in.cap).end);
        lists.push_back(i);
      }
    rc.count = (int)lists.size() - rc.first;
    // Clusters are placed kernel by kernel: while clusters of 16 wait for one of
    // the 7 places there are, the SMs beside them idle unless the grid ends at 7.
    rc.clusters = 2 * c > cmax ? std::min(rc.count, active[c]) : rc.count;
    if (rc.count) classes.push_back(rc);
  }
  w->nqueue[k] = nb - (int)lists.size();
  w->on_chip[k] = w->nqueue[k] == 0;
  for (int i = 0; i < nb; ++i) w->on_chip[k] = w->on_chip[k] && info[i].cap >= info[i].share;
  for (int i : by_cost)
    if (!cl[i]) lists.push_back(i);
  w->turns.alloc(RMAXC + 1);
  upload(ctx, w->lists[k], lists.data(), nb);
  upload(ctx, w->info[k], info.data(), nb);  // (pageable copies are staged before they return)
}

template <class T>
void launch_resident(fcu_ctx ctx, BatchWorkspace* w, const ResidentClass& rc, const BatchArgs& a,
                     cudaStream_t stream) {
  const int k = sizeof(T) == 4 ? 1 : 0;
  resident_limit<T>(ctx);
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = resident_config<T>(ctx, &attr, rc.cluster, rc.clusters, rc.smem, stream);
  CUDA_CHECK(cudaLaunchKernelEx(&cfg, k_batch_resident<T>, a, (const int*)(w->lists[k].p + rc.first),
                                (const ResidentInfo*)w->info[k].p, rc.count, w->turns.p + rc.cluster));
}

// Every launch of the batch: the resident classes, largest clusters first, and
// the queue kernel, side by side on branches of the context's stream.
void launch_all(fcu_matrix m, BatchWorkspace* w, bool mixed, double tol, i64 max_iter, double* x) {
  fcu_ctx ctx = m->ctx;
  const int k = mixed ? 1 : 0;
  BatchArgs a = make_args(m, w, mixed, tol, max_iter);
  a.x = x;
  const size_t branches = w->classes[k].size() + (w->nqueue[k] ? 1 : 0);
  while (w->side.size() + 1 < branches) {
    cudaStream_t t;
    CUDA_CHECK(cudaStreamCreateWithFlags(&t, cudaStreamNonBlocking));
    w->side.push_back(t);
  }
  while (w->joins.size() < branches) {
    cudaEvent_t e;
    CUDA_CHECK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    w->joins.push_back(e);
  }
  CUDA_CHECK(cudaMemsetAsync(w->turns.p, 0, (RMAXC + 1) * sizeof(int), ctx->stream));
  if (branches > 1) CUDA_CHECK(cudaEventRecord(w->joins[branches - 1], ctx->stream));  // fork
  for (size_t b = 0; b < branches; ++b) {
    cudaStream_t st = b == 0 ? ctx->stream : w->side[b - 1];
    if (b > 0) CUDA_CHECK(cudaStreamWaitEvent(st, w->joins[branches - 1], 0));
    if (b < w->classes[k].size()) {
      if (mixed) launch_resident<float>(ctx, w, w->classes[k][b], a, st);
      else launch_resident<double>(ctx, w, w->classes[k][b], a, st);
    } else {
      const BatchConfig c = w->cfg[k];
      BatchKernel kern = pick_kernel(mixed, c, w->nqueue[k]);
      const int grid = batch_grid(ctx, kern, c, w->nqueue[k]);
      if (grid <= 0) fail(FCU_ERR_UNSUPPORTED, "batched PCG configuration does not fit this device");
      launch_batch(st, w, kern, c, grid, a);
    }
  }
  for (size_t b = 1; b < branches; ++b) {  // join
    CUDA_CHECK(cudaEventRecord(w->joins[b - 1], w->side[b - 1]));
    CUDA_CHECK(cudaStreamWaitEvent(ctx->stream, w->joins[b - 1], 0));
  }
}

}  // namespace

// Batched PCG driver; b, x and the per-instance outputs are device or host
// buffers handled by the caller (api.cu) through staging.
int batch_pcg_impl(fcu_matrix m, i64 nb, const i64* offsets_host, const double* b_dev, double* x_dev, double tol,
                   i64 max_iter, int precision, i64* iters_host, double* relres_host, int* status_host,
                   fcu_solve_info* info, bool on_chip_only) {
  fcu_ctx ctx = m->ctx;
  const bool mixed = precision == FCU_MIXED;
  if (m->bs != 1) fail(FCU_ERR_UNSUPPORTED, "batched PCG takes scalar (CSR) matrices");
  if (!m->has_values) fail(FCU_ERR_BAD_ARG, "matrix has no values");
  if (mixed && !m->val32.p) fail(FCU_ERR_BAD_ARG, "matrix has no FP32 copy");
  if (nb <= 0 || nb > (1 << 30)) fail(FCU_ERR_BAD_ARG, "bad instance count");
  if (offsets_host[0] != 0 || offsets_host[nb] != m->n) fail(FCU_ERR_BAD_ARG, "offsets must span the matrix rows");
  for (i64 i = 0; i < nb; ++i)
    if (offsets_host[i + 1] < offsets_host[i]) fail(FCU_ERR_BAD_ARG, "offsets must not decrease");
  if (max_iter < 0) fail(FCU_ERR_BAD_ARG, "max_iter must be non-negative");

  // (a single system, tried on every small solve, leaves the caller's batch in place)
  BatchWorkspace*& kept = on_chip_only ? m->bws_single : m->bws;
  const bool same = kept && kept->nb == nb && std::equal(kept->off.begin(), kept->off.end(), offsets_host);
  if (!same) {
    delete kept;
    kept = nullptr;
    std::unique_ptr<BatchWorkspace> w(new BatchWorkspace());  // kept once it is complete
    w->nb = (int)nb;
    w->off.assign(offsets_host, offsets_host + nb + 1);
    upload(ctx, w->off_d, w->off.data(), nb + 1);
    DBuf<int> chk;  // [4 per instance: entries, longest row, bandwidth, -][a column outside its block]
    chk.alloc(4 * nb + 1);
    CUDA_CHECK(cudaMemsetAsync(chk.p, 0, chk.bytes(), ctx->stream));
    const unsigned per = (unsigned)std::max<i64>(1, std::min<i64>(64, 4 * ctx->num_sms / nb));
    k_batch_check<<<dim3((unsigned)nb, per), 256, 0, ctx->stream>>>(m->row_ptr, m->col_idx, w->off_d.p, (int)nb,
                                                                   chk.p + 4 * nb, chk.p);
    LAUNCH_CHECK(ctx);
    std::vector<int> hc(4 * nb + 1);
    download(ctx, hc.data(), chk.p, hc.size());
    CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
    if (hc[4 * nb]) fail(FCU_ERR_BAD_ARG, "matrix is not block diagonal over the given offsets");
    w->nnz.resize(nb);
    w->width.resize(nb);
    w->band.resize(nb);
    for (i64 i = 0; i < nb; ++i) {
      w->nnz[i] = hc[4 * i];
      w->width[i] = hc[4 * i + 1];
      w->band[i] = hc[4 * i + 2];
    }
    const i64 n = m->n;
    w->b.alloc(n);
    w->invd.alloc(n);
    w->counter.alloc(1);
    w->results.alloc(5 * nb);
    kept = w.release();
  }
  BatchWorkspace* const w = kept;
  const int k = mixed ? 1 : 0;
  if (!w->planned[k]) {
    // largest first by estimated cost: stored entries x sqrt(rows), the 2D
    // iteration growth
    std::vector<double> cost(nb);
    std::vector<int> ord(nb);
    for (i64 i = 0; i < nb; ++i) {
      const double rows = (double)(offsets_host[i + 1] - offsets_host[i]);
      cost[i] = ((double)w->nnz[i] + rows) * std::sqrt(std::max(rows, 1.0));
      ord[i] = (int)i;
    }
    std::stable_sort(ord.begin(), ord.end(), [&](int p, int q) { return cost[p] > cost[q]; });
    if (mixed) plan_resident<float>(m, w, ord);
    else plan_resident<double>(m, w, ord);
    w->planned[k] = true;
  }
  if (on_chip_only && !w->on_chip[k]) return BATCH_NOT_ON_CHIP;
  const i64 n = m->n;
  cudaEvent_t e0, e1;
  CUDA_CHECK(cudaEventCreate(&e0));
  CUDA_CHECK(cudaEventCreate(&e1));
  CUDA_CHECK(cudaEventRecord(e0, ctx->stream));
  const bool one_launch = w->classes[k].size() == 1 && w->nqueue[k] == 0;  // straight into x_dev
  if (!one_launch) w->x.alloc(n);
  if (w->nqueue[k]) w->r.alloc(n);
  k_batch_invd<<<grid_for(n, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(m->diag_pos, m->val64.p, n, w->invd.p);
  LAUNCH_CHECK(ctx);
  if (mixed) build_rowsum32(m);
  CUDA_CHECK(cudaMemcpyAsync(w->b.p, b_dev, n * sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream));
  if (!w->tuned[k]) {
    if (w->nqueue[k] && mixed) {
      w->z32.alloc(n);
      w->p32.alloc(n);
      w->q32.alloc(n);
      w->ap32.alloc(n);
    } else if (w->nqueue[k]) {
      w->z64.alloc(n);
      w->p64.alloc(n);
      w->q64.alloc(n);
      w->ap64.alloc(n);
    }
    if (w->nqueue[k] == 0) {
      w->cfg[k].vpr = 1;
      w->cfg[k].threads = RNT;
      w->cfg[k].cluster = w->classes[k][0].cluster;
    } else {
      w->cfg[k] = autotune(m, w, mixed, tol);
    }
    w->tuned[k] = true;
  }
  if (one_launch) {
    launch_all(m, w, mixed, tol, max_iter, x_dev);  // nothing to capture
  } else {
    if (!w->graph[k] || w->tol_g[k] != tol || w->iters_g[k] != max_iter) {
      if (w->graph[k]) {
        cudaGraphExecDestroy(w->graph[k]);
        w->graph[k] = nullptr;
      }
      cudaGraph_t g;
      CUDA_CHECK(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
      try {
        launch_all(m, w, mixed, tol, max_iter, w->x.p);
      } catch (...) {
        cudaStreamEndCapture(ctx->stream, &g);
        throw;
      }
      CUDA_CHECK(cudaStreamEndCapture(ctx->stream, &g));
      CUDA_CHECK(cudaGraphInstantiate(&w->graph[k], g, 0));
      cudaGraphDestroy(g);
      w->tol_g[k] = tol;
      w->iters_g[k] = max_iter;
    }
    CUDA_CHECK(cudaGraphLaunch(w->graph[k], ctx->stream));
  }
  ctx->launches += (i64)w->classes[k].size() + (w->nqueue[k] ? 1 : 0);
  if (!one_launch)
    CUDA_CHECK(cudaMemcpyAsync(x_dev, w->x.p, n * sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream));
  CUDA_CHECK(cudaEventRecord(e1, ctx->stream));
  std::vector<i64> results(5 * nb);
  download(ctx, results.data(), w->results.p, results.size());
  CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
  float ms = 0.f;
  CUDA_CHECK(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  const i64* const it = results.data();
  const i64* const up = it + nb;
  const double* const rel = reinterpret_cast<const double*>(it + 2 * nb);
  const double* const res = reinterpret_cast<const double*>(it + 3 * nb);
  const int* const st = reinterpret_cast<const int*>(it + 4 * nb);
  if (iters_host) std::copy(it, it + nb, iters_host);
  if (relres_host) std::copy(rel, rel + nb, relres_host);
  if (status_host) std::copy(st, st + nb, status_host);
  int worst = FCU_OK;
  i64 max_it = 0, sum_it = 0, sum_up = 0;
  double max_rel = 0.0, max_res = 0.0;
  double bytes = 0.0;
  const double w8 = mixed ? 4.0 : 8.0;
  for (i64 i = 0; i < nb; ++i) {
    if (st[i] != FCU_OK && worst == FCU_OK) worst = st[i];
    max_it = std::max(max_it, it[i]);
    sum_it += it[i];
    sum_up += up[i];
    max_rel = std::max(max_rel, rel[i]);
    max_res = std::max(max_res, res[i]);
    // per iteration: values + columns + row pointers, then the vector passes
    // (direction 3w, SpMV p and Ap 2w, update 40 + 3w bytes per row)
    const double rows = (double)(offsets_host[i + 1] - offsets_host[i]);
    bytes += (double)it[i] * (rows * (8.0 * w8 + 44.0));
  }
  if (info) {
    info->iterations = max_it;
    info->outer_updates = sum_up;
    info->residual = max_res;
    info->rel_residual = max_rel;
    info->kernel_ms = ms;
    info->effective_bw_gbps = ms > 0 ? bytes / (ms * 1e-3) / 1e9 : 0.0;
    info->status = worst;
  }
  (void)sum_it;
  return worst;
}

void batch_config(fcu_matrix m, int precision, int* vpr, int* threads, int* cluster) {
  const int k = precision == FCU_MIXED ? 1 : 0;
  const BatchWorkspace* w = m->bws && m->bws->tuned[k] ? m->bws : m->bws_single;
  if (!w || !w->tuned[k]) {
    *vpr = *threads = *cluster = 0;
    return;
  }
  *vpr = w->cfg[k].vpr;
  *threads = w->cfg[k].threads;
  *cluster = w->cfg[k].cluster;
}
