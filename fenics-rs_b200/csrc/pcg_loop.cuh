// The PCG iteration loop in one cooperative launch (included by solver.cu).
//
// One CTA per SM stays resident for the whole solve, the residual
// replacements of the mixed solver included. Warp 0 streams the CTA's tiles of
// the matrix (row ranges; row pointers, columns, values) through a
// shared-memory ring with bulk asynchronous copies; the consumer warps form
// the products and then update the vectors. Per iteration, in two forms:
//
//   plain   product    Ap = A p, shares of p.Ap                  -> sum over CTAs
//           update     r -= alpha Ap, shares of r.z and r.r      -> sum over CTAs
//                      (x += alpha p while the sums travel)
//           direction  p = D^-1 r + beta p                       -> arrival only
//   pairs   product    Ap = A p with p = z + beta p_old formed from (z, p_old)
//                      where it is read, shares of p.Ap          -> sum over CTAs
//           update     r -= alpha Ap, (z, p) stored, shares of r.z and r.r
//                                                                -> sum over CTAs
//
// An iteration is bound by the stream of the matrix (from HBM, or from L2 or
// shared memory when it fits there), the latency of the operand gathers, and
// the grid-wide exchanges of about 2.5 us each. Hence:
//  - The matrix stays in shared memory when every CTA's tiles fit the ring
//    (up to about 30 MB over 148 SMs): nothing is streamed at all.
//  - Otherwise the sweep over the tiles turns round at every iteration, so the
//    tiles read last, still in L2, are read first by the next product.
//  - Small matrices take the pairs, which save an exchange; large ones the
//    plain direction, whose gathers are half as wide (PAIR_BYTES).
//  - All CTAs add the partial sums of an exchange in one fixed order, so they
//    take the same decisions and a solve repeats bit for bit.
//  - What a phase needs and nobody else writes is loaded while the exchange
//    before it is under way.
// Against the kernels it replaced, on B200, per iteration: elasticity FP64
// 56k dofs 16.5 -> 11.2 us, 421k 47.7 -> 36.0, 1.57M 140.6 -> 118; mixed 56k
// 11.6 -> 9.6, 421k 31.9 -> 26.6, 1.57M 87.5 -> 78.4; heat on 1.05M dofs FP64
// 44.2 -> 33.6.
// Every wait is bounded. A CTA whose ring wait gives up says so in its next
// exchange, from which all CTAs end the loop; one whose exchange gives up ends
// it at once, and the others' next exchange gives up in turn. Either way the
// solve's fault flag is set.
#pragma once

constexpr int MAX_RING = 16;            // stages of the loop's ring
constexpr unsigned EX_LIMIT = 1u << 22;  // polls of an exchange (~0.7 us each) before giving up
constexpr unsigned long long EX_FAULT = 1ull << 40;
constexpr int EX_MAX_CTAS = 256;

// Named barrier of the consumer warps (warp 0, the producer, does not join).
template <int W>
__device__ __forceinline__ void consumer_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(32 * W) : "memory");
}

// The grid-wide exchanges of one CTA: every CTA contributes up to two sums and
// gets all CTAs' totals, added in one fixed order. A CTA stores its sums,
// counts itself with a releasing atomic add, polls the count with one thread
// and then reads all sums. Measured with two sums, 148 CTAs of 480 threads, the
// CTA's own reduction included: 2.5 us, and no more than the skew on top when
// the CTAs arrive up to 1.6 us apart. Reading the sums themselves until they
// carry the right epoch (no count, one trip less) took 2.1 us with one sum and
// no skew, but 2.9 us with two and 4.7 us under that skew, against 4.0 us
// here: the polls of 148 lines by 148 CTAs hold up the late stores. Pairs of
// CTAs joined as clusters took 3.9 us, a mailbox per reader 3.7 us.
// Sums alternate between two buffers: a CTA stores for exchange e + 2 where it
// stored for e only after it has seen every CTA's arrival at e + 1, which each
// CTA makes after it has read all of e.
struct ExchangeMem {
  unsigned long long count;  // arrivals; a CTA that met a fault adds EX_FAULT as well
  unsigned long long pad[15];
  double2 sums[2][EX_MAX_CTAS];
};

template <int W>
struct Exchange {
  ExchangeMem* mem;  // zeroed before the launch
  unsigned epoch = 0;
  int G, ctid;

  // The consumer threads' values summed over the CTA and handed over, with
  // everything the CTA wrote before. A fault the CTA has met (*failed) travels
  // along, so that every CTA, this one included, learns of it in this exchange.
  template <int NV>
  __device__ __forceinline__ void post(double (&v)[NV], double (*red)[W], const int* failed) {
    const int lane = ctid & 31, w = ctid >> 5;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const double s = warp_sum(v[j]);
      if (lane == 0) red[j][w] = s;
    }
    consumer_sync<W>();
    if (w == 0) {
      double s[2] = {0.0, 0.0};
#pragma unroll
      for (int j = 0; j < NV; ++j) s[j] = warp_sum(lane < W ? red[j][lane] : 0.0);
      if (lane == 0) {
        mem->sums[(epoch + 1) & 1][blockIdx.x] = make_double2(s[0], s[1]);
        arrive(failed);
      }
    }
    ++epoch;
  }
  __device__ __forceinline__ void post_arrival(const int* failed) {
    consumer_sync<W>();
    if (ctid == 0) arrive(failed);
    ++epoch;
  }
  __device__ __forceinline__ void arrive(const int* failed) {
    const unsigned long long one = *reinterpret_cast<const volatile int*>(failed) ? 1ull + EX_FAULT : 1ull;
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(&mem->count), "l"(one) : "memory");
  }
  // Waits until every CTA has arrived; what they wrote before is then visible.
  // False from the exchange on in which the poll gave up or a CTA reported a
  // fault: *bad is written between two barriers, so all threads of the CTA
  // get the same answer. `limit` bounds the polls.
  __device__ __forceinline__ bool wait_arrivals(int* bad, unsigned limit = EX_LIMIT) {
    if (ctid == 0) {
      const unsigned long long target = (unsigned long long)epoch * (unsigned)G;
      bool ok = false;
      for (unsigned i = 0; i < limit && !ok; ++i) {
        unsigned long long c;
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(&mem->count) : "memory");
        if (c >= EX_FAULT) break;
        ok = c >= target;
      }
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      if (!ok) *bad = 1;
    }
    consumer_sync<W>();
    return *reinterpret_cast<volatile int*>(bad) == 0;
  }
  // The same, and all CTAs' values added: 32 CTAs at a time by a fixed shuffle
  // tree, then group by group; valid in every consumer thread.
  template <int NV>
  __device__ __forceinline__ bool wait(double (&tot)[NV], double (*ws)[EX_MAX_CTAS / 32], int* bad) {
    static_assert(EX_MAX_CTAS <= 32 * W && NV <= 2, "one reading thread per CTA");
    const bool ok = wait_arrivals(bad);
    const int lane = ctid & 31, w = ctid >> 5;
    const int gw = (G + 31) >> 5;  // warps that read
    if (w < gw) {
      double2 s = make_double2(0.0, 0.0);
      if (ctid < G) s = __ldcg(&mem->sums[epoch & 1][ctid]);
      s.x = warp_sum(s.x);
      if (NV > 1) s.y = warp_sum(s.y);
      if (lane == 0) {
        ws[0][w] = s.x;
        if (NV > 1) ws[1][w] = s.y;
      }
    }
    consumer_sync<W>();
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      double s = 0.0;
      for (int q = 0; q < gw; ++q) s += ws[j][q];
      tot[j] = s;
    }
    return ok;
  }
};

template <class T>
struct Pair;
template <>
struct Pair<float> {
  using type = float2;
};
template <>
struct Pair<double> {
  using type = double2;
};

template <class T>
struct LoopArgs {
  const int* rp;
  const int* ci;
  const T* val;
  const int* tb;  // tile t is rows [tb[t], tb[t + 1]), or (null) [t tr, t tr + tr)
  i64 nrows, ntiles, n;
  int tr;
  int nstage;
  int resident;  // every CTA's tiles fit the ring: loaded once, tile k in stage k
  unsigned off_c, off_v, stage;  // byte offsets of columns and values in a stage; its size
  const double* val64;  // the FP64 values and the right-hand side (residual replacement)
  const double* b;
  double* x;
  double* r;
  const double* invd;
  T* p;
  typename Pair<T>::type* zp;
  T* ap;
  CgState* st;
  ExchangeMem* ex;
};

// Two (z, p) pairs side by side: 16 or 32 bytes.
struct alignas(32) quad64 {
  double x, y, z, w;
};
template <class T>
struct Quad;
template <>
struct Quad<float> {
  using type = float4;
};
template <>
struct Quad<double> {
  using type = quad64;
};
__device__ __forceinline__ float4 ldcg4(const float4* p) { return __ldcg(p); }
__device__ __forceinline__ void stg4(float4* p, const float4& v) { *p = v; }
__device__ __forceinline__ quad64 ldcg4(const quad64* p) {
  const double2* q = reinterpret_cast<const double2*>(p);
  const double2 a = __ldcg(q), b = __ldcg(q + 1);
  return quad64{a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ void stg4(quad64* p, const quad64& v) {
  double2* q = reinterpret_cast<double2*>(p);
  q[0] = make_double2(v.x, v.y);
  q[1] = make_double2(v.z, v.w);
}

__device__ __forceinline__ float dir_fma(float beta, float pold, float z) { return __fmaf_rn(beta, pold, z); }
__device__ __forceinline__ double dir_fma(double beta, double pold, double z) { return __fma_rn(beta, pold, z); }

// Sum of three values over the LPR lanes of a row (LPR = 8 or 16): the first
// two steps halve the number of values a lane carries (five shuffles instead
// of twelve for 16 lanes). Lane 0 of the row ends with a0, lane 2 with a1 and
// lane 1 with a2.
template <int LPR, class T>
__device__ __forceinline__ T row_sum3(T a0, T a1, T a2, int sub) {
  const bool odd = sub & 1, hi = sub & 2;
  const T r0 = __shfl_xor_sync(FULL, odd ? a0 : a2, 1);
  const T r1 = __shfl_xor_sync(FULL, odd ? a1 : T(0), 1);
  const T k0 = (odd ? a2 : a0) + r0;
  const T k1 = (odd ? T(0) : a1) + r1;
  T s = (hi ? k1 : k0) + __shfl_xor_sync(FULL, hi ? k0 : k1, 2);
#pragma unroll
  for (int o = 4; o < LPR; o <<= 1) s += __shfl_xor_sync(FULL, s, o);
  return s;
}

// What a consumer lane holds of one row of a tile: its range of the row's
// entries and the operands of the first E of them.
template <int BS, int LPR, int E, bool DIFF, class T>
struct RowFetch {
  int kb, kb1;
  int row;        // -1: no such row
  unsigned diag;  // bit e: fetched entry e is the diagonal (DIFF)
  T y[E * BS];
  T own[BS == 3 && DIFF ? 3 : 1];

  template <class OP>
  __device__ __forceinline__ void fetch(const unsigned char* base, unsigned off_c, const OP& op, int rit, int sub) {
    const TileHeader* h = reinterpret_cast<const TileHeader*>(base);
    const int* rps = reinterpret_cast<const int*>(base + align128(sizeof(TileHeader))) + h->rp_off;
    const int* cis = reinterpret_cast<const int*>(base + off_c + h->col_off);
    kb = kb1 = 0;
    row = -1;
    diag = 0;
    if (rit >= h->rows) return;
    row = h->r0 + rit;
    const int b0 = h->b0;
    kb = rps[rit] - b0 + sub;
    kb1 = rps[rit + 1] - b0;
    int c[E];
#pragma unroll
    for (int e = 0; e < E; ++e) c[e] = kb + e * LPR < kb1 ? cis[kb + e * LPR] : -1;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      if (c[e] >= 0) {
#pragma unroll
        for (int d = 0; d < BS; ++d) y[e * BS + d] = op(BS * (i64)c[e] + d);
      }
      if (DIFF && c[e] == row) diag |= 1u << e;
    }
    const i64 i = BS * (i64)row;
    if constexpr (BS == 3 && DIFF) {
      own[0] = op(i);
      own[1] = op(i + 1);
      own[2] = op(i + 2);
    } else if constexpr (BS == 3) {
      if (sub < 3) own[0] = op(i + (sub == 0 ? 0 : 3 - sub));
    } else {
      own[0] = op(i);
    }
  }

  // The row's product from the tile's values: the lane's sums. The operands
  // of entries beyond the first E are fetched E at a time.
  template <class OP>
  __device__ __forceinline__ void sum(const unsigned char* base, unsigned off_c, unsigned off_v, const OP& op,
                                      T (&acc)[BS]) const {
    const TileHeader* h = reinterpret_cast<const TileHeader*>(base);
    const T* vls = reinterpret_cast<const T*>(base + off_v + h->val_off);
#pragma unroll
    for (int d = 0; d < BS; ++d) acc[d] = T(0);
    auto add = [&](int q, const T* g, bool dg) {
      const T* v = vls + BS * BS * q;
      T t[BS];
#pragma unroll
      for (int d = 0; d < BS; ++d) {
        if constexpr (DIFF) t[d] = dg ? own[BS == 3 ? d : 0] : g[d] - own[BS == 3 ? d : 0];
        else t[d] = g[d];
      }
#pragma unroll
      for (int d = 0; d < BS; ++d) {
        if constexpr (BS == 3) acc[d] += v[3 * d] * t[0] + v[3 * d + 1] * t[1] + v[3 * d + 2] * t[2];
        else acc[d] += v[0] * t[0];
      }
    };
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (kb + e * LPR < kb1) add(kb + e * LPR, y + e * BS, DIFF && ((diag >> e) & 1u));
    const int* cis = reinterpret_cast<const int*>(base + off_c + h->col_off);
#pragma unroll 1
    for (int q = kb + E * LPR; q < kb1; q += E * LPR) {
      T g[E * BS];
      int c[E];
#pragma unroll
      for (int e = 0; e < E; ++e) c[e] = q + e * LPR < kb1 ? cis[q + e * LPR] : -1;
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (c[e] >= 0) {
#pragma unroll
          for (int d = 0; d < BS; ++d) g[e * BS + d] = op(BS * (i64)c[e] + d);
        }
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (c[e] >= 0) add(q + e * LPR, g + e * BS, c[e] == row);
    }
  }

  // The sums over the row's lanes; the lanes that end with a result store it
  // in Ap and add p.Ap.
  __device__ __forceinline__ void emit(const T (&acc)[BS], T* ap, int sub, double& dot) const {
    if constexpr (BS == 1) {
      T s = acc[0];
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
      if (row >= 0 && sub == 0) {
        ap[row] = s;
        dot += (double)own[0] * (double)s;
      }
    } else {
      const T s = row_sum3<LPR>(acc[0], acc[1], acc[2], sub);
      if (row >= 0 && sub < 3) {
        const int comp = sub == 0 ? 0 : 3 - sub;
        T o;
        if constexpr (DIFF) o = comp == 0 ? own[0] : comp == 1 ? own[1] : own[2];
        else o = own[0];
        ap[3 * (i64)row + comp] = s;
        dot += (double)o * (double)s;
      }
    }
  }
};

// Operand of the product at a vector element: the direction itself, or (PAIR)
// formed from the pair (z, p_old) where it is read. Written by other CTAs
// before the last exchange: ordinary coherent loads, never the read-only path.
template <class T>
struct Plain {
  const T* p;
  __device__ __forceinline__ T operator()(i64 i) const { return p[i]; }
};
template <class T>
struct FromPair {
  const typename Pair<T>::type* zp;
  T beta;
  __device__ __forceinline__ T operator()(i64 i) const {
    const typename Pair<T>::type v = zp[i];
    return dir_fma(beta, v.y, v.x);
  }
};

// Shape of the loop by block size and value type: consumer warps W, entries a
// lane fetches in one go (E), rows a lane group takes of a tile (R).
//  - FP64 needs the registers of 16 warps (128 a thread): with 24 or 32 warps
//    the product spills, and a spilled operand is waited for at once. Its plain
//    scalar shapes spill 36 bytes even so, the others at most 8.
//  - FP32 plain shapes run 24 warps, which hide more of the gather latency than
//    the 72 bytes they spill (80 registers) cost: P2 system of 2.15M dofs 151 us
//    per iteration, with 20 warps 159, with 16 174. Pairs keep 16.
//  - 3x3 blocks: one FP64 block per lane of a 16-lane row keeps the 72-byte
//    blocks free of bank conflicts, two rows at once hide the latency; FP32
//    takes two blocks per lane of an 8-lane row.
//  - Fetching the next tile's operands before the current tile is summed was
//    slower in every shape: the consumer then holds a stage while it waits
//    for the next one (421k-dof elasticity, FP64: 48.7 against 37.5 us).
template <int BS, bool PAIR, class T>
struct LoopShape {
  static constexpr int W = sizeof(T) == 8 || PAIR ? 15 : 23;
  static constexpr int E = BS == 1 ? 8 : sizeof(T) == 4 ? 2 : 1;
  static constexpr int R = BS == 3 && sizeof(T) == 8 ? 2 : 1;
  static constexpr int LPR3 = sizeof(T) == 8 ? 16 : 8;  // lanes per row of 3x3 blocks
};

// What the consumer threads share.
template <class T, int W>
struct LoopShared {
  double* x;
  double* r;
  const double* invd;
  T* p;
  typename Pair<T>::type* zp;
  const T* ap;
  ExchangeMem* mem;
  int n, step, G;        // vector elements; stride between a thread's elements; CTAs
  int tp, own;           // pairs of vector elements per tile; in the CTA's tiles
  unsigned epoch;        // exchanges so far
  double rz, rr, beta, bnorm, tol, maxr, delta;
  i64 iter, max_iter, updates;
  int gpus, timing;
  int done, pause, status;
  int bad;               // written by the polls of an exchange
  int failed;            // a ring wait of this CTA gave up
  double red[2][W];
  double ws[2][EX_MAX_CTAS / 32];
};

// On entry: p = z + beta p for the thread's elements; with pairs only
// z = D^-1 r (and p = 0 at the start of a solve, else as the last launch left it).
template <bool PAIR, class T, int W>
__device__ __forceinline__ void enter(const LoopShared<T, W>& S, int first) {
  const T bt = (T)S.beta;
  for (int i = first; i < S.n; i += S.step) {
    const T z = (T)(S.r[i] * S.invd[i]);
    if (!PAIR) {
      S.p[i] = dir_fma(bt, S.p[i], z);
    } else {
      if (S.iter == 0) S.zp[i].y = T(0);
      S.zp[i].x = z;
    }
  }
}

struct Decision {
  int done, pause, status;
  __device__ __forceinline__ bool end() const { return done || pause; }
};

// The decisions of decide_after_update(_mixed) on r.z and r.r, the same in
// every thread of every CTA.
template <bool MIXED, class T, int W>
__device__ __forceinline__ Decision decide(const LoopShared<T, W>& S, const double (&v)[2], bool ok, i64 iter, double rz,
                                          double* beta) {
  const double res = sqrt(v[1]);
  const double rel = S.bnorm > 0.0 ? res / S.bnorm : res;
  Decision d{0, 0, 0};
  if (!ok) {
    d.done = 1;
    d.status = FCU_ERR_CUDA;
  } else if (MIXED && (rel < S.tol || res < S.delta * S.maxr)) {
    d.pause = 1;  // a residual replacement comes first
  } else if (!MIXED && rel < S.tol) {
    d.done = 1;
    d.status = FCU_OK;
  } else if (iter >= S.max_iter) {
    d.done = 1;
    d.status = S.gpus ? FCU_OK : FCU_ERR_NO_CONVERGENCE;
  }
  *beta = v[0] / (S.gpus ? fmax(rz, 1e-30) : rz);
  return d;
}
// The state after the iteration, written by one thread: the others read it
// after the barrier here, and read the old one last before their post of
// r.z and r.r. True when the loop goes on.
template <class T, int W>
__device__ __forceinline__ bool record(LoopShared<T, W>& S, const Decision& d, const double (&v)[2], bool ok, i64 iter,
                                       double beta, unsigned epoch) {
  if (threadIdx.x == 32) {
    if (ok) {
      S.rr = v[1];
      S.iter = iter;
    }
    if (!d.end()) {
      S.beta = beta;
      S.rz = v[0];
    }
    S.epoch = epoch;
    S.done = d.done;
    S.pause = d.pause;
    S.status = d.status;
  }
  consumer_sync<W>();
  return !d.end();
}

// The vector half of an iteration, from this thread's share of p.Ap to the new
// direction: both sums, alpha, beta and the decisions. Returns false when the
// loop ends (S says how). Inlined: the elements of r, D^-1, p and z that a
// thread keeps across the exchanges (K pairs) are dead during the product.
template <bool MIXED, class T, int W>
__device__ __forceinline__ bool vector_phase(LoopShared<T, W>& S, double dot) {
  constexpr int K = 1;  // pairs of vector elements a thread keeps in registers
  using T2 = typename Pair<T>::type;
  const int ctid = (int)threadIdx.x - 32;
  const int np = (S.n + 1) >> 1, step = S.step;  // pairs (the arrays are padded past their end)
  const bool odd = S.n & 1;
  const int i0 = (int)blockIdx.x * 32 * W + ctid;
  double2* const r2 = reinterpret_cast<double2*>(S.r);
  const double2* const d2 = reinterpret_cast<const double2*>(S.invd);
  double2* const x2 = reinterpret_cast<double2*>(S.x);
  T2* const p2 = reinterpret_cast<T2*>(S.p);
  const T2* const ap2 = reinterpret_cast<const T2*>(S.ap);
  Exchange<W> ex;
  ex.mem = S.mem;
  ex.G = S.G;
  ex.ctid = ctid;
  ex.epoch = S.epoch;
  double v1[1] = {dot};
  ex.post(v1, S.red, &S.failed);
  // own elements of r, D^-1 and p while the sum is under way
  double2 rv[K], dv[K];
  T2 pc[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = i0 + k * step;
    if (i < np) {
      rv[k] = __ldcg(r2 + i);
      dv[k] = __ldcg(d2 + i);
      pc[k] = __ldcg(p2 + i);
    }
  }
  bool ok = ex.wait(v1, S.ws, &S.bad);
  // cg.rs:102-107: |p.Ap| < 1e-30 is a breakdown (Err); the GPU solvers
  // (gpu.rs:1326-1329, 1034-1037) stop with Ok when p.Ap <= 1e-30, the
  // iteration counting as done
  const double pap = v1[0];
  if (!ok || (!S.timing && (S.gpus ? !(pap > 1e-30) : fabs(pap) < 1e-30))) {
    if (ctid == 0) {
      S.done = 1;
      S.status = !ok ? FCU_ERR_CUDA : S.gpus ? FCU_OK : FCU_ERR_BREAKDOWN;
      if (ok) S.iter += 1;
    }
    return false;
  }
  const double rz = S.rz;
  const i64 iter = S.iter + 1;
  const double alpha = rz / pap;
  // r -= alpha Ap ; z = D^-1 r ; shares of r.z and r.r
  double v2[2] = {0.0, 0.0};
  auto residual = [&](int i, double2 r, double2 d, T2 ap) {
    r.x -= alpha * (double)ap.x;
    r.y -= alpha * (double)ap.y;
    const double2 z = make_double2(r.x * d.x, r.y * d.y);
    r2[i] = r;
    v2[0] += r.x * z.x;
    v2[1] += r.x * r.x;
    if (!(odd && i == np - 1)) {
      v2[0] += r.y * z.y;
      v2[1] += r.y * r.y;
    }
    return z;
  };
  auto direction = [&](int i, T bt, T2 p, T zx, T zy) {
    p.x = dir_fma(bt, p.x, zx);
    p.y = dir_fma(bt, p.y, zy);
    p2[i] = p;
  };
  T2 zc[K];
  {
    T2 av[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = i0 + k * step;
      if (i < np) av[k] = __ldcg(ap2 + i);
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = i0 + k * step;
      if (i < np) {
        const double2 z = residual(i, rv[k], dv[k], av[k]);
        zc[k].x = (T)z.x;
        zc[k].y = (T)z.y;
      }
    }
    // the elements beyond, two pairs at a time with their loads first
#pragma unroll 1
    for (int i = i0 + K * step; i < np; i += 2 * step) {
      const int j = i + step;
      const double2 ra = __ldcg(r2 + i), da = __ldcg(d2 + i);
      const T2 aa = __ldcg(ap2 + i);
      double2 rb, db;
      T2 ab;
      if (j < np) {
        rb = __ldcg(r2 + j);
        db = __ldcg(d2 + j);
        ab = __ldcg(ap2 + j);
      }
      residual(i, ra, da, aa);
      if (j < np) residual(j, rb, db, ab);
    }
  }
  ex.post(v2, S.red, &S.failed);
  // x += alpha p while the sums are under way
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = i0 + k * step;
    if (i < np) {
      double2 x = __ldcg(x2 + i);
      x.x += alpha * (double)pc[k].x;
      x.y += alpha * (double)pc[k].y;
      x2[i] = x;
    }
  }
#pragma unroll 2
  for (int i = i0 + K * step; i < np; i += step) {
    double2 x = __ldcg(x2 + i);
    const T2 p = __ldcg(p2 + i);
    x.x += alpha * (double)p.x;
    x.y += alpha * (double)p.y;
    x2[i] = x;
  }
  ok = ex.wait(v2, S.ws, &S.bad);
  double beta;
  const Decision d = decide<MIXED>(S, v2, ok, iter, rz, &beta);
  if (!d.end()) {
    // p = z + beta p
    const T bt = (T)beta;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = i0 + k * step;
      if (i < np) direction(i, bt, pc[k], zc[k].x, zc[k].y);
    }
#pragma unroll 1
    for (int i = i0 + K * step; i < np; i += 2 * step) {
      const int j = i + step;
      const double2 ra = __ldcg(r2 + i), da = __ldcg(d2 + i);
      const T2 pa = __ldcg(p2 + i);
      double2 rb, db;
      T2 pb;
      if (j < np) {
        rb = __ldcg(r2 + j);
        db = __ldcg(d2 + j);
        pb = __ldcg(p2 + j);
      }
      direction(i, bt, pa, (T)(ra.x * da.x), (T)(ra.y * da.y));
      if (j < np) direction(j, bt, pb, (T)(rb.x * db.x), (T)(rb.y * db.y));
    }
    ex.post_arrival(&S.failed);
    ex.wait_arrivals(&S.bad);  // a fault shows in the next sum
  }
  return record(S, d, v2, ok, iter, beta, ex.epoch);
}

// The same with the direction left to the product: z and p are kept as pairs
// and the CTA updates the elements of its own tiles' rows, so that Ap never
// leaves the CTA. Two exchanges per iteration instead of three; the price is
// the product's gathers of pairs.
template <bool MIXED, class T, int W>
__device__ __forceinline__ bool vector_phase_pair(LoopShared<T, W>& S, double dot) {
  using T2 = typename Pair<T>::type;
  using T4 = typename Quad<T>::type;
  constexpr int NCT = 32 * W;
  const int ctid = (int)threadIdx.x - 32;
  const int np = (S.n + 1) >> 1, own = S.own;
  const bool odd = S.n & 1;
  double2* const r2 = reinterpret_cast<double2*>(S.r);
  const double2* const d2 = reinterpret_cast<const double2*>(S.invd);
  double2* const x2 = reinterpret_cast<double2*>(S.x);
  T4* const zp4 = reinterpret_cast<T4*>(S.zp);
  const T2* const ap2 = reinterpret_cast<const T2*>(S.ap);
  // pair e of the CTA's tiles as a pair of the whole vectors (>= np: none)
  auto at = [&](int e) {
    const int t = e / S.tp;
    return ((int)blockIdx.x + t * S.G) * S.tp + (e - t * S.tp);
  };
  Exchange<W> ex;
  ex.mem = S.mem;
  ex.G = S.G;
  ex.ctid = ctid;
  ex.epoch = S.epoch;
  double v1[1] = {dot};
  ex.post(v1, S.red, &S.failed);
  // the first own pair while the sum is under way
  const T bt = (T)S.beta;
  int i0 = ctid < own ? at(ctid) : np;
  double2 r0, d0, x0;
  T4 zp0;
  T2 ap0;
  if (i0 < np) {
    r0 = __ldcg(r2 + i0);
    d0 = __ldcg(d2 + i0);
    zp0 = ldcg4(zp4 + i0);
    ap0 = __ldcg(ap2 + i0);
    x0 = __ldcg(x2 + i0);
  }
  bool ok = ex.wait(v1, S.ws, &S.bad);
  const double pap = v1[0];
  if (!ok || (!S.timing && (S.gpus ? !(pap > 1e-30) : fabs(pap) < 1e-30))) {  // as in vector_phase
    if (ctid == 0) {
      S.done = 1;
      S.status = !ok ? FCU_ERR_CUDA : S.gpus ? FCU_OK : FCU_ERR_BREAKDOWN;
      if (ok) S.iter += 1;
    }
    return false;
  }
  const double rz = S.rz;
  const i64 iter = S.iter + 1;
  const double alpha = rz / pap;
  // r -= alpha Ap ; z = D^-1 r ; (z, p) ; shares of r.z and r.r
  double v2[2] = {0.0, 0.0};
  auto update = [&](int i, double2& r, const double2& d, T4& zp, const T2& ap) {
    zp.y = dir_fma(bt, zp.y, zp.x);
    zp.w = dir_fma(bt, zp.w, zp.z);
    r.x -= alpha * (double)ap.x;
    r.y -= alpha * (double)ap.y;
    const double2 z = make_double2(r.x * d.x, r.y * d.y);
    zp.x = (T)z.x;
    zp.z = (T)z.y;
    stg4(zp4 + i, zp);
    v2[0] += r.x * z.x;
    v2[1] += r.x * r.x;
    if (!(odd && i == np - 1)) {
      v2[0] += r.y * z.y;
      v2[1] += r.y * r.y;
    }
  };
  auto advance = [&](int i, const double2& r, double2& x, const T4& zp) {
    x.x += alpha * (double)zp.y;
    x.y += alpha * (double)zp.w;
    r2[i] = r;
    x2[i] = x;
  };
  if (i0 < np) update(i0, r0, d0, zp0, ap0);
#pragma unroll 1
  for (int e = ctid + NCT; e < own; e += NCT) {
    const int i = at(e);
    if (i >= np) break;
    double2 r = __ldcg(r2 + i), x = __ldcg(x2 + i);
    const double2 d = __ldcg(d2 + i);
    T4 zp = ldcg4(zp4 + i);
    const T2 ap = __ldcg(ap2 + i);
    update(i, r, d, zp, ap);
    advance(i, r, x, zp);
  }
  ex.post(v2, S.red, &S.failed);  // the pairs go with it
  if (i0 < np) advance(i0, r0, x0, zp0);            // read by this thread alone
  ok = ex.wait(v2, S.ws, &S.bad);
  double beta;
  const Decision d = decide<MIXED>(S, v2, ok, iter, rz, &beta);
  return record(S, d, v2, ok, iter, beta, ex.epoch);
}

// The residual replacement of the mixed solver, as k_mx_replace: r = b - A64 x
// with the FP64 matrix, the decisions on it, and the next direction from the
// new z. Runs a few times per solve; a call of its own keeps its registers
// apart from the iteration's. Returns false when the solve ends.
template <int BS, bool PAIR, class T, int W>
__device__ __noinline__ bool replace_residual(LoopShared<T, W>& S, const int* __restrict__ rp,
                                              const int* __restrict__ ci, const double* __restrict__ val64,
                                              const double* __restrict__ b, i64 nrows) {
  struct Emit {
    const double* b;
    const double* invd;
    double* r;
    double v[2];
    __device__ __forceinline__ void operator()(i64 node, int a, double s) {
      const i64 i = node * BS + a;
      const double ri = b[i] - s;
      r[i] = ri;
      v[0] += ri * (ri * invd[i]);
      v[1] += ri * ri;
    }
  };
  const int ctid = (int)threadIdx.x - 32;
  Exchange<W> ex;
  ex.mem = S.mem;
  ex.G = S.G;
  ex.ctid = ctid;
  ex.epoch = S.epoch;
  ex.post_arrival(&S.failed);  // x of all CTAs
  ex.wait_arrivals(&S.bad);
  Emit em{b, S.invd, S.r, {0.0, 0.0}};
  warp_rows<BS, 8, false, double>(rp, ci, val64, nrows, (i64)blockIdx.x * W + (ctid >> 5), (i64)S.G * W,
                                  XPlain<double>{S.x}, em);
  ex.post(em.v, S.red, &S.failed);
  const bool ok = ex.wait(em.v, S.ws, &S.bad);
  const double res = sqrt(em.v[1]);
  const double rel = S.bnorm > 0.0 ? res / S.bnorm : res;
  const bool conv = rel < S.tol, limit = S.iter >= S.max_iter;
  const bool end = !ok || conv || limit;
  consumer_sync<W>();  // everybody has read the state
  if (ctid == 0) {
    S.pause = 0;
    S.epoch = ex.epoch + (end ? 0 : 1);
    if (ok) {
      S.updates += 1;
      S.rr = em.v[1];
    }
    if (end) {
      S.done = 1;
      S.status = !ok ? FCU_ERR_CUDA : conv ? FCU_OK : FCU_ERR_NO_CONVERGENCE;
    } else {
      S.maxr = res;
      S.beta = em.v[0] / S.rz;
      S.rz = em.v[0];
    }
  }
  consumer_sync<W>();
  if (end) return false;
  enter<PAIR>(S, (int)blockIdx.x * 32 * W + ctid);
  ex.post_arrival(&S.failed);
  ex.wait_arrivals(&S.bad);  // a fault shows in the next sum
  return true;
}

template <int BS, int LPR, bool DIFF, bool PAIR, class T>
__global__ void __launch_bounds__(32 * (LoopShape<BS, PAIR, T>::W + 1), 1)
    k_pcg_loop(const __grid_constant__ LoopArgs<T> a) {
  using Shape = LoopShape<BS, PAIR, T>;
  constexpr int W = Shape::W;
  constexpr int NCT = 32 * W;  // consumer threads
  constexpr int VPB = BS * BS;
  extern __shared__ __align__(128) unsigned char tile_smem[];
  __shared__ unsigned long long full[MAX_RING], empty[MAX_RING];
  __shared__ LoopShared<T, W> S;
  __shared__ volatile int ended_s;   // consumers -> producer: no more tiles are needed
  __shared__ volatile int pfault_s;  // producer -> consumers: a ring wait gave up
  CgState* const st = a.st;
  const i64 G = gridDim.x;
  const int mytiles = blockIdx.x < a.ntiles ? (int)((a.ntiles - blockIdx.x + G - 1) / G) : 0;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool run0 = !(st->done || st->pause);
  if (tid == 0) {
    for (int s = 0; s < a.nstage; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], W);
    }
    fence_mbar_init();
    S.x = a.x;
    S.r = a.r;
    S.invd = a.invd;
    S.p = a.p;
    S.zp = a.zp;
    S.tp = a.tr * BS / 2;
    S.own = mytiles * (a.tr * BS / 2);
    S.ap = a.ap;
    S.mem = a.ex;
    S.n = (int)a.n;  // the plan admits no larger n
    S.step = (int)G * NCT;
    S.G = (int)G;
    S.epoch = 1;
    S.rz = st->rz;
    S.rr = st->rr;
    S.beta = st->beta;
    S.bnorm = st->bnorm;
    S.tol = st->tol;
    S.maxr = st->maxr;
    S.delta = st->delta;
    S.iter = st->iter;
    S.max_iter = st->max_iter;
    S.updates = st->updates;
    S.gpus = st->gpu_semantics;
    S.timing = st->timing;
    S.done = S.pause = S.status = S.bad = S.failed = 0;
    ended_s = 0;
    pfault_s = 0;
  }
  __syncthreads();
  if (!run0) return;

  if (warp == 0) {
    // producer: the CTA's tiles forwards, backwards, forwards, ...
    if (mytiles == 0) return;
    int pb0 = 0, pb1 = 0, pr0 = 0, pr1 = 0, grp = -1;  // lane j: bounds of tile 32 grp + j
    int q = 0;
    bool back = false;
    int s = 0;        // ring stage
    unsigned ph = 0;  // phase parity of the stage's current use
    int issued = 0;   // copies issued, counted up to nstage
    for (;;) {
      const int k = back ? mytiles - 1 - q : q;
      if ((k >> 5) != grp) {
        grp = k >> 5;
        const i64 t = blockIdx.x + (i64)(32 * grp + lane) * G;
        if (t < a.ntiles) {
          pr0 = a.tb ? a.tb[t] : (int)(t * a.tr);
          pr1 = a.tb ? a.tb[t + 1] : (int)min(t * a.tr + a.tr, a.nrows);
          pb0 = a.rp[pr0];
          pb1 = a.rp[pr1];
        }
      }
      int state = 1;  // 1: stage free, 2: loop ended, 3: wait gave up
      if (lane == 0) {
        if (issued >= a.nstage) {
          state = 3;
          for (unsigned i = 0; i < WAIT_LIMIT; ++i) {
            if (mbar_try_wait(&empty[s], ph ^ 1u)) {
              state = 1;
              break;
            }
            if (ended_s) {
              state = 2;
              break;
            }
          }
        } else if (ended_s) {
          state = 2;
        }
      }
      state = __shfl_sync(FULL, state, 0);
      if (state != 1) {
        if (state == 3 && lane == 0) {
          atomicExch(&st->fault, 1);
          pfault_s = 1;
        }
        break;
      }
      const int b0 = __shfl_sync(FULL, pb0, k & 31), b1 = __shfl_sync(FULL, pb1, k & 31);
      const int r0 = __shfl_sync(FULL, pr0, k & 31), r1 = __shfl_sync(FULL, pr1, k & 31);
      if (lane == 0) {
        unsigned char* base = tile_smem + (size_t)s * a.stage;
        TileHeader* h = reinterpret_cast<TileHeader*>(base);
        const int rp_off = r0 & 3;  // rp + r0 - rp_off is 16-byte aligned
        const unsigned rp_bytes = (unsigned)(((r1 - r0 + 1 + rp_off) * 4 + 15) & ~15);
        const uintptr_t c_lo = reinterpret_cast<uintptr_t>(a.ci + b0) & ~(uintptr_t)15;
        const uintptr_t c_hi = (reinterpret_cast<uintptr_t>(a.ci + b1) + 15) & ~(uintptr_t)15;
        const uintptr_t v_lo = reinterpret_cast<uintptr_t>(a.val + VPB * (i64)b0) & ~(uintptr_t)15;
        const uintptr_t v_hi = (reinterpret_cast<uintptr_t>(a.val + VPB * (i64)b1) + 15) & ~(uintptr_t)15;
        h->b0 = b0;
        h->rows = r1 - r0;
        h->r0 = r0;
        h->rp_off = rp_off;
        h->col_off = (int)(reinterpret_cast<uintptr_t>(a.ci + b0) - c_lo);
        h->val_off = (int)(reinterpret_cast<uintptr_t>(a.val + VPB * (i64)b0) - v_lo);
        const unsigned cb = (unsigned)(c_hi - c_lo), vb = (unsigned)(v_hi - v_lo);
        fence_proxy_async();
        mbar_arrive_expect_tx(&full[s], rp_bytes + cb + vb);
        bulk_load(base + align128(sizeof(TileHeader)), a.rp + (r0 - rp_off), rp_bytes, &full[s]);
        if (cb) bulk_load(base + a.off_c, reinterpret_cast<const void*>(c_lo), cb, &full[s]);
        if (vb) bulk_load(base + a.off_v, reinterpret_cast<const void*>(v_lo), vb, &full[s]);
      }
      if (issued < a.nstage) ++issued;
      if (++s == a.nstage) {
        s = 0;
        ph ^= 1u;
      }
      if (++q == mytiles) {
        if (a.resident) break;
        q = 0;
        back = !back;
      }
    }
    // copies still in flight (at most one per stage) land before the CTA exits
    if (lane == 0)
      for (int i = 1; i <= issued; ++i) {
        int s2 = s - i;
        unsigned p2 = ph;
        if (s2 < 0) {
          s2 += a.nstage;
          p2 ^= 1u;
        }
        mbar_wait(&full[s2], p2);
      }
    return;
  }

  // consumer warps
  constexpr int R = Shape::R;
  constexpr int RPP = NCT / LPR;  // rows of a tile the lane groups take at once
  using Row = RowFetch<BS, LPR, Shape::E, DIFF, T>;
  using Op = typename std::conditional<PAIR, FromPair<T>, Plain<T>>::type;
  const int ctid = tid - 32;
  const int sub = lane % LPR;
  const int rit = ctid / LPR;  // the lane group's row in every tile
  int cs = 0;                  // ring stage of the next tile
  unsigned cph = 0;            // its phase parity
  enter<PAIR>(S, (int)blockIdx.x * NCT + ctid);
  {
    Exchange<W> ex;
    ex.mem = a.ex;
    ex.G = (int)G;
    ex.ctid = ctid;
    ex.post_arrival(&S.failed);
    ex.wait_arrivals(&S.bad);
  }
  auto wait_full = [&](int s, unsigned ph) {
    bool got = false;
    for (unsigned i = 0; i < WAIT_LIMIT && !got && !pfault_s; ++i) got = mbar_try_wait(&full[s], ph);
    return __all_sync(FULL, got) != 0;  // one answer per warp: its lanes shuffle together
  };
  for (;;) {
    // Ap = A p and this thread's share of p.Ap
    double dot = 0.0;
    bool ok = true;
    if (a.resident) cs = 0, cph = 0;
    Op op;
    if constexpr (PAIR) {
      op.zp = a.zp;
      op.beta = (T)S.beta;
    } else {
      op.p = a.p;
    }
    for (int k = 0; k < mytiles; ++k) {
      ok = wait_full(cs, cph);
      if (!ok) break;
      const unsigned char* base = tile_smem + (size_t)cs * a.stage;
      Row rows[R];
#pragma unroll
      for (int r = 0; r < R; ++r) rows[r].fetch(base, a.off_c, op, rit + r * RPP, sub);
      T acc[R][BS];
#pragma unroll
      for (int r = 0; r < R; ++r) rows[r].sum(base, a.off_c, a.off_v, op, acc[r]);
      if (!a.resident) {  // the stage is free once its values are read
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&empty[cs])) : "memory");
      }
#pragma unroll
      for (int r = 0; r < R; ++r) rows[r].emit(acc[r], a.ap, sub, dot);
      if (++cs == a.nstage) {
        cs = 0;
        if (!a.resident) cph ^= 1u;
      }
    }
    if (!ok) S.failed = 1;
    if (PAIR ? vector_phase_pair<DIFF>(S, dot) : vector_phase<DIFF>(S, dot)) continue;
    if (!(DIFF && S.pause)) break;
    if (!replace_residual<BS, PAIR>(S, a.rp, a.ci, a.val64, a.b, a.nrows)) break;
  }
  consumer_sync<W>();
  if (ctid == 0) {
    ended_s = 1;
    if (S.status == FCU_ERR_CUDA) atomicExch(&st->fault, 1);
    if (blockIdx.x == 0) {
      st->rz = S.rz;
      st->beta = S.beta;
      st->rr = S.rr;
      st->iter = S.iter;
      st->done = S.done;
      st->status = S.status;
      st->updates = S.updates;
      st->maxr = S.maxr;
    }
  }
}
