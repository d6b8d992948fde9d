// Krylov drivers whose vectors stay on chip: Cg, BiCgStab and Gmres for
// operators whose rows all lie in the thread bin of the SELL layout, in row
// order (stencils, bands), and are few enough.
//
// One CTA per SM owns a contiguous run of slices (128 rows each) for the whole
// solve.  The vectors of its rows live in its shared memory, and so does its
// part of the matrix where that fits too.  Only what other CTAs gather goes
// through global memory: the operand of the product, whose entries outside the
// CTA's rows are read from L2, all of a row's at once.  A phase that used to
// be a pass over L2 is a few hundred cycles of shared memory, so that the grid
// barriers and one L2 trip per product are what is left.
//
// Layout in shared memory: row 4q + j of the CTA at plane j, index q.  A lane
// of the quad-row SELL product owns rows 4q..4q+3 and reads, for each entry of
// a stencil, four columns at the same offset from them: consecutive lanes then
// read consecutive words.  The vector passes take the same quads, a thread
// always the same ones.
//
// The arithmetic is the fused kernels' (and so the reference's), operation by
// operation; only the grouping of the reductions differs.
//
// Measured in turn with the fused kernels, on the same barrier and with Jacobi (us
// per iteration, 7- or 5-point operators): Cg 512^2 18.7 -> 10.7, 48^3 16.7 -> 10.8;
// BiCgStab 32^3 13.8 -> 10.4, 512^2 16.0 -> 11.9; Gmres(30) 32^3 66 -> 52, 64^3 74 ->
// 60, and with the matrix streamed 96^3 117 -> 93, 112^3 152 -> 139, 128^3 188 ->
// 183 (short restarts lose there: see resident_solve).  Cg and BiCgStab with the matrix streamed gained nothing (80^3
// 20.8 -> 21.4, 90^3 32 -> 33): there the product sets the pace, and with the
// shared memory taken its gathers lose the L1.
#pragma once

namespace sb2 {

constexpr int kResSmem = 226 * 1024;     // dynamic shared memory a CTA may take

// What a CTA knows of the operator.
struct ResOp {
  const long long* sptr;
  const uint2* qinfo;
  const int* scol;
  const double* sval;
  const double* diag;  // nullptr: identity, else Jacobi
  int nslice, n;
  int per;             // slices per CTA
  int groups;          // groups (one entry of 4 rows) the shared copy holds, 0: none
};

#ifdef __CUDACC__

struct ResCta {
  int s0, s1, r0;  // slices and first row
  int nq, NQ;      // quads, plane stride
  int rows;        // 4 * nq
};

__device__ __forceinline__ ResCta res_cta(const ResOp& A) {
  ResCta c;
  c.s0 = min((int)blockIdx.x * A.per, A.nslice);
  c.s1 = min(c.s0 + A.per, A.nslice);
  c.r0 = c.s0 * kQuadRows;
  c.nq = (c.s1 - c.s0) * 32;
  c.NQ = A.per * 32;
  c.rows = 4 * c.nq;
  return c;
}

// One vector of the CTA's rows in shared memory.
struct ResVec {
  double* p;
  int NQ;
  __device__ __forceinline__ double& at(int q, int j) const { return p[j * NQ + q]; }
  __device__ __forceinline__ void get(int q, double (&v)[4]) const {
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = p[j * NQ + q];
  }
  __device__ __forceinline__ void set(int q, const double (&v)[4]) const {
#pragma unroll
    for (int j = 0; j < 4; j++) p[j * NQ + q] = v[j];
  }
};

// Rows row..row+3 of a caller's vector (any alignment; zero past the end).
__device__ __forceinline__ void res_load(const double* g, int row, int n, double (&v)[4]) {
#pragma unroll
  for (int j = 0; j < 4; j++) v[j] = row + j < n ? __ldcg(g + row + j) : 0.0;
}
__device__ __forceinline__ void res_store(double* g, int row, int n, const double (&v)[4]) {
#pragma unroll
  for (int j = 0; j < 4; j++)
    if (row + j < n) g[row + j] = v[j];
}

__device__ __forceinline__ double res_prec(bool jac, double r, double d) {
  return jac ? __ddiv_rn(r, d) : r;
}

// Operand of a product: the CTA's rows from shared memory, the others from
// global memory, by one generic load each: no branch keeps a row's loads from
// being in flight together.
struct ResGather {
  const double* own;  // the vector's planes in shared memory
  int NQ;
  const double* g;
  int r0, rows;
  __device__ __forceinline__ void operator()(const int4& c, double (&o)[4]) const {
    const int cc[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int i = cc[j] - r0;
      o[j] = *((unsigned)i < (unsigned)rows ? own + ((i & 3) * NQ + (i >> 2)) : g + cc[j]);
    }
  }
};

// The same for p = beta p + z, formed where it is read for rows of other CTAs
// (their p of this step is not published yet): Cg saves a barrier.
struct ResGatherP {
  const double* own;
  int NQ;
  const double *p, *z;
  double beta;
  bool first;
  int r0, rows;
  __device__ __forceinline__ void operator()(const int4& c, double (&o)[4]) const {
    const int cc[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int i = cc[j] - r0;
      const bool in = (unsigned)i < (unsigned)rows;
      o[j] = *(in ? own + ((i & 3) * NQ + (i >> 2)) : z + cc[j]);
      if (!in && !first) o[j] = add_rn(mul_rn(p[cc[j]], beta), o[j]);
    }
  }
};

// The vector in global memory only.
struct ResGatherAll {
  const double* g;
  __device__ __forceinline__ void operator()(const int4& c, double (&o)[4]) const {
    o[0] = __ldca(g + c.x);
    o[1] = __ldca(g + c.y);
    o[2] = __ldca(g + c.z);
    o[3] = __ldca(g + c.w);
  }
};

__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

// Bulk copies of basis vectors into shared memory, one mbarrier a buffer.
__device__ __forceinline__ void bulk_init(unsigned long long* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ void bulk_get(unsigned dst, const void* src, unsigned bytes,
                                         unsigned long long* bar) {
  proxy_fence();
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   dst),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
// false: the copy did not come
__device__ __forceinline__ bool bulk_wait(unsigned long long* bar, unsigned parity) {
  for (int tries = 0; tries < 4000000; tries++) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// Copies the CTA's part of the matrix to shared memory.
template <int NTR>
__device__ __forceinline__ void res_matrix(const ResOp& A, const ResCta& C, int4* mcol, double* mval) {
  const long long g0 = __ldg(A.sptr + C.s0), g1 = __ldg(A.sptr + C.s1);
  const int4* c4 = reinterpret_cast<const int4*>(A.scol) + g0;
  const double2* v2 = reinterpret_cast<const double2*>(A.sval + 4 * g0);
  const int ng = (int)(g1 - g0);
  for (int i = threadIdx.x; i < ng; i += NTR) mcol[i] = __ldcs(c4 + i);
  for (int i = threadIdx.x; i < 2 * ng; i += NTR) reinterpret_cast<double2*>(mval)[i] = __ldcs(v2 + i);
}

// One row sum per row of the CTA (divided by the row's diagonal entry with
// `diag`), entries in stored order, U groups' gathers in flight together;
// out(q, t) takes quad q's four values.
template <int NTR, bool MS, int U, class G, class Out>
__device__ __forceinline__ void res_rows(const ResOp& A, int s0, int s1, const int4* mcol,
                                         const double* mval, const G& gather, const double* diag,
                                         Out&& out) {
  const int lane = threadIdx.x & 31;
  const int4* __restrict__ col4 = MS ? mcol : reinterpret_cast<const int4*>(A.scol);
  const double* __restrict__ val = MS ? mval : A.sval;
  const long long base = MS ? __ldg(A.sptr + s0) : 0;
#pragma unroll 1
  for (int s = s0 + (threadIdx.x >> 5); s < s1; s += NTR / 32) {
    const uint2 inf = __ldg(A.qinfo + (size_t)s * 32 + lane);
    const int ln[4] = {(int)(inf.y & 255u), (int)((inf.y >> 8) & 255u), (int)((inf.y >> 16) & 255u),
                       (int)(inf.y >> 24)};
    const int L = max(max(ln[0], ln[1]), max(ln[2], ln[3]));
    const long long g0 = __ldg(A.sptr + s) - base + lane;
    double t[4] = {0.0, 0.0, 0.0, 0.0}, d[4] = {1.0, 1.0, 1.0, 1.0};
    if (diag) {
      const int row = s * kQuadRows + 4 * lane;
      if (row + 3 < A.n) {
        vld4_cs(diag + row, d);
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (row + j < A.n) d[j] = __ldg(diag + row + j);
      }
    }
#pragma unroll 1
    for (int k0 = 0; k0 < L; k0 += U) {
      int4 c[U];
      double v[U][4], xv[U][4];
#pragma unroll
      for (int u = 0; u < U; u++)
        if (k0 + u < L) {
          const long long g = g0 + (long long)(k0 + u) * 32;
          if (MS) {
            c[u] = col4[g];
          } else {
            c[u] = __ldcs(col4 + g);
            vld4_cs(val + g * 4, v[u]);
          }
        }
#pragma unroll
      for (int u = 0; u < U; u++)
        if (k0 + u < L) gather(c[u], xv[u]);
#pragma unroll
      for (int u = 0; u < U; u++)
        if (k0 + u < L) {
          if (MS) {
            const double2* m2 = reinterpret_cast<const double2*>(val) + 2 * (g0 + (long long)(k0 + u) * 32);
            const double2 a = m2[0], b = m2[1];
            v[u][0] = a.x; v[u][1] = a.y; v[u][2] = b.x; v[u][3] = b.y;
          }
#pragma unroll
          for (int j = 0; j < 4; j++)
            if (k0 + u < ln[j]) t[j] = add_rn(t[j], mul_rn(v[u][j], xv[u][j]));
        }
    }
    const int q = (s - s0) * 32 + lane;
    if (diag) {
#pragma unroll
      for (int j = 0; j < 4; j++) t[j] = __ddiv_rn(t[j], d[j]);
    }
    out(q, t);
  }
}

// The same into planes of shared memory, as a function of its own: inlined
// into the kernels with many vectors its batches of loads spill, and with the
// shared memory taken there is little L1 left to spill to.
template <int NTR, bool MS, int U, class G>
__device__ __noinline__ void res_product(const ResOp& A, int s0, int s1, const int4* mcol,
                                         const double* mval, const G gather, double* out, int NQ,
                                         const double* diag) {
  res_rows<NTR, MS, U>(A, s0, s1, mcol, mval, gather, diag, [&](int q, const double (&t)[4]) {
#pragma unroll
    for (int j = 0; j < 4; j++) out[j * NQ + q] = t[j];
  });
}

#define SB2_RES_DECL                                   \
  extern __shared__ __align__(16) double s_res[];      \
  __shared__ double s_red[2 * (NTR / 32)];             \
  __shared__ double s_vals[kMaxRed];                   \
  const int tid = threadIdx.x;                         \
  const ResCta C = res_cta(A);                         \
  int4* mcol = nullptr;                                \
  double* mval = nullptr;                              \
  const bool lead = (blockIdx.x == 0 && tid == 0);     \
  const bool jac = A.diag != nullptr;                  \
  constexpr std::integral_constant<int, MS ? 4 : 1> kRound; \
  unsigned epoch = 0;                                  \
  int hlen = 0;                                        \
  /* fence: another CTA's vector is read before the next barrier */ \
  auto reduce1 = [&](double a, bool fence = true) {    \
    grid_arrive_sums<NTR, 1>(P, epoch, {a}, s_red);    \
    return grid_wait<NTR, kPollerSums>(P, epoch, 1, s_vals, fence); \
  };                                                   \
  auto reduce2 = [&](double a, double b, bool fence = true) { \
    grid_arrive_sums<NTR, 2>(P, epoch, {a, b}, s_red); \
    return grid_wait<NTR, kPollerSums>(P, epoch, 2, s_vals, fence); \
  };                                                   \
  /* t = A v, t and v in shared memory planes */ \
  auto product = [&](auto uc, const auto& g, const ResVec& t, const double* diag = nullptr) { \
    __syncthreads();                                   \
    res_product<NTR, MS, decltype(uc)::value>(A, C.s0, C.s1, mcol, mval, g, t.p, C.NQ, diag); \
    __syncthreads();                                   \
  };                                                   \
  /* rows past the end add nothing, whatever the scalars are */ \
  auto live = [&](int q, int j) { return C.r0 + 4 * q + j < A.n; }; \
  /* quads of this thread */                           \
  auto quads = [&](auto&& f) {                         \
    _Pragma("unroll 1") for (int q = tid; q < C.nq; q += NTR) f(q, C.r0 + 4 * q); \
  }

// ----------------------------------------------------------------- Cg (Cg.cxx:45-116)

struct CgResVecs {
  const double* b;
  double *x, *z, *p[2];  // z, p: padded work vectors that other CTAs read
};

// Vectors in shared memory: x, r, p, q, and with Jacobi z and the diagonal.
constexpr int res_cg_vecs(bool jac) { return jac ? 6 : 4; }

template <int NTR, bool MS>
__global__ void __launch_bounds__(NTR, 1) cg_resident_kernel(ResOp A, CgResVecs v, IterArgs it,
                                                             Persist P, History H, SolveOut* out) {
  constexpr bool kPollerSums = true;
  SB2_RES_DECL;
  const size_t plane = 4 * (size_t)C.NQ;
  const ResVec xs{s_res, C.NQ}, rs{s_res + plane, C.NQ}, ps{s_res + 2 * plane, C.NQ},
      qs{s_res + 3 * plane, C.NQ}, zs{jac ? s_res + 4 * plane : rs.p, C.NQ}, ds{s_res + 5 * plane, C.NQ};
  mval = s_res + (jac ? 6 : 4) * plane;
  mcol = reinterpret_cast<int4*>(mval + 4 * (size_t)A.groups);
  if (MS) res_matrix<NTR>(A, C, mcol, mval);

  // iter.Init(b): facteur_reste = 1/||b|| (Iterative.cxx:235-249)
  double acc = 0.0;
  quads([&](int q, int row) {
    double bv[4], dv[4];
    res_load(v.b, row, A.n, bv);
    rs.set(q, bv);
    if (jac) {
      res_load(A.diag, row, A.n, dv);
#pragma unroll
      for (int j = 0; j < 4; j++) dv[j] = row + j < A.n ? dv[j] : 1.0;
      ds.set(q, dv);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) acc = add_rn(acc, mul_rn(bv[j], bv[j]));
  });
  if (!reduce1(acc)) return;
  const double normb = sqrt(s_vals[0]);
  if (normb == 0.0) {
    if (lead) { out->init_failed = 1; out->hist_len = 0; }
    return;
  }
  const double facteur = 1.0 / normb;

  // r = b - A x (or x = 0, r = b), with ||r||^2 and (r, z)
  if (!it.init_guess_null) product(kRound, ResGatherAll{v.x}, qs);
  double rr = 0.0, rz = 0.0;
  quads([&](int q, int row) {
    double rv[4], zv[4], xv[4] = {0.0, 0.0, 0.0, 0.0};
    rs.get(q, rv);
    if (!it.init_guess_null) {
#pragma unroll
      for (int j = 0; j < 4; j++) rv[j] = add_rn(rv[j], -qs.at(q, j));
      rs.set(q, rv);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      zv[j] = res_prec(jac, rv[j], jac ? ds.at(q, j) : 1.0);
      rr = add_rn(rr, mul_rn(rv[j], rv[j]));
      rz = add_rn(rz, mul_rn(rv[j], zv[j]));
    }
    if (jac) zs.set(q, zv);
    vst4(v.z + row, zv);
    if (!it.init_guess_null) res_load(v.x, row, A.n, xv);
    xs.set(q, xv);
  });
  if (!reduce2(rr, rz)) return;
  rr = s_vals[0];
  double rho = s_vals[1], rho_1 = 1.0;

  int nb_iter = 0, fail = 0;
  double reste;
  for (;;) {
    reste = facteur * sqrt(rr);
    if (lead) hist_push(H, &hlen, nb_iter, reste);
    if (reste < it.tol || nb_iter >= it.max_iter) break;
    if (rho == 0.0) { fail = 1; break; }
    // p = z (first) | p = beta*p + z: Mlt(beta, p); Add(1, z, p)
    const bool first = nb_iter == 0;
    const double beta = first ? 0.0 : rho / rho_1;
    double* pg = v.p[nb_iter & 1];
    quads([&](int q, int row) {
      double pv[4], zv[4];
      zs.get(q, zv);
      ps.get(q, pv);
#pragma unroll
      for (int j = 0; j < 4; j++) pv[j] = first ? zv[j] : add_rn(mul_rn(pv[j], beta), zv[j]);
      ps.set(q, pv);
      vst4(pg + row, pv);
    });
    __syncthreads();
    // q = A p fused with delta = (p, q)
    double d = 0.0;
    res_rows<NTR, MS, kRound()>(
        A, C.s0, C.s1, mcol, mval,
        ResGatherP{ps.p, C.NQ, v.p[(nb_iter & 1) ^ 1], v.z, beta, first, C.r0, C.rows}, nullptr,
        [&](int q, const double (&t)[4]) {
          qs.set(q, t);
#pragma unroll
          for (int j = 0; j < 4; j++)
            if (live(q, j)) d = add_rn(d, mul_rn(ps.at(q, j), t[j]));
        });
    if (!reduce1(d, false)) return;
    const double delta = s_vals[0];
    if (delta == 0.0) { fail = 2; break; }
    const double alpha = rho / delta;
    // Add(alpha, p, x); Add(-alpha, q, r); then ||r||^2 and (r, z) for the next test
    rr = 0.0;
    rz = 0.0;
    quads([&](int q, int row) {
      double xv[4], pv[4], rv[4], qv[4], zv[4];
      xs.get(q, xv);
      ps.get(q, pv);
      rs.get(q, rv);
      qs.get(q, qv);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (alpha != 0.0) {
          xv[j] = add_rn(xv[j], mul_rn(alpha, pv[j]));
          rv[j] = add_rn(rv[j], mul_rn(-alpha, qv[j]));
        }
        zv[j] = res_prec(jac, rv[j], jac ? ds.at(q, j) : 1.0);
        if (live(q, j)) {
          rr = add_rn(rr, mul_rn(rv[j], rv[j]));
          rz = add_rn(rz, mul_rn(rv[j], zv[j]));
        }
      }
      xs.set(q, xv);
      rs.set(q, rv);
      if (jac) zs.set(q, zv);
      vst4(v.z + row, zv);
    });
    if (!reduce2(rr, rz)) return;
    rr = s_vals[0];
    rho_1 = rho;
    rho = s_vals[1];
    nb_iter++;
  }
  quads([&](int q, int row) {
    double xv[4];
    xs.get(q, xv);
    res_store(v.x, row, A.n, xv);
  });
  if (lead) write_out(out, nb_iter, it.max_iter, fail, facteur, reste, hlen);
}

// ----------------------------------------------------------------- BiCgStab (BiCgStab.cxx:43-145)

struct BicgResVecs {
  const double* b;
  double *x, *rt, *ph, *sh;  // rt: only its owner reads it; ph, sh: gathered
};

// Vectors in shared memory: p, r (s in its place), v, t, and with Jacobi
// phat and shat.
constexpr int res_bicg_vecs(bool jac) { return jac ? 6 : 4; }

template <int NTR, bool MS>
__global__ void __launch_bounds__(NTR, 1) bicgstab_resident_kernel(ResOp A, BicgResVecs v,
                                                                   IterArgs it, Persist P,
                                                                   History H, SolveOut* out) {
  constexpr bool kPollerSums = true;
  SB2_RES_DECL;
  const size_t plane = 4 * (size_t)C.NQ;
  const ResVec ps{s_res, C.NQ}, rs{s_res + plane, C.NQ}, vs{s_res + 2 * plane, C.NQ},
      ts{s_res + 3 * plane, C.NQ}, phs{jac ? s_res + 4 * plane : ps.p, C.NQ},
      shs{jac ? s_res + 5 * plane : rs.p, C.NQ};
  mval = s_res + (jac ? 6 : 4) * plane;
  mcol = reinterpret_cast<int4*>(mval + 4 * (size_t)A.groups);
  if (MS) res_matrix<NTR>(A, C, mcol, mval);
  auto diag_of = [&](int row, double (&d)[4]) {
#pragma unroll
    for (int j = 0; j < 4; j++) d[j] = jac && row + j < A.n ? __ldg(A.diag + row + j) : 1.0;
  };

  double acc = 0.0;
  quads([&](int q, int row) {
    double bv[4];
    res_load(v.b, row, A.n, bv);
    rs.set(q, bv);
#pragma unroll
    for (int j = 0; j < 4; j++) acc = add_rn(acc, mul_rn(bv[j], bv[j]));
  });
  if (!reduce1(acc)) return;
  const double normb = sqrt(s_vals[0]);
  if (normb == 0.0) {
    if (lead) { out->init_failed = 1; out->hist_len = 0; }
    return;
  }
  const double facteur = 1.0 / normb;

  // r = b - A x (or x = 0); rtilde = r; ||r||^2 and (rtilde, r)
  if (!it.init_guess_null) product(kRound, ResGatherAll{v.x}, ts);
  double rr = 0.0;
  quads([&](int q, int row) {
    double rv[4];
    rs.get(q, rv);
    if (!it.init_guess_null) {
#pragma unroll
      for (int j = 0; j < 4; j++) rv[j] = add_rn(rv[j], -ts.at(q, j));
      rs.set(q, rv);
    }
    vst4(v.rt + row, rv);
    if (it.init_guess_null) {
      const double zero[4] = {0.0, 0.0, 0.0, 0.0};
      res_store(v.x, row, A.n, zero);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) rr = add_rn(rr, mul_rn(rv[j], rv[j]));
  });
  if (!reduce2(rr, rr)) return;
  rr = s_vals[0];
  double rho_1 = s_vals[1];  // (rtilde, r) with rtilde = r
  double rho_2 = 0.0, alpha = 0.0, omega = 0.0;

  int nb_iter = 0, fail = 0;
  double reste;
  for (;;) {
    reste = facteur * sqrt(rr);
    if (lead) hist_push(H, &hlen, nb_iter, reste);
    if (reste < it.tol || nb_iter >= it.max_iter) break;
    if (rho_1 == 0.0) { fail = 1; break; }
    const bool first = nb_iter == 0;
    if (!first && omega == 0.0) { fail = 2; break; }
    // Copy(r, p), or Add(-omega, v, p); Mlt(beta, p); Add(1, r, p); phat = M^{-1} p
    const double beta = first ? 0.0 : (rho_1 / rho_2) * (alpha / omega);
    quads([&](int q, int row) {
      double pv[4], vv[4], rv[4], dv[4];
      rs.get(q, rv);
      diag_of(row, dv);
      if (first) {
#pragma unroll
        for (int j = 0; j < 4; j++) pv[j] = rv[j];
      } else {
        ps.get(q, pv);
        vs.get(q, vv);
#pragma unroll
        for (int j = 0; j < 4; j++) {
          pv[j] = add_rn(pv[j], mul_rn(-omega, vv[j]));
          pv[j] = add_rn(mul_rn(pv[j], beta), rv[j]);
        }
      }
      ps.set(q, pv);
#pragma unroll
      for (int j = 0; j < 4; j++) pv[j] = res_prec(jac, pv[j], dv[j]);
      if (jac) phs.set(q, pv);
      vst4(v.ph + row, pv);
    });
    if (!grid_sync<NTR>(P, epoch, 0, s_vals)) return;
    // v = A phat, sigma = (rtilde, v)
    product(kRound, ResGather{phs.p, C.NQ, v.ph, C.r0, C.rows}, vs);
    double d = 0.0;
    quads([&](int q, int row) {
      double wv[4];
      vld4_cg(v.rt + row, wv);
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (live(q, j)) d = add_rn(d, mul_rn(wv[j], vs.at(q, j)));
    });
    if (!reduce1(d, false)) return;
    const double sigma = s_vals[0];
    if (sigma == 0.0) { fail = 3; break; }
    alpha = rho_1 / sigma;
    // Copy(r, s); Add(-alpha, v, s); shat = M^{-1} s; ||s||^2
    double ss = 0.0;
    quads([&](int q, int row) {
      double sv[4], vv[4], dv[4];
      rs.get(q, sv);
      vs.get(q, vv);
      diag_of(row, dv);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (alpha != 0.0) sv[j] = add_rn(sv[j], mul_rn(-alpha, vv[j]));
        if (live(q, j)) ss = add_rn(ss, mul_rn(sv[j], sv[j]));
      }
      rs.set(q, sv);
#pragma unroll
      for (int j = 0; j < 4; j++) sv[j] = res_prec(jac, sv[j], dv[j]);
      if (jac) shs.set(q, sv);
      vst4(v.sh + row, sv);
    });
    if (!reduce1(ss)) return;
    nb_iter++;
    reste = facteur * sqrt(s_vals[0]);
    if (lead) hist_push(H, &hlen, nb_iter, reste);
    if (reste < it.tol || nb_iter >= it.max_iter) {
      // Add(alpha, phat, x)
      if (alpha != 0.0)
        quads([&](int q, int row) {
          double xv[4];
          res_load(v.x, row, A.n, xv);
#pragma unroll
          for (int j = 0; j < 4; j++) xv[j] = add_rn(xv[j], mul_rn(alpha, phs.at(q, j)));
          res_store(v.x, row, A.n, xv);
        });
      break;
    }
    // t = A shat; omega = (t, s) / (t, t)
    product(kRound, ResGather{shs.p, C.NQ, v.sh, C.r0, C.rows}, ts);
    double t0 = 0.0, t1 = 0.0;
    quads([&](int q, int) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (!live(q, j)) continue;
        const double t = ts.at(q, j);
        t0 = add_rn(t0, mul_rn(rs.at(q, j), t));
        t1 = add_rn(t1, mul_rn(t, t));
      }
    });
    if (!reduce2(t0, t1, false)) return;
    omega = s_vals[0] / s_vals[1];
    // Add(alpha, phat, x); Add(omega, shat, x); Copy(s, r); Add(-omega, t, r)
    rr = 0.0;
    double rtr = 0.0;
    quads([&](int q, int row) {
      double xv[4], rv[4], tv[4], wv[4];
      res_load(v.x, row, A.n, xv);
      vld4_cg(v.rt + row, wv);
      rs.get(q, rv);
      ts.get(q, tv);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (alpha != 0.0) xv[j] = add_rn(xv[j], mul_rn(alpha, phs.at(q, j)));
        if (omega != 0.0) {
          xv[j] = add_rn(xv[j], mul_rn(omega, shs.at(q, j)));
        }
        if (-omega != 0.0) rv[j] = add_rn(rv[j], mul_rn(-omega, tv[j]));
        if (!live(q, j)) continue;
        rr = add_rn(rr, mul_rn(rv[j], rv[j]));
        rtr = add_rn(rtr, mul_rn(wv[j], rv[j]));
      }
      res_store(v.x, row, A.n, xv);
      rs.set(q, rv);
    });
    if (!reduce2(rr, rtr, false)) return;
    rr = s_vals[0];
    rho_2 = rho_1;
    rho_1 = s_vals[1];
    nb_iter++;
  }
  if (lead) write_out(out, nb_iter, it.max_iter, fail, facteur, reste, hlen);
}

// ----------------------------------------------------------------- Gmres (Gmres.cxx:44-183)

struct GmresResVecs {
  const double* b;
  double *x, *V;   // V: m + 1 padded vectors, `ld` apart
  double* H;       // the Hessenberg matrix of each CTA, (m + 1) x (m + 1)
  long long ld;
};

// Modified Gram-Schmidt in the reference's order with w in registers and the
// two basis vectors of a pass in shared memory: V_k, which was there the pass
// before, and V_{k+1}, which a bulk copy brings while the grid sums the dot of
// V_k.  A pass reads one basis vector once, where it read two and read and
// wrote w.
// QR: quads a thread owns at most.
template <int NTR, int QR, bool MS>
__global__ void __launch_bounds__(NTR, 1) gmres_resident_kernel(ResOp A, GmresResVecs v, IterArgs it,
                                                                Persist P, History H, SolveOut* out) {
  constexpr bool kPollerSums = false;
  SB2_RES_DECL;
  const int m = it.restart, ld = m + 1;
  const size_t plane = 4 * (size_t)C.NQ;
  // the product's result and operand; between products the basis vectors
  // fetched, V_k in part k % 2; between cycles M^{-1} r in the first
  const ResVec ws{s_res, C.NQ}, us{s_res + plane, C.NQ};
  double* hc = s_res + 2 * plane;       // column i of H
  double* sv = hc + ld;                 // s(0..m)
  double* cs = sv + ld;
  double* sn = cs + ld;
  mval = s_res + 2 * plane + 4 * (size_t)((ld + 3) / 4 * 4);
  mcol = reinterpret_cast<int4*>(mval + 4 * (size_t)A.groups);
  double* Hm = v.H + (size_t)blockIdx.x * ld * ld;
  __shared__ unsigned long long s_full[2];
  if (tid == 0) {
    bulk_init(&s_full[0]);
    bulk_init(&s_full[1]);
  }
  if (MS) res_matrix<NTR>(A, C, mcol, mval);
  auto diag_of = [&](int row, double (&d)[4]) {
    if (jac && row + 3 < A.n) {
      vld4_ldg(A.diag + row, d);
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++) d[j] = jac && row + j < A.n ? __ldg(A.diag + row + j) : 1.0;
    }
  };
  // the CTA's rows of basis vector k into buffer k % 2 (thread 0)
  unsigned parity = 0u;  // bit b: the phase of buffer b to wait for
  unsigned inflight = 0u;
  bool late = false;
  auto fetch = [&](int k) {
    inflight |= 1u << (k & 1);
    if (tid == 0)
      bulk_get(smem_addr(s_res + (k & 1) * plane), v.V + (size_t)k * v.ld + C.r0,
               8u * (unsigned)C.rows, &s_full[k & 1]);
  };
  auto arrived = [&](int k) {
    if (!bulk_wait(&s_full[k & 1], parity >> (k & 1) & 1u)) late = true;
    parity ^= 1u << (k & 1);
    inflight &= ~(1u << (k & 1));
  };
  // a CTA that leaves early waits for its own copies first
  auto drain = [&]() {
    for (int b = 0; b < 2; b++)
      if (inflight >> b & 1u) arrived(b);
  };
  // a thread's rows are pairs 2e, 2e + 1, e = tid + r * NTR
  auto fetched = [&](int k, int e) {
    return reinterpret_cast<const double2*>(s_res + (k & 1) * plane)[e];
  };
  const int pairs = 2 * C.nq;
  auto live2 = [&](int e, int j) { return C.r0 + 2 * e + j < A.n; };
  auto arrive1 = [&](double a) { grid_arrive_sums<NTR, 1>(P, epoch, {a}, s_red); };

  // w = b (- A x); r = M^{-1} w; beta = ||r|| (Gmres.cxx:82-90)
  double rr = 0.0;
  auto residual = [&](bool ax) {  // w holds A x, or is not read
    quads([&](int q, int row) {
      double rv[4], dv[4];
      res_load(v.b, row, A.n, rv);
      diag_of(row, dv);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (ax) rv[j] = add_rn(rv[j], -ws.at(q, j));
        rv[j] = res_prec(jac, rv[j], dv[j]);
        rr = add_rn(rr, mul_rn(rv[j], rv[j]));
      }
      ws.set(q, rv);
      if (!ax) {
        const double zero[4] = {0.0, 0.0, 0.0, 0.0};
        res_store(v.x, row, A.n, zero);
      }
    });
  };
  if (!it.init_guess_null) product(kRound, ResGatherAll{v.x}, ws);
  residual(!it.init_guess_null);
  if (!reduce1(rr)) return;
  double beta = sqrt(s_vals[0]);
  // outer.Init(r)
  if (beta == 0.0) {
    if (lead) { out->init_failed = 1; out->hist_len = 0; }
    return;
  }
  const double facteur = 1.0 / beta;

  int nb_iter = 0;
  double reste;
  for (;;) {
    // while (!outer.Finished(beta))
    reste = facteur * beta;
    if (lead) hist_push(H, &hlen, nb_iter, reste);
    if (reste < it.tol || nb_iter >= it.max_iter) break;
    // V0 = r * (1/beta); s = beta e0
    const double inv_beta = 1.0 / beta;
    quads([&](int q, int row) {
      double wv[4];
      ws.get(q, wv);
#pragma unroll
      for (int j = 0; j < 4; j++) wv[j] = mul_rn(wv[j], inv_beta);
      us.set(q, wv);
      vst4(v.V + row, wv);
    });
    proxy_fence();
    if (tid == 0) {
      for (int k = 0; k < ld; k++) sv[k] = 0.0;
      sv[0] = beta;
    }
    const int inner_max = nb_iter + m;
    int i = 0;
    if (!grid_sync<NTR>(P, epoch, 0, s_vals)) return;
    for (;;) {
      // w = M^{-1} A V_i
      product(kRound, ResGather{us.p, C.NQ, v.V + (size_t)i * v.ld, C.r0, C.rows}, ws, A.diag);
      // modified Gram-Schmidt: H(k,i) = (V_k, w); Add(-H(k,i), V_k, w)
      double w[2 * QR][2];
#pragma unroll
      for (int r = 0; r < 2 * QR; r++) {
        const int e = tid + r * NTR;
        if (e < pairs) {
          w[r][0] = ws.at(e >> 1, 2 * (e & 1));
          w[r][1] = ws.at(e >> 1, 2 * (e & 1) + 1);
        }
      }
      proxy_fence();
      __syncthreads();  // w is out of the shared memory that V_0 and V_1 go to
      fetch(0);
      if (i > 0) fetch(1);
      arrived(0);
      double acc = 0.0;
#pragma unroll
      for (int r = 0; r < 2 * QR; r++) {
        const int e = tid + r * NTR;
        if (e < pairs) {
          const double2 vn = fetched(0, e);
          if (live2(e, 0)) acc = add_rn(acc, mul_rn(vn.x, w[r][0]));
          if (live2(e, 1)) acc = add_rn(acc, mul_rn(vn.y, w[r][1]));
        }
      }
      arrive1(acc);
      if (!grid_wait<NTR>(P, epoch, 1, s_vals, false)) {
        drain();
        return;
      }
#pragma unroll 1
      for (int k = 0; k <= i; k++) {
        const double h = s_vals[0];
        if (tid == 0) {
          hc[k] = h;
          if (k > 0) apply_rot(hc[k - 1], hc[k], cs[k - 1], sn[k - 1]);
        }
        acc = 0.0;
        if (k < i) arrived(k + 1);
#pragma unroll
        for (int r = 0; r < 2 * QR; r++) {
          const int e = tid + r * NTR;
          if (e < pairs) {
            if (-h != 0.0) {
              const double2 vk = fetched(k, e);
              w[r][0] = add_rn(w[r][0], mul_rn(-h, vk.x));
              w[r][1] = add_rn(w[r][1], mul_rn(-h, vk.y));
            }
            double2 vn = make_double2(w[r][0], w[r][1]);
            if (k < i) vn = fetched(k + 1, e);
            if (live2(e, 0)) acc = add_rn(acc, mul_rn(vn.x, w[r][0]));
            if (live2(e, 1)) acc = add_rn(acc, mul_rn(vn.y, w[r][1]));
          }
        }
        arrive1(acc);  // every thread has read V_k
        if (k + 2 <= i) fetch(k + 2);
        if (!grid_wait<NTR>(P, epoch, 1, s_vals, false)) {
          drain();
          return;
        }
      }
      if (__syncthreads_or(late)) {
        if (tid == 0) atomicExch(&P.sync->status, 1);
        return;
      }
      // h_{i+1,i} = ||w||; V_{i+1} = w / h, published and kept for the product
      double hi_ip1 = sqrt(s_vals[0]);
      const double inv_h = hi_ip1 != 0.0 ? 1.0 / hi_ip1 : 1.0;
      double* Vn = v.V + (size_t)(i + 1) * v.ld + C.r0;
#pragma unroll
      for (int r = 0; r < 2 * QR; r++) {
        const int e = tid + r * NTR;
        if (e < pairs) {
          if (hi_ip1 != 0.0) {
            w[r][0] = mul_rn(w[r][0], inv_h);
            w[r][1] = mul_rn(w[r][1], inv_h);
          }
          us.at(e >> 1, 2 * (e & 1)) = w[r][0];
          us.at(e >> 1, 2 * (e & 1) + 1) = w[r][1];
          *reinterpret_cast<double2*>(Vn + 2 * e) = make_double2(w[r][0], w[r][1]);
        }
      }
      proxy_fence();
      grid_arrive<NTR>(P, epoch, 0, s_vals);
      // rotations, while the grid arrives (every CTA computes the same scalars;
      // those of the earlier columns were applied to column i as it came)
      if (tid == 0) {
        double hii = hc[i];
        if (hi_ip1 != 0.0) {
          gen_rot(hii, hi_ip1, cs[i], sn[i]);
          hc[i] = hii;
          apply_rot(sv[i], sv[i + 1], cs[i], sn[i]);
        }
      }
      if (!grid_wait<NTR>(P, epoch, 0, s_vals, true)) return;  // V_{i+1} complete
      if (tid <= i) Hm[tid + i * ld] = hc[tid];
      for (int k = NTR + tid; k <= i; k += NTR) Hm[k + i * ld] = hc[k];
      i++;
      nb_iter++;
      // inner.Finished(|s(i)|): inner counts alongside outer, max = start + m
      const double rin = facteur * fabs(sv[i]);
      if (lead) hist_push(H, &hlen, nb_iter, rin);
      reste = rin;
      if ((rin < it.tol) || (nb_iter >= inner_max)) break;
    }
    // Solve(H, s): netlib DTRSV column sweep on the leading i x i block
    __syncthreads();
    if (tid == 0) {
      for (int j = i - 1; j >= 0; j--)
        if (sv[j] != 0.0) {
          sv[j] = sv[j] / Hm[j + j * ld];
          const double t = sv[j];
          for (int r = j - 1; r >= 0; r--) sv[r] = __dsub_rn(sv[r], mul_rn(t, Hm[r + j * ld]));
        }
    }
    __syncthreads();
    // x += sum_k s(k) V_k (Add skipped when s(k) == 0)
    quads([&](int q, int row) {
      double xv[4];
      res_load(v.x, row, A.n, xv);
#pragma unroll 4
      for (int k = 0; k < i; k++)
        if (sv[k] != 0.0) {
          double vv[4];
          vld4_cg(v.V + (size_t)k * v.ld + row, vv);
#pragma unroll
          for (int j = 0; j < 4; j++) xv[j] = add_rn(xv[j], mul_rn(sv[k], vv[j]));
        }
      res_store(v.x, row, A.n, xv);
    });
    if (!grid_sync<NTR>(P, epoch, 0, s_vals)) return;
    // w = b - A x; r = M^{-1} w; beta = ||r||
    rr = 0.0;
    product(kRound, ResGatherAll{v.x}, ws);
    residual(true);
    if (!reduce1(rr)) return;
    beta = sqrt(s_vals[0]);
  }
  if (lead) write_out(out, nb_iter, it.max_iter, 0, facteur, reste, hlen);
}

#endif  // __CUDACC__

}  // namespace sb2
