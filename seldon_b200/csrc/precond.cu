// Preconditioners: identity, Jacobi, SOR and the ILUT apply.
//
// SOR reproduces the reference's strictly sequential sweeps
// (Relaxation_MatVect.cxx:41-95 RowSparse, :176-298 RowSymSparse) bit for
// bit: a sweep writes its values into a vector of its own, so a row reads the
// updated rows there and the others in the vector the sweep started from,
// and each row repeats the reference's own operation order with separately
// rounded products.
//
// The ILUT apply runs Seldon's SolveLU (computation/solver/SparseSolver.cxx:
// 533-611 and 852-882) on a factor computed on the host.  Its loops are
// either row gathers (x_i -= v * x_c over row i) or column scatters
// (x_c -= v * x_i for each entry of row i).  Every sweep is put in gather
// form: target j collects its updates in the order the sequential loop
// would have applied them (the scatter sources in increasing or decreasing
// row order, each row's entries in stored order).  Each row then repeats the
// reference's own operations with separately rounded products, so the result
// is the reference's bit for bit.
//
// Both run as persistent launches whose rows wait for the values they read, or
// level by level where levels are few and wide or rows long (sweep.cuh:
// SweepForm).  The device factorization of ILU(0) runs level by level.
#include <algorithm>
#include <vector>

#include "sweep.cuh"

namespace sb2 {

struct LevelPlan {
  int nlev = 0;
  std::vector<int> h_lvl;      // [nlev+1] offsets into rows
  int* d_rows = nullptr;       // rows ordered by level
  int* d_lvl = nullptr;        // device copy of h_lvl
  void release() {
    cudaFree(d_rows);
    cudaFree(d_lvl);
    d_rows = d_lvl = nullptr;
    h_lvl.clear();
    nlev = 0;
  }
};

static int upload_plan(const std::vector<int>& level, int n, LevelPlan* P) {
  int nlev = 0;
  for (int i = 0; i < n; i++) nlev = std::max(nlev, level[i] + 1);
  P->nlev = nlev;
  P->h_lvl.assign(nlev + 1, 0);
  for (int i = 0; i < n; i++) P->h_lvl[level[i] + 1]++;
  for (int l = 0; l < nlev; l++) P->h_lvl[l + 1] += P->h_lvl[l];
  std::vector<int> rows(std::max(n, 1)), fill(P->h_lvl.begin(), P->h_lvl.end() - 1);
  for (int i = 0; i < n; i++) rows[fill[level[i]]++] = i;  // increasing row in a level
  SB2_CUDA_TRY(cudaMalloc(&P->d_rows, sizeof(int) * std::max(n, 1)));
  SB2_CUDA_TRY(cudaMalloc(&P->d_lvl, sizeof(int) * (nlev + 1)));
  SB2_CUDA_TRY(cudaMemcpy(P->d_rows, rows.data(), sizeof(int) * std::max(n, 1), cudaMemcpyHostToDevice));
  SB2_CUDA_TRY(cudaMemcpy(P->d_lvl, P->h_lvl.data(), sizeof(int) * (nlev + 1), cudaMemcpyHostToDevice));
  return SB2_OK;
}

// Levels of a sweep: row j depends on the entries of `ptr/ind` on the side
// already swept (lower: c < j, upper: c > j).
static void tri_levels(int n, const int* ptr, const int* ind, bool lower,
                       std::vector<int>& level) {
  level.assign(n, 0);
  for (int s = 0; s < n; s++) {
    const int j = lower ? s : n - 1 - s;
    int lev = 0;
    for (int k = ptr[j]; k < ptr[j + 1]; k++) {
      const int c = ind[k];
      if (lower ? (c < j) : (c > j)) lev = std::max(lev, level[c] + 1);
    }
    level[j] = lev;
  }
}

// Levels of the mirrored entries of symmetric storage (row j, stored columns
// >= j): row c depends on each j < c that stores column c.
static void mirrored_levels(int n, const int* ptr, const int* ind, std::vector<int>& level) {
  level.assign(n, 0);
  for (int j = 0; j < n; j++)
    for (int k = ptr[j]; k < ptr[j + 1]; k++)
      if (ind[k] > j) level[ind[k]] = std::max(level[ind[k]], level[j] + 1);
}

// Levels of a sweep that works in place: row j comes after the rows whose new
// value it reads and before the rows that it reads old.
static void in_place_levels(int n, const int* ptr, const int* ind, bool forward, std::vector<int>& level) {
  level.assign(n, 0);
  std::vector<int> least(n, 0);
  for (int q = 0; q < n; q++) {
    const int j = forward ? q : n - 1 - q;
    int lev = least[j];
    for (int k = ptr[j]; k < ptr[j + 1]; k++) {
      const int c = ind[k];
      if (forward ? c < j : c > j) lev = std::max(lev, level[c] + 1);
    }
    level[j] = lev;
    for (int k = ptr[j]; k < ptr[j + 1]; k++) {
      const int c = ind[k];
      if (forward ? c > j : c < j) least[c] = std::max(least[c], lev + 1);
    }
  }
}

static int count_levels(const std::vector<int>& level) {
  int most = 0;
  for (int l : level) most = std::max(most, l + 1);
  return std::max(most, 1);
}

// ------------------------------------------------------------------ row ops

#ifdef __CUDACC__
// Plain loads: within one CTA (all levels in one launch) the SM's L1 holds
// the CTA's own stores, and across launches every write is visible.
__device__ __forceinline__ double ldx(const double* p) { return *p; }

template <class Op>
__global__ void level_kernel(int begin, int end, const int* __restrict__ rows, Op op) {
  int i = begin + blockIdx.x * blockDim.x + threadIdx.x;
  if (i < end) op(rows[i]);
}

// All levels in one CTA, separated by __syncthreads (small systems).
template <class Op>
__global__ void __launch_bounds__(1024) level_single_cta(int nlev, const int* __restrict__ lvl,
                                                         const int* __restrict__ rows, Op op) {
  for (int l = 0; l < nlev; l++) {
    for (int i = lvl[l] + threadIdx.x; i < lvl[l + 1]; i += blockDim.x) op(rows[i]);
    __syncthreads();
  }
}

// One row of GetIlu0 (IlutPreconditioning.cxx:1115-1176) or, with
// `modified`, of GetMilu0 (:1178-1243), in place on the CSR values: rows
// sorted by column with the diagonal at dpos.  For each L entry (stored
// order) tl = a_ij / u_jj (1/u_jj is already stored), then a_ic -= tl * u_jc
// for the columns c of row j's U part that row i holds; MILU(0) sums the
// others into s and takes s off the diagonal.  Finally the diagonal is
// inverted.  A zero pivot is recorded in *status (row + 1) and left as it is.
struct Ilu0Row {
  const int* ptr; const int* ind; double* val; const int* dpos; int* status; int modified;
  __device__ void operator()(int i) const {
    const int d = dpos[i], e = ptr[i + 1];
    double s = 0.0;
    for (int j = ptr[i]; j < d; j++) {
      const int jr = ind[j];
      const double tl = mul_rn(ldx(val + j), ldx(val + dpos[jr]));
      val[j] = tl;
      int q = j + 1;
      for (int k = dpos[jr] + 1; k < ptr[jr + 1]; k++) {
        const int c = ind[k];
        while (q < e && ind[q] < c) q++;
        if (q < e && ind[q] == c)
          val[q] = __dsub_rn(ldx(val + q), mul_rn(tl, ldx(val + k)));
        else if (modified)
          s = add_rn(s, mul_rn(tl, ldx(val + k)));
        else if (q == e)
          break;  // ILU(0): no column of row i is left to update
      }
    }
    double piv = ldx(val + d);
    if (modified) {
      piv = __dsub_rn(piv, s);
      val[d] = piv;
    }
    if (piv == 0.0) {
      atomicCAS(status, 0, i + 1);
      return;
    }
    val[d] = __ddiv_rn(1.0, piv);
  }
};

__global__ void jacobi_kernel(int n, const double* __restrict__ r,
                              const double* __restrict__ d, double* __restrict__ z) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    z[i] = __ddiv_rn(r[i], d[i]);
}
#endif

constexpr int kSingleCtaMaxN = 65536;

template <class Op>
static int run_factor_levels(const LevelPlan& P, int n, const Op& op, cudaStream_t s) {
  if (n == 0 || P.nlev == 0) return SB2_OK;
  if (n <= kSingleCtaMaxN) {
    level_single_cta<Op><<<1, 1024, 0, s>>>(P.nlev, P.d_lvl, P.d_rows, op);
  } else {
    for (int l = 0; l < P.nlev; l++) {
      const int cnt = P.h_lvl[l + 1] - P.h_lvl[l];
      level_kernel<Op><<<(cnt + 255) / 256, 256, 0, s>>>(P.h_lvl[l], P.h_lvl[l + 1], P.d_rows, op);
    }
  }
  SB2_CUDA_TRY(cudaGetLastError());
  return SB2_OK;
}

}  // namespace sb2

namespace sb2 {
// One triangular sweep in gather form: the rows' update lists, stored in the
// order the rows are taken.
struct GatherSweep {
  int* d_ind = nullptr;
  double* d_val = nullptr;
  SweepPlan plan;
  void release() {
    cudaFree(d_ind);
    cudaFree(d_val);
    d_ind = nullptr;
    d_val = nullptr;
    plan.release();
  }
};
}  // namespace sb2

struct sb2_precond {
  const sb2_csr* A = nullptr;
  int kind = 0;
  double omega = 1.0;
  int nb_iter = 1;
  int symmetric = 1;
  sb2::SweepGrid grid;      // row blocks and work vectors of the sweeps
  sb2::SweepPlan fwd, bwd;  // SOR
  double* d_tmp = nullptr;    // SOR, several launches: their other target
  int form = -1;              // SweepForm (-1: not planned yet)
  double* d_sdiag = nullptr;  // SOR, symmetric storage: diagonal of each stored row
  std::mutex mu;
  // ILUT: order, storage, permutations (and the inverse of the row one),
  // 1/U(i,i) or 1/D(i), and the sweeps (unsymmetric: L forward, U backward,
  // U^T forward, L^T backward; symmetric: L forward through the transposed
  // rows, L^T backward)
  int n_ilu = 0;
  int ilu_sym = 0;
  int* d_iprow = nullptr;
  int* d_pcol = nullptr;
  double* d_dinv = nullptr;
  sb2::GatherSweep s_lf, s_ub, s_utf, s_ltb;
};

namespace sb2 {

static int place_rows(const SweepGrid& G, const SweepPlan& P, int4* span, const int* ptr, const int* uptr) {
  if (G.n == 0) return SB2_OK;
  sweep_place_kernel<<<std::min((G.n + 255) / 256, 1184), 256>>>(G.n, P.d_rows, P.d_pos, span, ptr, uptr);
  SB2_CUDA_TRY(cudaGetLastError());
  return SB2_OK;
}

// Plans the sweeps not planned yet of those asked for.
static int plan_sor(sb2_precond* M, bool fwd, bool bwd) {
  std::lock_guard<std::mutex> g(M->mu);
  fwd = fwd && !M->fwd.d_buf;
  bwd = bwd && !M->bwd.d_buf;
  if (!fwd && !bwd) return SB2_OK;
  const sb2_csr* A = M->A;
  const int n = A->m;
  const CsrArrays &f = A->full, &src = A->sym ? A->upper : A->full;
  std::vector<int> ptr(n + 1), ind(std::max<long long>(src.nnz, 1));
  SB2_CUDA_TRY(cudaMemcpy(ptr.data(), src.d_ptr, sizeof(int) * (n + 1), cudaMemcpyDeviceToHost));
  if (src.nnz) SB2_CUDA_TRY(cudaMemcpy(ind.data(), src.d_ind, sizeof(int) * src.nnz, cudaMemcpyDeviceToHost));
  if (!M->grid.d_state) SB2_TRY(make_sweep_grid(n, &M->grid));
  if (A->sym && !M->d_sdiag) {
    // values of symmetric storage never change (sb2_csr_set_values)
    SB2_CUDA_TRY(cudaMalloc(&M->d_sdiag, sizeof(double) * std::max(n, 1)));
    if (n > 0)
      sym_diag_kernel<<<std::min((n + 255) / 256, 1184), 256>>>(n, src.d_ptr, src.d_ind, src.d_val, M->d_sdiag);
    SB2_CUDA_TRY(cudaGetLastError());
  }
  std::vector<int> level;
  SweepOrder order;
  SweepPlan made[2];
  int longest = 0;
  if (A->sym) {
    std::vector<int> len(n);  // stored and mirrored entries
    for (int j = 0; j < n; j++) {
      len[j] += ptr[j + 1] - ptr[j];
      for (int k = ptr[j]; k < ptr[j + 1]; k++)
        if (ind[k] > j) len[ind[k]]++;
    }
    for (int l : len) longest = std::max(longest, l);
  } else {
    for (int j = 0; j < n; j++) longest = std::max(longest, ptr[j + 1] - ptr[j]);
  }
  int st = SB2_OK;
  for (int k = 0; k < 2 && st == SB2_OK; k++) {
    if (!(k ? bwd : fwd)) continue;
    if (k == 0 && A->sym) mirrored_levels(n, ptr.data(), ind.data(), level);
    else tri_levels(n, ptr.data(), ind.data(), k == 0, level);
    if (M->form < 0)
      M->form = sweep_form(n, count_levels(level), (double)f.nnz / std::max(n, 1), A->sym ? 1 : 0);
    if (M->form == kFormSweep) {
      make_sweep_order(M->grid, level, &order);
      st = upload_sweep_plan(M->grid, order, nullptr, &made[k]);
    } else {
      if (M->form == kFormInPlace && !A->sym) in_place_levels(n, ptr.data(), ind.data(), k == 0, level);
      std::vector<int> rows, lvl;
      make_level_order(n, level, &rows, &lvl);
      st = upload_level_plan(n, rows, lvl, nullptr, &made[k]);
    }
    made[k].max_len = longest;
    if (st == SB2_OK && M->form == kFormSweep)
      st = place_rows(M->grid, made[k], made[k].d_span, f.d_ptr, A->sym ? src.d_ptr : nullptr);
  }
  // complete before any stream reads it
  if (st == SB2_OK) st = map_cuda_error(cudaStreamSynchronize(nullptr));
  for (int k = 0; k < 2; k++) {
    if (st != SB2_OK) made[k].release();
    else if (made[k].d_buf) (k ? M->bwd : M->fwd) = made[k];
  }
  return st;
}

// SOR(A, X, B, omega, iter, type_ssor) on the device: the sweeps from x0
// (null: zero) into x, two a launch.  x0 is null or x itself.
static int sor_apply(sb2_precond* M, const double* x0, double* x, const double* b, double omega,
                     int iter, int type_ssor, int late, cudaStream_t s) {
  const int nf = type_ssor % 2 == 0 ? std::max(iter, 0) : 0;
  const int total = nf + (type_ssor % 3 == 0 ? std::max(iter, 0) : 0);
  SB2_TRY(plan_sor(M, nf > 0, total > nf));
  const sb2_csr* A = M->A;
  const int n = A->m;
  if (!A->sym) SB2_TRY(ensure_diag(A));
  const SweepGrid& G = M->grid;
  const int launches = (total + 1) / 2;
  // targets alternate between x and a work vector, so that none is the
  // vector its launch starts from; from zero the last one is x
  if ((M->form == kFormSweep ? launches : M->form == kFormLevels ? total : 2 * (int)A->sym) > (x0 ? 0 : 1) && !M->d_tmp) {
    std::lock_guard<std::mutex> g(M->mu);
    if (!M->d_tmp) SB2_CUDA_TRY(cudaMalloc(&M->d_tmp, sizeof(double) * std::max(n, 1)));
  }
  const double* cur = x0;
  const CsrArrays &u = A->upper, &f = A->full;
  const double rest = 1.0 - omega, ratio = rest / omega;
  if (M->form == kFormLevels) {
    // the same, a sweep at a time
    const LevelSpan span{nullptr, f.d_ptr, A->sym ? u.d_ptr : nullptr};
    for (int q = 0; q < total; q++) {
      const bool fwd = q < nf;
      double* out = (x0 ? q % 2 == 1 : (total - 1 - q) % 2 == 0) ? x : M->d_tmp;
      const SweepPlan& P = fwd ? M->fwd : M->bwd;
      if (A->sym)
        SB2_TRY(run_levels(P, n, 0, fwd, span, cur, out,
                           SymmetricSor{u.d_ind, u.d_val, f.d_ind, f.d_val, M->d_sdiag, b, cur, omega, ratio}, s));
      else
        SB2_TRY(run_levels(P, n, 0, fwd, span, cur, out,
                           GeneralSor{f.d_ind, f.d_val, A->d_diag, b, cur, omega, rest}, s));
      cur = out;
    }
  } else if (M->form == kFormInPlace) {
    if (!x0) SB2_CUDA_TRY(cudaMemsetAsync(x, 0, sizeof(double) * n, s));
    for (int q = 0; q < total; q++) {
      const bool fwd = q < nf;
      const SweepPlan& P = fwd ? M->fwd : M->bwd;
      if (A->sym) {
        InPlaceSymmetricSor op{u.d_ptr, u.d_ind, u.d_val, f.d_ptr, f.d_ind, f.d_val, M->d_sdiag,
                           b, x, M->d_tmp, omega, ratio, fwd, true};
        all_rows_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, op);
        SB2_CUDA_TRY(cudaGetLastError());
        op.start = false;
        SB2_TRY(run_in_place(P, n, op, s));
      } else {
        SB2_TRY(run_in_place(P, n, InPlaceSor{f.d_ptr, f.d_ind, f.d_val, A->d_diag, b, x, omega, rest}, s));
      }
    }
    cur = x;
  }
  for (int l = 0, done = 0; l < launches && M->form == kFormSweep; l++, done += 2) {
    const int sweeps = done + 1 < total ? 2 : 1;
    const bool fwd[2] = {done < nf, done + 1 < nf};
    const SweepPlan* const plan[2] = {fwd[0] ? &M->fwd : &M->bwd, fwd[1] ? &M->fwd : &M->bwd};
    const bool into_x = x0 ? l % 2 == 1 : (launches - 1 - l) % 2 == 0;
    double* last = into_x ? x : M->d_tmp;
    if (A->sym) {
      SB2_TRY(launch_sweeps(G, sweeps, plan, fwd, last,
                            SymmetricSor{u.d_ind, u.d_val, f.d_ind, f.d_val, M->d_sdiag, b, cur, omega, ratio}, late, s));
    } else {
      SB2_TRY(launch_sweeps(G, sweeps, plan, fwd, last,
                            GeneralSor{f.d_ind, f.d_val, A->d_diag, b, cur, omega, rest}, late, s));
    }
    cur = last;
  }
  if (launches == 0 && !x0) SB2_CUDA_TRY(cudaMemsetAsync(x, 0, sizeof(double) * n, s));
  if (launches > 0 && cur != x)
    SB2_CUDA_TRY(cudaMemcpyAsync(x, cur, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
  return SB2_OK;
}

// Levels of a gather sweep: row j waits for every row it reads; rows are
// visited in dependency order (increasing j when reads are of smaller
// rows, decreasing otherwise).
static void gather_levels(int n, const std::vector<int>& ptr, const std::vector<int>& ind,
                          bool ascending, std::vector<int>& level) {
  level.assign(n, 0);
  for (int s = 0; s < n; s++) {
    const int j = ascending ? s : n - 1 - s;
    int lev = 0;
    for (int k = ptr[j]; k < ptr[j + 1]; k++) lev = std::max(lev, level[ind[k]] + 1);
    level[j] = lev;
  }
}

static int upload_sweep(sb2_precond* M, const std::vector<int>& ptr,
                        const std::vector<int>& ind, const std::vector<double>& val,
                        bool ascending, GatherSweep* S) {
  const SweepGrid& G = M->grid;
  std::vector<int> level, pos(std::max(G.n, 1));
  gather_levels(G.n, ptr, ind, ascending, level);
  if (M->form < 0) M->form = sweep_form(G.n, count_levels(level), (double)ind.size() / std::max(G.n, 1), 2);
  const bool levels = M->form == kFormLevels;
  SweepOrder order;
  std::vector<int> lvl;
  if (levels) make_level_order(G.n, level, &order.rows, &lvl);
  else make_sweep_order(G, level, &order);
  // the values are by position, or by row when run by levels
  for (int i = 0; i < G.n; i++) pos[order.rows[i]] = levels ? order.rows[i] : i;
  // the lists in the order the rows are taken
  std::vector<int> pind;
  std::vector<double> pval;
  std::vector<int4> span(std::max(G.n, 1));
  pind.reserve(ind.size());
  pval.reserve(val.size());
  for (int i = 0; i < G.n; i++) {
    const int j = order.rows[i], k0 = (int)pind.size();
    for (int k = ptr[j]; k < ptr[j + 1]; k++) pind.push_back(pos[ind[k]]);
    pval.insert(pval.end(), val.begin() + ptr[j], val.begin() + ptr[j + 1]);
    span[i] = make_int4(k0, (int)pind.size(), 0, 0);
  }
  if (levels) {
    std::vector<int> lists(G.n + 1, 0);
    for (int i = 0; i < G.n; i++) lists[i + 1] = span[i].y;
    SB2_TRY(upload_level_plan(G.n, order.rows, lvl, lists.data(), &S->plan));
  } else {
    SB2_TRY(upload_sweep_plan(G, order, span.data(), &S->plan));
    SB2_TRY(place_rows(G, S->plan, nullptr, nullptr, nullptr));
  }
  for (int i = 0; i < G.n; i++) S->plan.max_len = std::max(S->plan.max_len, span[i].y - span[i].x);
  const size_t nz = pind.size();
  SB2_CUDA_TRY(cudaMalloc(&S->d_ind, sizeof(int) * std::max<size_t>(nz, 1)));
  SB2_CUDA_TRY(cudaMalloc(&S->d_val, sizeof(double) * std::max<size_t>(nz, 1)));
  if (nz) {
    SB2_CUDA_TRY(cudaMemcpy(S->d_ind, pind.data(), sizeof(int) * nz, cudaMemcpyHostToDevice));
    SB2_CUDA_TRY(cudaMemcpy(S->d_val, pval.data(), sizeof(double) * nz, cudaMemcpyHostToDevice));
  }
  return SB2_OK;
}

// Update lists of a column scatter: entry (i -> c, v) for the rows i in the
// order the sequential loop visits them, each row's entries in stored order.
struct ListBuilder {
  int n;
  std::vector<int> to, from;
  std::vector<double> v;
  explicit ListBuilder(int order) : n(order) {}
  void add(int target, int source, double value) {
    to.push_back(target);
    from.push_back(source);
    v.push_back(value);
  }
  // the lists one after the other, each in the order of its entries' arrival
  void flatten(std::vector<int>& ptr, std::vector<int>& ind, std::vector<double>& val) const {
    ptr.assign(n + 1, 0);
    for (int j : to) ptr[j + 1]++;
    for (int j = 0; j < n; j++) ptr[j + 1] += ptr[j];
    ind.resize(to.size());
    val.resize(to.size());
    std::vector<int> at(ptr.begin(), ptr.end() - 1);
    for (size_t e = 0; e < to.size(); e++) {
      const int q = at[to[e]]++;
      ind[q] = from[e];
      val[q] = v[e];
    }
  }
};

static bool is_permutation(int n, const int* p) {
  std::vector<char> seen(n, 0);
  for (int i = 0; i < n; i++) {
    if (p[i] < 0 || p[i] >= n || seen[p[i]]) return false;
    seen[p[i]] = 1;
  }
  return true;
}

// Builds every sweep of the factor (host arrays in Seldon's stored order).
static int plan_ilut(sb2_precond* M, int n, const int* fp, const int* fi, const double* fv,
                     const int* prow, const int* pcol) {
  if (fp[0] != 0) return SB2_ERR_INVALID_CSR;
  for (int i = 0; i < n; i++)
    if (fp[i + 1] < fp[i]) return SB2_ERR_INVALID_CSR;
  if (!is_permutation(n, prow) || (!M->ilu_sym && !is_permutation(n, pcol)))
    return SB2_ERR_INVALID_VALUE;
  SB2_TRY(make_sweep_grid(n, &M->grid));
  std::vector<double> dinv(n);
  std::vector<int> ptr, ind;
  std::vector<double> val;
  if (M->ilu_sym) {
    // row i: 1/D(i) at the first position, then row i of L^T (columns > i)
    ListBuilder fwd(n);
    std::vector<int> bptr(n + 1, 0), bind;
    std::vector<double> bval;
    for (int i = 0; i < n; i++) {
      if (fp[i + 1] <= fp[i]) return SB2_ERR_INVALID_CSR;
      dinv[i] = fv[fp[i]];
      for (int k = fp[i] + 1; k < fp[i + 1]; k++) {
        if (fi[k] <= i || fi[k] >= n) return SB2_ERR_INVALID_CSR;
        fwd.add(fi[k], i, fv[k]);  // L y = b: x(j) -= A(i,k) x(i), i increasing
        bind.push_back(fi[k]);
        bval.push_back(fv[k]);
      }
      bptr[i + 1] = (int)bind.size();
    }
    fwd.flatten(ptr, ind, val);
    SB2_TRY(upload_sweep(M, ptr, ind, val, true, &M->s_lf));
    SB2_TRY(upload_sweep(M, bptr, bind, bval, false, &M->s_ub));
  } else {
    // row i: L part (columns < i), then 1/U(i,i), then the U part
    std::vector<int> lptr(n + 1, 0), lind, uptr(n + 1, 0), uind;
    std::vector<double> lval, uval;
    ListBuilder utf(n), ltb(n);
    std::vector<int> dpos(n);
    for (int i = 0; i < n; i++) {
      int k = fp[i];
      while (k < fp[i + 1] && fi[k] < i) {
        if (fi[k] < 0) return SB2_ERR_INVALID_CSR;
        lind.push_back(fi[k]);
        lval.push_back(fv[k]);
        k++;
      }
      if (k == fp[i + 1]) return SB2_ERR_INVALID_CSR;  // no diagonal position
      dpos[i] = k;
      dinv[i] = fv[k];
      for (int q = k + 1; q < fp[i + 1]; q++) {
        if (fi[q] <= i || fi[q] >= n) return SB2_ERR_INVALID_CSR;
        uind.push_back(fi[q]);
        uval.push_back(fv[q]);
        utf.add(fi[q], i, fv[q]);  // U^T: x(c) -= U(i,c) x(i), i increasing
      }
      lptr[i + 1] = (int)lind.size();
      uptr[i + 1] = (int)uind.size();
    }
    for (int i = n - 1; i >= 0; i--)  // L^T: x(k) -= L(i,k) x(i), i decreasing
      for (int k = fp[i]; k < dpos[i]; k++) ltb.add(fi[k], i, fv[k]);
    SB2_TRY(upload_sweep(M, lptr, lind, lval, true, &M->s_lf));
    SB2_TRY(upload_sweep(M, uptr, uind, uval, false, &M->s_ub));
    utf.flatten(ptr, ind, val);
    SB2_TRY(upload_sweep(M, ptr, ind, val, true, &M->s_utf));
    ltb.flatten(ptr, ind, val);
    SB2_TRY(upload_sweep(M, ptr, ind, val, false, &M->s_ltb));
  }
  std::vector<int> iprow(n);
  for (int i = 0; i < n; i++) iprow[prow[i]] = i;
  SB2_CUDA_TRY(cudaMalloc(&M->d_dinv, sizeof(double) * std::max(n, 1)));
  SB2_CUDA_TRY(cudaMalloc(&M->d_iprow, sizeof(int) * std::max(n, 1)));
  SB2_CUDA_TRY(cudaMemcpy(M->d_dinv, dinv.data(), sizeof(double) * n, cudaMemcpyHostToDevice));
  SB2_CUDA_TRY(cudaMemcpy(M->d_iprow, iprow.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
  if (!M->ilu_sym) {
    SB2_CUDA_TRY(cudaMalloc(&M->d_pcol, sizeof(int) * std::max(n, 1)));
    SB2_CUDA_TRY(cudaMemcpy(M->d_pcol, pcol, sizeof(int) * n, cudaMemcpyHostToDevice));
  }
  SB2_CUDA_TRY(cudaStreamSynchronize(nullptr));  // complete before any stream reads it
  return SB2_OK;
}

// GetIlu0 on the device: rows in levels of their L dependencies, each row
// factored by one thread in the reference's operation order.  The factor
// (A's pattern, Seldon's ArrayRowSparse layout) is returned on the host.
static int ilu0_factor(const sb2_csr* A, int modified, std::vector<int>& ptr,
                       std::vector<int>& ind, std::vector<double>& val, cudaStream_t s) {
  const int n = A->m;
  const CsrArrays& f = A->full;
  ptr.resize(n + 1);
  ind.resize(f.nnz);
  val.resize(f.nnz);
  SB2_CUDA_TRY(cudaMemcpy(ptr.data(), f.d_ptr, sizeof(int) * (n + 1), cudaMemcpyDeviceToHost));
  if (f.nnz) {
    SB2_CUDA_TRY(cudaMemcpy(ind.data(), f.d_ind, sizeof(int) * f.nnz, cudaMemcpyDeviceToHost));
  }
  // GetIlu0 reads the row prefix before the diagonal as L and needs every
  // row sorted, with its diagonal, and no repeated column
  std::vector<int> dpos(n, -1), lptr(n + 1, 0), lind;
  for (int i = 0; i < n; i++) {
    for (int k = ptr[i]; k < ptr[i + 1]; k++) {
      if (ind[k] < 0 || ind[k] >= n) return SB2_ERR_INVALID_CSR;
      if (k > ptr[i] && ind[k] <= ind[k - 1]) return SB2_ERR_INVALID_CSR;
      if (ind[k] == i) dpos[i] = k;
      if (ind[k] < i) lind.push_back(ind[k]);
    }
    if (dpos[i] < 0) return SB2_ERR_INVALID_CSR;
    lptr[i + 1] = (int)lind.size();
  }
  std::vector<int> level;
  gather_levels(n, lptr, lind, true, level);
  LevelPlan plan;
  int st = upload_plan(level, n, &plan);
  double* d_val = nullptr;
  int *d_dpos = nullptr, *d_status = nullptr;
  cudaError_t e = cudaMalloc(&d_val, sizeof(double) * std::max<long long>(f.nnz, 1));
  if (e == cudaSuccess) e = cudaMalloc(&d_dpos, sizeof(int) * std::max(n, 1));
  if (e == cudaSuccess) e = cudaMalloc(&d_status, sizeof(int));
  if (e == cudaSuccess && f.nnz)
    e = cudaMemcpyAsync(d_val, f.d_val, sizeof(double) * f.nnz, cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d_dpos, dpos.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_status, 0, sizeof(int), s);
  if (st == SB2_OK) st = map_cuda_error(e);
  int status = 0;
  if (st == SB2_OK)
    st = run_factor_levels(plan, n, Ilu0Row{f.d_ptr, f.d_ind, d_val, d_dpos, d_status, modified}, s);
  if (st == SB2_OK) {
    e = cudaMemcpyAsync(&status, d_status, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && f.nnz)
      e = cudaMemcpyAsync(val.data(), d_val, sizeof(double) * f.nnz, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    st = map_cuda_error(e);
  }
  if (st == SB2_OK && status != 0) st = SB2_ERR_INVALID_VALUE;  // zero pivot
  cudaFree(d_val);
  cudaFree(d_dpos);
  cudaFree(d_status);
  plan.release();
  return st;
}

// IlutPreconditioning::Solve / TransSolve (IlutPreconditioning.cxx:329-374):
// both sweeps and both permutations in one launch.  Seldon's t[prow[i]] = r[i]
// and z[i] = t[prow[i]] are t[j] = r[iprow[j]] and z[iprow[j]] = t[j] for the
// thread that owns row j.
static int ilut_apply(sb2_precond* M, bool trans, const double* r, double* z, int late,
                      cudaStream_t s) {
  const bool sym = M->ilu_sym != 0;
  const GatherSweep& first = !sym && trans ? M->s_utf : M->s_lf;
  const GatherSweep& second = !sym && trans ? M->s_ltb : M->s_ub;
  const double* d = M->d_dinv;
  FactorSolve op{{first.d_ind, second.d_ind},
                 {first.d_val, second.d_val},
                 {nullptr, sym ? d : nullptr},
                 {!sym && trans ? d : nullptr, !sym && !trans ? d : nullptr},
                 r, !sym && trans ? M->d_pcol : M->d_iprow,
                 z, !sym && !trans ? M->d_pcol : M->d_iprow};
  const SweepPlan* const plan[2] = {&first.plan, &second.plan};
  const bool fwd[2] = {true, false};
  if (M->form == kFormLevels) {
    const SweepGrid& G = M->grid;
    SB2_TRY(run_levels(first.plan, G.n, 0, true, LevelSpan{first.plan.d_lists, nullptr, nullptr}, nullptr, G.d_new[0],
                       op, s));
    return run_levels(second.plan, G.n, 1, false, LevelSpan{second.plan.d_lists, nullptr, nullptr}, G.d_new[0],
                      G.d_new[1], op, s);
  }
  return launch_sweeps(M->grid, 2, plan, fwd, nullptr, op, late, s);
}

int precond_kind(const sb2_precond* M) { return M->kind; }
int precond_n(const sb2_precond* M) { return M->kind == SB2_PRECOND_ILUT ? M->n_ilu : M->A->m; }
const sb2_csr* precond_matrix(const sb2_precond* M) { return M->A; }

static int apply(const sb2_precond* cM, bool trans, const double* r, double* z, int late,
                 cudaStream_t s) {
  sb2_precond* M = const_cast<sb2_precond*>(cM);
  if (M->kind == SB2_PRECOND_ILUT) return M->n_ilu ? ilut_apply(M, trans, r, z, late, s) : SB2_OK;
  const int n = M->A->m;
  if (n == 0) return SB2_OK;
  if (M->kind == SB2_PRECOND_IDENTITY) {
    SB2_CUDA_TRY(cudaMemcpyAsync(z, r, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    return SB2_OK;
  }
  if (M->kind == SB2_PRECOND_JACOBI) {
    SB2_TRY(ensure_diag(M->A));
    int g = std::min((n + 255) / 256, num_sms(current_device()) * 8);
    jacobi_kernel<<<g, 256, 0, s>>>(n, r, M->A->d_diag, z);
    SB2_CUDA_TRY(cudaGetLastError());
    return SB2_OK;
  }
  // SorPreconditioner::Solve / TransSolve (Precond_Ssor.cxx:62-90)
  const int type = M->symmetric ? 0 : (trans ? 3 : 2);
  return sor_apply(M, nullptr, z, r, M->omega, M->nb_iter, type, late, s);
}

// An apply inside a solver.
int precond_apply(const sb2_precond* M, bool trans, const double* r, double* z, cudaStream_t s) {
  return apply(M, trans, r, z, kStLateSolve, s);
}

// Whether a wait of the preconditioner's sweeps ran out since the word was
// last read, which clears it (synchronizes the stream).
static int read_late(const sb2_precond* M, int word, unsigned* late, cudaStream_t s) {
  *late = 0;
  if (!M->grid.d_state) return SB2_OK;
  unsigned* d = M->grid.d_state + word;
  SB2_CUDA_TRY(cudaMemcpyAsync(late, d, sizeof(*late), cudaMemcpyDeviceToHost, s));
  SB2_CUDA_TRY(cudaStreamSynchronize(s));
  if (*late) SB2_CUDA_TRY(cudaMemsetAsync(d, 0, sizeof(*late), s));
  return SB2_OK;
}

// A solver with M starts: what an earlier one that ended with an error left in
// its word is not this one's.
int precond_begin(const sb2_precond* M, cudaStream_t s) {
  if (!M || !M->grid.d_state) return SB2_OK;
  SB2_CUDA_TRY(cudaMemsetAsync(M->grid.d_state + kStLateSolve, 0, sizeof(unsigned), s));
  return SB2_OK;
}

// A solver with M ends: whether a wait ran out in it.
int precond_check(const sb2_precond* M, cudaStream_t s) {
  unsigned late = 0;
  if (M) SB2_TRY(read_late(M, kStLateSolve, &late, s));
  return late ? SB2_ERR_TIMEOUT : SB2_OK;
}

}  // namespace sb2

using namespace sb2;

extern "C" {

int sb2_precond_create(const sb2_csr* A, int kind, double omega, int nb_iter,
                       int symmetric, sb2_precond** out) try {
  if (!out || !A) return SB2_ERR_INVALID_VALUE;
  *out = nullptr;
  if (kind < SB2_PRECOND_IDENTITY || kind > SB2_PRECOND_SOR) return SB2_ERR_INVALID_VALUE;
  if (A->m != A->n) return SB2_ERR_INVALID_VALUE;
  std::unique_ptr<sb2_precond, int (*)(sb2_precond*)> M(new sb2_precond(),
                                                         sb2_precond_destroy);
  M->A = A;
  M->kind = kind;
  M->omega = omega;
  M->nb_iter = nb_iter;
  M->symmetric = symmetric ? 1 : 0;
  if (kind == SB2_PRECOND_JACOBI) SB2_TRY(ensure_diag(A));
  *out = M.release();
  return SB2_OK;
} SB2_CATCH

int sb2_precond_create_ilut(const sb2_csr* A, int n, const int* fptr, const int* find,
                            const double* fval, const int* perm_row, const int* perm_col,
                            int symmetric, sb2_precond** out) try {
  SB2_TRACE("sb2_precond_create_ilut");
  if (!out || n < 0 || (n > 0 && (!fptr || !perm_row || (!symmetric && !perm_col))))
    return SB2_ERR_INVALID_VALUE;
  *out = nullptr;
  if (A && (A->m != n || A->n != n)) return SB2_ERR_INVALID_VALUE;
  if (n > 0 && fptr[n] > 0 && (!find || !fval)) return SB2_ERR_INVALID_VALUE;
  // every index the sweeps read is checked while they are built
  std::unique_ptr<sb2_precond, int (*)(sb2_precond*)> M(new sb2_precond(),
                                                         sb2_precond_destroy);
  M->A = A;
  M->kind = SB2_PRECOND_ILUT;
  M->n_ilu = n;
  M->ilu_sym = symmetric ? 1 : 0;
  if (n > 0) SB2_TRY(plan_ilut(M.get(), n, fptr, find, fval, perm_row, perm_col));
  *out = M.release();
  return SB2_OK;
} SB2_CATCH

int sb2_precond_create_ilu0(const sb2_csr* A, int modified, void* stream, sb2_precond** out) try {
  SB2_TRACE("sb2_precond_create_ilu0");
  if (!out || !A || A->m != A->n || A->sym) return SB2_ERR_INVALID_VALUE;
  *out = nullptr;
  const int n = A->m;
  std::vector<int> ptr, ind;
  std::vector<double> val;
  if (n > 0) SB2_TRY(ilu0_factor(A, modified ? 1 : 0, ptr, ind, val, (cudaStream_t)stream));
  std::vector<int> ident(std::max(n, 1));
  for (int i = 0; i < n; i++) ident[i] = i;
  if (ptr.empty()) ptr.assign(1, 0);
  // the factor no longer needs A: like the reference's preconditioner, it
  // applies to whichever matrix of order n the solver is given
  return sb2_precond_create_ilut(nullptr, n, ptr.data(), ind.empty() ? nullptr : ind.data(),
                                 val.empty() ? nullptr : val.data(), ident.data(), ident.data(), 0,
                                 out);
} SB2_CATCH

int sb2_precond_destroy(sb2_precond* M) try {
  if (!M) return SB2_OK;
  M->grid.release();
  M->fwd.release();
  M->bwd.release();
  cudaFree(M->d_sdiag);
  cudaFree(M->d_tmp);
  M->s_lf.release();
  M->s_ub.release();
  M->s_utf.release();
  M->s_ltb.release();
  cudaFree(M->d_iprow);
  cudaFree(M->d_pcol);
  cudaFree(M->d_dinv);
  delete M;
  return SB2_OK;
} SB2_CATCH

int sb2_precond_solve(const sb2_precond* M, const double* r, double* z, void* stream) try {
  SB2_TRACE("sb2_precond_solve");
  if (!M || (precond_n(M) > 0 && (!r || !z)) || (r == z && precond_n(M) > 0))
    return SB2_ERR_INVALID_VALUE;
  return apply(M, false, r, z, kStLateApply, (cudaStream_t)stream);
} SB2_CATCH

int sb2_precond_trans_solve(const sb2_precond* M, const double* r, double* z, void* stream) try {
  SB2_TRACE("sb2_precond_trans_solve");
  if (!M || (precond_n(M) > 0 && (!r || !z)) || (r == z && precond_n(M) > 0))
    return SB2_ERR_INVALID_VALUE;
  return apply(M, true, r, z, kStLateApply, (cudaStream_t)stream);
} SB2_CATCH

int sb2_precond_status(const sb2_precond* M, void* stream, int* status) try {
  if (!M || !status) return SB2_ERR_INVALID_VALUE;
  unsigned late = 0;
  SB2_TRY(read_late(M, kStLateApply, &late, (cudaStream_t)stream));
  if (!M->grid.d_state) SB2_CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
  *status = late ? 1 : 0;
  return SB2_OK;
} SB2_CATCH

int sb2_sor(const sb2_csr* A, double* x, const double* b, double omega, int iter,
            int type_ssor, void* stream) try {
  SB2_TRACE("sb2_sor");
  if (!A || A->m != A->n || (A->m > 0 && (!x || !b)) || x == b) return SB2_ERR_INVALID_VALUE;
  sb2_precond tmp;
  tmp.A = A;
  tmp.kind = SB2_PRECOND_SOR;
  int st = sor_apply(&tmp, x, x, b, omega, iter, type_ssor, kStLateSolve, (cudaStream_t)stream);
  // the plan is released after the stream has consumed it
  const int late = precond_check(&tmp, (cudaStream_t)stream);
  cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
  tmp.grid.release();
  tmp.fwd.release();
  tmp.bwd.release();
  cudaFree(tmp.d_sdiag);
  cudaFree(tmp.d_tmp);
  if (st == SB2_OK && e != cudaSuccess) st = map_cuda_error(e);
  if (st == SB2_OK) st = late;
  return st;
} SB2_CATCH

}  // extern "C"
