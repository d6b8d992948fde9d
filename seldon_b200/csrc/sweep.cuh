// Sequential sweeps (Gauss-Seidel, triangular solves) as one persistent launch
// whose rows wait for the values they read, not for levels.
//
// The rows are cut into one contiguous block per CTA.  Inside a block they
// are ordered by dependency level and dealt to the warps in items of up to 32
// rows of one level; a warp takes its items in order, one row per lane.
//  - Values of the CTA's own block live in its shared memory.  The items of
//    one level form a step with an mbarrier, and an item waits for the step
//    before its own, suspended by the hardware.
//  - Values of other blocks come through global memory.  The vector a sweep
//    writes was filled with a reserved NaN, so a value announces itself: the
//    row polls the entries it needs until they differ from the fill.  No
//    flag, fence or grid barrier stands between a value and its use.  The
//    vector is in the order the rows are taken: an item's values are one run
//    that is written once.  (By row, a line held values of 16 levels, and a
//    line that other SMs poll is slow to write: 3 us from CTA to CTA.)
// Each row repeats the reference's operations in the reference's order, so
// the result does not depend on the timing.
//
// What bounds it is the chain of dependent rows.  Inside a block a level costs
// what one row does between its turn and its barrier (430 cycles for three
// entries, measured with clock64): its loads, products, sums and exact
// division; everything that reads only old values comes before, while the
// warp's predecessors still work.  From one CTA to the next a value takes about
// a microsecond.  Two sweeps on a 7-point grid, against a graph of one launch
// per level before: ILU(0) apply 96^3 408 us (2070), 128^3 673 us (2970); SSOR on
// 64^3 with symmetric storage 288 us (1446), with general storage 265 us (1547).
// 384 threads for three-entry and symmetric rows: with 256 the small grids lose
// (ILU(0) 16^3 54 us against 45), with 768 and more the registers spill on the
// chain (83 us); general rows hold more and spill at 384 already (64^3 307 us).
// Rows of more entries than a lane holds have a kernel of their own (LONG): the
// others' is faster without its code (ILU(0) 64^3 199 us, 211 with), and it loads
// ahead: ILU(0) of 27-entry rows, 40^3 657 us, 1697 entry by entry.
//
// Progress: all CTAs are resident (cooperative launch), a warp's items are in
// level order and a row reads rows of smaller levels only.  Every wait is
// bounded: when no CTA has made progress for the wait limit (a long row that is
// being summed is progress), the waiting warp sets the status words and the
// grid leaves; the rows it did not finish come out as NaN.
#pragma once

#include <algorithm>
#include <vector>

#include "sb2_internal.cuh"

namespace sb2 {

constexpr int kSweepMaxCtas = 148;
constexpr int kSweepStep = 32;   // items of one step at most
constexpr int kSweepRing = 64;   // step barriers (more than the warps of a CTA)
constexpr int kSweepSmem = 224 * 1024;  // most shared memory a CTA takes for its values
constexpr int kSweepLong = 256;   // threads of a CTA where rows hold more entries than a lane does
constexpr int kSweepNote = 4096;  // entries of a long row between two notes of progress
// Words of SweepGrid::d_state: the grid leaves; a wait ran out since the word
// was last read, in a solver's apply and in a caller's own; then one word a
// CTA that changes as it gets on.
constexpr int kStLeave = 0, kStLateSolve = 1, kStLateApply = 2, kStProgress = 3;
// The fill: a signalling NaN, which no arithmetic produces.  A value that
// was copied from the caller with these very bits is stored as the quiet NaN.
constexpr unsigned long long kSweepFill = 0x7ff4b2005e1d0001ull;

// The rows of one sweep in the order they are taken (one allocation).
struct SweepPlan {
  void* d_buf = nullptr;
  int4* d_span = nullptr;     // [n] entry ranges of each position's row
  int4* d_item = nullptr;     // [items] first position, rows, step, arrivals (below)
  int* d_rows = nullptr;      // [n] row of each position
  int* d_pos = nullptr;       // [n] position of each row
  int* d_cta_item = nullptr;  // [ctas + 1] first item of each CTA
  int* d_steps = nullptr;     // [ctas] steps of each CTA
  int max_len = 0;            // entries of the longest row
  // by levels (SweepForm): d_rows in level order, and
  std::vector<int> h_lvl;     // [levels + 1] first position of each level
  int* d_lvl = nullptr;       // the same on the device
  int* d_lists = nullptr;     // [n + 1] first entry of each position's list
  void release() {
    cudaFree(d_buf);
    *this = SweepPlan();
  }
};

// The row blocks shared by all sweeps of one preconditioner, and the vectors
// the sweeps write (one allocation).
struct SweepGrid {
  int n = 0, ctas = 0, max_rows = 0;
  std::vector<int> h_blk;     // [ctas + 1] first row of each block
  double* d_new[2] = {nullptr, nullptr};
  int* d_blk = nullptr;
  unsigned* d_state = nullptr;  // [kStProgress + kSweepMaxCtas]
  void release() {
    cudaFree(d_new[0]);
    d_new[0] = d_new[1] = nullptr;
    d_blk = nullptr;
    d_state = nullptr;
  }
};

struct SweepPhase {
  const int* rows;
  const int4* span;
  const int4* item;
  const int* cta_item;
  const int* steps;
  const int* pos;       // position of each row here
  const int* pos_prev;  // and in the sweep before (of the same launch)
  int forward;     // new values are those of smaller rows
  double* out;     // values of this phase by position (filled before the launch)
};

struct SweepArgs {
  const int* blk;
  int max_rows;
  int nph;          // 1 or 2 sweeps in this launch
  double* result;   // the last sweep's values by row (may be null)
  SweepPhase ph[2];
  unsigned* state;
  int late;         // the word of state that tells of a wait that ran out
  unsigned long long wait_ns;
};

// ------------------------------------------------------------------ planning

// Cuts n rows into blocks of about 2048, one CTA each, and larger ones where
// the SMs run out.  SSOR on 7-point grids with a first form of the kernel, 2048
// / 4096 / 8192 rows a block: 20^3 123 / 177 / 238 us, 40^3 244 / 273 / 423,
// 64^3 395 / 413 / 499; smaller blocks add CTAs for a chain of rows to cross
// (1024: 433 us at 64^3).
inline int make_sweep_grid(int n, SweepGrid* G) {
  G->n = n;
  const int most = std::min(kSweepMaxCtas, num_sms(current_device()));
  G->ctas = std::max(1, std::min(most, (n + 2047) / 2048));
  const int per = (n + G->ctas - 1) / G->ctas;
  G->max_rows = per;
  G->h_blk.resize(G->ctas + 1);
  for (int c = 0; c <= G->ctas; c++) G->h_blk[c] = (int)std::min<long long>((long long)c * per, n);
  // d_new, then d_blk and d_state
  const size_t len = std::max(n, 1), words = G->ctas + 1 + kStProgress + kSweepMaxCtas;
  SB2_CUDA_TRY(cudaMalloc(&G->d_new[0], 2 * sizeof(double) * len + sizeof(int) * words));
  G->d_new[1] = G->d_new[0] + len;
  G->d_blk = reinterpret_cast<int*>(G->d_new[1] + len);
  G->d_state = reinterpret_cast<unsigned*>(G->d_blk + G->ctas + 1);
  std::vector<int> head(words, 0);
  std::copy(G->h_blk.begin(), G->h_blk.end(), head.begin());
  SB2_CUDA_TRY(cudaMemcpy(G->d_blk, head.data(), sizeof(int) * words, cudaMemcpyHostToDevice));
  return SB2_OK;
}

// The order of one sweep on the host.
struct SweepOrder {
  std::vector<int> rows, cta_item, steps;
  std::vector<int4> item;
};

// Each block's rows by level (increasing row in a level) and the items they
// make.  A call of SOR plans on the way, so that the passes stay within a block:
// 885,000 rows take 3 ms (11 with one sort over all rows).
inline void make_sweep_order(const SweepGrid& G, const std::vector<int>& level, SweepOrder* O) {
  const int n = G.n;
  O->rows.resize(std::max(n, 1));
  O->cta_item.assign(G.ctas + 1, 0);
  O->steps.assign(G.ctas, 0);
  O->item.clear();
  std::vector<int> at;
  for (int c = 0; c < G.ctas; c++) {
    const int r0 = G.h_blk[c], r1 = G.h_blk[c + 1];
    O->cta_item[c] = (int)O->item.size();
    if (r0 == r1) continue;
    int* rows = O->rows.data();
    const auto range = std::minmax_element(level.begin() + r0, level.begin() + r1);
    const int lo = *range.first;
    const long long span = (long long)*range.second - lo + 1;
    if (span <= 4LL * (r1 - r0)) {
      at.assign(span + 1, 0);
      for (int i = r0; i < r1; i++) at[level[i] - lo + 1]++;
      for (long long l = 0; l < span; l++) at[l + 1] += at[l];
      for (int i = r0; i < r1; i++) rows[r0 + at[level[i] - lo]++] = i;
    } else {
      for (int i = r0; i < r1; i++) rows[i] = i;
      std::stable_sort(rows + r0, rows + r1, [&](int a, int b) { return level[a] < level[b]; });
    }
    for (int i = r0; i < r1;) {
      // a step: up to kSweepStep items of one level; its last item makes up
      // the barrier's count
      const int lev = level[rows[i]];
      int q = 0;
      for (; q < kSweepStep && i < r1 && level[rows[i]] == lev; q++) {
        const int s = i;
        while (i < r1 && i - s < 32 && level[rows[i]] == lev) i++;
        O->item.push_back(make_int4(s, i - s, O->steps[c], 1));
      }
      O->item.back().w = kSweepStep - (q - 1);
      O->steps[c]++;
    }
  }
  O->cta_item[G.ctas] = (int)O->item.size();
}

// The order on the device.  d_pos and, without `span`, d_span are for the
// caller to fill (sweep_place_kernel).
inline int upload_sweep_plan(const SweepGrid& G, const SweepOrder& O, const int4* span, SweepPlan* P) {
  const size_t n = std::max(G.n, 1), items = O.item.size(), words = 2 * (size_t)G.ctas + 1;
  SB2_CUDA_TRY(cudaMalloc(&P->d_buf, sizeof(int4) * (n + items) + sizeof(int) * (2 * n + words)));
  P->d_span = static_cast<int4*>(P->d_buf);
  P->d_item = P->d_span + n;
  P->d_rows = reinterpret_cast<int*>(P->d_item + items);
  P->d_pos = P->d_rows + n;
  P->d_cta_item = P->d_pos + n;
  P->d_steps = P->d_cta_item + G.ctas + 1;
  std::vector<int> tail(O.cta_item);
  tail.insert(tail.end(), O.steps.begin(), O.steps.end());
  if (span) SB2_CUDA_TRY(cudaMemcpy(P->d_span, span, sizeof(int4) * G.n, cudaMemcpyHostToDevice));
  SB2_CUDA_TRY(cudaMemcpy(P->d_item, O.item.data(), sizeof(int4) * items, cudaMemcpyHostToDevice));
  SB2_CUDA_TRY(cudaMemcpy(P->d_rows, O.rows.data(), sizeof(int) * G.n, cudaMemcpyHostToDevice));
  SB2_CUDA_TRY(cudaMemcpy(P->d_cta_item, tail.data(), sizeof(int) * words, cudaMemcpyHostToDevice));
  return SB2_OK;
}

// ------------------------------------------------------------------ by levels

constexpr int kLevelCta = 65536;  // rows up to which one CTA takes all levels of a sweep in place

// How a sweep runs.  Bit for bit the same; what differs is what they wait for.
enum SweepForm {
  kFormSweep = 0,   // rows that wait for their values, above
  kFormLevels = 1,  // a launch per level
  kFormInPlace = 2  // x in place (SOR): all levels in one CTA, or a plain launch each
};

// The form for n rows of `entries` on the average in `levels`, kind 0 SOR, 1 SOR
// on symmetric storage, 2 a factor's solves.
//  - Few wide levels leave the sweep's one CTA per SM waiting for memory, where a
//    launch per level (2.4 us, its own loads ahead of the one before) fills the
//    GPU.  Forward SOR, sweep / launches: 1000^2 grid in red-black order, 2 levels,
//    189 / 26 us; 300^2 in random order, 14 levels, 73 / 37; 1000^2 so, 15 levels, 262 /
//    66; 10^6 diagonal rows 68 / 13.  Many levels: 40^3 convection-diffusion, 118, 94 /
//    288.  A sweep moves 5 rows a ns, which is a launch's time at 12,000 rows a
//    level.
//  - Rows of many entries in narrow levels are bound by the instructions of the
//    few lanes that have a row; one CTA whose operand stays in L1 needs the fewest.
//    SSOR, sweep / one CTA: 20^3 grid of 27-entry rows, symmetric storage, 1.80 / 1.01
//    ms, 40^3 4.0 / 3.2; bands of 31 entries, 2000 rows 6.6 / 4.9, of 81, 20,000 rows
//    412 / 196.  General storage with 60 and 234 rows a level 1.0 / 0.96, 2.3 / 4.4 ms;
//    with 262,144 rows more than one CTA is needed.
//  - Very wide levels are bound by their bytes, of which x in place takes the
//    fewest: SSOR, launches / in place: red-black 1000^2 54 / 42 us, 10^6 diagonal rows
//    29 / 21; random order, 66,667 rows a level, 144 / 183.
inline SweepForm sweep_form(int n, int levels, double entries, int kind) {
  if (kind != 2 && n >= 200000LL * levels) return kFormInPlace;
  if ((levels <= 16 && n >= 4096) || n >= 16000LL * levels) return kFormLevels;
  if (kind != 2 && n <= kLevelCta && entries >= 16.0 && (kind == 1 || n <= 32LL * levels)) return kFormInPlace;
  return kFormSweep;
}

// All rows by level (increasing row in a level), and the levels' offsets.
inline void make_level_order(int n, const std::vector<int>& level, std::vector<int>* rows,
                             std::vector<int>* lvl) {
  int levels = 0;
  for (int l : level) levels = std::max(levels, l + 1);
  lvl->assign(levels + 1, 0);
  for (int l : level) (*lvl)[l + 1]++;
  for (int l = 0; l < levels; l++) (*lvl)[l + 1] += (*lvl)[l];
  rows->resize(std::max(n, 1));
  std::vector<int> at(lvl->begin(), lvl->end());
  for (int i = 0; i < n; i++) (*rows)[at[level[i]]++] = i;
}

// lists: [n + 1] first entry of each position's list (null: the rows' own).
inline int upload_level_plan(int n, const std::vector<int>& rows, const std::vector<int>& lvl,
                             const int* lists, SweepPlan* P) {
  const size_t len = std::max(n, 1);
  SB2_CUDA_TRY(cudaMalloc(&P->d_buf, sizeof(int) * (2 * len + 1 + lvl.size())));
  P->d_rows = static_cast<int*>(P->d_buf);
  P->d_lvl = P->d_rows + len;
  P->h_lvl = lvl;
  SB2_CUDA_TRY(cudaMemcpy(P->d_rows, rows.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
  SB2_CUDA_TRY(cudaMemcpy(P->d_lvl, lvl.data(), sizeof(int) * lvl.size(), cudaMemcpyHostToDevice));
  if (lists) {
    P->d_lists = P->d_lvl + lvl.size();
    SB2_CUDA_TRY(cudaMemcpy(P->d_lists, lists, sizeof(int) * (n + 1), cudaMemcpyHostToDevice));
  }
  return SB2_OK;
}

#ifdef __CUDACC__

// ------------------------------------------------------------------ waiting

__device__ __forceinline__ bool is_fill(double v) {
  return (unsigned long long)__double_as_longlong(v) == kSweepFill;
}

// A value made by copying, never the fill.
__device__ __forceinline__ double not_fill(double v) {
  return is_fill(v) ? __longlong_as_double((long long)(kSweepFill | 0x0008000000000000ull)) : v;
}

__device__ __forceinline__ double ld_shared(unsigned at) {
  double v;
  asm volatile("ld.volatile.shared.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ void st_shared(unsigned at, double v) {
  asm volatile("st.volatile.shared.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}
__device__ __forceinline__ double ld_volatile(const double* p) {
  return *reinterpret_cast<const volatile double*>(p);
}

// Step barriers: mbarriers of this CTA.  A waiting warp is suspended by the
// hardware, where polling loops would take issue slots from the warp that the
// others wait for.
__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* b, unsigned count) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(count)
               : "memory");
}
// whether the phase of this parity is complete, suspended until it is or a
// system-defined time has passed; the second form does not wait
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n"
      " mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return ok != 0u;
}
__device__ __forceinline__ bool mbar_test_wait(unsigned long long* b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n"
      " mbarrier.test_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return ok != 0u;
}

// State of a warp's waits: gives up when the grid was told to leave, or when
// no CTA has finished an item for wait_ns.
struct SweepWait {
  unsigned* state;
  int late, ctas;
  unsigned long long wait_ns;
  __device__ __forceinline__ unsigned progress() const {
    unsigned s = 0;
    for (int c = 0; c < ctas; c++) s = s * 31u + *((volatile unsigned*)state + kStProgress + c);
    return s;
  }
  // called now and then by a waiting warp; false: leave.  (The progress words
  // are read only when the limit has passed: reading them takes microseconds.)
  __device__ __noinline__ bool go_on(unsigned long long& t0, unsigned& seen) const {
    if (*((volatile unsigned*)state + kStLeave) != 0u) return false;
    const unsigned long long t = global_timer_ns();
    if (t0 == 0ull) t0 = t;
    if (t - t0 <= wait_ns) return true;
    const unsigned p = progress() * 2u + 1u;  // never 0
    if (p != seen) {
      seen = p;
      t0 = t;
      return true;
    }
    atomicExch(state + kStLeave, 1u);
    atomicExch(state + late, 1u);
    return false;
  }
};

// The values of one vector: those of the CTA's own rows in its shared memory
// at `own`, all of them in global memory.
struct SweepSource {
  const double* g;
  unsigned own;
};

// ------------------------------------------------------------------ row operations
// An operation describes one row's new value as a sequence of entries (column,
// coefficient) to be taken in order:
//   Row r = op.load(ph, fwd, j, span)     what does not depend on other rows
//   op.entry(r, k, c, a)                  entry k of r.len; c is its column, or with
//                                         Op::kPositions the column's position
//   op.is_new(r, k, c)                    it reads this sweep's value of c
//   op.first(r, s, xj)                    xj: the row's value before the sweep
//   op.take(r, s, k, c, a, x)             entry k with the value x of column c
//   op.lead(r, s, k)                      entries 0..k-1 are taken, none new
//   op.last(r, s)                         the new value
//   op.store(r, v)                        where it goes beside
// The entries after the lead that are held in registers only add products to
// one number, so that nothing but loads, products and sums follows the row's
// turn:
//   op.skips(r, c)                        such an entry adds nothing
//   op.signed_value(r, a)                 what multiplies x
//   op.running(r, s), op.run_to(r, s, v)  that number, and what became of it

// Division by a divisor known ahead: y + z = 1 / b to twice the precision is
// made before the row's turn; then q = a y + a z is within an ulp of a / b, and
// one of Markstein's correction steps (IBM J. Res. Dev. 34, 1990: q' = q + y
// (a - b q), the remainder exact by fma) gives RN(a / b) where no intermediate
// leaves the normal range.  The full division, several hundred cycles of one
// warp, stays for the operands outside it.
struct Divisor {
  double b, y, z;  // y = 0: use the full division
  __device__ __forceinline__ explicit Divisor(double v) : b(v), y(0.0), z(0.0) {
    const double m = fabs(v);
    if (m > 0x1p-400 && m < 0x1p400) {
      y = __drcp_rn(v);
      z = __dmul_rn(__fma_rn(-v, y, 1.0), y);
    }
  }
  __device__ __forceinline__ Divisor() : b(1.0), y(0.0), z(0.0) {}
  __device__ __forceinline__ double divide(double a) const {
    const double m = fabs(a);
    if (y != 0.0 && m > 0x1p-400 && m < 0x1p400) {
      const double q = __fma_rn(a, y, __dmul_rn(a, z));
      return __fma_rn(__fma_rn(-b, q, a), y, q);
    }
    return __ddiv_rn(a, b);
  }
};

// RowSparse sweep (Relaxation_MatVect.cxx:69-77 / :83-91).  span.x..y: row j.
struct GeneralSor {
  static constexpr int kAhead = 8, kThreads = 256, kAheadLong = 8;
  static constexpr bool kTwoAhead = false, kTail = false;
  static constexpr bool kPositions = false;
  const int* ind; const double* val; const double* diag;
  const double* b; const double* x0; double omega, rest;  // rest = 1 - omega
  struct Row { int j, k0, len; bool fwd; double bj; Divisor ajj; };
  struct Sum { double temp, xj; };
  __device__ __forceinline__ Row load(int, bool fwd, int j, const int4& sp) const {
    return Row{j, sp.x, sp.y - sp.x, fwd, __ldg(b + j), Divisor(__ldg(diag + j))};
  }
  __device__ __forceinline__ void entry(const Row& r, int k, int& c, double& a) const {
    c = __ldg(ind + r.k0 + k);
    a = __ldg(val + r.k0 + k);
  }
  __device__ __forceinline__ bool is_new(const Row& r, int, int c) const {
    return r.fwd ? c < r.j : c > r.j;
  }
  __device__ __forceinline__ void first(const Row&, Sum& s, double xj) const {
    s.temp = 0.0;
    s.xj = xj;
  }
  __device__ __forceinline__ void take(const Row&, Sum& s, int, int, double a, double x) const {
    s.temp = add_rn(s.temp, mul_rn(a, x));
  }
  __device__ __forceinline__ void lead(const Row&, Sum&, int) const {}
  __device__ __forceinline__ bool skips(const Row&, int) const { return false; }
  __device__ __forceinline__ double signed_value(const Row&, double a) const { return a; }
  __device__ __forceinline__ double running(const Row&, const Sum& s) const { return s.temp; }
  __device__ __forceinline__ void run_to(const Row&, Sum& s, double v) const { s.temp = v; }
  __device__ __forceinline__ double last(const Row& r, const Sum& s) const {
    const double temp = add_rn(__dsub_rn(r.bj, s.temp), mul_rn(r.ajj.b, s.xj));
    return add_rn(mul_rn(rest, s.xj), r.ajj.divide(mul_rn(omega, temp)));
  }
  __device__ __forceinline__ void store(const Row&, double) const {}
};

// RowSymSparse sweeps.  span.x..y: the stored (upper) row j; span.z..w: the
// mirrored entries of row j (columns < j, increasing) in the full pattern;
// diag: the sum of the row's diagonal entries.
// Forward (Relaxation_MatVect.cxx:214-249): t = ((1-w)/w * ajj) * x_j +
// (b_j - sum_{p != j} a_jp x_p), x read old, then x_j = (t - sum a_kj x_k) *
// (w / ajj), the x_k new and k increasing: the stored entries, then the
// mirrored ones.  Backward (:257-294): y = sum a_kj x_k, old; t =
// (((1-w)/w * ajj) * x_j + b_j) - y; x_j = ((t - sum_{p != j} a_jp x_p) * w) /
// ajj, the x_p new: the mirrored entries, then the stored ones.
struct SymmetricSor {
  static constexpr int kAhead = 8, kThreads = 384, kAheadLong = 6;
  static constexpr bool kTwoAhead = true, kTail = true;
  static constexpr bool kPositions = false;
  const int* uind; const double* uval; const int* find; const double* fval;
  const double* diag; const double* b; const double* x0;
  double omega, ratio;  // ratio = (1 - omega) / omega
  struct Row { int j, u0, f0, nu, len; bool fwd; double bj, scale; Divisor ajj; };
  struct Sum { double temp, t, xj; bool started; };
  __device__ __forceinline__ Row load(int, bool fwd, int j, const int4& sp) const {
    const Divisor d(__ldg(diag + j));
    return Row{j, sp.x, sp.z, sp.y - sp.x, sp.y - sp.x + sp.w - sp.z, fwd, __ldg(b + j),
               fwd ? __ddiv_rn(omega, d.b) : 0.0, d};
  }
  __device__ __forceinline__ bool stored(const Row& r, int k) const {
    return r.fwd ? k < r.nu : k >= r.len - r.nu;
  }
  __device__ __forceinline__ void entry(const Row& r, int k, int& c, double& a) const {
    const bool st = stored(r, k);
    const int q = st ? r.u0 + (r.fwd ? k : k - (r.len - r.nu)) : r.f0 + (r.fwd ? k - r.nu : k);
    c = __ldg((st ? uind : find) + q);
    a = __ldg((st ? uval : fval) + q);
  }
  __device__ __forceinline__ bool is_new(const Row& r, int k, int c) const {
    return r.fwd ? k >= r.nu : stored(r, k) && c != r.j;
  }
  __device__ __forceinline__ void first(const Row&, Sum& s, double xj) const {
    s.temp = s.t = 0.0;
    s.xj = xj;
    s.started = false;
  }
  // t before the entries that read new values
  __device__ __forceinline__ void start(const Row& r, Sum& s) const {
    const double q = mul_rn(mul_rn(ratio, r.ajj.b), s.xj);
    s.t = r.fwd ? add_rn(q, __dsub_rn(r.bj, s.temp)) : __dsub_rn(add_rn(q, r.bj), s.t);
    s.started = true;
  }
  __device__ __forceinline__ int olds(const Row& r) const { return r.fwd ? r.nu : r.len - r.nu; }
  __device__ __forceinline__ void take(const Row& r, Sum& s, int k, int c, double a, double x) const {
    if (!s.started && k >= olds(r)) start(r, s);
    if (stored(r, k)) {
      if (c != r.j) s.temp = add_rn(s.temp, mul_rn(a, x));
    } else if (r.fwd) {
      s.t = __dsub_rn(s.t, mul_rn(a, x));
    } else {
      s.t = add_rn(s.t, mul_rn(a, x));
    }
  }
  __device__ __forceinline__ void lead(const Row& r, Sum& s, int k) const {
    if (!s.started && k >= olds(r)) start(r, s);
  }
  __device__ __forceinline__ bool skips(const Row& r, int c) const { return c == r.j; }
  __device__ __forceinline__ double signed_value(const Row& r, double a) const { return r.fwd ? -a : a; }
  // (an entry held in registers comes after the lead only once t is started)
  __device__ __forceinline__ double running(const Row& r, const Sum& s) const { return r.fwd ? s.t : s.temp; }
  __device__ __forceinline__ void run_to(const Row& r, Sum& s, double v) const {
    if (r.fwd) s.t = v;
    else s.temp = v;
  }
  __device__ __forceinline__ double last(const Row& r, Sum& s) const {
    if (!s.started) start(r, s);
    return r.fwd ? mul_rn(s.t, r.scale) : r.ajj.divide(mul_rn(__dsub_rn(s.t, s.temp), omega));
  }
  __device__ __forceinline__ void store(const Row&, double) const {}
};

// The two sweeps of an ILUT apply in gather form: x_j = (x_j * pre_j - v_1
// x_{c1} - v_2 x_{c2} - ...) * post_j, the subtractions in the listed order
// (pre and post may be null).  The first sweep starts from r through the
// input permutation, the second from the first's values; its results also go
// to z through the output permutation.  span.x..y: the row's update list.
struct FactorSolve {
  static constexpr int kAhead = 4, kThreads = 384, kAheadLong = 8;
  static constexpr bool kTwoAhead = true, kTail = false;
  static constexpr bool kPositions = true;
  const int* ind[2]; const double* val[2];
  const double* pre[2]; const double* post[2];
  const double* r; const int* in_at;
  double* z; const int* out_at;
  struct Row { int ph, k0, len, out; double in, pre, post; bool has_pre, has_post; };
  struct Sum { double t; };
  __device__ __forceinline__ Row load(int ph, bool, int j, const int4& sp) const {
    const double* pr = ph ? pre[1] : pre[0];
    const double* po = ph ? post[1] : post[0];
    return Row{ph, sp.x, sp.y - sp.x, ph ? __ldg(out_at + j) : 0,
               ph ? 0.0 : __ldg(r + __ldg(in_at + j)),
               pr ? __ldg(pr + j) : 0.0, po ? __ldg(po + j) : 0.0, pr != nullptr, po != nullptr};
  }
  __device__ __forceinline__ void entry(const Row& r, int k, int& c, double& a) const {
    c = __ldg((r.ph ? ind[1] : ind[0]) + r.k0 + k);
    a = __ldg((r.ph ? val[1] : val[0]) + r.k0 + k);
  }
  __device__ __forceinline__ bool is_new(const Row&, int, int) const { return true; }
  __device__ __forceinline__ void first(const Row& r, Sum& s, double xj) const {
    s.t = r.ph ? xj : r.in;
    if (r.has_pre) s.t = mul_rn(s.t, r.pre);
  }
  __device__ __forceinline__ void take(const Row&, Sum& s, int, int, double a, double x) const {
    s.t = __dsub_rn(s.t, mul_rn(a, x));
  }
  __device__ __forceinline__ void lead(const Row&, Sum&, int) const {}
  __device__ __forceinline__ bool skips(const Row&, int) const { return false; }
  __device__ __forceinline__ double signed_value(const Row&, double a) const { return -a; }
  __device__ __forceinline__ double running(const Row&, const Sum& s) const { return s.t; }
  __device__ __forceinline__ void run_to(const Row&, Sum& s, double v) const { s.t = v; }
  __device__ __forceinline__ double last(const Row& r, const Sum& s) const {
    return r.has_post ? mul_rn(s.t, r.post) : s.t;
  }
  __device__ __forceinline__ void store(const Row& r, double v) const {
    if (r.ph == 1) z[r.out] = v;
  }
};

// x0 of an operation that reads values from before the first sweep
template <class Op>
__device__ __forceinline__ const double* sweep_start(const Op& op) { return op.x0; }
__device__ __forceinline__ const double* sweep_start(const FactorSolve&) { return nullptr; }
// and where the last sweep's values go
template <class Op>
__device__ __forceinline__ double* sweep_out(const Op&, double* result, const int** at) {
  *at = nullptr;
  return result;
}
__device__ __forceinline__ double* sweep_out(const FactorSolve& op, double*, const int** at) {
  *at = op.out_at;
  return op.z;
}

// The rows of the last sweep that this warp did not finish, from item q of its
// own on, come out as NaN: out[at[row]], or out[row] with no `at`.
static __device__ __noinline__ void sweep_mark(const int4* items, const int* rows, int q, int q1,
                                               int step, double* out, const int* at) {
  const int lane = threadIdx.x & 31;
  for (; q < q1; q += step) {
    const int4 item = __ldg(items + q);
    if (lane < item.y) {
      const int j = __ldg(rows + item.x + lane);
      out[at ? __ldg(at + j) : j] = __longlong_as_double(0x7ff8000000000000ll);
    }
  }
}

// ------------------------------------------------------------------ the kernel

template <class Op, bool OWN, bool LONG>
__global__ void __launch_bounds__(LONG ? kSweepLong : Op::kThreads, 1) sweep_kernel(SweepArgs a, Op op) {
  extern __shared__ double s_own[];
  __shared__ unsigned long long s_bar[kSweepRing];  // step s completes s_bar[s % ring]
  constexpr int U = LONG ? Op::kAheadLong : Op::kAhead, W = (LONG ? kSweepLong : Op::kThreads) / 32;
  static_assert(W + 2 < kSweepRing, "a warp may be W items ahead of the oldest unfinished step");
  const int c0 = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r0 = __ldg(a.blk + c0), rows = __ldg(a.blk + c0 + 1) - r0;
  if (threadIdx.x < kSweepRing) mbar_init(&s_bar[threadIdx.x], kSweepStep);
  const SweepWait w{a.state, a.late, (int)gridDim.x, a.wait_ns};
  const double* x0 = sweep_start(op);
  SweepSource old{nullptr, 0u};
  int base = 0;  // this CTA's steps of the sweeps before
  bool ok = true;
  // this warp leaves: its items of the last sweep from the given one on
  auto mark = [&](int from) {
    const SweepPhase& P = a.nph > 1 ? a.ph[1] : a.ph[0];
    const int* at;
    double* out = sweep_out(op, a.result, &at);
    sweep_mark(P.item, P.rows, from, __ldg(P.cta_item + c0 + 1), W, out, at);
  };
  for (int ph = 0; ph < a.nph; ph++) {
    // every value of the CTA's rows from the sweep before is in place
    if (__syncthreads_or(!ok)) {
      mark(__ldg((a.nph > 1 ? a.ph[1] : a.ph[0]).cta_item + c0) + warp);
      return;
    }
    const SweepPhase P = ph ? a.ph[1] : a.ph[0];
    const SweepSource fresh{P.out, OWN ? smem_u32(s_own + (size_t)ph * a.max_rows) : 0u};
    const bool fwd = P.forward != 0;
    const int it0 = __ldg(P.cta_item + c0), it1 = __ldg(P.cta_item + c0 + 1);
    // the next item's row and entry ranges are loaded an item ahead
    int4 item = make_int4(0, 0, 0, 0);
    int j = -1;
    int4 span = make_int4(0, 0, 0, 0);
    auto fetch = [&](int q) {
      j = -1;
      if (q >= it1) return;
      item = __ldg(P.item + q);
      if (lane < item.y) {
        j = __ldg(P.rows + item.x + lane);
        span = __ldg(P.span + item.x + lane);
      }
    };
    // where the value of column c is: its position in this sweep, or in the
    // one before, or the row itself in the vector given
    auto place = [&](int c, bool nw) {
      return Op::kPositions ? c : nw ? __ldg(P.pos + c) : ph == 1 ? __ldg(P.pos_prev + c) : c;
    };
    fetch(it0 + warp);
    int it = it0 + warp;
    for (; it < it1 && ok; it += W) {
      const bool live = j >= 0;
      const int row = j, slot = item.x + lane;
      // this item's step, and what it adds to the step's barrier; the step
      // before must be complete (it waited for the one before it, and so on)
      const int step = base + item.z, arrivals = item.w;
      typename Op::Row R = {};
      typename Op::Sum s;
      int c[U], at[U];
      double f[U], x[U];
      unsigned isnew = 0u, far = 0u, near = 0u;  // far: awaited in L2, near: in shared memory
      double xj = 0.0;
      int before = 0;  // this row's position in the sweep before
      if (live) {
        R = op.load(ph, fwd, row, span);
        if (ph == 0 && x0) xj = __ldcg(x0 + row);
        if (ph == 1) before = __ldg(P.pos_prev + row);
#pragma unroll
        for (int u = 0; u < U; u++) {
          c[u] = 0;
          f[u] = 0.0;
          if (u < R.len) op.entry(R, u, c[u], f[u]);
        }
      }
      const int len = live ? R.len : 0;
      fetch(it + W);
#pragma unroll
      for (int u = 0; u < U; u++) {
        at[u] = 0;
        if (u < len) {
          const bool nw = op.is_new(R, u, c[u]);
          if (nw) isnew |= 1u << u;
          at[u] = place(c[u], nw);
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        x[u] = 0.0;
        if (u < len) {
          if ((isnew >> u & 1u) || ph == 1) {
            if (OWN && (unsigned)(at[u] - r0) < (unsigned)rows) near |= 1u << u;
            else far |= 1u << u;
          } else if (x0) {
            x[u] = __ldcg(x0 + at[u]);
          }
        }
      }
      // looks once at the values that other CTAs have yet to give
      auto look = [&]() {
        double y[U];
#pragma unroll
        for (int u = 0; u < U; u++)
          if (far >> u & 1u) y[u] = ld_volatile((isnew >> u & 1u ? fresh.g : old.g) + at[u]);
#pragma unroll
        for (int u = 0; u < U; u++)
          if ((far >> u & 1u) && !is_fill(y[u])) {
            x[u] = y[u];
            far &= ~(1u << u);
          }
      };
      unsigned long long t0 = 0ull;
      unsigned seen = 0u, spin = 0u;
      auto poll = [&](unsigned mask) -> bool {  // whether some lane still awaits an entry of `mask`
        if (far) look();
        if ((++spin & 1023u) == 0u && __any_sync(0xffffffffu, !w.go_on(t0, seen))) ok = false;
        return __any_sync(0xffffffffu, (far & mask) != 0u);
      };
      // the values of the sweep before, and the entries that lead the row
      // up to the first new one
      const int lead = isnew ? min(__ffs(isnew) - 1, len) : min(len, U);
      if (ph == 1) {
        while (poll(~isnew) && ok) {}
#pragma unroll
        for (int u = 0; u < U; u++)
          if ((near & ~isnew) >> u & 1u) x[u] = ld_shared(old.own + 8u * (unsigned)(at[u] - r0));
        if (live) {
          xj = OWN ? ld_shared(old.own + 8u * (unsigned)(before - r0)) : ld_volatile(old.g + before);
        }
      }
      if (live) {
        op.first(R, s, xj);
#pragma unroll
        for (int u = 0; u < U; u++)
          if (u < lead) op.take(R, s, u, c[u], f[u], x[u]);
        op.lead(R, s, lead);
      }
      near &= isnew;
      // the entries after the lead: which add, with what, and from where
      unsigned adds = 0u, from[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (u >= lead && u < len && !op.skips(R, c[u])) adds |= 1u << u;
        if (u >= lead) f[u] = op.signed_value(R, f[u]);
        from[u] = fresh.own + ((near >> u & 1u) ? 8u * (unsigned)(at[u] - r0) : 0u);
      }
      double sum = live ? op.running(R, s) : 0.0;
      // the first entries beyond, before the row's turn
      int c1[U], q1[U], c2[U];
      double f1[U], f2[U];
      if (LONG) {
#pragma unroll
        for (int u = 0; u < U; u++) {
          c1[u] = c2[u] = q1[u] = 0;
          f1[u] = f2[u] = 0.0;
          if (U + u < len) op.entry(R, U + u, c1[u], f1[u]);
          if (Op::kTwoAhead && 2 * U + u < len) op.entry(R, 2 * U + u, c2[u], f2[u]);
        }
        if (Op::kTwoAhead) {
#pragma unroll
          for (int u = 0; u < U; u++)
            if (U + u < len) q1[u] = place(c1[u], op.is_new(R, U + u, c1[u]));
        }
      }
      // wait for the other CTAs' new values and for this CTA's earlier steps
      while (ok) {
        const bool more = poll(~0u);
        unsigned long long* bar = &s_bar[(step - 1) & (kSweepRing - 1)];
        const unsigned parity = (unsigned)((step - 1) / kSweepRing) & 1u;
        const bool turn = step == 0 || (more ? mbar_test_wait(bar, parity) : mbar_try_wait(bar, parity));
        if (__all_sync(0xffffffffu, !more && turn)) break;
      }
      if (live && ok) {
        if (OWN) {
          double y[U];
#pragma unroll
          for (int u = 0; u < U; u++) y[u] = ld_shared(from[u]);
#pragma unroll
          for (int u = 0; u < U; u++) x[u] = (near >> u & 1u) ? y[u] : x[u];
        }
#pragma unroll
        for (int u = 0; u < U; u++) x[u] = mul_rn(f[u], x[u]);
#pragma unroll
        for (int u = 0; u < U; u++)
          if (adds >> u & 1u) sum = add_rn(sum, x[u]);
        if (adds) op.run_to(R, s, sum);
        // rows longer than the entries held in registers, U at a time: while the
        // values of U entries come, so do the places of the next U and the
        // entries after those
        if (LONG) {
          for (int k0 = U; k0 < len && ok; k0 += U) {
            if (k0 % kSweepNote == 0) *((volatile unsigned*)a.state + kStProgress + c0) = ~(unsigned)k0;
            unsigned wait = 0u;
#pragma unroll
            for (int u = 0; u < U; u++) {
              x[u] = 0.0;
              if (k0 + u < len) {
                if (!Op::kTwoAhead) q1[u] = place(c1[u], op.is_new(R, k0 + u, c1[u]));
                if (op.is_new(R, k0 + u, c1[u]) || ph == 1) {
                  if (OWN && (unsigned)(q1[u] - r0) < (unsigned)rows)
                    x[u] = ld_shared((op.is_new(R, k0 + u, c1[u]) ? fresh : old).own + 8u * (unsigned)(q1[u] - r0));
                  else
                    wait |= 1u << u;
                } else if (x0) {
                  x[u] = __ldcg(x0 + q1[u]);
                }
              }
            }
            int c3[U], q2[U];
            double f3[U];
            if (Op::kTwoAhead) {
#pragma unroll
              for (int u = 0; u < U; u++) {
                q2[u] = 0;
                if (k0 + U + u < len) q2[u] = place(c2[u], op.is_new(R, k0 + U + u, c2[u]));
              }
            }
            constexpr int kNext = (Op::kTwoAhead ? 2 : 1) * U;
#pragma unroll
            for (int u = 0; u < U; u++) {
              c3[u] = 0;
              f3[u] = 0.0;
              if (k0 + kNext + u < len) op.entry(R, k0 + kNext + u, c3[u], f3[u]);
            }
            for (unsigned n = 1; wait && ok; n++) {
              double y[U];
#pragma unroll
              for (int u = 0; u < U; u++)
                if (wait >> u & 1u) y[u] = ld_volatile((op.is_new(R, k0 + u, c1[u]) ? fresh : old).g + q1[u]);
#pragma unroll
              for (int u = 0; u < U; u++)
                if ((wait >> u & 1u) && !is_fill(y[u])) {
                  x[u] = y[u];
                  wait &= ~(1u << u);
                }
              if ((n & 255u) == 0u && wait && !w.go_on(t0, seen)) ok = false;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
              if (k0 + u < len) op.take(R, s, k0 + u, c1[u], f1[u], x[u]);
              c1[u] = Op::kTwoAhead ? c2[u] : c3[u];
              f1[u] = Op::kTwoAhead ? f2[u] : f3[u];
              if (Op::kTwoAhead) {
                q1[u] = q2[u];
                c2[u] = c3[u];
                f2[u] = f3[u];
              }
            }
          }
        }
        if (!LONG && Op::kTail) {
        for (int k = U; k < len && ok; k++) {
          if (k % kSweepNote == 0) *((volatile unsigned*)a.state + kStProgress + c0) = ~(unsigned)k;
          int cc;
          double ff, y = 0.0;
          op.entry(R, k, cc, ff);
          const bool nw = op.is_new(R, k, cc);
          if (nw || ph == 1) {
            const SweepSource& S = nw ? fresh : old;
            const int q = place(cc, nw);
            const bool here = OWN && (unsigned)(q - r0) < (unsigned)rows;
            y = here ? ld_shared(S.own + 8u * (unsigned)(q - r0)) : ld_volatile(S.g + q);
            for (unsigned n = 1; !here && is_fill(y); n++) {
              if ((n & 255u) == 0u && !w.go_on(t0, seen)) {
                ok = false;
                break;
              }
              y = ld_volatile(S.g + q);
            }
          } else if (x0) {
            y = __ldcg(x0 + cc);
          }
          op.take(R, s, k, cc, ff, y);
        }
        }
        if (ok) {
          const double v = not_fill(op.last(R, s));
          if (OWN) st_shared(fresh.own + 8u * (unsigned)(slot - r0), v);
          *((volatile double*)P.out + slot) = v;
          if (a.result && ph == a.nph - 1) a.result[row] = v;
          op.store(R, v);
        }
      }
      ok = __all_sync(0xffffffffu, ok) != 0;
      // every lane's value is ordered before lane 0's arrival, which publishes
      // them all (a vote orders no memory)
      __syncwarp();
      if (lane == 0 && ok) {
        mbar_arrive(&s_bar[step & (kSweepRing - 1)], arrivals);
        *((volatile unsigned*)a.state + kStProgress + c0) = (unsigned)step + 1u;
      }
    }
    if (!ok && ph == a.nph - 1) mark(it - W);
    base += __ldg(P.steps + c0);
    old = fresh;
  }
}

// Sum of the diagonal entries of each stored row, in stored order (the
// reference's ajj, Relaxation_MatVect.cxx:214-294).
__global__ void sym_diag_kernel(int n, const int* __restrict__ ptr, const int* __restrict__ ind,
                                const double* __restrict__ val, double* __restrict__ d) {
  for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < n;
       j += (long long)gridDim.x * blockDim.x) {
    double ajj = 0.0;
    for (int k = ptr[j]; k < ptr[j + 1]; k++)
      if (ind[k] == j) ajj = add_rn(ajj, val[k]);
    d[j] = ajj;
  }
}

// Positions of the rows, and with `span` the entry ranges of rows of the pattern
// `ptr` (with `uptr` of symmetric storage: the stored row, then the mirrored
// entries, which come first in the expanded one).
__global__ void __launch_bounds__(256) sweep_place_kernel(int n, const int* __restrict__ rows, int* pos,
                                                          int4* span, const int* __restrict__ ptr,
                                                          const int* __restrict__ uptr) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int j = __ldg(rows + i);
    pos[j] = (int)i;
    if (!span) continue;
    const int a = __ldg(ptr + j), e = __ldg(ptr + j + 1);
    if (uptr) {
      const int u = __ldg(uptr + j), ue = __ldg(uptr + j + 1);
      span[i] = make_int4(u, ue, a, e - (ue - u));
    } else {
      span[i] = make_int4(a, e, 0, 0);
    }
  }
}

__global__ void __launch_bounds__(256) sweep_fill_kernel(int n, double* x, double* y,
                                                         unsigned* state, int late) {
  // a solver's applies after one whose wait ran out leave at once: the solve is lost
  if (blockIdx.x == 0 && threadIdx.x == 0) state[kStLeave] = late == kStLateSolve ? state[late] : 0u;
  const double f = __longlong_as_double((long long)kSweepFill);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    x[i] = f;
    if (y) y[i] = f;
  }
}

// One sweep by levels: a row reads new values in `out` and the others in `old`
// (null: zero), both by row.  What does not depend on other rows is loaded by
// load(), before the level before is complete, the rest by finish().  (U entries
// in flight: with eight, a factor's solves hold 48 registers for 32, and 10^6
// diagonal rows take 23 us for 19.)
template <class Op, bool LONG>
struct LevelRow {
  static constexpr int U = Op::kAhead;
  typename Op::Row R;
  int j, c[U];
  double f[U];
  __device__ __forceinline__ void load(const Op& op, int ph, bool fwd, int row, const int4& span) {
    j = row;
    R = op.load(ph, fwd, row, span);
#pragma unroll
    for (int u = 0; u < U; u++) {
      c[u] = 0;
      f[u] = 0.0;
      if (u < R.len) op.entry(R, u, c[u], f[u]);
    }
  }
  __device__ __forceinline__ void finish(const Op& op, const double* old, double* out) {
    typename Op::Sum s;
    op.first(R, s, old ? old[j] : 0.0);
    int k0 = 0;
    do {
      int c2[U];
      double f2[U], x[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        x[u] = 0.0;
        if (k0 + u < R.len) {
          const double* p = op.is_new(R, k0 + u, c[u]) ? out : old;
          if (p) x[u] = p[c[u]];
        }
      }
      if (LONG) {
#pragma unroll
        for (int u = 0; u < U; u++) {
          c2[u] = 0;
          f2[u] = 0.0;
          if (k0 + U + u < R.len) op.entry(R, k0 + U + u, c2[u], f2[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (k0 + u < R.len) op.take(R, s, k0 + u, c[u], f[u], x[u]);
        if (LONG) {
          c[u] = c2[u];
          f[u] = f2[u];
        }
      }
      k0 += U;
    } while (LONG && k0 < R.len);
    const double v = op.last(R, s);
    out[j] = v;
    op.store(R, v);
  }
};

// Where a row's entries are: lists by position, or the rows' own with, for
// symmetric storage, the stored half.
struct LevelSpan {
  const int *lists, *ptr, *uptr;
  __device__ __forceinline__ int4 operator()(int i, int j) const {
    if (lists) return make_int4(__ldg(lists + i), __ldg(lists + i + 1), 0, 0);
    const int a = __ldg(ptr + j), e = __ldg(ptr + j + 1);
    if (!uptr) return make_int4(a, e, 0, 0);
    const int u = __ldg(uptr + j), ue = __ldg(uptr + j + 1);
    return make_int4(u, ue, a, e - (ue - u));
  }
};

// One level: what it needs of the level before is awaited by the hardware
// (programmatic dependent launch), after its own loads are under way.
template <class Op, bool LONG>
__global__ void __launch_bounds__(256) level_rows_kernel(int begin, int end, int ph, bool fwd, const int* rows,
                                                         LevelSpan span, const double* old, double* out, Op op) {
  const int i = begin + blockIdx.x * blockDim.x + threadIdx.x;
  LevelRow<Op, LONG> r;
  if (i < end) {
    const int j = __ldg(rows + i);
    r.load(op, ph, fwd, j, span(i, j));
  }
  pdl_release();
  pdl_wait();
  if (i < end) r.finish(op, old, out);
}

// One sweep, a launch per level.
template <class Op>
int run_levels(const SweepPlan& P, int n, int ph, bool fwd, const LevelSpan& span, const double* old, double* out,
               const Op& op, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  auto* kern = P.max_len > LevelRow<Op, true>::U ? level_rows_kernel<Op, true> : level_rows_kernel<Op, false>;
  for (int l = 0; l + 1 < (int)P.h_lvl.size(); l++) {
    const int begin = P.h_lvl[l], end = P.h_lvl[l + 1];
    cfg.gridDim = dim3((end - begin + 255) / 256);
    cfg.numAttrs = l > 0 ? 1 : 0;  // the first follows all that the caller queued
    SB2_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, begin, end, ph, fwd, (const int*)P.d_rows, span, old, out, op));
  }
  return SB2_OK;
}

// x in place: levels then separate a row from the rows that read its new value and
// from those that read its old one.  f(j): row j.
template <class Row>
__global__ void __launch_bounds__(1024) level_cta_kernel(int levels, const int* __restrict__ lvl,
                                                         const int* __restrict__ rows, Row f) {
  for (int l = 0; l < levels; l++) {
    for (int i = lvl[l] + threadIdx.x; i < lvl[l + 1]; i += 1024) f(rows[i]);
    __syncthreads();
  }
}

// A row of GeneralSor, x in place.
struct InPlaceSor {
  const int *ptr, *ind;
  const double *val, *diag, *b;
  double* x;
  double omega, rest;
  __device__ __forceinline__ void operator()(int j) const {
    double t = 0.0;
    for (int k = ptr[j], e = ptr[j + 1]; k < e; k++) t = add_rn(t, mul_rn(val[k], x[ind[k]]));
    const double xj = x[j], ajj = diag[j];
    t = add_rn(__dsub_rn(b[j], t), mul_rn(ajj, xj));
    x[j] = add_rn(mul_rn(rest, xj), __ddiv_rn(mul_rn(omega, t), ajj));
  }
};

// Rows of SymmetricSor in two passes: `start` makes t of every row from old
// values, `finish` takes the new ones.  Forward the stored entries are old and the
// mirrored ones (which lead the expanded row) new, backward the other way round.
struct InPlaceSymmetricSor {
  const int *uptr, *uind;
  const double* uval;
  const int *ptr, *ind;
  const double *val, *diag, *b;
  double *x, *t;
  double omega, ratio;
  bool fwd, start;
  __device__ __forceinline__ void operator()(int j) const {
    const double ajj = diag[j];
    double v = start || !fwd ? 0.0 : t[j];
    if (fwd == start) {
      for (int k = uptr[j], e = uptr[j + 1]; k < e; k++)
        if (uind[k] != j) v = add_rn(v, mul_rn(uval[k], x[uind[k]]));
    } else {
      const int e = ptr[j + 1] - (uptr[j + 1] - uptr[j]);
      for (int k = ptr[j]; k < e; k++) {
        const double p = mul_rn(val[k], x[ind[k]]);
        v = start ? add_rn(v, p) : __dsub_rn(v, p);
      }
    }
    if (start) {
      const double q = mul_rn(mul_rn(ratio, ajj), x[j]);
      t[j] = fwd ? add_rn(q, __dsub_rn(b[j], v)) : __dsub_rn(add_rn(q, b[j]), v);
    } else if (fwd) {
      x[j] = mul_rn(v, __ddiv_rn(omega, ajj));
    } else {
      x[j] = __ddiv_rn(mul_rn(__dsub_rn(t[j], v), omega), ajj);
    }
  }
};

template <class Row>
__global__ void __launch_bounds__(256) level_in_place_kernel(int begin, int end, const int* __restrict__ rows,
                                                             Row f) {
  const int i = begin + blockIdx.x * blockDim.x + threadIdx.x;
  if (i < end) f(rows[i]);
}

template <class Row>
int run_in_place(const SweepPlan& P, int n, const Row& f, cudaStream_t s) {
  const int levels = (int)P.h_lvl.size() - 1;
  if (n <= kLevelCta) {
    level_cta_kernel<<<1, 1024, 0, s>>>(levels, P.d_lvl, P.d_rows, f);
  } else {
    for (int l = 0; l < levels; l++) {
      const int begin = P.h_lvl[l], end = P.h_lvl[l + 1];
      level_in_place_kernel<<<(end - begin + 255) / 256, 256, 0, s>>>(begin, end, P.d_rows, f);
    }
  }
  SB2_CUDA_TRY(cudaGetLastError());
  return SB2_OK;
}

template <class Row>
__global__ void __launch_bounds__(256) all_rows_kernel(int n, Row f) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n) f(j);
}

// One launch of `sweeps` (1 or 2) sweeps; the last one's values go to `result`
// by row (null: the operation stores them).  late: kStLateSolve or kStLateApply.
template <class Op>
int launch_sweeps(const SweepGrid& G, int sweeps, const SweepPlan* const (&plan)[2],
                  const bool (&forward)[2], double* result, const Op& op, int late, cudaStream_t s) {
  const int n = G.n;
  if (n == 0) return SB2_OK;
  SweepArgs a;
  a.blk = G.d_blk;
  a.max_rows = G.max_rows;
  a.nph = sweeps;
  a.result = result;
  for (int k = 0; k < 2; k++) {
    const int q = k < sweeps ? k : 0;
    const SweepPlan& P = *plan[q];
    a.ph[k] = SweepPhase{P.d_rows, P.d_span, P.d_item, P.d_cta_item, P.d_steps, P.d_pos,
                         plan[0]->d_pos, forward[q] ? 1 : 0, G.d_new[k]};
  }
  a.state = G.d_state;
  a.late = late;
  a.wait_ns = ring_wait_ns();
  // values of the CTA's own rows stay in shared memory when both sweeps' fit
  const size_t smem = sizeof(double) * (size_t)a.nph * G.max_rows;
  const bool own = smem <= (size_t)kSweepSmem;
  const int g = std::min((n + 255) / 256, num_sms(current_device()) * 8);
  sweep_fill_kernel<<<g, 256, 0, s>>>(n, G.d_new[0], sweeps > 1 ? G.d_new[1] : nullptr, G.d_state,
                                   late);
  SB2_CUDA_TRY(cudaGetLastError());
  const bool lng = plan[0]->max_len > Op::kAhead || plan[sweeps - 1]->max_len > Op::kAhead;
  const void* kern = lng ? (own ? (const void*)sweep_kernel<Op, true, true> : (const void*)sweep_kernel<Op, false, true>)
                         : (own ? (const void*)sweep_kernel<Op, true, false> : (const void*)sweep_kernel<Op, false, false>);
  if (own && smem > 48 * 1024) SB2_CUDA_TRY(allow_shared(kern, kSweepSmem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(G.ctas);
  cfg.blockDim = dim3(lng ? kSweepLong : Op::kThreads);
  cfg.dynamicSmemBytes = own ? smem : 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;  // the CTAs wait for one another
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* args[2] = {(void*)&a, (void*)const_cast<Op*>(&op)};
  SB2_CUDA_TRY(cudaLaunchKernelExC(&cfg, kern, args));
  return SB2_OK;
}

#endif  // __CUDACC__

}  // namespace sb2
