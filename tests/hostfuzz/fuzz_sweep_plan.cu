// The order of a sweep's rows and its items on the host, over random levels:
// rows stay in their block, sorted by level and by row within one; items hold up
// to 32 rows of one level, up to 32 items a step, and each step's arrivals make up
// its barrier's count.  And the levels of symmetric storage against those of the
// expanded pattern.  Argument: the number of trials.  Test infrastructure only.
#include "../../seldon_b200/csrc/precond.cu"
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace sb2;
#define CHECK(c)                                             \
  do {                                                       \
    if (!(c)) {                                              \
      printf("FAILED trial %d line %d\n", trial, __LINE__);  \
      return 1;                                              \
    }                                                        \
  } while (0)
int main(int argc, char** argv) {
  const int trials = argc > 1 ? atoi(argv[1]) : 200;
  std::mt19937_64 g(11);
  long long sorted = 0;
  for (int trial = 0; trial < trials; trial++) {
    const int n = trial % 10 == 0 ? (int)(g() % 30000) : (int)(g() % 3000);
    SweepGrid G;
    CHECK(make_sweep_grid(n, &G) == SB2_OK);
    CHECK(G.h_blk[0] == 0 && G.h_blk[G.ctas] == n);
    const int most = trial % 3 == 0 ? 5 : trial % 3 == 1 ? n + 1 : 1000000000;
    std::vector<int> level(n);
    for (int& l : level) l = (int)(g() % most);
    SweepOrder O;
    make_sweep_order(G, level, &O);
    CHECK((int)O.cta_item.size() == G.ctas + 1 && (int)O.steps.size() == G.ctas);
    for (int c = 0; c < G.ctas; c++) {
      int at = G.h_blk[c], step = -1, items = 0, arrivals = 0;
      for (int i = G.h_blk[c]; i < G.h_blk[c + 1]; i++) {
        CHECK(O.rows[i] >= G.h_blk[c] && O.rows[i] < G.h_blk[c + 1]);
        if (i == G.h_blk[c]) continue;
        const int a = O.rows[i - 1], b = O.rows[i];
        CHECK(level[a] < level[b] || (level[a] == level[b] && a < b));
      }
      for (int k = O.cta_item[c]; k < O.cta_item[c + 1]; k++) {
        const int4 t = O.item[k];
        CHECK(t.x == at && t.y >= 1 && t.y <= 32);
        for (int q = 0; q < t.y; q++) CHECK(level[O.rows[at + q]] == level[O.rows[at]]);
        if (t.z != step) {
          CHECK(t.z == step + 1 && (step < 0 || arrivals == kSweepStep));
          step = t.z;
          items = arrivals = 0;
        }
        items++;
        arrivals += t.w;
        CHECK(items <= kSweepStep && t.w >= 1);
        at += t.y;
      }
      CHECK(at == G.h_blk[c + 1] && O.steps[c] == step + 1 && (step < 0 || arrivals == kSweepStep));
      sorted += G.h_blk[c + 1] > G.h_blk[c];
    }
    G.release();
    // symmetric storage: row j's columns >= j; expanded rows list the mirrored ones too
    std::vector<int> uptr(1, 0), uind;
    std::vector<std::vector<int>> full(n);
    for (int j = 0; j < n; j++) {
      uind.push_back(j);
      for (int q = (int)(g() % 4); q > 0 && j + 1 < n; q--) {
        uind.push_back(j + 1 + (int)(g() % std::min(n - j - 1, 50)));
        full[uind.back()].push_back(j);
      }
      uptr.push_back((int)uind.size());
    }
    std::vector<int> fptr(1, 0), find;
    for (int j = 0; j < n; j++) {
      find.insert(find.end(), full[j].begin(), full[j].end());
      find.insert(find.end(), uind.begin() + uptr[j], uind.begin() + uptr[j + 1]);
      fptr.push_back((int)find.size());
    }
    std::vector<int> a, b;
    mirrored_levels(n, uptr.data(), uind.data(), a);
    tri_levels(n, fptr.data(), find.data(), true, b);
    CHECK(a == b);
  }
  printf("blocks %lld\n", sorted);
  return 0;
}
