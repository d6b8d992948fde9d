// CTAs the persistent solvers take for a matrix: rows and entries a row as
// arguments, the rule's answer for 148 SMs on stdout.  Test infrastructure only.
#include "../../seldon_b200/csrc/csr.cu"
#include <cstdio>
#include <cstdlib>
#include "../../seldon_b200/csrc/persist.cuh"
int main(int argc, char** argv) {
  for (int k = 1; k + 1 < argc; k += 2) {
    const int rows = atoi(argv[k]), len = atoi(argv[k + 1]);
    std::vector<int> ptr(rows + 1);
    for (int i = 0; i <= rows; i++) ptr[i] = i * len;
    sb2::Partition P;
    if (sb2::build_partition_host(ptr.data(), rows, &P) != SB2_OK) return 1;
    cudaFree(P.d_blk);
    cudaFree(P.d_kind);
    printf("%d\n", sb2::persist_ctas(rows, P.nblk, 148));
  }
  return 0;
}
