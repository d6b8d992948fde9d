// Makes one value of an ILUT preconditioner's sweeps one that never comes: an
// entry of the plan (not of the factor) is pointed at a row that comes after its
// own, so that the two rows wait for one another until the wait limit.  Every
// position written lies in the vector.  Test infrastructure only; the kernels
// that run are the library's.
#include "../../seldon_b200/csrc/precond.cu"

// The value that entry `entry` of the first (sweep 0) or second sweep of Solve
// reads becomes that of position `at`; *old receives the position it read.
extern "C" int break_sweep(sb2_precond* M, int sweep, int entry, int at, int* old) {
  if (!M || M->kind != SB2_PRECOND_ILUT || at < 0 || at >= M->n_ilu || entry < 0) return -1;
  int* d = (sweep ? M->s_ub : M->s_lf).d_ind + entry;
  if (cudaMemcpy(old, d, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -2;
  return cudaMemcpy(d, &at, sizeof(int), cudaMemcpyHostToDevice) == cudaSuccess ? 0 : -2;
}
