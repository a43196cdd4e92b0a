// Two-step row and middle passes (apply_fast.cuh): dispatch over the compiled lengths, and their
// first group.
#include <initializer_list>

#include "apply_fast.cuh"

namespace mrsr {

MRSR_ROWS_GROUP(0)

// the lengths the fp16-storage operator takes
bool fast_length(int L) { return L == 64 || L == 128 || L == 256 || L == 384 || L == 512 || L == 768 || L == 1024; }

template <class... A>
static int first_group(std::initializer_list<int (*)(A...)> groups, A... a) {
  for (auto* f : groups) {
    const int s = f(a...);
    if (s != MRSR_ERR_UNSUPPORTED) return s;
  }
  return MRSR_ERR_UNSUPPORTED;
}

int fast_rows_fwd(const RowsFwdArgs& a, int64_t nrows, int ncg, cudaStream_t st) {
  return first_group<const RowsFwdArgs&, int64_t, int, cudaStream_t>(
      {rows_fwd_group_0, rows_fwd_group_1, rows_fwd_group_2, rows_fwd_group_3, rows_fwd_group_4, rows_fwd_group_5}, a, nrows,
      ncg, st);
}

int fast_rows_inv(const RowsInvArgs& a, int64_t nrows, cudaStream_t st) {
  return first_group<const RowsInvArgs&, int64_t, cudaStream_t>(
      {rows_inv_group_0, rows_inv_group_1, rows_inv_group_2, rows_inv_group_3, rows_inv_group_4, rows_inv_group_5}, a, nrows, st);
}

int fast_mid(const MidArgs& a, int nplanes, cudaStream_t st) {
  return first_group<const MidArgs&, int, cudaStream_t>(
      {mid_group_0, mid_group_1, mid_group_2, mid_group_3, mid_group_4, mid_group_5}, a, nplanes, st);
}

}  // namespace mrsr
