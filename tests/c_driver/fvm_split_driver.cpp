// The engine's column split (fvm_split.h) behind C entry points, for CPU tests.
#include "fvm_split.h"

namespace {
std::vector<fvm::ZColumn> columns(int n, const int* nz) {
  std::vector<fvm::ZColumn> c;
  for (int i = 0; i < n; ++i) c.push_back({i, 0, 0, nz[i]});
  return c;
}
int copy_out(const std::vector<fvm::Task>& t, int* out, int cap) {
  for (size_t i = 0; i < t.size() && (int)i < cap; ++i) {
    out[3 * i] = t[i].blk;
    out[3 * i + 1] = t[i].z0;
    out[3 * i + 2] = t[i].z1;
  }
  return (int)t.size();
}
}  // namespace

extern "C" {
// (column, z0, z1) per task into out (room for cap); returns the task count.
int even_split_c(int n, const int* nz, int slots, double ovh, int* out, int cap, double* share, int* tries) {
  std::vector<fvm::Task> t;
  const fvm::Split s = fvm::even_split(columns(n, nz), slots, ovh, t);
  *share = s.share;
  *tries = s.tries;
  return copy_out(t, out, cap);
}
int split_columns_c(int n, const int* nz, int slots, int prec, double ovh, int* out, int cap) {
  std::vector<fvm::Task> t;
  fvm::split_columns(columns(n, nz), slots, prec, ovh, t);
  return copy_out(t, out, cap);
}
}
