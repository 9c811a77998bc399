// Host check of csrc/handles.h's rule for the records (test_records_cpu.py).
#include "../mantaray_gb300/csrc/handles.h"

int main() {
  using mr::split_records_fit;
  const size_t mb = size_t(1) << 20;
  const bool small = split_records_fit(32 * mb, 0) && !split_records_fit(32 * mb + 1, 0);
  const bool share = split_records_fit(100 * mb, 800 * mb) && !split_records_fit(100 * mb + 1, 800 * mb);
  // 32,768^2 nodes' records (86 GB of current) beside 200 GB free
  const bool large = !split_records_fit(size_t(80) << 30, size_t(200) << 30);
  return small && share && large ? 0 : 1;
}
