// key_range.cuh — the keys of one query row in equal ranges (attn.cu attn_row_kernel): plain arithmetic, for the device and the host alike.
#pragma once

namespace b200 {

struct KeyRange {
  int first, n;      // the range's keys: the row sees `cached` rows of the cache and, where `append`, one new one behind them
  int n_cached;      // those of them that are cached
  bool owns_new;     // the new key is the last of this range: true for one range
};

#ifdef __CUDACC__
__host__ __device__
#endif
inline KeyRange key_range(int cached, bool append, int range, int log_ranges) {
  const int nkeys = cached + (append ? 1 : 0);
  const int per = (((nkeys + (1 << log_ranges) - 1) >> log_ranges) + 15) & ~15;   // whole warps' worth: the first ranges are full, the last may be empty
  KeyRange r;
  r.first = range * per < nkeys ? range * per : nkeys;
  r.n = (r.first + per < nkeys ? r.first + per : nkeys) - r.first;
  r.n_cached = (cached < r.first + r.n ? cached : r.first + r.n) - r.first;
  r.owns_new = append && r.n > 0 && r.n > r.n_cached;   // of a range behind the last key n_cached is n - 1 too
  return r;
}

}  // namespace b200
