// Internal entry of the forward launcher, shared by fa_fwd() and the tiled path of fa_kvcache().
#pragma once

#include "common.h"

namespace fa {

// Same as fa_fwd(); seqused_k_add is added to every seqused_k[b] on the device.  overlap: the previous kernel of the stream
// lets this one start early (launch_overlapped).  checked: the host refuses lengths beyond the capacity; they are neither read nor
// reported.
int run_fwd(const FaFwdParams* p, int seqused_k_add, cudaStream_t stream, bool overlap = false, bool checked = false);

#ifdef __CUDACC__
// What a sequence of a cache holds, limited to what it can hold; in 64 bits, a length may be any int32.  Beyond the capacity:
// nothing when the host refuses the call for it, which has to read no page that its caller never filled in, else the capacity.
struct CacheLength {
  int len;
  bool report;  // it was limited, and the host does not refuse the call for that
};
__device__ __forceinline__ CacheLength cache_length(int cached, int added, int capacity, bool checked) {
  const int64_t n = static_cast<int64_t>(cached) + added;
  if (n < 0) return {0, true};
  if (n > capacity) return {checked ? 0 : capacity, !checked};
  return {static_cast<int>(n), false};
}
#endif

}  // namespace fa
