// Internal entry of the forward launcher, shared by fa_fwd() and the tiled path of fa_kvcache().
#pragma once

#include "common.h"

namespace fa {

// Same as fa_fwd(); seqused_k_add is added to every seqused_k[b] on the device.  overlap: the previous kernel of the stream
// lets this one start early (launch_overlapped).  checked: the host refuses lengths beyond the capacity, the status word need not
// tell of them.
int run_fwd(const FaFwdParams* p, int seqused_k_add, cudaStream_t stream, bool overlap = false, bool checked = false);

}  // namespace fa
