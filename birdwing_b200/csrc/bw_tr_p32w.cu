// bw_tr_p32w.cu -- transform launches: 32-bit path, 64-bit coefficients (six primes).
#include "bw_transform.cuh"

namespace bw {

template int bw_set_transform_attrs<Ar32, false>();
template int bw_enqueue_transform<Ar32, false, true>(bw_ctx*, const uint32_t*, const uint32_t*,
                                                     bool, bool, const HostIO*);

}  // namespace bw
