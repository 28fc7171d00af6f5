// The number that a kernel writes to mapped host memory after its results.
#pragma once

namespace lfx {

// Acquire: what was written before the number is read after it, also on a host
// CPU that reorders loads.
inline unsigned host_number(const unsigned* p) { return __atomic_load_n(p, __ATOMIC_ACQUIRE); }

}  // namespace lfx
