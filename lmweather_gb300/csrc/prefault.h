#pragma once
#include <cstddef>

namespace lmw {

// Faults the pages of a host buffer of `bytes` about to be filled by a device copy, if its ends are not resident: the copy
// engine faults fresh pages one by one (1 GB/s), the kernel a range at once, and several ranges in parallel. The contents
// are left alone. Where memory or threads run out it does less: the copy faults what is left.
void prefault(void *p, std::size_t bytes) noexcept;

}  // namespace lmw
