// Pages of host arrays (host_pages.cpp).
#pragma once

#include <cstddef>

namespace simp {

// Ranges smaller than this are left alone (their faults cost less than looking).
constexpr size_t kPagesFrom = 256 * 1024;

struct HostRange { const void *p; size_t bytes; };

// Gives the large ones of the ranges their pages, if they look as if they had
// none.  Never fails.
void make_resident(const HostRange *v, int n);

}  // namespace simp
