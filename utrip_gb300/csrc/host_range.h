// Whether a host array may be read or written in place by a kernel.
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace cans {

// Device address of the host array p of n doubles if all of it is page-locked and
// lies in one piece for the device, else nullptr.  alias(q) is the device address of
// the byte at q if it is page-locked, else nullptr.  Registrations cover whole pages,
// so besides the ends one byte of every page in between is asked for: two
// registrations may hold the ends of an array whose middle neither covers.
template <class Alias>
double *mapped_range(double *p, size_t n, uintptr_t page, Alias alias) {
  if (((uintptr_t)p & 7) || n == 0) return nullptr;
  char *const dev = (char *)alias(p);
  if (!dev) return nullptr;
  const uintptr_t first = (uintptr_t)p, last = first + sizeof(double) * n - 1;
  for (uintptr_t q = (first / page + 1) * page; q < last; q += page)
    if ((char *)alias((void *)q) != dev + (q - first)) return nullptr;
  return (char *)alias((void *)last) == dev + (last - first) ? (double *)dev : nullptr;
}

}  // namespace cans
