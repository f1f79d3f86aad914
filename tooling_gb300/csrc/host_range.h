// Which host arrays a kernel may touch in place.
#pragma once
#include <cstddef>
#include <cstdint>

// A page-locked host range as the device sees it, looked up by an address in
// it: that address on the device, and the range's start and bytes there (0
// where the address is not page-locked memory that the device can reach).
struct HostRange {
  uintptr_t at, start;
  size_t bytes;
};

// The device's address of `bytes` bytes at p if one range holds all of them,
// else 0.  Looking at both ends is not enough: under unified addressing they
// can lie in two ranges, at the same distance on the device, with memory
// between them that the device cannot reach.
template <class Lookup>
uintptr_t device_address(const void* p, size_t bytes, Lookup lookup) {
  const HostRange r = lookup(p);
  if (bytes == 0 || r.at < r.start || bytes > r.bytes || r.at - r.start > r.bytes - bytes) return 0;
  return r.at;
}
