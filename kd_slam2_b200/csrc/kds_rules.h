// Rules that choose between two forms of a call, as plain host functions (no CUDA), so that they
// can be checked without a device.
#pragma once

#include <atomic>
#include <cstdint>

namespace kds {

// Devices on which something that each one needs has been done (a kernel's limits belong to a
// device).  Safe with several threads; a device above the 64th is never in it.
class DeviceSet {
 public:
  bool has(int device) const { return in(device) && ((bits_.load() >> device) & 1u); }
  void add(int device) {
    if (in(device)) bits_.fetch_or(1ull << device);
  }

 private:
  static bool in(int device) { return device >= 0 && device < 64; }
  std::atomic<uint64_t> bits_{0};
};

// Whether a request's first stamp is found by a kernel on the calling thread's device: the
// scratch that the kernel writes is the server's, so the caller, the server and both ends of
// the stamps must be on one device.  Between two devices the pointers of one are not the
// other's to read or write; the host copy works from any of them.
inline bool first_stamp_on_device(int current, int server, int first, int last) {
  return current == server && first == server && last == server;
}

// Blocks of the largest cluster that the device schedules (fits(n)), 0 for none: 16 where it
// gives leave, else the portable 8.  A device that is shared or partitioned may have room for
// neither beside the shared memory that a block needs.
template <class Fits>
int largest_cluster(Fits fits) {
  return fits(16) ? 16 : (fits(8) ? 8 : 0);
}

}  // namespace kds
