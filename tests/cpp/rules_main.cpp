// Prints the decisions of kds_rules.h for the arguments given, one per line.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "kds_rules.h"

int main(int argc, char** argv) {
  if (argc == 6 && !strcmp(argv[1], "first_stamp")) {
    std::printf("%d\n", kds::first_stamp_on_device(atoi(argv[2]), atoi(argv[3]), atoi(argv[4]), atoi(argv[5])) ? 1 : 0);
    return 0;
  }
  if (argc == 3 && !strcmp(argv[1], "cluster")) {  // the largest size that fits
    std::printf("%d\n", kds::largest_cluster([&](int n) { return n <= atoi(argv[2]); }));
    return 0;
  }
  if (argc > 2 && !strcmp(argv[1], "devices")) {  // per device: was it new?  (added then)
    kds::DeviceSet set;
    for (int i = 2; i < argc; ++i) {
      std::printf("%d\n", set.has(atoi(argv[i])) ? 0 : 1);
      set.add(atoi(argv[i]));
    }
    return 0;
  }
  return 2;
}
