// Which ranks of a job run on one device: every rank contributes the identity of its own.
#pragma once
#include <cstring>
#include <vector>

namespace hetuCTR {

struct DeviceIdentity {
  char uuid[16];
};

inline bool shares_device(const std::vector<DeviceIdentity> &of_rank, int rank) {
  for (size_t p = 0; p < of_rank.size(); p++)
    if ((int)p != rank && std::memcmp(of_rank[p].uuid, of_rank[rank].uuid, sizeof(of_rank[p].uuid)) == 0) return true;
  return false;
}

}  // namespace hetuCTR
