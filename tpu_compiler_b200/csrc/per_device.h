// Set-up that the driver keeps for each device by itself (a kernel's attributes): done once for every device, by whichever
// thread comes first, while the others wait. One that throws is done again by the next caller.
#pragma once
#include <mutex>
#include <set>

namespace tpucb {

class OncePerDevice {
public:
  template <class Work> void run(int device, Work work) {
    std::lock_guard<std::mutex> g(m_);
    if (done_.count(device)) return;
    work();
    done_.insert(device);
  }

private:
  std::mutex m_;
  std::set<int> done_;
};

} // namespace tpucb
