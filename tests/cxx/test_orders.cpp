// The epochs' sample orders (adg_orders.hpp) over a queue that reads its
// sources as late as a stream may: when it is waited for, and at the end.
#include <algorithm>
#include <cstdio>
#include <deque>
#include <numeric>
#include <random>
#include <vector>

#include "adg_orders.hpp"

struct LatePort {
  size_t n;
  std::vector<int> host[2];
  struct Copy {
    int b;
  };
  std::deque<Copy> queue;
  std::vector<std::vector<int>> received;
  explicit LatePort(size_t count) : n(count) { host[0].resize(n), host[1].resize(n); }
  void run() {
    received.push_back(host[queue.front().b]);
    queue.pop_front();
  }
  bool wait(int b) {
    size_t upto = 0;  // in stream order, up to the buffer's last copy
    for (size_t i = 0; i < queue.size(); ++i)
      if (queue[i].b == b) upto = i + 1;
    for (; upto; --upto) run();
    return true;
  }
  int* buffer(int b, size_t) { return host[b].data(); }
  bool copy(int b, size_t) {
    queue.push_back({b});
    return true;
  }
};

int main() {
  std::vector<int> order(1000);
  std::iota(order.begin(), order.end(), 0);
  std::mt19937_64 rng(7);
  LatePort port(order.size());
  std::vector<std::vector<int>> sent;
  for (int epoch = 0; epoch < 9; ++epoch) {
    std::shuffle(order.begin(), order.end(), rng);
    sent.push_back(order);
    if (!adg::send_order(port, order.data(), order.size(), epoch)) return 1;
    if (port.queue.empty()) {
      std::printf("nothing overlaps\n");
      return 1;
    }
  }
  while (!port.queue.empty()) port.run();
  if (port.received != sent) {
    std::printf("an epoch got another order than its own\n");
    return 1;
  }
  std::printf("ok\n");
  return 0;
}
