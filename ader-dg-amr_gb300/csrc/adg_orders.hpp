// The sample orders of training epochs on their way to the GPU.
#pragma once

#include <cstddef>
#include <cstring>

namespace adg {

// Queues the copy of an epoch's order; the caller may rewrite `order` at once.
// A queued copy reads its source when the stream comes to it, which is behind
// the kernels of the epochs before, so the order goes through two host
// buffers in turn and a buffer is rewritten only after its last copy is done.
// Port: wait(b) for buffer b's last copy, buffer(b, n), copy(b, n) queues one.
template <class Port>
bool send_order(Port& port, const int* order, size_t n, int epoch) {
  const int b = epoch & 1;
  if (!port.wait(b)) return false;
  std::memcpy(port.buffer(b, n), order, n * sizeof(int));
  return port.copy(b, n);
}

}  // namespace adg
