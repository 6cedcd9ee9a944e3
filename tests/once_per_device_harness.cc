// OncePerDevice (plum_gb300/csrc/per_device.h), compiled here for the host, against a
// fake of the call it guards. Exits 1 with a line on what went wrong.
#include <cstdio>
#include <map>
#include <thread>
#include <vector>

#include "../plum_gb300/csrc/per_device.h"

static int bad(const char* what) {
  std::printf("%s\n", what);
  return 1;
}

int main() {
  plum::OncePerDevice a, b;
  std::map<int, int> calls;
  const auto on = [&](plum::OncePerDevice& o, int dev, int rc) {
    return o.run(dev, [&] {
      calls[dev]++;
      return rc;
    });
  };
  for (int i = 0; i < 3; i++)
    if (on(a, 0, 0)) return bad("device 0");
  if (calls[0] != 1) return bad("device 0 is set once");
  if (on(a, 1, 0) || calls[1] != 1) return bad("device 1 is set after device 0");
  if (on(a, 63, 0) || on(a, 63, 0) || calls[63] != 1) return bad("the last device");
  if (on(b, 0, 0) || calls[0] != 2) return bad("each kernel has its own flag");
  if (on(a, 2, 7) != 7 || on(a, 2, 0) != 0 || on(a, 2, 0) != 0 || calls[2] != 2)
    return bad("a failed call is made again");
  for (int dev : {-1, 64, 1000})
    if (on(a, dev, 0) || on(a, dev, 0) || calls[dev] != 2) return bad("a device out of range");
  // threads on two devices: every thread finds its device set on return
  plum::OncePerDevice c;
  std::atomic<int> set[2] = {};
  std::atomic<int> missed{0};
  std::vector<std::thread> t;
  for (int i = 0; i < 8; i++)
    t.emplace_back([&, i] {
      for (int k = 0; k < 1000; k++) {
        c.run(i & 1, [&] { return set[i & 1]++, 0; });
        if (set[i & 1] == 0) missed++;
      }
    });
  for (auto& x : t) x.join();
  if (missed || set[0] < 1 || set[1] < 1 || set[0] > 4 || set[1] > 4) return bad("threads");
  return 0;
}
