// Upward passes of different degrees by two threads (csrc/hr_aux.cu,
// csrc/hr_moments_tc.cu): the launch of one between the other's setting of the
// kernel's shared-memory limit and its launch.
#include <cstdio>
#include <functional>

#include "../../high-order-regularization_b200/csrc/hr_device.h"
#include "fake_launch.h"

using namespace hr;

int main() {
  for (int channels : {6, 9, 106, 109}) {  // 100 +: on the tensor cores
    auto pass = [&](int P1) {
      MomTree t{};
      t.nitems = 1;
      if (channels < 100) launch_moments(channels, P1, t, MomTree{}, nullptr);
      else
        launch_moments_tc(channels == 109, nullptr, 1, P1, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                          nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
    };
    for (int P1 = 2; P1 <= (channels < 100 ? 16 : 11); P1++)
      for (int other : {2, 11}) {
        fake_launch = FakeLaunch{};
        fake_launch.between = [&] { pass(other); };
        pass(P1);
        if (fake_launch.launches != 2 || fake_launch.refused || fake_launch.most > (227 << 10)) {
          printf("channels %d: P + 1 = %d beside %d: %d of %d launches refused\n", channels, P1, other,
                 fake_launch.refused, fake_launch.launches);
          return 1;
        }
      }
  }
  return 0;
}
