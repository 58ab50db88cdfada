// Sine-transform plans of several sizes in use at once (csrc/hr_poisson.cu).
#include <cstdio>
#include <vector>

#include "../../high-order-regularization_b200/csrc/hr_runtime.h"
#include "fake_launch.h"

namespace hr {
struct Dst1Plan;
Dst1Plan* dst1_plan_create(Ctx& C, int n);
void dst1_plan_destroy(Dst1Plan* D);
void dst1_execute(Ctx& C, Dst1Plan* D, const double* in_host, double* out_host);
}  // namespace hr

int main() {
  hr::Ctx C;
  // pairs that share a kernel: the general one, and that of lines of 64 R - 1 points
  for (auto sizes : {std::pair<int, int>(265, 3), {127, 127}}) {
    hr::Dst1Plan* a = hr::dst1_plan_create(C, sizes.first);
    hr::Dst1Plan* b = hr::dst1_plan_create(C, sizes.second);
    const size_t m = (size_t)sizes.first * sizes.first * sizes.first;
    std::vector<double> in(m), out(m);
    for (hr::Dst1Plan* p : {a, b, a}) {
      fake_launch.launches = fake_launch.refused = 0;
      try {
        hr::dst1_execute(C, p, in.data(), out.data());
      } catch (const hr::Error& e) {
        fake_launch.refused++;
      }
      if (fake_launch.launches != 3 || fake_launch.refused || fake_launch.most > (227 << 10)) {
        printf("n = %d beside %d: %d of %d launches refused\n", sizes.first, sizes.second, fake_launch.refused,
               fake_launch.launches);
        return 1;
      }
    }
    hr::dst1_plan_destroy(a);
    hr::dst1_plan_destroy(b);
  }
  return 0;
}
