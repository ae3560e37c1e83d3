// Host-side check (no GPU) of the divisions written out in radio_device.cuh:
// over_light_speed and divide3 against the processor's own quotients, bit for
// bit, over random operands of every magnitude and at the edges of their
// ranges.  Prints "ok" or the first failed quotients; exit status 1 on a
// failure.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>

#include "radio_device.cuh"

using namespace c8r;

namespace {

int failures = 0;

void expect_same(double got, double want, char const* what, double a, double b) {
  if (std::memcmp(&got, &want, sizeof got) == 0 || (std::isnan(got) && std::isnan(want))) return;
  if (++failures <= 10) std::printf("FAIL %s %a / %a: %a, not %a\n", what, a, b, got, want);
}

void check_vector(double x, double y, double z) {
  double const d = std::sqrt(x * x + y * y + z * z);
  double kx = x, ky = y, kz = z;
  divide3(kx, ky, kz, d);
  expect_same(kx, x / d, "divide3 x", x, d);
  expect_same(ky, y / d, "divide3 y", y, d);
  expect_same(kz, z / d, "divide3 z", z, d);
}

}  // namespace

int main() {
  std::mt19937_64 rng(20240607);
  // a random mantissa, one in four of them near all ones or near a power of two
  auto number = [&](int low, int high) {
    uint64_t mantissa = rng() & 0xfffffffffffffull;
    unsigned const kind = rng() & 7u;
    if (kind == 0) mantissa = 0xfffffffffffffull - (mantissa & 15u);
    if (kind == 1) mantissa &= 15u;
    double const m = 1. + static_cast<double>(mantissa) * 0x1p-52;
    int const e = low + static_cast<int>(rng() % static_cast<uint64_t>(high - low + 1));
    return std::ldexp((rng() & 1u) ? -m : m, e);
  };
  for (int i = 0; i < 4000000; ++i) {  // the magnitudes of a shower
    double const x = number(-20, 60);
    expect_same(over_light_speed(x), x / kSpeedOfLight, "over_light_speed", x, kSpeedOfLight);
    check_vector(number(-20, 20), number(-20, 20), number(-20, 20));
  }
  for (int i = 0; i < 1000000; ++i) {  // every magnitude
    double const x = number(-1074, 1023);
    expect_same(over_light_speed(x), x / kSpeedOfLight, "over_light_speed", x, kSpeedOfLight);
    check_vector(number(-1074, 1023), number(-1074, 1023), number(-1074, 1023));
    check_vector(number(-640, -360), number(-640, 640), number(-640, 640));
    check_vector(number(-640, -520), number(-640, -520), number(-640, -520));
  }
  double const special[] = {0., -0., 1., -1., 0x1p-400, 0x1.fffffffffffffp-401, 0x1p400, 0x1.fffffffffffffp399, 0x1p-600,
                            0x1p600, std::numeric_limits<double>::min(), std::numeric_limits<double>::denorm_min(),
                            std::numeric_limits<double>::max(), std::numeric_limits<double>::infinity(),
                            std::numeric_limits<double>::quiet_NaN()};
  for (double x : special) {
    expect_same(over_light_speed(x), x / kSpeedOfLight, "over_light_speed", x, kSpeedOfLight);
    for (double y : special)
      for (double z : special) check_vector(x, y, z);
  }
  if (failures) return 1;
  std::printf("ok\n");
  return 0;
}
