// Host checks of the double -> float-pair splits of dd.h: reads doubles, writes
// hi, lo of dd_from_double, dd_from_double_z, dd_from_double_near and of
// dd_from_double3 over consecutive triples.
#include <cstdio>
#include <vector>

#include "dd.h"

int main() {
  std::vector<double> x;
  double v;
  while (std::fread(&v, sizeof v, 1, stdin) == 1) x.push_back(v);
  std::vector<float> out;
  auto put = [&](nw::dd a) {
    out.push_back(a.hi);
    out.push_back(a.lo);
  };
  for (double d : x) put(nw::dd_from_double(d));
  for (double d : x) put(nw::dd_from_double_z(d));
  for (double d : x) put(nw::dd_from_double_near(d));
  for (size_t i = 0; i + 2 < x.size(); i += 3) {
    nw::dd t[3];
    nw::dd_from_double3(&x[i], t);
    for (const nw::dd& a : t) put(a);
  }
  return std::fwrite(out.data(), sizeof(float), out.size(), stdout) == out.size() ? 0 : 1;
}
