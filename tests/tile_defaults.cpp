// The default tile of a mesh: rows "kind threads" for (key, p, elements per SM,
// one more element, boundary sides) arguments; the first line is the SM count.
#include <cstdio>
#include <cstdlib>

#include "../dgm_b200/csrc/dgmx_internal.hpp"

int main(int argc, char **argv) {
  const int sms = dgmx::sm_count(0);
  std::printf("%d\n", sms);
  for (int i = 1; i + 4 < argc; i += 5) {
    const int key = std::atoi(argv[i]), p = std::atoi(argv[i + 1]);
    const int ne = std::atoi(argv[i + 2]) * sms + std::atoi(argv[i + 3]);
    const dgmx::KernelOps *o = dgmx::default_ops(key, p + 1, p + 2, ne, std::atoi(argv[i + 4]) != 0, 0);
    std::printf("%d %d\n", o ? o->warp : -1, o ? o->nt : -1);
  }
}
