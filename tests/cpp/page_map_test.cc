// A tensor map over a paged cache counts every page that starts within 32 TB of the first: of one kv head and of many.
#include <cstdio>
#include <initializer_list>

#include "page_map.h"

int main() {
  const unsigned long long reach = 1ull << 45;
  for (unsigned long long hd : {128, 256})
    for (unsigned long long hkv : {1, 2, 3, 4, 16, 32, 1000}) {
      const unsigned long long bytes = hkv * 256 * hd * 2, pages = b200lm::map_pages(bytes), last = (reach - 1) / bytes;
      if (pages <= last || pages > 1ull << 31) {
        std::printf("%llu kv heads of %llu: %llu pages, the last one to reach is %llu\n", hkv, hd, pages, last);
        return 1;
      }
    }
  return 0;
}
