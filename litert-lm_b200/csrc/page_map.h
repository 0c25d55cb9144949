// How many pages a tensor map over a paged cache counts.  Only the caller knows how many there are, and a page past the map's
// count reads as zeros instead of failing, so the map takes in every page that starts within 32 TB of the first, whatever a
// page's size: far more than a GPU and its host hold.
#pragma once

namespace b200lm {

constexpr unsigned long long kMapBytes = 1ull << 45;
// A page number is an int; the smallest page of the kernels that use a map (one kv head of 128 in bf16) has 64 KB.
constexpr unsigned long long map_pages(unsigned long long page_bytes) {
  return (kMapBytes + page_bytes - 1) / page_bytes < 1ull << 31 ? (kMapBytes + page_bytes - 1) / page_bytes : 1ull << 31;
}

}  // namespace b200lm
