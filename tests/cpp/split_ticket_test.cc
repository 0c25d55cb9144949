// Arrivals of two calls in every order (exhaustive for few splits, random beyond): all tickets must be zero when both
// are done, and a call that runs alone afterwards joins each unit once, at its last arrival.
#include <cstdio>
#include <random>
#include <vector>

#include "split_ticket.h"

using namespace b200lm;

static unsigned inc(unsigned* t, unsigned top) {      // atomicInc
  const unsigned v = *t;
  *t = v >= top ? 0u : v + 1u;
  return v;
}

struct Call { int units, nsplit; };

static bool clean(const std::vector<unsigned>& t) {
  for (unsigned v : t)
    if (v) return false;
  return true;
}

static bool alone(std::vector<unsigned>& t, Call c) {
  for (int u = 0; u < c.units; ++u)
    for (int s = 0; s < c.nsplit; ++s)
      if (ticket_last(ticket_row(t.data(), c.nsplit) + u, c.nsplit, inc) != (s == c.nsplit - 1)) return false;
  return clean(t);
}

int main() {
  const Call calls[] = {{1, 2}, {1, 3}, {1, 4}, {2, 3}, {4, 31}, {37, 4}, {74, 2}, {128, 2}, {1, 148}, {1, 256}};
  std::vector<unsigned> t(kTicketWords, 0u);
  std::mt19937 rng(1);
  for (const Call& a : calls)
    for (const Call& b : calls) {
      const int na = a.units * a.nsplit, nb = b.units * b.nsplit;
      const bool all = na + nb <= 12;
      for (long order = 0; order < (all ? 1L << (na + nb) : 50); ++order) {
        if (all && __builtin_popcountl(order) != na) continue;
        int ia = 0, ib = 0;
        for (int i = 0; i < na + nb; ++i) {
          const bool first = all ? order >> i & 1 : (int)(rng() % (unsigned)(na - ia + nb - ib)) < na - ia;
          int& at = first ? ia : ib;
          const Call& c = first ? a : b;
          ticket_last(ticket_row(t.data(), c.nsplit) + at / c.nsplit, c.nsplit, inc);
          ++at;
        }
        if (!clean(t)) { printf("off zero after %dx%d and %dx%d\n", a.units, a.nsplit, b.units, b.nsplit); return 1; }
      }
      if (!alone(t, a) || !alone(t, b)) { printf("joined early after %dx%d and %dx%d\n", a.units, a.nsplit, b.units, b.nsplit); return 1; }
    }
  printf("ok\n");
  return 0;
}
