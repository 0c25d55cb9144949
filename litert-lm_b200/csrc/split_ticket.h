// Arrival tickets of a kernel whose key splits are joined by the last CTA to finish.  The tickets live in one array per
// GPU that every call shares, so they have to come back to zero whatever the calls do.  A unit (kv head, row tile) has
// a ticket of its own for every split count, and an arrival adds one modulo that count: a ticket only ever sees calls of
// one modulus, each of which arrives exactly that often, so it is at zero when they are done, also when two calls
// overlapped (which the entry point forbids) and each took the other's arrivals for its own.  One ticket per unit, set
// to zero by the last arrival, stayed off zero after such a pair and joined the splits of all later calls too early.
#pragma once

#ifdef __CUDACC__
#define B2_TICKET_FN __host__ __device__ inline
#else
#define B2_TICKET_FN inline
#endif

namespace b200lm {

constexpr int kTicketSplits = 256;         // most splits of a unit
constexpr int kTicketUnits = 128;          // most units of a call with splits: two splits each fill 256 SMs

constexpr int kTicketWords = (kTicketSplits + 1) * kTicketUnits;
// The tickets of a call, one per unit.
B2_TICKET_FN unsigned* ticket_row(unsigned* tickets, int nsplit) { return tickets + nsplit * kTicketUnits; }

// Arrival of one split; true for the last one.  `inc` is atomicInc: returns the old value v and stores v >= top ? 0 : v + 1.
template <typename Inc>
B2_TICKET_FN bool ticket_last(unsigned* ticket, int nsplit, const Inc& inc) {
  return (int)inc(ticket, (unsigned)(nsplit - 1)) == nsplit - 1;
}

}  // namespace b200lm
