// serve_ticket.h -- how a worker of the element-mode request loop waits for
// its next load case (serve_modes.cu).  Plain C++, so that the rule can be run
// without a device.
#pragma once

#ifdef __CUDACC__
#define SP_HOST_DEVICE __host__ __device__
#else
#define SP_HOST_DEVICE
#endif

namespace sp {

struct ServeWait {
  long long ticket = -1;  // taken and not yet published
  long long idle = 0;     // polls since the last publication
  long long seen = -1;    // published load cases at the last poll
};

constexpr long long SERVE_WAIT = -1;   // poll again
constexpr long long SERVE_LEAVE = -2;  // no work, and none to come
constexpr long long SERVE_LOST = -3;   // gave up a ticket

// Polls after which a worker leaves, in idle limits of the dispatcher (its
// polls since the last publication): without a ticket nothing is lost with it.
// With one, its load case would be: the counter has moved past the ticket.  So
// it leaves with the dispatcher, which leaves by its own limit and frees what
// is unpublished.  A poll of the dispatcher (two reads of host memory) may take
// many of a worker's; the bound here is for a dispatcher that does not run.
constexpr long long SERVE_IDLE_FREE = 8, SERVE_IDLE_HELD = 4096;

// One poll.  gone: the dispatcher had left, read before `end`, the load cases
// published; claimed() reads the ticket counter, take() advances it.  Returns
// the load case to solve (>= 0) or one of the above.
template <typename Claimed, typename Take>
SP_HOST_DEVICE inline long long serve_poll(ServeWait &w, bool gone, long long end,
                                           long long idle_limit, const Claimed &claimed,
                                           const Take &take) {
  if (end != w.seen) w.idle = 0;
  w.seen = end;
  if (w.ticket < 0 && claimed() < end) w.ticket = take();
  if (w.ticket >= 0 && w.ticket < end) return w.ticket;
  if (gone) return SERVE_LEAVE;
  w.idle++;
  if (w.ticket < 0) return w.idle > SERVE_IDLE_FREE * idle_limit ? SERVE_LEAVE : SERVE_WAIT;
  return w.idle > SERVE_IDLE_HELD * idle_limit ? SERVE_LOST : SERVE_WAIT;
}

}  // namespace sp
