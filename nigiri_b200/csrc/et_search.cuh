// get_earliest_transport of one stop of one route for one query, shared by
// the batched route scan and the single-query no-allocation search.
#pragma once

#include "engine.cuh"

namespace b2r::dev {

// The service days of a bitfield around `day` in search direction: bit i =
// day + i (forward) or day - i (backward), i < 6; days outside the bitfield
// are 0.
__device__ __forceinline__ uint32_t six_days(dtt const& T, uint32_t bf, bool fwd, uint16_t day) {
  static_assert(B2R_MAX_DAYS == 512);
  auto const lo = static_cast<int>(day) - (fwd ? 0 : 5);
  auto const word = lo >> 6, sh = lo & 63;
  auto const at = [&](int w) { return w >= 0 && w < 8 ? __ldg(T.bf + 8ull * bf + w) : 0ull; };
  auto x = at(word) >> sh;
  if (sh > 58) x |= at(word + 1) << (64 - sh);
  auto const six = static_cast<uint32_t>(x) & 63u;
  return fwd ? six : __brev(six) >> 26;
}

// get_earliest_transport, raptor.h:1351-1442.  Event columns are ordered by
// minutes after midnight (loader/get_index.h), so the reference's
// linear_lb is a lower bound found by binary search; the scan that follows
// visits events in the reference's order with the same prune / skip / day
// rules.  Routes flagged unsorted use the reference's linear seek.
// Two shortcuts leave the result as it is: the route's six service days are
// read at once, and a later day whose first possible minute is already
// pruned ends the search (every event from there on is later still).
__device__ __forceinline__ bool et_search(dtt const& T, bool fwd, route_rec const& R, uint32_t si, uint16_t day_at_stop,
                                          int mam, int lbv, int tad_k, uint16_t base, uint32_t& out_off,
                                          uint16_t& out_day, uint32_t& n_ev, uint32_t& n_days) {
  auto const n = R.n_t;
  auto const* col = T.st + (R.st + n * (si * 2u - (fwd ? 0u : 1u)));
  auto days = six_days(T, R.bf, fwd, day_at_stop);
  ++n_days;
  for (; days != 0u; days &= days - 1u) {
    auto const i = __ffs(days) - 1;
    auto const day = static_cast<uint16_t>(fwd ? day_at_stop + i : day_at_stop - i);
    uint32_t j = 0;
    if (i != 0) {
      if (to_delta_key(fwd, day, base, fwd ? 0 : 1439) + lbv > tad_k) return false;
    } else if ((R.flags & kRouteSorted) != 0u) {
      // forward: the first index with mam >= m; backward, from the end, the
      // first with mam <= m: n - upper_bound(m).  An event's minutes are
      // the bits above its 5 days, so it is compared as a whole.
      auto const m = static_cast<uint32_t>(fwd ? mam : mam + 1) << 5;
      uint32_t lo = 0, len = n;
      while (len != 0u) {
        auto const half = len >> 1;
        ++n_ev;
        auto const below = static_cast<uint32_t>(__ldg(col + lo + half)) < m;
        lo = below ? lo + half + 1u : lo;
        len = below ? len - half - 1u : half;
      }
      j = fwd ? lo : n - lo;
    } else {
      for (j = 0; j < n; ++j) {
        auto const em = static_cast<int>(__ldg(col + (fwd ? j : n - 1 - j)) >> 5);
        if (!(fwd ? em < mam : em > mam)) break;
      }
    }
    for (; j < n; ++j) {
      auto const idx = fwd ? j : n - 1u - j;
      auto const e = __ldg(col + idx);
      ++n_ev;
      auto const em = static_cast<int>(e >> 5);
      if (to_delta_key(fwd, day, base, em) + lbv > tad_k) return false;
      if (i == 0 && !(fwd ? mam <= em : mam >= em)) continue;
      auto const sday = static_cast<uint16_t>(static_cast<int>(day) - static_cast<int>(e & 31u));
      // the route runs on `day`; a transport with the route's days does too
      if ((R.flags & kRouteOneDays) != 0u) {
        if (sday != day && !bf_test(T, R.bf, sday)) continue;
      } else if (!bf_test(T, __ldg(T.transport_bf + R.t0 + idx), sday)) {
        continue;
      }
      out_off = idx;
      out_day = sday;
      return true;
    }
  }
  return false;
}

__device__ __forceinline__ route_rec load_route(dtt const& T, uint32_t r) {
  auto const* p = reinterpret_cast<uint4 const*>(T.routes + r);
  auto const a = __ldg(p), b = __ldg(p + 1);
  return {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
}

}  // namespace b2r::dev
