// Device-side journey reconstruction: a group of NW warps per journey walks
// the round times of its query backwards (src/routing/raptor/reconstruct.cc:
// 22-877 for Vias = 0) and then applies the footpath optimisations of
// src/routing/raptor/optimize_footpaths.cc.
//
// A journey is a chain of dependent loads, leg after leg, so what bounds the
// kernel is that chain's length, not bandwidth.  The search for the
// transport that produced a label -- every (route, stop position) pair of
// every footpath candidate, several hundred at a busy stop -- is split
// across the group's threads and the first success in the reference's
// iteration order taken; each pair's record (lrs_rec) holds what its search
// needs, so no route array stands between the pair and its event column.
// The sequential parts run redundantly on all threads; the legs live in
// shared memory until the journey is finished.  NW = 4 where journeys are
// few and their latency counts (4 x 32 pairs a pass), NW = 1 where there
// are more journeys than the device has room for groups of four.
#pragma once

#include "engine.cuh"

namespace b2r::dev {

// a (route, stop position) pair whose event column holds the wanted minute
struct recon_cand {
  uint32_t t, day, i, sec, r, owner, is_rt;
  uint4 rec;
};

template <int NW>
struct recon_smem {
  b2r_leg legs[kMaxLegs];
  recon_cand cand[NW * 32];
  uint32_t mask[NW];
  double pen[NW];
  uint32_t pen_at[NW];
};

template <int NW>
struct recon_ctx {
  static constexpr uint32_t kT = NW * 32u;  // threads of the group
  state const* st;
  dtt const* T;
  slot_t const* sl;
  uint32_t s;          // slot
  bool fwd;
  uint16_t qtag;
  int32_t base_days;
  uint16_t base;
  bool ontrip;
  journey_rec* j;
  recon_smem<NW>* sm;
  b2r_leg* legs;       // sm->legs, written by thread 0
  int n_legs;
  bool failed;
  uint32_t lane, wid, tid;
  b2r_leg last;        // last pushed leg (all threads)

  __device__ static void sync() {
    if constexpr (NW == 1) __syncwarp();
    else __syncthreads();
  }
  __device__ static bool any(bool x) {
    if constexpr (NW == 1) return __any_sync(kFull, x);
    else return __syncthreads_or(x) != 0;
  }

  // ------------------------------------------------------------- access
  __device__ int rt_t(unsigned k, uint32_t l) const {  // delta_t of round_times[k][l]
    auto const key = dec(st->rt[(static_cast<size_t>(k) * T->n_loc + l) * st->S + s], qtag);
    return from_key(fwd, key);
  }
  __device__ int inv() const { return fwd ? 32767 : -32768; }
  __device__ bool beq(int a, int b) const { return fwd ? a <= b : a >= b; }
  __device__ int dir(int a) const { return fwd ? a : -a; }
  __device__ uint32_t n_stops(uint32_t r) const { return T->route_stop_idx[r + 1] - T->route_stop_idx[r]; }
  __device__ uint32_t stopw(uint32_t r, uint32_t i) const { return T->route_stops[T->route_stop_idx[r] + i]; }
  __device__ int32_t day_time(uint16_t day, uint16_t e) const {
    return (T->internal_from_days + static_cast<int32_t>(day)) * 1440 + (e & 31) * 1440 + (e >> 5);
  }
  __device__ int unix_to_delta(int32_t t) const { return clamp16(t - base_days * 1440); }
  __device__ int32_t delta_to_unix(int d) const { return base_days * 1440 + d; }
  __device__ b2r_offset const* start_offs() const { return st->off_pool + sl->soff_off; }
  __device__ b2r_offset const* dest_offs() const { return st->off_pool + sl->doff_off; }

  __device__ uint32_t root(uint32_t idx) const {
    if (T->parent == nullptr) return idx;
    auto l = idx;
    for (int i = 0;; ++i) {
      auto const p = T->parent[l];
      if (p == B2R_INVALID_IDX) break;
      if (p == idx || i > 20) {
        l = T->parent[idx];
        break;
      }
      l = p;
    }
    return l;
  }
  // matches(tt, mode, a, b), for_each_meta.h:47-70 (no equivalence lists)
  __device__ bool matches(uint8_t mode, uint32_t a, uint32_t b) const {
    if (a == b) return true;
    if (mode == B2R_MATCH_EXACT || T->children_idx == nullptr) {
      if (mode == B2R_MATCH_EQUIVALENT) return root(a) == b;
      return false;
    }
    if (mode == B2R_MATCH_INTERMODAL) {
      for (auto i = T->children_idx[a]; i != T->children_idx[a + 1]; ++i) {
        auto const c = T->children[i];
        if (T->loc_type != nullptr && T->loc_type[c] == B2R_LOC_GENERATED_TRACK && c == b) return true;
      }
      return false;
    }
    auto const r = mode == B2R_MATCH_EQUIVALENT ? root(a) : a;
    if (r == b) return true;
    for (auto i = T->children_idx[r]; i != T->children_idx[r + 1]; ++i) {
      auto const c = T->children[i];
      if (c == b) return true;
      for (auto j = T->children_idx[c]; j != T->children_idx[c + 1]; ++j) {
        if (T->children[j] == b) return true;
      }
    }
    return false;
  }
  __device__ bool is_journey_start(uint32_t l) const {
    auto const* o = start_offs();
    for (auto i = 0U; i != sl->n_soff; ++i) {
      if (matches(sl->start_mode, o[i].target, l)) return true;
    }
    return false;
  }

  // -------------------------------------------------------------- legs
  __device__ b2r_leg make_leg(uint32_t a, uint32_t b, int32_t ta, int32_t tb) const {
    b2r_leg l{};
    l.rt_transport = B2R_INVALID_IDX;
    l.from = fwd ? a : b;
    l.to = fwd ? b : a;
    l.dep_time = fwd ? ta : tb;
    l.arr_time = fwd ? tb : ta;
    return l;
  }
  __device__ static void set_run(b2r_leg& l, uint32_t t, uint16_t day, uint32_t a, uint32_t b) {
    l.kind = B2R_LEG_TRANSPORT;
    l.transport = t;
    l.day = day;
    l.stop_from = static_cast<uint16_t>(a < b ? a : b);
    l.stop_to = static_cast<uint16_t>((a < b ? b : a) + 1u);
  }
  __device__ static void set_fp(b2r_leg& l, uint32_t target, int dur) {
    l.kind = B2R_LEG_FOOTPATH;
    l.transport = target;
    l.duration = static_cast<int16_t>(dur > 511 ? 511 : dur);
    l.transport_mode_id = 0;
  }
  __device__ static void set_off(b2r_leg& l, b2r_offset const& o) {
    l.kind = B2R_LEG_OFFSET;
    l.transport = o.target;
    l.duration = o.duration;
    l.transport_mode_id = o.transport_mode_id;
  }
  __device__ void push(b2r_leg const& l) {
    if (n_legs >= kMaxLegs) {
      failed = true;
      return;
    }
    if (tid == 0) legs[n_legs] = l;
    ++n_legs;
    last = l;
  }

  // reconstruct.cc:180-280 (single pass: no vias).  The stops before the
  // exit stop are split across the lanes; the ballot keeps the first one in
  // the reference's order.  A section lacking one of the flags `sec` ends
  // the ride (reconstruct.cc:239-250): stops at or past the first such
  // section do not count.  rec: the exit stop's pair record.  Called by
  // whole warps with equal arguments.
  __device__ bool find_start_in_prev_round(unsigned k, uint4 rec, uint32_t t, uint16_t day, uint32_t finish,
                                           uint32_t sec, b2r_leg& out) const {
    auto const sb = T->route_stop_idx[rec.x];
    auto const size = T->route_stop_idx[rec.x + 1] - sb;
    // event column entry of trip t at stop i: evs[2 i n_t], its arrival n_t before
    auto const n_t = rec.w;
    auto const* evs = T->st + (rec.y - 2u * finish * n_t) + (t - rec.z);
    auto const n = fwd ? finish + 1u : size - finish;
    for (auto i0 = 1u; i0 < n; i0 += 32u) {
      auto const i = i0 + lane;
      bool ok = false, cut = false;
      uint32_t si = 0, l = 0;
      int event_time = 0;
      if (i < n) {
        si = fwd ? finish - i : finish + i;
        auto const w = T->route_stops[sb + si];
        auto const e = evs[fwd ? 2u * si * n_t : (2u * si - 1u) * n_t];
        l = B2R_STOP_LOC(w);
        // departure section forward, arrival section backward
        cut = sec != 0u && !section_ok(*T, sb, fwd ? si : si - 1u, sec);
        // plain in / out bits for every profile: reconstruct.cc:252-253
        // passes the bool is_wheelchair as a profile index (0 or 1)
        if (!cut && !((fwd && !B2R_STOP_IN(w)) || (!fwd && !B2R_STOP_OUT(w)))) {
          event_time = unix_to_delta(day_time(day, e));
          auto const round_time = rt_t(k - 1, l);
          ok = beq(round_time, event_time) ||
               (k == 1 && sl->start_mode == B2R_MATCH_EQUIVALENT && is_journey_start(l) &&
                (ontrip ? beq(round_time, event_time) : round_time == event_time));
        }
      }
      auto m = __ballot_sync(kFull, ok);
      auto const cuts = __ballot_sync(kFull, cut);
      if (cuts != 0u) m &= (1u << (__ffs(cuts) - 1)) - 1u;  // lanes before the first cut
      if (m != 0u) {
        auto const src = __ffs(m) - 1;
        si = __shfl_sync(kFull, si, src);
        l = __shfl_sync(kFull, l, src);
        event_time = __shfl_sync(kFull, event_time, src);
        auto const e = evs[fwd ? (2u * finish - 1u) * n_t : 2u * finish * n_t];
        out = make_leg(l, B2R_STOP_LOC(T->route_stops[sb + finish]), delta_to_unix(event_time), day_time(day, e));
        set_run(out, t, day, si, finish);
        return true;
      }
      if (cuts != 0u) return false;
    }
    return false;
  }

  // find_start_in_prev_round on a real-time run (rt::frun::from_rt): the
  // run's own stops and event times, as above.
  __device__ bool find_start_in_prev_round_rt(unsigned k, uint32_t x, uint32_t finish, uint32_t sec,
                                              b2r_leg& out) const {
    auto const sb = T->rt_stop_idx[x];
    auto const size = T->rt_stop_idx[x + 1] - sb;
    auto const* tm = T->rt_times + 2ull * (sb - x);
    auto const n = fwd ? finish + 1u : size - finish;
    for (auto i0 = 1u; i0 < n; i0 += 32u) {
      auto const i = i0 + lane;
      bool ok = false, cut = false;
      uint32_t si = 0, l = 0;
      int event_time = 0;
      if (i < n) {
        si = fwd ? finish - i : finish + i;
        auto const w = T->rt_stops[sb + si];
        l = B2R_STOP_LOC(w);
        cut = sec != 0u && (static_cast<uint32_t>(T->rt_sec[sb + (fwd ? si : si - 1u)]) & sec) != sec;
        if (!cut && !((fwd && !B2R_STOP_IN(w)) || (!fwd && !B2R_STOP_OUT(w)))) {
          event_time = unix_to_delta(tm[2u * si - (fwd ? 0u : 1u)]);
          auto const round_time = rt_t(k - 1, l);
          ok = beq(round_time, event_time) ||
               (k == 1 && sl->start_mode == B2R_MATCH_EQUIVALENT && is_journey_start(l) &&
                (ontrip ? beq(round_time, event_time) : round_time == event_time));
        }
      }
      auto m = __ballot_sync(kFull, ok);
      auto const cuts = __ballot_sync(kFull, cut);
      if (cuts != 0u) m &= (1u << (__ffs(cuts) - 1)) - 1u;
      if (m != 0u) {
        auto const src = __ffs(m) - 1;
        si = __shfl_sync(kFull, si, src);
        l = __shfl_sync(kFull, l, src);
        event_time = __shfl_sync(kFull, event_time, src);
        out = make_leg(l, B2R_STOP_LOC(T->rt_stops[sb + finish]), delta_to_unix(event_time),
                       tm[2u * finish - (fwd ? 1u : 0u)]);
        set_run(out, T->rt_static[x], T->rt_static_day[x], si, finish);
        out.rt_transport = x;
        return true;
      }
      if (cuts != 0u) return false;
    }
    return false;
  }

  // The transports of a pair's route whose event at its stop has the minutes
  // after midnight of `time` (reconstruct.cc:292-373), one at a time from
  // `cursor`: columns are ordered by minutes after midnight (kLrsSorted), so
  // they form one run found by binary search and visited in index order.
  __device__ uint16_t const* pair_col(uint4 rec) const { return T->st + rec.y - (fwd ? rec.w : 0u); }
  __device__ uint32_t first_cursor(int time, uint4 rec, bool sorted) const {
    if (!sorted) return 0u;
    auto const mam = static_cast<int16_t>((static_cast<int>(base) * 1440 + time) % 1440);
    auto const* col = pair_col(rec);
    uint32_t lo = 0, hi = rec.w;
    while (lo < hi) {
      auto const mid = (lo + hi) >> 1;
      if ((col[mid] >> 5) < static_cast<uint16_t>(mam < 0 ? 0 : mam)) lo = mid + 1;
      else hi = mid;
    }
    return lo;
  }
  __device__ bool next_transport(int time, uint4 rec, bool sorted, uint32_t& cursor, uint32_t& t,
                                 uint32_t& tday) const {
    auto const minutes = static_cast<int>(base) * 1440 + time;
    auto const day = static_cast<uint16_t>(minutes / 1440);
    auto const mam = static_cast<int16_t>(minutes % 1440);
    auto const* col = pair_col(rec);
    for (auto x = cursor; x < rec.w; ++x) {
      auto const cnt = delta_count(col[x]);
      auto const m = static_cast<int16_t>(cnt % 1440);
      if (m != mam) {
        if (sorted && m > mam) break;
        continue;
      }
      auto const td = static_cast<uint16_t>(static_cast<int>(day) - cnt / 1440);
      if (!bf_test(*T, T->transport_bf[rec.z + x], td)) continue;
      cursor = x + 1u;
      t = rec.z + x;
      tday = td;
      return true;
    }
    cursor = rec.w;
    return false;
  }

  // get_transport (reconstruct.cc:375-545) for a list of footpath
  // candidates, tried in order: candidate f reaches location `target(f)` at
  // `time(f)`; its real-time (run, stop position) pairs and then its (route,
  // stop position) pairs are visited in the reference's order
  // (reconstruct.cc:381-452 first).  All pairs of all candidates form one
  // sequence that the group takes kT at a time; the first success in
  // sequence order wins.
  // get(f, target, time) describes candidate f (lane-local; false: no such
  // candidate); returns the winning candidate or -1.
  template <typename Get>
  __device__ int get_transport(unsigned k, uint32_t n_cand, Get&& get, b2r_leg& out) const {
    for (auto f0 = 0u; f0 < n_cand; f0 += 32u) {
      // lane f: candidate f0 + f, its pair range and the inclusive prefix sum
      auto const f = f0 + lane;
      uint32_t tg = 0, pb = 0, cnt = 0, rb = 0, rcnt = 0;
      int tm = 0;
      if (f < n_cand && get(f, tg, tm)) {
        pb = T->lrs_idx[tg];
        rb = T->lrs_rt_idx[tg];
        rcnt = T->lrs_rt_idx[tg + 1] - rb;
        cnt = rcnt + (T->lrs_idx[tg + 1] - pb);
      }
      auto end = cnt;
      for (auto o = 1u; o < 32u; o <<= 1) {
        auto const v = __shfl_up_sync(kFull, end, o);
        if (lane >= o) end += v;
      }
      auto const total = __shfl_sync(kFull, end, 31);
      for (auto p0 = 0u; p0 < total; p0 += kT) {
        auto const p = p0 + tid;
        // owner candidate of pair p: the first lane whose prefix end > p
        uint32_t owner = 0;
        for (auto b = 16u; b > 0u; b >>= 1) {
          auto const probe = owner + b - 1u;
          auto const e = __shfl_sync(kFull, end, static_cast<int>(probe));
          if (e <= p) owner += b;
        }
        auto const o_tm = __shfl_sync(kFull, tm, static_cast<int>(owner));
        auto const o_pb = __shfl_sync(kFull, pb, static_cast<int>(owner));
        auto const o_end = __shfl_sync(kFull, end, static_cast<int>(owner));
        auto const o_cnt = __shfl_sync(kFull, cnt, static_cast<int>(owner));
        auto const o_rb = __shfl_sync(kFull, rb, static_cast<int>(owner));
        auto const o_rcnt = __shfl_sync(kFull, rcnt, static_cast<int>(owner));
        bool has = false, sorted = false;
        recon_cand c{};
        c.owner = owner;
        uint32_t cursor = 0;
        if (p < total && p - (o_end - o_cnt) < o_rcnt) {  // a real-time run at the stop
          auto const x = o_rb + (p - (o_end - o_cnt));
          c.is_rt = 1u;
          c.r = T->lrs_rt[x];
          c.i = static_cast<uint32_t>(T->lrs_rt_stop[x]);
          auto const sb = T->rt_stop_idx[c.r];
          auto const n = T->rt_stop_idx[c.r + 1] - sb;
          auto const w = T->rt_stops[sb + c.i];
          auto const allowed = (sl->allowed_claszes == 0xFFFFu && sl->req_flags == 0u) ||
                               filter_allowed(T->rt_filter[c.r], sl->allowed_claszes, sl->req_flags, c.sec);
          // an earlier arrival than the label is accepted (reconstruct.cc:437-440)
          has = allowed &&
                !((fwd && (c.i == 0u || !B2R_STOP_OUT(w))) || (!fwd && (c.i + 1u == n || !B2R_STOP_IN(w)))) &&
                beq(T->rt_times[2ull * (sb - c.r) + 2u * c.i - (fwd ? 1u : 0u)], delta_to_unix(o_tm));
        } else if (p < total) {
          auto const x = o_pb + (p - (o_end - o_cnt) - o_rcnt);
          c.rec = T->lrs_rec[x];
          auto const w = T->lrs_stop[x];
          c.r = c.rec.x;
          c.i = w & 0xFFFFu;
          sorted = (w & kLrsSorted) != 0u;
          auto const allowed = (sl->allowed_claszes == 0xFFFFu && sl->req_flags == 0u) ||
                               route_allowed(*T, c.r, sl->allowed_claszes, sl->req_flags, c.sec);
          // arrivals: not at the first stop, and alighting allowed (backward: departures)
          if (allowed && (w & (fwd ? kLrsAlight : kLrsBoard)) != 0u) {
            cursor = first_cursor(o_tm, c.rec, sorted);
            has = next_transport(o_tm, c.rec, sorted, cursor, c.t, c.day);
          }
        }
        if (!any(has)) continue;
        if (has) sm->cand[tid] = c;
        auto const mine = __ballot_sync(kFull, has);
        if (lane == 0u) sm->mask[wid] = mine;
        sync();
        while (true) {
          uint32_t w = 0, m = 0;
          for (; w != NW; ++w) {
            m = sm->mask[w];
            if (m != 0u) break;
          }
          if (m == 0u) break;
          auto const src = w * 32u + static_cast<uint32_t>(__ffs(m) - 1);
          auto const& b = sm->cand[src];
          if (b.is_rt != 0u ? find_start_in_prev_round_rt(k, b.r, b.i, b.sec, out)
                            : find_start_in_prev_round(k, b.rec, b.t, static_cast<uint16_t>(b.day), b.i, b.sec, out)) {
            auto const won = static_cast<int>(f0 + b.owner);
            sync();  // read by all before the next search writes
            return won;
          }
          sync();
          if (tid == src) {  // its next trip at the same minute
            if (c.is_rt == 0u && next_transport(o_tm, c.rec, sorted, cursor, c.t, c.day)) sm->cand[tid] = c;
            else sm->mask[w] = m & (m - 1u);
          }
          sync();
        }
        sync();
      }
    }
    return -1;
  }

  // check_fp (reconstruct.cc:547-666, no vias) for one footpath
  __device__ bool check_fp(unsigned k, uint32_t l, int curr_time, uint32_t target, int dur_raw,
                           bool adjust, b2r_leg& fp_leg, b2r_leg& tr_leg) const {
    auto const d = adjust ? static_cast<int>(adjusted<int16_t>(sl->tts, static_cast<int16_t>(dur_raw)))
                          : static_cast<int>(static_cast<int16_t>(dur_raw));
    auto const fp_start = static_cast<int>(static_cast<int16_t>(curr_time - dir(d)));
    auto const one = [&](uint32_t, uint32_t& tg, int& tm) {
      tg = target;
      tm = fp_start;
      return true;
    };
    if (get_transport(k, 1u, one, tr_leg) < 0) return false;
    fp_leg = make_leg(target, l, delta_to_unix(fp_start), delta_to_unix(fp_start + dir(d)));
    set_fp(fp_leg, target, dur_raw);
    return true;
  }

  // reconstruct.cc:700-790
  __device__ bool get_legs(unsigned k, uint32_t l, b2r_leg& fp_leg, b2r_leg& tr_leg) const {
    auto const curr = rt_t(k, l);
    if (sl->dest_mode == B2R_MATCH_INTERMODAL && k == j->transfers + 1u) {
      auto const* o = dest_offs();
      // destinations without generated tracks: their offsets are the
      // candidates of one search, in order
      auto tracks = false;
      if (T->children_idx != nullptr && T->loc_type != nullptr) {
        for (auto i = lane; i < sl->n_doff; i += 32u) {
          for (auto c = T->children_idx[o[i].target]; c != T->children_idx[o[i].target + 1]; ++c) {
            tracks = tracks || T->loc_type[T->children[c]] == B2R_LOC_GENERATED_TRACK;
          }
        }
        tracks = __any_sync(kFull, tracks);
      }
      if (!tracks) {
        auto const start_of = [&](b2r_offset const& x) {
          return static_cast<int>(static_cast<int16_t>(curr - dir(static_cast<int>(x.duration))));
        };
        auto const get = [&](uint32_t f, uint32_t& tg, int& tm) {
          auto const x = o[f];
          tg = x.target;
          tm = start_of(x);
          return x.duration < 511;
        };
        auto const f = get_transport(k, sl->n_doff, get, tr_leg);
        if (f < 0) return false;
        auto const x = o[f];
        auto const fp_start = start_of(x);
        fp_leg = make_leg(x.target, l, delta_to_unix(fp_start), delta_to_unix(fp_start + dir(static_cast<int>(x.duration))));
        set_off(fp_leg, x);
        return true;
      }
      for (auto i = 0u; i != sl->n_doff; ++i) {
        if (o[i].duration >= 511) continue;
        auto found = false;
        // for_each_meta(kIntermodal): the location and its generated tracks;
        // the last matching meta wins (reconstruct.cc:680-696)
        auto const try_eq = [&](uint32_t eq) {
          b2r_leg f, t;
          if (check_fp(k, l, curr, eq, o[i].duration, false, f, t)) {
            b2r_offset oo = o[i];
            oo.target = eq;
            set_off(f, oo);
            fp_leg = f;
            tr_leg = t;
            found = true;
          }
        };
        try_eq(o[i].target);
        if (T->children_idx != nullptr) {
          for (auto c = T->children_idx[o[i].target]; c != T->children_idx[o[i].target + 1]; ++c) {
            auto const ch = T->children[c];
            if (T->loc_type != nullptr && T->loc_type[ch] == B2R_LOC_GENERATED_TRACK) try_eq(ch);
          }
        }
        if (found) return true;
      }
      return false;
    }
    // candidate 0: staying at l (transfer time, or none at the destination);
    // candidates 1..: the footpaths into l, in order
    auto const same = (k == j->transfers + 1u)
                          ? 0
                          : static_cast<int>(adjusted<uint8_t>(sl->tts, T->transfer_time[l]));
    auto const* idx = fp_index(*T, sl->prf, !fwd);  // the query's profile (reconstruct.cc:81, 761)
    auto const* fps = fp_words(*T, sl->prf, !fwd);
    auto const fb = idx[l];
    auto const raw = [&](uint32_t f, uint32_t& tg, int& dur) {
      if (f == 0u) {
        tg = l;
        dur = same;
      } else {
        auto const w = fps[fb + f - 1u];
        tg = B2R_FP_TARGET(w);
        dur = static_cast<int>(B2R_FP_DURATION(w));
      }
    };
    auto const eff = [&](uint32_t f, int dur) {
      return f == 0u ? static_cast<int>(static_cast<int16_t>(dur))
                     : static_cast<int>(adjusted<int16_t>(sl->tts, static_cast<int16_t>(dur)));
    };
    auto const get = [&](uint32_t f, uint32_t& tg, int& tm) {
      int dur = 0;
      raw(f, tg, dur);
      tm = static_cast<int>(static_cast<int16_t>(curr - dir(eff(f, dur))));
      return true;
    };
    auto const f = get_transport(k, 1u + (idx[l + 1] - fb), get, tr_leg);
    if (f < 0) return false;
    uint32_t tg = 0;
    int dur = 0;
    raw(static_cast<uint32_t>(f), tg, dur);
    auto const d = eff(static_cast<uint32_t>(f), dur);
    auto const fp_start = static_cast<int>(static_cast<int16_t>(curr - dir(d)));
    fp_leg = make_leg(tg, l, delta_to_unix(fp_start), delta_to_unix(fp_start + dir(d)));
    set_fp(fp_leg, tg, dur);
    return true;
  }

  // reconstruct.cc:30-160 (no vias)
  __device__ bool find_start_footpath(b2r_leg& out, bool& has) const {
    has = false;
    auto const& back = last;
    auto const lsl = fwd ? back.from : back.to;
    auto const lst = fwd ? back.dep_time : back.arr_time;
    if (sl->start_mode != B2R_MATCH_INTERMODAL && is_journey_start(lsl) && beq(j->start_time, lst)) {
      return true;
    }
    auto const* o = start_offs();
    if (sl->start_mode == B2R_MATCH_INTERMODAL) {
      for (auto i = 0u; i != sl->n_soff; ++i) {
        if (matches(sl->start_mode, o[i].target, lsl) && beq(j->start_time, lst - dir(o[i].duration))) {
          out = make_leg(B2R_SPECIAL_START, lsl, lst - dir(o[i].duration), lst);
          set_off(out, o[i]);
          has = true;
          return true;
        }
      }
      return false;
    }
    auto const jst = unix_to_delta(j->start_time);
    auto const fp_target_time = rt_t(0, lsl);
    auto const* idx = fp_index(*T, sl->prf, !fwd);  // the query's profile (reconstruct.cc:81, 761)
    auto const* fps = fp_words(*T, sl->prf, !fwd);
    for (auto i = idx[lsl]; i != idx[lsl + 1]; ++i) {
      auto const tgt = B2R_FP_TARGET(fps[i]);
      auto const d = static_cast<int>(adjusted<int16_t>(sl->tts, static_cast<int16_t>(B2R_FP_DURATION(fps[i]))));
      auto const lhs = jst + static_cast<int16_t>(dir(d));
      if (is_journey_start(tgt) && fp_target_time != inv() &&
          (ontrip ? beq(lhs, fp_target_time) : lhs == fp_target_time)) {
        out = make_leg(tgt, lsl, j->start_time, delta_to_unix(fp_target_time));
        set_fp(out, tgt, d);
        has = true;
        return true;
      }
    }
    return false;
  }

  // ---------------------------------------------- optimize_footpaths.cc
  // The stops and event times of a leg's run (rt::frun): a real-time run's
  // own, else the static trip's.
  struct run_view {
    uint32_t const* words;
    uint32_t size;
    int32_t const* rt;    // real-time: departure of stop i at [2 i], arrival before it
    uint16_t const* evs;  // static: departure of stop i at [2 i n_t], arrival n_t before it
    uint32_t n_t;
    int32_t day_min;
    __device__ uint32_t word(uint32_t i) const { return words[i]; }
    __device__ int32_t time(uint32_t i, bool arr) const {
      if (rt != nullptr) return rt[2u * i - (arr ? 1u : 0u)];
      auto const e = evs[(2u * i - (arr ? 1u : 0u)) * n_t];
      return day_min + (e & 31) * 1440 + (e >> 5);
    }
  };
  __device__ run_view view_of(b2r_leg const& l) const {
    run_view v{};
    if (l.rt_transport != B2R_INVALID_IDX) {
      auto const x = l.rt_transport;
      auto const sb = T->rt_stop_idx[x];
      v.words = T->rt_stops + sb;
      v.size = T->rt_stop_idx[x + 1] - sb;
      v.rt = T->rt_times + 2ull * (sb - x);
    } else {
      auto const r = T->transport_route[l.transport];
      auto const sb = T->route_stop_idx[r];
      auto const t0 = T->route_tr_from[r];
      v.words = T->route_stops + sb;
      v.size = T->route_stop_idx[r + 1] - sb;
      v.n_t = T->route_tr_to[r] - t0;
      v.evs = T->st + T->route_st_from[r] + (l.transport - t0);
      v.day_min = (T->internal_from_days + static_cast<int32_t>(l.day)) * 1440;
    }
    return v;
  }

  // The four passes over the first / last ride (optimize_footpaths.cc:
  // 15-257) by one warp: the reference walks the ride's stops and takes every
  // improvement in order; few stops can be reached by the offset or footpath
  // at all, so the lanes look for those 32 stops at a time and the walk
  // visits only them.
  //
  // offsets at the ride's stops: departure side (15-60), arrival side
  // (122-187); `offs` = start / destination offsets of the journey query
  __device__ void opt_offset(b2r_offset const* offs, uint32_t n_offs, bool dep) {
    if (n_legs <= 1) return;
    auto& ol = legs[dep ? 0 : n_legs - 1];
    auto& tl = legs[dep ? 1 : n_legs - 2];
    if (ol.kind != B2R_LEG_OFFSET || tl.kind != B2R_LEG_TRANSPORT) return;
    auto const v = view_of(tl);
    auto const from = dep ? 0u : static_cast<uint32_t>(tl.stop_from + 1u);
    auto const end = dep ? static_cast<uint32_t>(tl.stop_to - 1u) : v.size;
    auto best = static_cast<int>(ol.duration);
    auto bound = dep ? ol.dep_time : ol.arr_time;
    uint32_t at = B2R_INVALID_IDX, at_loc = 0, which = 0;
    int32_t at_time = 0;
    for (auto s0 = from; s0 < end; s0 += 32u) {
      auto const si = s0 + lane;
      auto has = false;
      uint32_t loc = 0;
      int32_t tm = 0;
      if (si < end) {
        auto const w = v.word(si);
        loc = B2R_STOP_LOC(w);
        if (dep ? B2R_STOP_IN(w) : B2R_STOP_OUT(w)) {
          for (auto i = 0u; i != n_offs; ++i) has = has || (offs[i].target == loc && offs[i].duration < best);
        }
        if (has) tm = v.time(si, !dep);
      }
      for (auto m = __ballot_sync(kFull, has); m != 0u; m &= m - 1u) {
        auto const src = __ffs(m) - 1;
        auto const x_loc = __shfl_sync(kFull, loc, src);
        auto const x_tm = __shfl_sync(kFull, tm, src);
        for (auto i = 0u; i != n_offs; ++i) {
          auto const o = offs[i];
          if (best <= o.duration || o.target != x_loc) continue;
          auto const o_time = dep ? x_tm - o.duration : x_tm + o.duration;
          if (dep ? bound <= o_time : o_time <= bound) {
            bound = o_time;
            best = o.duration;
            at = s0 + static_cast<uint32_t>(src);
            at_loc = x_loc;
            at_time = x_tm;
            which = i;
          }
        }
      }
    }
    __syncwarp();
    if (at == B2R_INVALID_IDX || lane != 0u) return;
    set_off(ol, offs[which]);
    if (dep) {
      ol.to = tl.from = at_loc;
      ol.dep_time = bound;
      ol.arr_time = tl.dep_time = at_time;
      tl.stop_from = static_cast<uint16_t>(at);
    } else {
      ol.from = tl.to = at_loc;
      ol.dep_time = tl.arr_time = at_time;
      ol.arr_time = bound;
      tl.stop_to = static_cast<uint16_t>(at + 1u);
    }
  }

  // footpaths between the journey's start / destination and the ride's
  // stops: departure side (62-120), arrival side (189-257)
  __device__ void opt_footpath(bool dep) {
    if (n_legs <= 1) return;
    auto& fl = legs[dep ? 0 : n_legs - 1];
    auto& tl = legs[dep ? 1 : n_legs - 2];
    if (fl.kind != B2R_LEG_FOOTPATH || tl.kind != B2R_LEG_TRANSPORT) return;
    auto const v = view_of(tl);
    auto const end_loc = dep ? fl.from : fl.to;
    auto const from = dep ? 0u : static_cast<uint32_t>(tl.stop_from + 1u);
    auto const end = dep ? static_cast<uint32_t>(tl.stop_to - 1u) : v.size;
    auto const* idx = fp_index(*T, sl->prf, dep);  // optimize_footpaths.cc:91, 215
    auto const* fps = fp_words(*T, sl->prf, dep);
    auto const fb = idx[end_loc], fe = idx[end_loc + 1];
    auto best = static_cast<int>(adjusted<int16_t>(sl->tts, fl.duration));
    auto bound = dep ? fl.dep_time : fl.arr_time;
    uint32_t at = B2R_INVALID_IDX, at_loc = 0;
    int32_t at_time = 0;
    for (auto s0 = from; s0 < end; s0 += 32u) {
      auto const si = s0 + lane;
      auto has = false;
      uint32_t loc = 0;
      int32_t tm = 0;
      int d = 0;
      if (si < end) {
        auto const w = v.word(si);
        loc = B2R_STOP_LOC(w);
        if (dep ? B2R_STOP_IN(w) : B2R_STOP_OUT(w)) {
          for (auto i = fb; i != fe; ++i) {
            if (B2R_FP_TARGET(fps[i]) != loc) continue;
            d = static_cast<int>(adjusted<int16_t>(sl->tts, static_cast<int16_t>(B2R_FP_DURATION(fps[i]))));
            has = d < best;
            break;
          }
        }
        if (has) tm = v.time(si, !dep);
      }
      for (auto m = __ballot_sync(kFull, has); m != 0u; m &= m - 1u) {
        auto const src = __ffs(m) - 1;
        auto const x_loc = __shfl_sync(kFull, loc, src);
        auto const x_tm = __shfl_sync(kFull, tm, src);
        auto const x_d = __shfl_sync(kFull, d, src);
        auto const f_time = dep ? x_tm - x_d : x_tm + x_d;
        if (x_d < best && (dep ? bound <= f_time : f_time <= bound)) {
          bound = f_time;
          best = x_d;
          at = s0 + static_cast<uint32_t>(src);
          at_loc = x_loc;
          at_time = x_tm;
        }
      }
    }
    __syncwarp();
    if (at == B2R_INVALID_IDX || lane != 0u) return;
    set_fp(fl, dep ? at_loc : end_loc, best);
    if (dep) {
      fl.to = tl.from = at_loc;
      fl.dep_time = bound;
      fl.arr_time = tl.dep_time = at_time;
      tl.stop_from = static_cast<uint16_t>(at);
    } else {
      fl.from = tl.to = at_loc;
      fl.dep_time = tl.arr_time = at_time;
      fl.arr_time = bound;
      tl.stop_to = static_cast<uint16_t>(at + 1u);
    }
  }

  // get_penalty, optimize_footpaths.cc:259-283, with IEEE double operations
  // spelled out (no contraction) so the result equals the host's.
  __device__ double penalty(int duration, int buffer, uint32_t from, uint32_t to) const {
    auto w = static_cast<double>(duration);
    if (matches(B2R_MATCH_EQUIVALENT, from, to)) {
      auto const x = root(from);
      auto const imp = T->importance == nullptr ? 0u : T->importance[x];
      auto const q = __ddiv_rn(static_cast<double>(imp), static_cast<double>(T->max_importance));
      w = __dsub_rn(w, __dmul_rn(q, 3.0));
    }
    auto const b = buffer < 0 ? 0 : (buffer > 15 ? 15 : buffer);
    return __dsub_rn(w, __dmul_rn(0.2, static_cast<double>(b)));
  }

  // optimize_footpaths.cc:285-450 (no vias).  For each transport-footpath-
  // transport triple the (exit stop, entry stop) pairs are split across the
  // group; pairs do not depend on each other except through the running best
  // penalty, so the sequential loop keeps the first pair (in its order) with
  // the smallest penalty below the initial one, which is what the reduction
  // over (penalty, pair index) selects.  Called by the whole group; the
  // winning pair's thread writes the legs.
  __device__ void opt_transfers() {
    for (auto i = 0; i + 2 < n_legs; ++i) {
      sync();
      auto const lf = legs[i];
      auto const lp = legs[i + 1];
      auto const lt = legs[i + 2];
      if (lf.kind != B2R_LEG_TRANSPORT || lp.kind != B2R_LEG_FOOTPATH || lt.kind != B2R_LEG_TRANSPORT) continue;
      auto const vf = view_of(lf), vt = view_of(lt);
      auto const from_start = static_cast<uint32_t>(lf.stop_from + 1u);
      auto const to_end = static_cast<uint32_t>(lt.stop_to - 1u);
      auto const pbest0 = penalty(lp.duration, lt.dep_time - lp.arr_time, lf.from, lt.to);
      auto const n_sf = vf.size > from_start ? vf.size - from_start : 0u;
      auto const n_pairs = n_sf * to_end;
      auto const* oidx = fp_index(*T, sl->prf, true);  // optimize_footpaths.cc:405
      auto const* ofp = fp_words(*T, sl->prf, true);
      double best = pbest0;
      uint32_t best_idx = 0xFFFFFFFFu, best_fp = 0;
      int32_t best_arr = 0, best_dep = 0, best_d = 0;
      for (auto x = tid; x < n_pairs; x += kT) {
        auto const sf = from_start + x / to_end, s2 = x % to_end;
        auto const wf = vf.word(sf), wt = vt.word(s2);
        if (!B2R_STOP_OUT(wf) || !B2R_STOP_IN(wt)) continue;
        auto const a = B2R_STOP_LOC(wf), b = B2R_STOP_LOC(wt);
        for (auto y = oidx[a], ye = oidx[a + 1]; y != ye; ++y) {
          auto const fp = ofp[y];
          if (B2R_FP_TARGET(fp) != b) continue;
          auto const d = static_cast<int>(adjusted<int16_t>(sl->tts, static_cast<int16_t>(B2R_FP_DURATION(fp))));
          auto const arr = vf.time(sf, true);
          auto const dep = vt.time(s2, false);
          auto const arr_fp = arr + d;
          if (arr_fp <= dep) {
            auto const pen = penalty(d, dep - arr_fp, a, b);
            if (pen < best) {  // threads visit their pairs in increasing order
              best = pen;
              best_idx = x;
              best_fp = fp;
              best_arr = arr;
              best_dep = dep;
              best_d = d;
            }
          }
          break;
        }
      }
      // (penalty, pair index) minimum over the group
      auto win_pen = best;
      auto win_idx = best_idx;
      auto const take = [&](double op, uint32_t oi) {
        if (op < win_pen || (op == win_pen && oi < win_idx)) {
          win_pen = op;
          win_idx = oi;
        }
      };
      for (auto o = 16; o > 0; o >>= 1) {
        take(__shfl_xor_sync(kFull, win_pen, o), __shfl_xor_sync(kFull, win_idx, o));
      }
      if constexpr (NW > 1) {
        if (lane == 0u) {
          sm->pen[wid] = win_pen;
          sm->pen_at[wid] = win_idx;
        }
        sync();
        for (auto w = 0; w != NW; ++w) take(sm->pen[w], sm->pen_at[w]);
      } else {
        sync();  // the legs are read by all before they change
      }
      if (win_idx != 0xFFFFFFFFu && win_idx % kT == tid) {  // a pair below the initial penalty
        auto const sf = from_start + win_idx / to_end, s2 = win_idx % to_end;
        auto const a = B2R_STOP_LOC(vf.word(sf)), b = B2R_STOP_LOC(vt.word(s2));
        auto& wf = legs[i];
        auto& wp = legs[i + 1];
        auto& wt = legs[i + 2];
        wf.to = a;
        wf.arr_time = best_arr;
        wf.stop_to = static_cast<uint16_t>(sf + 1u);
        wt.from = b;
        wt.dep_time = best_dep;
        wt.stop_from = static_cast<uint16_t>(s2);
        wp.from = a;
        wp.to = b;
        wp.dep_time = best_arr;
        wp.arr_time = best_arr + best_d;
        set_fp(wp, B2R_FP_TARGET(best_fp), static_cast<int>(B2R_FP_DURATION(best_fp)));
      }
    }
    sync();
  }

  // reconstruct.cc:792-877 + optimize_footpaths(journey_q)
  __device__ void run() {
    n_legs = 0;
    failed = false;
    auto l = j->dest;
    for (auto i = 0u; i <= j->transfers && !failed; ++i) {
      auto const k = j->transfers + 1u - i;
      b2r_leg fp_leg, tr_leg;
      if (!get_legs(k, l, fp_leg, tr_leg)) {
        failed = true;
        break;
      }
      l = fwd ? tr_leg.from : tr_leg.to;
      if (i != 0 || fp_leg.from != fp_leg.to || fp_leg.dep_time != fp_leg.arr_time) push(fp_leg);
      push(tr_leg);
    }
    if (!failed) {
      b2r_leg init;
      bool has = false;
      if (!find_start_footpath(init, has)) failed = true;
      else if (has) push(init);
    }
    if (failed) return;
    sync();
    if (wid == 0u) {
      if (fwd) {
        for (auto a = static_cast<int>(lane); a < n_legs / 2; a += 32) {
          auto const x = legs[a];
          legs[a] = legs[n_legs - 1 - a];
          legs[n_legs - 1 - a] = x;
        }
      } else if (lane == 0u) {
        for (auto i = 1; i < n_legs; ++i) {
          if (legs[i].kind != B2R_LEG_FOOTPATH) continue;
          auto const diff = legs[i].dep_time - legs[i - 1].arr_time;
          legs[i].dep_time -= diff;
          legs[i].arr_time -= diff;
        }
      }
      __syncwarp();
      // optimize_footpaths on the journey query (flipped for backward search)
      opt_offset(fwd ? start_offs() : dest_offs(), fwd ? sl->n_soff : sl->n_doff, true);
      __syncwarp();
      opt_footpath(true);
      __syncwarp();
      opt_offset(fwd ? dest_offs() : start_offs(), fwd ? sl->n_doff : sl->n_soff, false);
      __syncwarp();
      opt_footpath(false);
    }
    opt_transfers();
  }
};

}  // namespace b2r::dev
