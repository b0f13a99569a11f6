// Per-round kernels of the batched RAPTOR super-step.  One super-step runs
// one RAPTOR round (raptor::execute's loop body, raptor.h:218-387) for every
// resident query whose current start-time group is still running, then
// collects, reconstructs and seeds the next start-time group of queries
// whose rounds ended (search.h:436-475).
#pragma once

#include "engine.cuh"
#include "et_search.cuh"
#include "reconstruct.cuh"

namespace b2r::dev {

// C_PAR: which of the two station-mark arrays the next marks go to (k_routes
// flips it between a step's reads and its writes); C_RECON0 + parity: the
// journeys listed for reconstruction; C_RPAR: the parity of those the step
// rebuilds
enum : uint32_t {
  C_PAR = 0, C_Y = 1, C_R = 2, C_RECON0 = 3, C_F0 = 5, C_F1 = 6, C_RT = 7, C_RECON1 = 8, C_RPAR = 9
};
constexpr uint32_t recon_counter(uint32_t par) { return par == 0u ? C_RECON0 : C_RECON1; }

// The round kernels' way to fail a query (a buffer of theirs is too small for
// it): the slot ends at the end of the step (k_end), its neighbours go on.
__device__ __forceinline__ void fail_slot(state const& st, uint32_t s) {
  st.slots[s].error = B2R_ERR_DEVICE_STATUS;
}

// The first thing every super-step kernel does.  The kernels of a step are
// launched with programmatic dependencies (enqueue_superstep): the next one
// may take its place on the SMs from here on, so that its launch does not
// wait for this one's end, and this one reads and writes nothing before all
// kernels ahead of it are complete.
__device__ __forceinline__ void step_begin() {
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
}

__device__ __forceinline__ size_t li(state const& st, uint32_t l, uint32_t s) {
  return static_cast<size_t>(l) * st.S + s;
}
__device__ __forceinline__ size_t rti(state const& st, uint32_t k, uint32_t l, uint32_t s) {
  return (static_cast<size_t>(k) * st.tt.n_loc + l) * st.S + s;
}

__device__ __forceinline__ void mark(state const& st, uint32_t* M, uint32_t* list, uint32_t counter,
                                     uint32_t e, uint32_t bits) {
  auto const old = atomicOr(&M[e], bits);
  if (old == 0u) list[atomicAdd(&st.counters[counter], 1u)] = e;
}

// warp-aggregated mark: lanes with `want` OR their bit into M[e(lane)];
// lanes sharing the same word combine into one atomic.
__device__ __forceinline__ void mark_warp(state const& st, uint32_t* M, uint32_t* list,
                                          uint32_t counter, bool want, uint32_t e, uint32_t lane) {
  auto const key = want ? e : 0xFFFFFFFFu;
  auto const peers = __match_any_sync(kFull, key);
  if (want && lane == static_cast<uint32_t>(__ffs(peers) - 1)) mark(st, M, list, counter, e, peers);
}

// position of the n-th (from 0) set bit of m
__device__ __forceinline__ uint32_t nth_bit(uint32_t m, uint32_t n) {
  uint32_t pos = 0;
#pragma unroll
  for (auto w = 16u; w != 0u; w >>= 1) {
    auto const c = static_cast<uint32_t>(__popc(m & ((1u << w) - 1u)));
    if (n >= c) {
      n -= c;
      m >>= w;
      pos += w;
    }
  }
  return pos;
}

// Visits the (entry, query) pairs of a frontier list: a warp takes up to 32
// list entries (a location or route with a group of 32 queries; 8 when the
// list is short, to keep more warps busy), and its lanes take their set
// query bits, one pair per lane per pass.  Resident queries
// are unrelated, so an entry holds few of its 32 queries; a lane per query of
// one entry would leave most lanes idle.  word(e) returns the entry's query
// bits; f(e, b) runs for every set bit b.  f must not synchronise the warp.
template <typename Word, typename F>
__device__ __forceinline__ void for_each_pair(uint32_t const* list, uint32_t n, Word&& word, F&& f) {
  auto const lane = threadIdx.x & 31u;
  auto const warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  auto const n_warps = (gridDim.x * blockDim.x) >> 5;
  auto const per = n >= n_warps * 8u ? 32u : 8u;
  for (auto w0 = warp * per; w0 < n; w0 += n_warps * per) {
    auto const w = w0 + lane;
    uint32_t e = 0, mask = 0;
    if (lane < per && w < n) {
      e = list[w];
      mask = word(e);
    }
    auto const cnt = static_cast<uint32_t>(__popc(mask));
    auto end = cnt;  // inclusive prefix sum of the pair counts
    for (auto o = 1u; o < 32u; o <<= 1) {
      auto const v = __shfl_up_sync(kFull, end, o);
      if (lane >= o) end += v;
    }
    auto const total = __shfl_sync(kFull, end, 31);
    for (auto p0 = 0u; p0 < total; p0 += 32u) {
      auto const p = p0 + lane;
      uint32_t owner = 0;  // first lane whose prefix end exceeds p
      for (auto b = 16u; b > 0u; b >>= 1) {
        if (__shfl_sync(kFull, end, static_cast<int>(owner + b - 1u)) <= p) owner += b;
      }
      auto const o_e = __shfl_sync(kFull, e, static_cast<int>(owner));
      auto o_mask = __shfl_sync(kFull, mask, static_cast<int>(owner));
      auto const o_first = __shfl_sync(kFull, end, static_cast<int>(owner)) -
                           __shfl_sync(kFull, cnt, static_cast<int>(owner));
      if (p < total) {
        for (auto x = p - o_first; x != 0u; --x) o_mask &= o_mask - 1u;
        f(o_e, static_cast<uint32_t>(__ffs(o_mask) - 1));
      }
    }
  }
}

// A slot keeps its round times for a later start-time group unless it runs
// one group and nothing after it: a one-to-one query at one start time whose
// journeys are collected as usual, or a one-to-all query at one start time.
// Range queries, interval extension, pong phases and step-driven searches
// keep them (raptor.h:174-177: only reset_arrivals clears them).
__device__ __forceinline__ bool keeps_round_times(slot_t const& sl) {
  if (sl.ontrip && sl.one_to_all) return false;
  return !(sl.ontrip && sl.recon_mode == 0);
}

// the touched bit of a round-time write (k, l) of slot s
__device__ __forceinline__ void touch(state const& st, lane_t const& ln, uint32_t k, uint32_t l, uint32_t s) {
  if (!(ln.mode & 128u)) return;
  auto* w = st.touched + (static_cast<size_t>(k) * st.G + (s >> 5)) * st.tt.n_loc + l;
  auto const bit = 1u << (s & 31u);
  if ((*w & bit) == 0u) atomicOr(w, bit);
}

__device__ __forceinline__ void update_tad(slot_t& sl, uint32_t k, int key) {  // raptor.h:1479-1486
  if (sl.one_to_all) return;
  for (auto i = k; i < kK; ++i) {
    if (key < sl.tad[i]) sl.tad[i] = static_cast<int16_t>(key);
  }
}

// The compact view of a slot that every lane of the round kernels reads.
__device__ __forceinline__ lane_t lane_of(slot_t const& sl) {
  lane_t ln{};
  if (sl.state != S_RUN) return ln;
  ln.run = static_cast<uint8_t>(kLaneRun | (sl.k + 1u >= sl.end_k ? kLaneLast : 0u));
  ln.fwd = sl.fwd;
  ln.k = sl.k;
  ln.base = sl.base;
  ln.gtag = tagcode(sl.gen_group);
  ln.qtag = tagcode(sl.gen_query);
  ln.mode = (sl.intermodal_dest ? 1u : 0u) |
            ((!sl.intermodal_dest && !sl.one_to_all && sl.n_dest != 0) ? 2u : 0u) |
            (sl.tts.is_default ? 4u : 0u) | (sl.no_lb ? 8u : 0u) | (static_cast<uint32_t>(sl.prf) << 4) |
            (keeps_round_times(sl) ? 128u : 0u);
  ln.tad_k = sl.tad[sl.k];
  ln.claszes = sl.allowed_claszes;
  ln.req = sl.req_flags;
  ln.blast = sl.blast;
  return ln;
}

// best <- min(best, round_times[k]) over all locations (raptor.h:219-223)
// for the slots whose earlier start-time groups left round times behind
// (range queries).  Only locations whose touched word of (round, slot group)
// has the slot's bit can hold such a round time, so a warp reads the words
// of 32 locations at once (one coalesced load) and spreads their set bits,
// the (location, slot) pairs, over its lanes: every lane loads one round
// time and best label, independent of the others.  Bits whose entry belongs
// to an earlier query of the slot (its tag no longer matches) are cleared
// here; any later write sets them again.  The slots of one group that are
// at the same round (sweep_k) are taken together, and each (group, round)
// pair gets its share of the warps, so that slots at a dozen different
// rounds do not queue behind each other.
__device__ __forceinline__ void sweep(state const& st, uint32_t lane, uint32_t warp, uint32_t n_warps) {
  auto const n_loc = st.tt.n_loc;
  auto const n_chunks = (n_loc + 31u) / 32u;
  // the (group, round) pairs to sweep: how many, and the warp's
  auto const n_words = st.G * kK;
  uint32_t n_pairs = 0;
  for (auto q0 = 0u; q0 < n_words; q0 += 32u) {
    auto const w = q0 + lane < n_words ? st.sweep_k[q0 + lane] : 0u;
    n_pairs += static_cast<uint32_t>(__popc(__ballot_sync(kFull, w != 0u)));
  }
  if (n_pairs == 0u) return;
  auto const per = max(1u, n_warps / n_pairs);  // warps of a pair
  for (auto pair = warp / per; pair < n_pairs; pair += n_warps / per) {
    uint32_t same = 0, at_word = 0;
    for (auto q0 = 0u, seen = 0u; q0 < n_words; q0 += 32u) {
      auto const w = q0 + lane < n_words ? st.sweep_k[q0 + lane] : 0u;
      auto const q = __ballot_sync(kFull, w != 0u);
      auto const c = static_cast<uint32_t>(__popc(q));
      if (pair < seen + c) {
        auto const src = nth_bit(q, pair - seen);
        same = __shfl_sync(kFull, w, static_cast<int>(src));
        at_word = q0 + src;
        break;
      }
      seen += c;
    }
    auto const g = at_word / kK, k = at_word % kK;
    auto* tw = st.touched + (static_cast<size_t>(k) * st.G + g) * n_loc;
    auto const ln = st.lanes[g * 32u + lane];
    for (auto c = warp % per; c < n_chunks; c += per) {
      auto const l = c * 32u + lane;
      auto const word = l < n_loc ? (tw[l] & same) : 0u;
      if (__ballot_sync(kFull, word != 0u) == 0u) continue;
      auto const cnt = static_cast<uint32_t>(__popc(word));
      auto end = cnt;  // inclusive prefix sum of the pair counts
      for (auto o = 1u; o < 32u; o <<= 1) {
        auto const y = __shfl_up_sync(kFull, end, o);
        if (lane >= o) end += y;
      }
      auto const total = __shfl_sync(kFull, end, 31);
      for (auto p0 = 0u; p0 < total; p0 += 32u) {
        auto const p = p0 + lane;
        uint32_t owner = 0;  // first lane whose prefix end exceeds p
        for (auto b = 16u; b > 0u; b >>= 1) {
          if (__shfl_sync(kFull, end, static_cast<int>(owner + b - 1u)) <= p) owner += b;
        }
        auto o_word = __shfl_sync(kFull, word, static_cast<int>(owner));
        auto const o_first = __shfl_sync(kFull, end, static_cast<int>(owner)) -
                             __shfl_sync(kFull, cnt, static_cast<int>(owner));
        uint32_t b = 0u;
        if (p < total) {
          for (auto x = p - o_first; x != 0u; --x) o_word &= o_word - 1u;
          b = static_cast<uint32_t>(__ffs(o_word) - 1);
        }
        auto const qtag = __shfl_sync(kFull, static_cast<uint32_t>(ln.qtag), static_cast<int>(b));
        auto const gtag = __shfl_sync(kFull, static_cast<uint32_t>(ln.gtag), static_cast<int>(b));
        if (p < total) {
          auto const at = c * 32u + owner;
          auto const s = g * 32u + b;
          auto const r = dec(st.rt[rti(st, k, at, s)], static_cast<uint16_t>(qtag));
          if (r == kKeyInv) {
            atomicAnd(tw + at, ~(1u << b));
          } else {
            auto& bw = st.best[li(st, at, s)];
            if (r < dec(bw, static_cast<uint16_t>(gtag))) bw = enc(static_cast<uint16_t>(gtag), r);
          }
        }
      }
    }
  }
}

// station marks -> route marks (raptor.h:228-241), then the sweep.
//
// A warp takes 32 words of the station marks ((location, group) pairs; most
// are zero, and 32 zero words cost one load and one ballot), and spreads the
// (word, route) pairs of the marked ones over its lanes, so that hub
// stations with many routes do not hold one lane.  Reading the marks where
// they lie saves a frontier list and its launch: the words of a step are
// read in full once here and once where they are cleared (k_reached).
// Where one pass takes all words, a warp's 32 lie n_warps apart: marks
// cluster (a query's frontier is a few districts), and a warp with 32
// neighbours of one cluster has 600 routes to mark one pass after the other
// while most warps have none (17.1 -> 14.5 us at 128 slots on 40,000
// stops).  With more words every warp has enough to do and neighbours are
// better: their marks fall on the same routes (31 us at 1,024 slots, 49 us
// apart).
// The per-group "any route marked" word is read before its atomicOr: it only
// gains bits during the kernel, so a read that shows the bits set makes the
// atomic redundant, and same-address atomics would queue in L2.  A marked
// real-time run (n_rt != 0) also keeps its queries in the round.
// Only queries whose label at the station time_at_dest does not rule out
// already mark its routes: a trip search from the others ends at its first
// event (every event is at or after the label, and the search prunes with
// this station's bound), so a pair marked by none but them reaches nothing.
// One look at the label here saves one in each of the station's 19 routes,
// and the pairs that drop out are never scanned.  The round loop's "any
// route marked" still counts every mark, as do the real-time runs' marks.
__global__ void __launch_bounds__(256) k_mark(state st) {
  step_begin();
  __shared__ uint32_t live_bits[8][32];
  auto const lane = threadIdx.x & 31u;
  auto const warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  auto const n_warps = (gridDim.x * blockDim.x) >> 5;
  auto* live = live_bits[threadIdx.x >> 5];
  auto const par = st.counters[C_PAR];
  auto const* X = st.X[par];
  auto const& T = st.tt;
  if (blockIdx.x == 0u && threadIdx.x == 0u) {  // this step's lists
    st.counters[C_Y] = 0u;
    st.counters[C_R] = 0u;
    st.counters[C_RT] = 0u;
    st.counters[recon_counter(par ^ 1u)] = 0u;
    st.counters[C_RPAR] = par;  // the list the last k_end filled
  }
  auto const n = T.n_loc * st.G;
  auto const step = n_warps * 32u;
  auto i = n <= step ? lane * n_warps + warp : warp * 32u + lane;
  auto x = i < n ? X[i] : 0u;
  for (auto w0 = 0u; w0 < n; w0 += step) {
    auto const e = i;
    auto w = x;
    i += step;
    x = i < n ? X[i] : 0u;  // the next pass's word, in flight during this one
    if (__ballot_sync(kFull, w != 0u) == 0u) continue;
    uint32_t g = 0, l = 0, rb = 0, cnt = 0;
    if (w != 0u) {
      g = e % st.G;
      l = e / st.G;
      w &= st.run_mask[g];
      if (w != 0u) {
        rb = __ldg(T.loc_routes_idx + l);
        cnt = __ldg(T.loc_routes_idx + l + 1) - rb;
        auto any = cnt;
        if (T.n_rt != 0u) {
          auto const b = T.loc_rt_idx[l], m = T.loc_rt_idx[l + 1] - b;
          any += m;
          for (auto j = 0u; j != m; ++j) atomicOr(&st.RT_R[T.loc_rt[b + j] * st.G + g], w);
        }
        if (any != 0u && (st.any_mask[g] & w) != w) atomicOr(&st.any_mask[g], w);
        if (cnt == 0u) w = 0u;
      }
    }
    // the live queries of each word, its (word, query) pairs spread over the lanes
    {
      live[lane] = 0u;
      auto const bits = static_cast<uint32_t>(__popc(w));
      auto end = bits;
      for (auto o = 1u; o < 32u; o <<= 1) {
        auto const v = __shfl_up_sync(kFull, end, o);
        if (lane >= o) end += v;
      }
      auto const total = __shfl_sync(kFull, end, 31);
      __syncwarp();
      for (auto p0 = 0u; p0 < total; p0 += 32u) {
        auto const p = p0 + lane;
        uint32_t owner = 0;  // first lane whose prefix end exceeds p
        for (auto b = 16u; b > 0u; b >>= 1) {
          if (__shfl_sync(kFull, end, static_cast<int>(owner + b - 1u)) <= p) owner += b;
        }
        auto const o_first = __shfl_sync(kFull, end, static_cast<int>(owner)) -
                             __shfl_sync(kFull, bits, static_cast<int>(owner));
        auto const o_w = __shfl_sync(kFull, w, static_cast<int>(owner));
        auto const o_g = __shfl_sync(kFull, g, static_cast<int>(owner));
        auto const o_l = __shfl_sync(kFull, l, static_cast<int>(owner));
        if (p < total) {
          auto const b = nth_bit(o_w, p - o_first);
          auto const s = o_g * 32u + b;
          auto const ln = st.lanes[s];
          auto const at = li(st, o_l, s);
          auto const prt = dec(st.rt[static_cast<size_t>(ln.k - 1u) * T.n_loc * st.S + at], ln.qtag);
          auto const lbv = (ln.mode & 8u) ? uint16_t{0} : st.lb[at];
          if (prt != kKeyInv && lbv != 0xFFFFu && prt + static_cast<int>(lbv) <= ln.tad_k) {
            atomicOr(&live[owner], 1u << b);
          }
        }
      }
      __syncwarp();
      w = live[lane];
      __syncwarp();
      if (w == 0u) cnt = 0u;
    }
    auto end = cnt;  // inclusive prefix sum of the route counts
    for (auto o = 1u; o < 32u; o <<= 1) {
      auto const v = __shfl_up_sync(kFull, end, o);
      if (lane >= o) end += v;
    }
    auto const total = __shfl_sync(kFull, end, 31);
    for (auto p0 = 0u; p0 < total; p0 += 32u) {
      auto const p = p0 + lane;
      uint32_t owner = 0;  // first lane whose prefix end exceeds p
      for (auto b = 16u; b > 0u; b >>= 1) {
        if (__shfl_sync(kFull, end, static_cast<int>(owner + b - 1u)) <= p) owner += b;
      }
      auto const o_first = __shfl_sync(kFull, end, static_cast<int>(owner)) -
                           __shfl_sync(kFull, cnt, static_cast<int>(owner));
      auto const o_rb = __shfl_sync(kFull, rb, static_cast<int>(owner));
      auto const o_g = __shfl_sync(kFull, g, static_cast<int>(owner));
      auto const o_w = __shfl_sync(kFull, w, static_cast<int>(owner));
      if (p < total) {
        auto const r = __ldg(T.loc_routes + o_rb + (p - o_first));
        // a corridor's stops mark the same routes over and over: a read that
        // shows the bits saves the atomic
        auto* rw = &st.R[r * st.G + o_g];
        if ((*rw & o_w) != o_w) atomicOr(rw, o_w);  // listed by k_routes
      }
    }
  }
  sweep(st, lane, warp, n_warps);
}

// The non-zero words of W[0, n) listed in no particular order: emit(at, i,
// word) fills the items(word) places from `at` on.  Each thread reads 4 words with one 16-byte load (W comes from
// cudaMalloc and i is a multiple of 4), the block scans the counts and
// reserves its range with one atomicAdd per 4 * blockDim words.
// Block `block` of `n_blocks`.
template <typename Items, typename Emit>
__device__ __forceinline__ void list_nonzero(state const& st, uint32_t const* W, uint32_t n, uint32_t counter,
                                             uint32_t block, uint32_t n_blocks, Items&& items, Emit&& emit) {
  __shared__ uint32_t warp_off[32];
  __shared__ uint32_t base;
  auto const lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
  auto const per_block = blockDim.x * 4u;
  for (auto b0 = block * per_block; b0 < n; b0 += n_blocks * per_block) {
    auto const i = b0 + threadIdx.x * 4u;
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (i + 3u < n) {
      auto const v = *reinterpret_cast<uint4 const*>(W + i);
      w[0] = v.x;
      w[1] = v.y;
      w[2] = v.z;
      w[3] = v.w;
    } else {
      for (auto j = 0u; j != 4u; ++j) w[j] = i + j < n ? W[i + j] : 0u;
    }
    auto const cnt = items(w[0]) + items(w[1]) + items(w[2]) + items(w[3]);
    auto incl = cnt;  // inclusive scan over the warp
    for (auto d = 1u; d < 32u; d <<= 1) {
      auto const y = __shfl_up_sync(kFull, incl, d);
      if (lane >= d) incl += y;
    }
    if (lane == 31u) warp_off[warp] = incl;
    __syncthreads();
    if (warp == 0u) {  // scan of the warp totals, then the block's reservation
      auto const ws = lane < n_warps ? warp_off[lane] : 0u;
      auto x = ws;
      for (auto d = 1u; d < 32u; d <<= 1) {
        auto const y = __shfl_up_sync(kFull, x, d);
        if (lane >= d) x += y;
      }
      if (lane < n_warps) warp_off[lane] = x - ws;
      if (lane == 31u) base = x != 0u ? atomicAdd(&st.counters[counter], x) : 0u;
    }
    __syncthreads();
    auto at = base + warp_off[warp] + (incl - cnt);
    for (auto j = 0u; j != 4u; ++j) {
      if (w[j] != 0u) {
        emit(at, i + j, w[j]);
        at += items(w[j]);
      }
    }
    __syncthreads();  // warp_off and base are reused by the next pass
  }
}

struct one_item {
  __device__ __forceinline__ uint32_t operator()(uint32_t word) const { return word != 0u ? 1u : 0u; }
};

// Per slot, a warp: destination times into time_at_dest (raptor.h:224-226;
// a minimum, so the lanes take the destinations in any order), and a slot
// with no marked route leaves the round loop (raptor.h:243-246).
__device__ __forceinline__ void dest_slot(state const& st, uint32_t s, uint32_t lane) {
  auto& sl = st.slots[s];
  if (sl.state != S_RUN) return;
  auto const k = static_cast<uint32_t>(sl.k);
  if (!sl.one_to_all) {
    auto const gtag = tagcode(sl.gen_group);
    int key = kKeyInv;
    if (sl.intermodal_dest) {
      key = dec(st.best[li(st, B2R_SPECIAL_END, s)], gtag);
    } else {
      for (auto i = lane; i < sl.n_dest; i += 32u) {
        key = min(key, dec(st.best[li(st, st.dest_pool[sl.dest_off + i].loc, s)], gtag));
      }
    }
    key = __reduce_min_sync(kFull, key);
    if (lane >= k && lane < kK && key < sl.tad[lane]) sl.tad[lane] = static_cast<int16_t>(key);
    if (lane == 0u && key < st.lanes[s].tad_k) st.lanes[s].tad_k = static_cast<int16_t>(key);
  }
  if (lane == 0u) {
    ++sl.n_rounds;
    if (!((st.any_mask[s >> 5] >> (s & 31u)) & 1u)) {
      sl.state = S_COLLECT;
      st.lanes[s].run = 0;
    }
  }
}

// The round's marked (route, group) words, in entries of up to kEntryMarks
// queries, and (real-time run, group) words listed, the slots' destination
// times, and the station-mark arrays swapped: from here to the end of the
// step X[C_PAR ^ 1] holds the marks the round reads and X[C_PAR] takes the
// marks it makes.  The first blocks take the slots, 8 each, the others the
// lists, so that neither waits for the other.
__global__ void __launch_bounds__(256) k_routes(state st) {
  step_begin();
  auto const lane = threadIdx.x & 31u;
  if (blockIdx.x == 0u && threadIdx.x == 0u) st.counters[C_PAR] ^= 1u;
  if (blockIdx.x == 0u) {
    for (auto g = threadIdx.x; g < st.G; g += blockDim.x) st.made_mask[g] = 0u;
  }
  auto const slot_blocks = (st.S + 7u) / 8u;
  if (blockIdx.x < slot_blocks) {
    auto const s = blockIdx.x * 8u + (threadIdx.x >> 5);
    if (s < st.S) dest_slot(st, s, lane);
    return;
  }
  auto const block = blockIdx.x - slot_blocks, n_blocks = gridDim.x - slot_blocks;
  list_nonzero(
      st, st.R, st.tt.n_routes * st.G, C_R, block, n_blocks,
      [](uint32_t marks) { return (static_cast<uint32_t>(__popc(marks)) + kEntryMarks - 1u) / kEntryMarks; },
      [&](uint32_t at, uint32_t e, uint32_t marks) {
        st.R[e] = 0u;
        while (marks != 0u) {
          auto rest = marks;  // the marks of a later entry
          for (auto i = 0u; i != kEntryMarks; ++i) rest &= rest - 1u;
          st.rlist[at++] = uint2{e, marks ^ rest};
          marks = rest;
        }
      });
  if (st.tt.n_rt != 0u) {
    list_nonzero(st, st.RT_R, st.tt.n_rt * st.G, C_RT, block, n_blocks, one_item{},
                 [&](uint32_t at, uint32_t e, uint32_t) { st.rtlist[at] = e; });
  }
}

// ------------------------------------------------------------ route scan
// update_route, raptor.h:1177-1349 (no vias), for every (route, query) pair
// marked this round.
//
// The reference walks a route's stops in order, carrying the trip it rides
// (et).  At a stop marked last round it looks up the earliest trip
// boardable there (get_earliest_transport) and switches to it when that
// trip is at least as good at this stop as the current one; at every stop
// it improves the arrival label with the current trip.  Walked like that,
// one (route, query) pair is a chain of dependent loads as long as the
// route.
//
// Here 8 lanes take one pair, a warp four pairs, 32 stops at a time (32
// lanes and one pair where there are few, kFewPerSm):
// * the lanes read the stops' marks, four stops each;
// * the marked boardable stops of the four pairs are numbered through, and
//   the warp's lanes take 32 of them at once: the label to board from and,
//   unless time_at_dest rules it out, the search (it depends only on its
//   stop's labels; what it needs of its pair lies in shared memory);
// * on a route whose trips keep one order at every event
//   (kRouteOrder), "switch when at least as good at this
//   stop" is "keep the best trip so far", whatever stop compares them (on a
//   tie both are the same trip or equal at every event), so a prefix
//   minimum over the stops gives the trip each stop is reached by;
// * every stop then reads its arrival event of that trip.
// A section that lacks a flag the query requires drops the trip carried
// into it (raptor.h:1194-1217): the minimum starts anew there.
// The result equals the sequential walk's; routes without that order take
// the sequential walk (k_route_scan_seq).
// Labels are combined with atomicMin and marks with atomicOr, so the order
// of the pairs does not matter.
//
// The kernel is bound by instruction issue, and the trip searches are most
// of it.  With a warp per pair a pair cost about 890 warp instructions, its
// searches running on the few lanes whose stops were marked; on the
// regional batch of 1,024 a warp's four pairs bring 24 searches per 32
// stops, so numbering them fills the lanes.

struct scan_ctr {
  uint32_t stops, ev, days, writes, warp_steps;
};

// the stop word at position i of route (sb, n) in search direction; for the
// wheelchair profile with its wheelchair bits in place of the in / out bits
// (can_start / can_finish, raptor.h:1252, 1304)
__device__ __forceinline__ uint32_t scan_stop_word(dtt const& T, uint32_t sb, uint32_t n, bool fwd, uint32_t i,
                                                   uint32_t sec) {
  auto const w = __ldg(T.route_stops + sb + (fwd ? i : n - 1u - i));
  return (sec & 0x100u) != 0u ? (w & 0xCFFFFFFFu) | ((w >> 2) & 0x30000000u) : w;
}

// the arrival-side label update of one stop (raptor.h:1242-1302)
template <bool Prof>
__device__ __forceinline__ void scan_arrive(state const& st, lane_t const& ln, uint32_t s, uint32_t g, uint32_t bit,
                                            uint32_t l, uint16_t lbv, int by, scan_ctr& pc) {
  if (by <= ln.tad_k && lbv != 0xFFFFu && by + static_cast<int>(lbv) <= ln.tad_k &&
      (ln.blast == 0u || within_bounds(st, s, ln.blast, ln.k, l, by))) {
    auto const word = enc(ln.gtag, by);
    auto* tp = &st.tmp[li(st, l, s)];
    if constexpr (Prof) {
      if (word < atomicMin(tp, word)) ++pc.writes;
    } else {
      atomicMin(tp, word);  // result unused: no round trip
    }
    atomicOr(&st.Y[l * st.G + g], bit);  // listed by k_reached
  }
}

// The filters of a (route, query) pair: false if the route is filtered
// out; sec receives the flags checked per section (bits 0-3) and bit 8 for
// the wheelchair profile's stop bits.
__device__ __forceinline__ bool scan_filters(uint32_t filter, lane_t const& ln, uint32_t& sec) {
  sec = 0u;
  if ((ln.claszes != 0xFFFFu || ln.req != 0u) && !filter_allowed(filter, ln.claszes, ln.req, sec)) return false;
  if ((ln.mode & 0x70u) == (B2R_PROFILE_WHEELCHAIR << 4)) sec |= 0x100u;
  return true;
}

// The reference's sequential walk of one (route, query) pair.
__device__ __forceinline__ void scan_walk_seq(state const& st, uint32_t const* X, lane_t const& ln, route_rec const& R,
                                              uint32_t g, uint32_t b, uint32_t sec, scan_ctr& pc) {
  auto const& T = st.tt;
  auto const s = g * 32u + b;
  auto const bit = 1u << b;
  auto const fwd = ln.fwd != 0;
  auto const k = static_cast<uint32_t>(ln.k);
  auto const sb = R.sb, n = R.n, n_t = R.n_t;
  auto const* colbase = T.st + R.st;
  auto const lb_off = (ln.mode & 8u) != 0u;
  bool et_valid = false;
  uint32_t et_off = 0;
  uint16_t et_day = 0;
  for (auto i = 0u; i < n; ++i) {
    ++pc.stops;
    ++pc.warp_steps;
    auto const stp = scan_stop_word(T, sb, n, fwd, i, sec);
    auto const si = fwd ? i : n - 1u - i;
    auto const l = B2R_STOP_LOC(stp);
    auto const lbv = lb_off ? uint16_t{0} : st.lb[li(st, l, s)];
    auto const can_finish = fwd ? B2R_STOP_OUT(stp) : B2R_STOP_IN(stp);
    auto const can_start = fwd ? B2R_STOP_IN(stp) : B2R_STOP_OUT(stp);
    if ((sec & 15u) != 0u && i != 0u && !section_ok(T, sb, fwd ? i - 1u : si, sec & 15u)) {
      et_valid = false;  // raptor.h:1194-1217: the section ridden lacks a flag
    }
    bool arrival_ran = false;
    if (et_valid && can_finish) {
      arrival_ran = true;
      auto const ev = colbase[n_t * (si * 2u - (fwd ? 1u : 0u)) + et_off];
      scan_arrive<true>(st, ln, s, g, bit, l, lbv, to_delta_key(fwd, et_day, ln.base, delta_count(ev)), pc);
    }
    if (i + 1u == n || !can_start || !(X[l * st.G + g] & bit)) continue;
    if (lbv == 0xFFFFu) break;  // raptor.h:1309-1311: no later stop of this query
    auto const board_col = n_t * (si * 2u - (fwd ? 0u : 1u));
    auto const et_time =
        et_valid ? to_delta_key(fwd, et_day, ln.base, delta_count(colbase[board_col + et_off])) : kKeyInv;
    auto const prt = dec(st.rt[rti(st, k - 1u, l, s)], ln.qtag);
    if (prt == kKeyInv || prt > et_time) continue;
    auto const minutes = static_cast<int>(ln.base) * 1440 + from_key(fwd, prt);
    uint32_t nt = 0;
    uint16_t nd = 0;
    if (!et_search(T, fwd, R, si, static_cast<uint16_t>(minutes / 1440), minutes % 1440, static_cast<int>(lbv),
                   ln.tad_k, ln.base, nt, nd, pc.ev, pc.days)) {
      continue;
    }
    // current_best (raptor.h:1328-1329) is valid whenever the arrival part
    // ran or the station carries a label of this start time
    auto const cb_valid = arrival_ran || dec(st.best[li(st, l, s)], ln.gtag) != kKeyInv ||
                          dec(st.tmp[li(st, l, s)], ln.gtag) != kKeyInv;
    if (!cb_valid || to_delta_key(fwd, nd, ln.base, delta_count(colbase[board_col + nt])) <= et_time) {
      et_valid = true;
      et_off = nt;
      et_day = nd;
    }
  }
}

// The pairs the parallel scan leaves to the sequential walk: routes without
// one trip order at every event (launched only if the timetable has any).
// A thread per marked (route, group) entry.
__global__ void __launch_bounds__(256) k_route_scan_seq(const __grid_constant__ state st) {
  step_begin();
  auto const& T = st.tt;
  auto const nr = st.counters[C_R];
  auto const* X = st.X[st.counters[C_PAR] ^ 1u];
  scan_ctr pc{0u, 0u, 0u, 0u, 0u};
  for (auto w = blockIdx.x * blockDim.x + threadIdx.x; w < nr; w += gridDim.x * blockDim.x) {
    auto const en = st.rlist[w];
    auto const R = load_route(T, en.x / st.G);
    if ((R.flags & kRouteOrder) != 0u) continue;  // k_route_scan's
    auto const g = en.x % st.G;
    for (auto mask = en.y; mask != 0u; mask &= mask - 1u) {
      auto const b = static_cast<uint32_t>(__ffs(mask) - 1);
      auto const ln = st.lanes[g * 32u + b];
      uint32_t sec = 0u;
      if (!ln.run || !scan_filters(R.filter, ln, sec)) continue;
      scan_walk_seq(st, X, ln, R, g, b, sec, pc);
    }
  }
  if (st.profile && (pc.stops | pc.ev | pc.days | pc.writes) != 0u) {
    atomicAdd(&st.prof[0], static_cast<unsigned long long>(pc.stops));
    atomicAdd(&st.prof[1], static_cast<unsigned long long>(pc.ev));
    atomicAdd(&st.prof[2], static_cast<unsigned long long>(pc.days));
    atomicAdd(&st.prof[3], static_cast<unsigned long long>(pc.writes));
    atomicAdd(&st.prof[5], static_cast<unsigned long long>(pc.warp_steps));
  }
}

// The parallel scan (above) with kTile lanes per pair.  Every loop that
// shuffles or ballots is uniform over the warp; a tile without work takes
// part idle.
template <uint32_t kTile>
struct scan_smem {  // of a warp
  static constexpr uint32_t kPer = 32u / kTile;
  uint4 pair[kPer][4];      // route record (2), lane record, {first stop of the 32, slot, 0, 0}
  uint32_t key[kPer][32];   // per stop: its location, then the candidate (order key << 6 | stop),
                            // kNone without one, kShut where the query cannot go on from
  uint2 trip[kPer][33];     // per stop: the candidate's offset and day; 32: the trip carried in
};
template <uint32_t kTile, bool Prof>
__device__ __forceinline__ void scan_tiles(state const& st, scan_smem<kTile>& sm, uint32_t nr, scan_ctr& pc) {
  constexpr uint32_t kPer = 32u / kTile;  // stops a lane takes of each 32; pairs of a warp
  constexpr uint32_t kTileBits = kTile == 32u ? kFull : (1u << (kTile % 32u)) - 1u;
  constexpr uint32_t kNone = 0xFFFFFFFFu, kShut = 0xFFFFFFFEu;
  constexpr uint32_t kCarried = 32u;
  auto const& T = st.tt;
  auto const lane = threadIdx.x & 31u;
  auto const tile = lane / kTile, tl = lane % kTile;
  auto const n_tiles = (gridDim.x * blockDim.x) / kTile;
  auto const* X = st.X[st.counters[C_PAR] ^ 1u];
  auto const tile_bits = [&](bool x) { return (__ballot_sync(kFull, x) >> (tile * kTile)) & kTileBits; };
  auto const tile_shfl = [&](uint32_t x, uint32_t src) {
    return __shfl_sync(kFull, x, static_cast<int>(src), static_cast<int>(kTile));
  };
  // With fewer entries than tiles, an entry's queries are shared by 2^split
  // tiles, each taking the ones in its part of the group: a short frontier
  // lasts as long as its longest entry, one pair after the other.
  uint32_t split = 0;
  while (split < 5u && (nr << (split + 1u)) <= n_tiles) ++split;
  auto const n_items = nr << split;
  auto const part_bits = 32u >> split;
  // the tile's entry and pair
  auto w = (blockIdx.x * blockDim.x + threadIdx.x) / kTile;
  uint32_t g = 0, mask = 0, s = 0, sec = 0, i0 = 0;
  route_rec R{};
  lane_t ln{};
  bool have = false;
  // The trips' order key, below 2^21, smaller is better: with
  // kRouteOffsetOrder (service day - base + 64) * n_t + transport offset (the service
  // day lies within 64 days of the base day, n_t < 2^14), else the time at
  // the route's first departure event (|t| < 2^20 minutes) + 2^20; both
  // mirrored backward, where later is better.
  uint32_t carry = kNone;  // the trip carried over from the earlier stops: key << 6 | kCarried
  while (true) {
    while (!have) {
      if (mask == 0u) {
        if (w >= n_items) break;
        auto const en = st.rlist[w >> split];
        mask = en.y & ((split == 0u ? kFull : (1u << part_bits) - 1u) << ((w & ((1u << split) - 1u)) * part_bits));
        w += n_tiles;
        if (mask == 0u) continue;
        g = en.x % st.G;
        R = load_route(T, en.x / st.G);
        if ((R.flags & kRouteOrder) == 0u) mask = 0u;  // k_route_scan_seq's
        continue;
      }
      auto const b = static_cast<uint32_t>(__ffs(mask) - 1);
      mask &= mask - 1u;
      s = g * 32u + b;
      ln = st.lanes[s];
      if (!ln.run || !scan_filters(R.filter, ln, sec)) continue;
      have = true;
      i0 = 0u;
      carry = kNone;
    }
    if (!__any_sync(kFull, have)) break;
    auto const fwd = ln.fwd != 0;
    auto const bit = 1u << (s & 31u);
    auto const lb_off = (ln.mode & 8u) != 0u;
    auto const n_blk = have ? min(32u, R.n - i0) : 0u;
    // the block's stop words and its marked boardable stops
    uint32_t sw[kPer];
    uint32_t m = 0, cuts = 0;
#pragma unroll
    for (auto c = 0u; c != kPer; ++c) {
      auto const p = c * kTile + tl;
      sw[c] = p < n_blk ? scan_stop_word(T, R.sb, R.n, fwd, i0 + p, sec) : 0u;
    }
#pragma unroll
    for (auto c = 0u; c != kPer; ++c) {
      auto const p = c * kTile + tl;
      auto const board = p < n_blk && i0 + p + 1u != R.n && (fwd ? B2R_STOP_IN(sw[c]) : B2R_STOP_OUT(sw[c])) != 0u;
      m |= tile_bits(board && (X[B2R_STOP_LOC(sw[c]) * st.G + g] & bit) != 0u) << (c * kTile);
      sm.key[tile][p] = B2R_STOP_LOC(sw[c]);
    }
    bool ends = false;
    if constexpr (Prof) {
      if (lane == 0u) pc.warp_steps += kPer;  // 32 stops of each of its pairs
      if (tl == 0u) pc.stops += n_blk;
    }
    if (__any_sync(kFull, m != 0u || carry != kNone)) {
      if (__any_sync(kFull, have && (sec & 15u) != 0u)) {
#pragma unroll
        for (auto c = 0u; c != kPer; ++c) {
          auto const i = i0 + c * kTile + tl;
          auto const check = c * kTile + tl < n_blk && (sec & 15u) != 0u && i != 0u;
          cuts |= tile_bits(check && !section_ok(T, R.sb, fwd ? i - 1u : R.n - 1u - i, sec & 15u)) << (c * kTile);
        }
      }
      // the searches (raptor.h:1313-1327), 32 at a time over the warp's pairs
      if (tl == 0u && m != 0u) {
        sm.pair[tile][0] = uint4{R.sb, R.n, R.st, R.t0};
        sm.pair[tile][1] = uint4{R.n_t, R.bf, R.flags, R.filter};
        sm.pair[tile][2] = *reinterpret_cast<uint4 const*>(&ln);
        sm.pair[tile][3] = uint4{i0, s, 0u, 0u};
      }
      __syncwarp();
      auto const cnt = static_cast<uint32_t>(__popc(m));
      uint32_t ends_at[kPer];  // searches up to each pair's last
#pragma unroll
      for (auto x = 0u; x != kPer; ++x) {
        ends_at[x] = (x == 0u ? 0u : ends_at[x - 1u]) + __shfl_sync(kFull, cnt, static_cast<int>(x * kTile));
      }
      auto const total = ends_at[kPer - 1u];
      for (auto q0 = 0u; q0 < total; q0 += 32u) {
        auto const q = q0 + lane;
        uint32_t o = 0, first = 0;  // the search's pair and that pair's first search
#pragma unroll
        for (auto x = 0u; x + 1u < kPer; ++x) {
          if (q >= ends_at[x]) {
            o = x + 1u;
            first = ends_at[x];
          }
        }
        auto const om = __shfl_sync(kFull, m, static_cast<int>(o * kTile));
        if (q < total) {
          auto const pos = nth_bit(om, q - first);
          auto const a = sm.pair[o][0], b = sm.pair[o][1], c = sm.pair[o][2];
          route_rec const oR{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
          auto const oln = *reinterpret_cast<lane_t const*>(&c);
          auto const ofwd = oln.fwd != 0;
          auto const i = sm.pair[o][3].x + pos;
          auto const at = li(st, sm.key[o][pos], sm.pair[o][3].y);
          auto const lbv = (oln.mode & 8u) ? uint16_t{0} : st.lb[at];
          auto const prt = dec(st.rt[static_cast<size_t>(oln.k - 1u) * T.n_loc * st.S + at], oln.qtag);
          auto const has_best = dec(st.best[at], oln.gtag) != kKeyInv;
          auto const minutes = static_cast<int>(oln.base) * 1440 + from_key(ofwd, prt);
          uint32_t nt = 0, v = lbv == 0xFFFFu ? kShut : kNone, n_ev = 0, n_days = 0;
          uint16_t nd = 0;
          // every event of the search is at or after prt: pruned with it
          if (lbv != 0xFFFFu && prt != kKeyInv && prt + static_cast<int>(lbv) <= oln.tad_k &&
              et_search(T, ofwd, oR, ofwd ? i : oR.n - 1u - i, static_cast<uint16_t>(minutes / 1440), minutes % 1440,
                        static_cast<int>(lbv), oln.tad_k, oln.base, nt, nd, n_ev, n_days)) {
            // a marked station always carries a best label of its start time
            // (marks come with best updates), so the boarding rule never meets
            // an invalid current_best; were it to, the query is failed loudly
            if (!has_best && dec(st.tmp[at], oln.gtag) == kKeyInv) fail_slot(st, sm.pair[o][3].y);
            uint32_t key;
            if ((oR.flags & kRouteOffsetOrder) != 0u) {
              auto const x = static_cast<uint32_t>(static_cast<int>(nd) - static_cast<int>(oln.base) + 64) * oR.n_t + nt;
              key = ofwd ? x : (1u << 21) - 1u - x;
            } else {
              auto const t =
                  (static_cast<int>(nd) - static_cast<int>(oln.base)) * 1440 + delta_count(__ldg(T.st + oR.st + nt));
              key = static_cast<uint32_t>((ofwd ? t : -t) + (1 << 20));
            }
            v = (key << 6) | pos;
            sm.trip[o][pos] = uint2{nt, nd};
          }
          sm.key[o][pos] = v;
          if constexpr (Prof) {
            pc.ev += n_ev;
            pc.days += n_days;
          }
        }
      }
      __syncwarp();
      // the trip each stop is reached by: the minimum over the stops before
      // it, from the last cut on
      uint32_t by[kPer];
      uint32_t closed = 0;  // boardable stops the query cannot reach
      auto run = carry;
#pragma unroll
      for (auto c = 0u; c != kPer; ++c) {
        auto const cc = (cuts >> (c * kTile)) & kTileBits;
        auto v = ((m >> (c * kTile + tl)) & 1u) != 0u ? sm.key[tile][c * kTile + tl] : kNone;
        closed |= tile_bits(v == kShut) << (c * kTile);
        if (v == kShut) v = kNone;
#pragma unroll
        for (auto o = 1u; o < kTile; o <<= 1) {
          auto const y = __shfl_up_sync(kFull, v, o, kTile);
          if (tl >= o && ((cc >> (tl + 1u - o)) & ((1u << o) - 1u)) == 0u) v = min(v, y);
        }
        auto const up = __shfl_up_sync(kFull, v, 1, kTile);
        auto const before = tl == 0u || ((cc >> tl) & 1u) != 0u ? kNone : up;
        by[c] = (cc & ((2u << tl) - 1u)) == 0u ? min(before, run) : before;
        auto const last = tile_shfl(v, kTile - 1u);
        run = cc == 0u ? min(run, last) : last;
      }
      // raptor.h:1309-1311: the walk ends at the first boardable stop the
      // query cannot reach, after that stop's arrival
      ends = closed != 0u;
      auto const limit = ends ? static_cast<uint32_t>(__ffs(closed)) : n_blk;
      if constexpr (Prof) {
        if (tl == 0u) pc.stops -= n_blk - limit;
      }
      // arrivals (raptor.h:1219-1302)
      uint16_t ev[kPer], lbs[kPer], day[kPer];
      bool go[kPer];
#pragma unroll
      for (auto c = 0u; c != kPer; ++c) {
        auto const p = c * kTile + tl;
        go[c] = p < limit && by[c] != kNone && (fwd ? B2R_STOP_OUT(sw[c]) : B2R_STOP_IN(sw[c])) != 0u;
        ev[c] = lbs[c] = day[c] = 0;
        if (go[c]) {
          auto const t = sm.trip[tile][by[c] & 63u];
          auto const i = i0 + p;
          day[c] = static_cast<uint16_t>(t.y);
          ev[c] = __ldg(T.st + (R.st + R.n_t * (fwd ? 2u * i - 1u : 2u * (R.n - 1u - i)) + t.x));
          if (!lb_off) lbs[c] = st.lb[li(st, B2R_STOP_LOC(sw[c]), s)];
        }
      }
#pragma unroll
      for (auto c = 0u; c != kPer; ++c) {
        if (!go[c]) continue;
        scan_arrive<Prof>(st, ln, s, g, bit, B2R_STOP_LOC(sw[c]), lbs[c],
                          to_delta_key(fwd, day[c], ln.base, delta_count(ev[c])), pc);
      }
      __syncwarp();  // the trips are read before the one carried on is put aside
      if (run != kNone && (run & 63u) != kCarried) {
        if (tl == 0u) sm.trip[tile][kCarried] = sm.trip[tile][run & 63u];
        run = (run & ~63u) | kCarried;
      }
      carry = run;
    }
    __syncwarp();  // before the next block's labels
    if (have) {
      i0 += 32u;
      if (ends || i0 >= R.n) have = false;
    }
  }
}

// Above this many entries per SM the scan takes 8 lanes per pair, else a
// warp: a step of a warp is about 1,500 instructions for four pairs and 700
// for one, so with warps to spare one pair ends sooner.  Device time with 0
// (never a warp), 48, 96, 192, 384 and no limit (always a warp): 32.1, 31.4,
// 31.3, 31.2, 31.3, 31.3 ms for 96 range queries; 3.70, 3.79, 3.77, 3.79,
// 3.91, 4.50 for 1,024 on 40,009 stops; 1.57, 1.60, 1.59, 1.59, 1.68, 1.84 for
// 1,000 on 1,009 stops.  The same run repeats within 0.5%: the line lies
// anywhere between 48 and 192.
constexpr uint32_t kFewPerSm = 96;

// Builds with four, five or six blocks of 256 threads resident per SM (the
// launch shape picks one), and with work counters for profiling engines
// (Prof).
template <int MinBlocks, bool Prof>
__global__ void __launch_bounds__(256, MinBlocks) k_route_scan(const __grid_constant__ state st) {
  step_begin();
  __shared__ union {
    scan_smem<8> few[8];
    scan_smem<32> one[8];
  } sm;
  auto const lane = threadIdx.x & 31u;
  auto const nr = st.counters[C_R];
  scan_ctr pc{0u, 0u, 0u, 0u, 0u};
  if (nr > kFewPerSm * st.sms) scan_tiles<8, Prof>(st, sm.few[threadIdx.x >> 5], nr, pc);
  else scan_tiles<32, Prof>(st, sm.one[threadIdx.x >> 5], nr, pc);
  if constexpr (Prof) {  // work counters for the roofline (warp-reduced)
    __syncwarp();
    for (auto o = 16; o > 0; o >>= 1) {
      pc.stops += __shfl_xor_sync(kFull, pc.stops, o);
      pc.ev += __shfl_xor_sync(kFull, pc.ev, o);
      pc.days += __shfl_xor_sync(kFull, pc.days, o);
      pc.writes += __shfl_xor_sync(kFull, pc.writes, o);
      pc.warp_steps += __shfl_xor_sync(kFull, pc.warp_steps, o);
    }
    if (lane == 0 && pc.warp_steps != 0u) {
      atomicAdd(&st.prof[0], static_cast<unsigned long long>(pc.stops));
      atomicAdd(&st.prof[1], static_cast<unsigned long long>(pc.ev));
      atomicAdd(&st.prof[2], static_cast<unsigned long long>(pc.days));
      atomicAdd(&st.prof[3], static_cast<unsigned long long>(pc.writes));
      atomicAdd(&st.prof[5], static_cast<unsigned long long>(pc.warp_steps));  // warp stop steps
    }
  }
}

// update_rt_transport, raptor.h:1068-1175 (no vias), a warp per marked
// (rt transport, query) pair, the lanes over the run's stops: et is whether
// the query rides the run when it passes the stop, i.e. whether it could
// board at an earlier stop with no section in between that lacks a required
// flag.  The walk ends at the first stop the query cannot reach, boardable
// or not (raptor.h:1156-1158).  The filters are loop_rt_routes'
// (raptor.h:583-626): the class of the first section and the route flags,
// section by section where set on some sections only.
// A lane per pair walked the run one stop at a time, four dependent loads
// each.
__global__ void __launch_bounds__(256) k_rt_scan(const __grid_constant__ state st) {
  step_begin();
  auto const& T = st.tt;
  auto const* X = st.X[st.counters[C_PAR] ^ 1u];
  auto const lane = threadIdx.x & 31u;
  auto const n_warps = (gridDim.x * blockDim.x) >> 5;
  auto const n_list = st.counters[C_RT];
  scan_ctr pc{};
  for (auto w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n_list; w += n_warps) {
    auto const e = st.rtlist[w];
    auto mask = st.RT_R[e];
    __syncwarp();
    if (lane == 0u) st.RT_R[e] = 0u;
    auto const g = e % st.G, x = e / st.G;
    auto const sb = T.rt_stop_idx[x];
    auto const n = T.rt_stop_idx[x + 1] - sb;
    auto const* tm = T.rt_times + 2ull * (sb - x);
    for (; mask != 0u; mask &= mask - 1u) {
      auto const b = static_cast<uint32_t>(__ffs(mask) - 1);
      auto const s = g * 32u + b;
      auto const ln = st.lanes[s];
      uint32_t sec = 0u;
      if (!ln.run || !scan_filters(T.rt_filter[x], ln, sec)) continue;
      auto const bit = 1u << b;
      auto const fwd = ln.fwd != 0;
      auto const base_min = (T.internal_from_days + static_cast<int32_t>(ln.base)) * 1440;
      auto const lb_off = (ln.mode & 8u) != 0u;
      bool carried = false;  // riding into the chunk
      for (auto i0 = 0u; i0 < n; i0 += 32u) {
        auto const i = i0 + lane;
        auto const act = i < n;
        auto const si = fwd ? i : n - 1u - i;
        uint32_t sw = 0, l = 0;
        uint16_t lbv = 0;
        bool cut = false, marked = false;
        if (act) {
          sw = T.rt_stops[sb + si];
          if ((sec & 0x100u) != 0u) sw = (sw & 0xCFFFFFFFu) | ((sw >> 2) & 0x30000000u);
          l = B2R_STOP_LOC(sw);
          if (!lb_off) lbv = st.lb[li(st, l, s)];
          marked = (X[l * st.G + g] & bit) != 0u;
          cut = (sec & 15u) != 0u && i != 0u &&
                (static_cast<uint32_t>(T.rt_sec[sb + (fwd ? si - 1u : si)]) & (sec & 15u)) != (sec & 15u);
        }
        auto const closed = __ballot_sync(kFull, act && lbv == 0xFFFFu);
        auto const end = closed != 0u ? static_cast<uint32_t>(__ffs(closed) - 1) : 32u;
        auto board = act && lane < end && i + 1u != n && marked && (fwd ? B2R_STOP_IN(sw) : B2R_STOP_OUT(sw)) != 0u;
        if (board) {
          auto const dep = to_key(fwd, clamp16(tm[2u * si - (fwd ? 0u : 1u)] - base_min));
          board = dec(st.rt[rti(st, ln.k - 1u, l, s)], ln.qtag) <= dep;
        }
        auto const boards = __ballot_sync(kFull, board), cuts = __ballot_sync(kFull, cut);
        if (!carried && boards == 0u) {
          if (end != 32u) break;
          continue;
        }
        auto const cut_to = cuts & ((2u << lane) - 1u);  // cuts up to this stop (lane 31: all)
        auto const from = cut_to != 0u ? 31u - static_cast<uint32_t>(__clz(cut_to)) : 0u;
        auto const et = ((boards & ((1u << lane) - 1u)) >> from) != 0u || (carried && cut_to == 0u);
        if (et && act && lane < end && (fwd ? si != 0u : si + 1u != n) &&
            (fwd ? B2R_STOP_OUT(sw) : B2R_STOP_IN(sw)) != 0u) {
          auto const by = to_key(fwd, clamp16(tm[2u * si - (fwd ? 1u : 0u)] - base_min));
          scan_arrive<false>(st, ln, s, g, bit, l, lbv, by, pc);
        }
        if (end != 32u) break;
        carried = (boards >> (cuts != 0u ? 31u - static_cast<uint32_t>(__clz(cuts)) : 0u)) != 0u ||
                  (carried && cuts == 0u);
      }
    }
  }
}

// ------------------------------------- stations reached, destination passes
// tad in effect at position (hi, lo) of phase `ph`'s processing order (0:
// transfers, 1: footpaths)
__device__ __forceinline__ int tad_at(state const& st, uint32_t ph, uint32_t s, uint32_t hi, uint32_t lo) {
  auto const n = st.timeline_n[ph * st.S + s];
  int tad = st.tad_phase[ph * st.S + s];
  auto const* tl = st.timeline + (static_cast<size_t>(ph) * st.S + s) * kMaxTimeline;
  for (auto i = 0u; i != n; ++i) {
    if (tl[i].pos_hi < hi || (tl[i].pos_hi == hi && tl[i].pos_lo < lo)) tad = tl[i].tad;
    else break;
  }
  return tad;
}

// one label of a destination station (key at d), in the phase's order:
// round times, best label, mark, time_at_dest and the phase's timeline
// (raptor.h:690-740, 790-840).  One lane.
__device__ __forceinline__ void dest_label(state const& st, uint32_t* X, slot_t& sl, lane_t const& ln, uint32_t s,
                                           uint32_t d, int key, uint32_t ph, uint32_t pos_hi, uint32_t pos_lo,
                                           uint32_t& tl_n) {
  auto const k = static_cast<uint32_t>(ln.k);
  auto const bk = dec(st.best[li(st, d, s)], ln.gtag);
  auto& rtw = st.rt[rti(st, k, d, s)];
  if (ln.blast == 0u && key < bk && key < dec(rtw, ln.qtag)) {
    rtw = enc(ln.qtag, key);
    touch(st, ln, k, d, s);
  }
  auto const tad = static_cast<int>(sl.tad[k]);
  if (key >= bk || key > tad) return;
  auto const lbv = (ln.mode & 8u) ? uint16_t{0} : st.lb[li(st, d, s)];
  if (lbv == 0xFFFFu || key + static_cast<int>(lbv) > tad) return;
  if (!within_bounds(st, s, ln.blast, k, d, key)) return;
  rtw = enc(ln.qtag, key);
  touch(st, ln, k, d, s);
  st.best[li(st, d, s)] = enc(ln.gtag, key);
  if ((ln.run & kLaneLast) == 0u) {
    atomicOr(&X[d * st.G + (s >> 5)], 1u << (s & 31u));
    atomicOr(&st.made_mask[s >> 5], 1u << (s & 31u));
  }
  if (key < tad) {
    if (tl_n < kMaxTimeline) {
      st.timeline[(static_cast<size_t>(ph) * st.S + s) * kMaxTimeline + tl_n++] = {pos_hi, pos_lo, key};
    } else {
      fail_slot(st, s);
    }
  }
  update_tad(sl, k, key);
}

// update_intermodal_footpaths, raptor.h:954-1026: the best of the egress
// stations' END labels (every label at or below time_at_dest replaces it,
// so the last one kept is their minimum).  A warp.
__device__ __forceinline__ void intermodal_slot(state const& st, slot_t& sl, lane_t const& ln, uint32_t s,
                                                uint32_t lane, int tad0) {
  auto const g = s >> 5;
  auto const bit = 1u << (s & 31u);
  int key = kKeyInv + 1;
  for (auto i = lane; i < sl.n_dest; i += 32u) {
    auto const dr = st.dest_pool[sl.dest_off + i];
    if (!(st.Y[dr.loc * st.G + g] & bit)) continue;
    auto const tk = dec(st.tmp[li(st, dr.loc, s)], ln.gtag);
    if (tk != kKeyInv) key = min(key, key_add(tk, static_cast<int>(dr.dist)));
  }
  key = __reduce_min_sync(kFull, key);
  if (key > tad0) return;  // tad0 <= kKeyInv: nothing reached
  if (lane == 0u) {
    st.rt[rti(st, ln.k, B2R_SPECIAL_END, s)] = enc(ln.qtag, key);
    touch(st, ln, ln.k, B2R_SPECIAL_END, s);
    st.best[li(st, B2R_SPECIAL_END, s)] = enc(ln.gtag, key);
    st.tad_phase[st.S + s] = static_cast<int16_t>(key);
  }
  if (lane >= ln.k && lane < kK && key < sl.tad[lane]) sl.tad[lane] = static_cast<int16_t>(key);
}

struct fp_cand {
  uint32_t src, pos, dest;
  int key;
};
constexpr uint32_t kMaxFpCand = 64;

// The destination stations of a station-to-station query ahead of all other
// stations: their transfers in location order, then the footpaths into them
// in the reference's order (source location, position in the source's
// list), so that the time_at_dest updates they make (raptor.h:737-739) are
// seen by the other stations exactly as in the sequential loops; each
// phase's timeline of those updates is kept per query.  The lanes look for
// the labels, lane 0 takes them in order.
__device__ __forceinline__ void station_dests_slot(state const& st, uint32_t* X, slot_t& sl, lane_t const& ln,
                                                   uint32_t s, uint32_t lane, fp_cand* c) {
  auto const& T = st.tt;
  auto const g = s >> 5;
  auto const bit = 1u << (s & 31u);
  uint32_t tl_n = 0;
  for (auto i0 = 0u; i0 < sl.n_dest; i0 += 32u) {
    auto const i = i0 + lane;
    uint32_t d = 0;
    int tk = kKeyInv;
    if (i < sl.n_dest) {
      d = st.dest_pool[sl.dest_off + i].loc;
      if (st.Y[d * st.G + g] & bit) tk = dec(st.tmp[li(st, d, s)], ln.gtag);
    }
    for (auto m = __ballot_sync(kFull, tk != kKeyInv); m != 0u; m &= m - 1u) {
      auto const src = __ffs(m) - 1;
      auto const xd = __shfl_sync(kFull, d, src);
      auto const xk = __shfl_sync(kFull, tk, src);
      if (lane == 0u) dest_label(st, X, sl, ln, s, xd, key_add(xk, 0), 0u, xd, 0u, tl_n);
    }
  }
  if (lane == 0u) {
    st.timeline_n[s] = tl_n;
    st.tad_phase[st.S + s] = sl.tad[ln.k];
  }
  __syncwarp();
  auto const fwd = ln.fwd != 0;
  auto const prf = (static_cast<uint32_t>(ln.mode) >> 4) & 7u;
  auto const* iidx = fp_index(T, prf, !fwd);
  auto const* idat = fp_words(T, prf, !fwd);
  auto const* oidx = fp_index(T, prf, fwd);
  auto const* odat = fp_words(T, prf, fwd);
  uint32_t nc = 0;
  for (auto i = 0u; i != sl.n_dest; ++i) {
    auto const d = st.dest_pool[sl.dest_off + i].loc;
    auto const xe = iidx[d + 1];
    for (auto x0 = iidx[d]; x0 < xe; x0 += 32u) {
      auto const x = x0 + lane;
      bool has = false;
      fp_cand cd{};
      if (x < xe) {
        auto const src = B2R_FP_TARGET(idat[x]);
        if (st.Y[src * st.G + g] & bit) {
          auto const tk = dec(st.tmp[li(st, src, s)], ln.gtag);
          if (tk != kKeyInv) {
            auto const o0 = oidx[src], o1 = oidx[src + 1];
            // the footpath in the source's own list: among several between
            // the two, the one of this duration
            auto at = o1;
            for (auto y = o0; y != o1; ++y) {
              if (B2R_FP_TARGET(odat[y]) != d) continue;
              if (at == o1) at = y;
              if (B2R_FP_DURATION(odat[y]) != B2R_FP_DURATION(idat[x])) continue;
              at = y;
              break;
            }
            if (at != o1) {
              auto const dur = adjusted<int>(sl.tts, static_cast<int>(B2R_FP_DURATION(odat[at])));
              cd = {src, at - o0, d, key_add(tk, dur)};
              has = true;
            }
          }
        }
      }
      auto const m = __ballot_sync(kFull, has);
      auto const at = nc + static_cast<uint32_t>(__popc(m & ((1u << lane) - 1u)));
      if (has && at < kMaxFpCand) c[at] = cd;
      if (has && at >= kMaxFpCand) fail_slot(st, s);
      nc = min(nc + static_cast<uint32_t>(__popc(m)), kMaxFpCand);
    }
  }
  __syncwarp();
  if (lane == 0u) {
    for (auto a = 1u; a < nc; ++a) {  // insertion sort by (src, pos)
      auto const x = c[a];
      auto b = a;
      while (b > 0u && (c[b - 1u].src > x.src || (c[b - 1u].src == x.src && c[b - 1u].pos > x.pos))) {
        c[b] = c[b - 1u];
        --b;
      }
      c[b] = x;
    }
    tl_n = 0;
    for (auto a = 0u; a != nc; ++a) {
      dest_label(st, X, sl, ln, s, c[a].dest, c[a].key, 1u, c[a].src, c[a].pos, tl_n);
    }
    st.timeline_n[st.S + s] = tl_n;
  }
}

// After the scan: the stations it reached listed (every nonzero word of Y),
// the station marks the round read cleared, and per slot (a warp each) what
// the round does at the query's destinations before all other stations.
// The destination passes of both phases can run ahead of the other
// stations' transfers because they alone write the destinations' labels:
// k_relax leaves out transfers at, and footpaths into, destinations.
// The first blocks take the slots, 8 each, the others the words.
__global__ void __launch_bounds__(256) k_reached(state st) {
  step_begin();
  __shared__ fp_cand cand[8][kMaxFpCand];
  auto const lane = threadIdx.x & 31u;
  auto const par = st.counters[C_PAR];
  auto const slot_blocks = (st.S + 7u) / 8u;
  if (blockIdx.x < slot_blocks) {
    auto const s = blockIdx.x * 8u + (threadIdx.x >> 5);
    if (s >= st.S) return;
    auto const ln = st.lanes[s];
    if (!ln.run) return;
    auto& sl = st.slots[s];
    auto const tad0 = static_cast<int>(sl.tad[ln.k]);
    if (lane < 2u) {
      st.timeline_n[lane * st.S + s] = 0u;
      st.tad_phase[lane * st.S + s] = static_cast<int16_t>(tad0);
    }
    __syncwarp();
    if (ln.mode & 1u) intermodal_slot(st, sl, ln, s, lane, tad0);
    else if (ln.mode & 2u) station_dests_slot(st, st.X[par], sl, ln, s, lane, cand[threadIdx.x >> 5]);
    return;
  }
  auto const block = blockIdx.x - slot_blocks, n_blocks = gridDim.x - slot_blocks;
  auto const n = st.tt.n_loc * st.G;
  auto* X = st.X[par ^ 1u];
  for (auto i = (block * blockDim.x + threadIdx.x) * 4u; i < n; i += n_blocks * blockDim.x * 4u) {
    if (i + 3u < n) {
      auto* p = reinterpret_cast<uint4*>(X + i);
      auto const v = *p;
      if ((v.x | v.y | v.z | v.w) != 0u) *p = uint4{0u, 0u, 0u, 0u};
    } else {
      for (auto j = i; j < n; ++j) X[j] = 0u;
    }
  }
  list_nonzero(st, st.Y, n, C_Y, block, n_blocks, one_item{}, [&](uint32_t at, uint32_t e, uint32_t) { st.ylist[at] = e; });
}

// ------------------------------------------------ transfers and footpaths
// update_transfers (raptor.h:680-743) and update_footpaths (raptor.h:745-
// 845): a lane per reached (station, query) pair takes the station's
// transfer, then walks its footpaths.  The pair's word of reached marks is
// cleared as it is read.
//
// The reference runs all transfers before all footpaths.  Taken together
// they give the same labels: both only lower round_times[k] and best, to
// the minimum of the candidates that beat best at the start of the round
// and pass the pruning, and a candidate that meets a label already lowered
// by another one of the round is above a value that is written anyway.  The
// pruning bounds differ between the phases, and each keeps its own
// (tad_phase, timelines; k_reached).
//
// A start-time group's last round marks nothing: no round of the group would
// read the marks, and left in place they would be the next search's of the
// slot, which starts from its own stations alone (raptor.h:179-188).
//
// Which queries marked a station is gathered per block and written once (a
// global word per group read and written by every pair doubled the kernel's
// time at 1,024 slots).
//
// Four blocks per SM (62 registers): left to itself the compiler took 80, three
// blocks, for a kernel that waits on gathers (device time of 1,024 queries 3.87
// -> 3.77 ms, of the national 256 44.0 -> 43.3, 333 filtered ones 2.68 -> 2.65;
// runs repeat within 0.5%).  48 registers with five blocks took the same, 40
// spill.
__global__ void __launch_bounds__(256, 4) k_relax(state st) {
  step_begin();
  __shared__ uint32_t made_bits[kMaxGroups];
  for (auto g = threadIdx.x; g < st.G; g += blockDim.x) made_bits[g] = 0u;
  __syncthreads();
  auto const& T = st.tt;
  auto* X = st.X[st.counters[C_PAR]];
  for_each_pair(
      st.ylist, st.counters[C_Y],
      [&](uint32_t e) {
        auto const m = st.Y[e];
        st.Y[e] = 0u;
        return m;
      },
      [&](uint32_t e, uint32_t b) {
        auto const g = e % st.G, src = e / st.G;
        auto const s = g * 32u + b;
        auto const ln = st.lanes[s];
        if (!ln.run) return;
        auto const tk = dec(st.tmp[li(st, src, s)], ln.gtag);
        if (tk == kKeyInv) return;
        auto const stations = (ln.mode & 2u) != 0u;
        auto const& tts = st.slots[s].tts;
        auto const marks = (ln.run & kLaneLast) == 0u;
        bool made = false;  // a station marked
        if (!stations || !((st.D[e] >> b) & 1u)) {
          auto const tt = static_cast<int>(T.transfer_time[src]);
          auto const fp = key_add(tk, (ln.mode & 4u) ? tt : static_cast<int>(adjusted<int>(tts, tt)));
          if (fp < dec(st.best[li(st, src, s)], ln.gtag)) {
            auto* rtw = &st.rt[rti(st, ln.k, src, s)];
            // the reference writes round_times ahead of its pruning only
            // when unbounded (raptor.h:710-714, 790-794)
            if (ln.blast == 0u) {
              atomicMin(rtw, enc(ln.qtag, fp));
              touch(st, ln, ln.k, src, s);
            }
            auto const tad = stations ? tad_at(st, 0u, s, src, 0u) : static_cast<int>(st.tad_phase[s]);
            auto const lbv = (ln.mode & 8u) ? uint16_t{0} : st.lb[li(st, src, s)];
            if (fp <= tad && lbv != 0xFFFFu && fp + static_cast<int>(lbv) <= tad &&
                within_bounds(st, s, ln.blast, ln.k, src, fp)) {
              if (ln.blast != 0u) {
                atomicMin(rtw, enc(ln.qtag, fp));
                touch(st, ln, ln.k, src, s);
              }
              atomicMin(&st.best[li(st, src, s)], enc(ln.gtag, fp));
              if (marks) {
                atomicOr(&X[e], 1u << b);
                made = true;
              }
            }
          }
        }
        auto const fwd = ln.fwd != 0;
        auto const prf = (static_cast<uint32_t>(ln.mode) >> 4) & 7u;
        auto const* idx = fp_index(T, prf, fwd);
        auto const* dat = fp_words(T, prf, fwd);
        auto const fb = idx[src], n = idx[src + 1] - fb;
        auto const tad_flat = static_cast<int>(st.tad_phase[st.S + s]);
        // four footpaths at a time: their targets' labels load together
        for (auto j0 = 0u; j0 < n; j0 += 4u) {
          uint32_t fps[4];
          int bks[4];
#pragma unroll
          for (auto x = 0u; x != 4u; ++x) fps[x] = j0 + x < n ? dat[fb + j0 + x] : B2R_INVALID_IDX;
#pragma unroll
          for (auto x = 0u; x != 4u; ++x) {
            bks[x] = j0 + x < n ? dec(st.best[li(st, B2R_FP_TARGET(fps[x]), s)], ln.gtag) : -32768;
          }
#pragma unroll
          for (auto x = 0u; x != 4u; ++x) {
            auto const j = j0 + x;
            auto const tgt = B2R_FP_TARGET(fps[x]);
            auto const dur = static_cast<int>(B2R_FP_DURATION(fps[x]));
            auto const key = key_add(tk, (ln.mode & 4u) ? dur : adjusted<int>(tts, dur));
            if (key >= bks[x]) continue;  // no key is below -32768: the places past the end too
            if (stations && ((st.D[tgt * st.G + g] >> b) & 1u)) continue;
            if (ln.blast == 0u) {
              atomicMin(&st.rt[rti(st, ln.k, tgt, s)], enc(ln.qtag, key));
              touch(st, ln, ln.k, tgt, s);
            }
            auto const tad = stations ? tad_at(st, 1u, s, src, j) : tad_flat;
            if (key > tad) continue;
            auto const lbv = (ln.mode & 8u) ? uint16_t{0} : st.lb[li(st, tgt, s)];
            if (lbv != 0xFFFFu && key + static_cast<int>(lbv) <= tad) {
              if (ln.blast != 0u) {
                if (!within_bounds(st, s, ln.blast, ln.k, tgt, key)) continue;
                atomicMin(&st.rt[rti(st, ln.k, tgt, s)], enc(ln.qtag, key));
                touch(st, ln, ln.k, tgt, s);
              }
              atomicMin(&st.best[li(st, tgt, s)], enc(ln.gtag, key));
              if (marks) {
                atomicOr(&X[tgt * st.G + g], 1u << b);
                made = true;
              }
            }
          }
        }
        if (made && ((made_bits[g] >> b) & 1u) == 0u) atomicOr(&made_bits[g], 1u << b);
      });
  __syncthreads();
  for (auto g = threadIdx.x; g < st.G; g += blockDim.x) {
    if (made_bits[g] != 0u) atomicOr(&st.made_mask[g], made_bits[g]);
  }
}

// ------------------------------------------------- round end / results
__host__ __device__ inline bool dominates(journey_rec const& a, journey_rec const& b) {  // journey.h:84-92
  if (a.start_time <= a.dest_time) {
    return a.transfers <= b.transfers && a.start_time >= b.start_time && a.dest_time <= b.dest_time;
  }
  return a.transfers <= b.transfers && a.start_time <= b.start_time && a.dest_time >= b.dest_time;
}

__device__ int alloc_block(state const& st, uint32_t s) {
  auto const words = (st.max_j + 31u) / 32u;
  for (auto w = 0u; w != words; ++w) {
    auto& u = st.blocks_used[s * words + w];
    auto const free_bits = ~u;
    if (free_bits != 0u) {
      auto const b = __ffs(free_bits) - 1;
      if (w * 32u + b >= st.max_j) break;
      u |= 1u << b;
      return static_cast<int>(w * 32u + b);
    }
  }
  return -1;
}

__device__ void free_block(state const& st, uint32_t s, uint16_t blk) {
  auto const words = (st.max_j + 31u) / 32u;
  st.blocks_used[s * words + blk / 32u] &= ~(1u << (blk % 32u));
}

// pareto_set::add, pareto_set.h:21-37, by a warp: the lanes compare the
// journeys 32 at a time.  A journey that dominates `el` leaves the set as it
// is (then none in the set is dominated by `el`, or the set would not be
// Pareto); the journeys `el` dominates go, the others keep their order.
__device__ bool pareto_add(state const& st, uint32_t s, uint32_t& n, journey_rec el, uint32_t lane) {
  auto* els = st.journeys + static_cast<size_t>(s) * st.max_j;
  for (auto i0 = 0u; i0 < n; i0 += 32u) {
    auto const i = i0 + lane;
    if (__any_sync(kFull, i < n && dominates(els[i], el))) return true;
  }
  auto kept = 0u;
  for (auto i0 = 0u; i0 < n; i0 += 32u) {
    auto const i = i0 + lane;
    journey_rec x{};
    bool keep = false, drop = false;
    if (i < n) {
      x = els[i];
      drop = dominates(el, x);
      keep = !drop;
    }
    auto const km = __ballot_sync(kFull, keep);
    for (auto dm = __ballot_sync(kFull, drop); dm != 0u; dm &= dm - 1u) {
      if (static_cast<int>(lane) == __ffs(dm) - 1) free_block(st, s, x.block);
      __syncwarp();
    }
    if (keep) els[kept + static_cast<uint32_t>(__popc(km & ((1u << lane) - 1u)))] = x;
    kept += static_cast<uint32_t>(__popc(km));
    __syncwarp();
  }
  n = kept;
  auto blk = -1;
  if (lane == 0u) blk = alloc_block(st, s);
  blk = __shfl_sync(kFull, blk, 0);
  if (blk < 0 || n >= st.max_j) return false;
  el.block = static_cast<uint16_t>(blk);
  if (lane == 0u) els[n] = el;
  ++n;
  __syncwarp();
  return true;
}

// whether journey j of the slot is to be reconstructed now (search.h:457-475;
// a pong phase rebuilds only the journey of its ping result, pong.cc:322-339)
__device__ __forceinline__ bool recon_wanted(slot_t const& sl, journey_rec const& j) {
  if (j.reconstructed || j.error) return false;
  auto const tt = j.dest_time > j.start_time ? j.dest_time - j.start_time : j.start_time - j.dest_time;
  return sl.recon_mode == 0 ? ((sl.ontrip || (sl.iv_from <= j.start_time && j.start_time < sl.iv_to)) &&
                               tt < sl.fastest_direct)
         : sl.recon_mode == 1 ? (j.transfers == sl.recon_transfers && j.start_time == sl.recon_start)
                              : false;
}

// result collection (raptor.h:393-413): the round times of the destinations
// in the reference's order (destination, then round), the lanes loading 32
// of them at once, into the slot's Pareto set.  A warp; false: out of
// journey capacity.
__device__ bool collect_slot(state const& st, slot_t& sl, uint32_t s, uint32_t lane) {
  auto const qtag = tagcode(sl.gen_query);
  auto const fwd = sl.fwd != 0;
  auto const n_k = static_cast<uint32_t>(sl.end_k) - 1u;
  auto const total = (sl.intermodal_dest ? 1u : sl.n_dest) * n_k;
  auto n = sl.n_journeys;
  __syncwarp();
  bool ok = true;
  for (auto p0 = 0u; ok && p0 < total; p0 += 32u) {
    auto const p = p0 + lane;
    int key = kKeyInv;
    uint32_t d = 0, k = 0;
    if (p < total) {
      k = 1u + p % n_k;
      d = sl.intermodal_dest ? B2R_SPECIAL_END : st.dest_pool[sl.dest_off + p / n_k].loc;
      key = dec(st.rt[rti(st, k, d, s)], qtag);
    }
    for (auto m = __ballot_sync(kFull, key != kKeyInv); ok && m != 0u; m &= m - 1u) {
      auto const src = __ffs(m) - 1;
      journey_rec j{};
      j.start_time = sl.cur_start_time;
      j.dest_time = sl.base_days * 1440 + from_key(fwd, __shfl_sync(kFull, key, src));
      j.dest = __shfl_sync(kFull, d, src);
      j.transfers = static_cast<uint8_t>(__shfl_sync(kFull, k, src) - 1u);
      ok = pareto_add(st, s, n, j, lane);
    }
  }
  if (lane == 0u) sl.n_journeys = n;
  __syncwarp();
  return ok;
}

// the reconstruction worklist (search.h:457-475): whether any journey of the
// slot is to be rebuilt before its next start-time group
__device__ bool list_recon(state const& st, slot_t const& sl, uint32_t s, uint32_t lane, uint32_t par) {
  auto const* els = st.journeys + static_cast<size_t>(s) * st.max_j;
  auto any = false;
  for (auto i0 = 0u; i0 < sl.n_journeys; i0 += 32u) {
    auto const i = i0 + lane;
    auto const want = i < sl.n_journeys && recon_wanted(sl, els[i]);
    if (want) st.recon_list[atomicAdd(&st.counters[recon_counter(par)], 1u)] = (s << 16) | i;
    any = __any_sync(kFull, want) || any;
  }
  return any;
}

// One journey (slot s, index ji) rebuilt by the calling group of NW warps.
template <int NW>
__device__ __forceinline__ void reconstruct_one(state const& st, recon_smem<NW>& sm, uint32_t s, uint32_t ji) {
  uint64_t t_begin = 0;
  if (st.profile) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_begin));
  auto& sl = st.slots[s];
  auto& j = st.journeys[static_cast<size_t>(s) * st.max_j + ji];
  recon_ctx<NW> c;
  c.st = &st;
  c.T = &st.tt;
  c.sl = &sl;
  c.s = s;
  c.fwd = sl.fwd != 0;
  c.qtag = tagcode(sl.gen_query);
  c.base_days = sl.base_days;
  c.base = sl.base;
  c.ontrip = sl.ontrip != 0;
  c.j = &j;
  c.tid = threadIdx.x % recon_ctx<NW>::kT;
  c.lane = threadIdx.x & 31u;
  c.wid = c.tid >> 5;
  c.sm = &sm;
  c.legs = sm.legs;
  c.run();  // ends with the group in step unless it failed
  c.sync();
  if (!c.failed) {
    auto* out = reinterpret_cast<uint32_t*>(st.legs + (static_cast<size_t>(s) * st.max_j + j.block) * kMaxLegs);
    auto const* in = reinterpret_cast<uint32_t const*>(sm.legs);
    auto const words = static_cast<uint32_t>(c.n_legs) * static_cast<uint32_t>(sizeof(b2r_leg) / 4u);
    for (auto i = c.tid; i < words; i += recon_ctx<NW>::kT) out[i] = in[i];
  }
  c.sync();  // before the next journey's legs
  if (c.tid == 0) {
    if (c.failed) {
      j.error = 1;
    } else {
      j.reconstructed = 1;
      j.n_legs = static_cast<uint16_t>(c.n_legs);
    }
    if (st.profile) {  // longest single reconstruction (ns), journeys
      uint64_t t_end = 0;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_end));
      atomicMax(&st.prof[6], static_cast<unsigned long long>(t_end - t_begin));
      atomicAdd(&st.prof[7], 1ull);
    }
  }
}

// The journeys listed at the end of the last super-step (queries with
// several start-time groups: their next group changes the round times), a
// block each.  Their slots wait (S_RECON) while the round kernels of the
// other slots run beside this one; the step's k_end joins both and sends
// them on.
constexpr int kReconWarps = 4;
__global__ void __launch_bounds__(kReconWarps * 32) k_reconstruct(state st) {
  __shared__ recon_smem<kReconWarps> sm;
  auto const n = st.counters[recon_counter(st.counters[C_RPAR])];
  for (auto i = blockIdx.x; i < n; i += gridDim.x) {
    auto const e = st.recon_list[i];
    reconstruct_one<kReconWarps>(st, sm, e >> 16, e & 0xFFFFu);
  }
}

// One given journey of slot s (index ji): the Algo interface's reconstruct.
__global__ void __launch_bounds__(kReconWarps * 32) k_reconstruct_one(state st, uint32_t s, uint32_t ji) {
  __shared__ recon_smem<kReconWarps> sm;
  reconstruct_one<kReconWarps>(st, sm, s, ji);
}

// The journeys of finished slots whose reconstruction was deferred, listed
// by the host as (slot << 16 | journey index): launched on the export stream
// while the next super-steps run.  A finished slot is left alone by the
// super-step kernels, so its round times are stable.  Blocks of 128 threads:
// one group of four warps, or four of one.
template <int NW>
__global__ void __launch_bounds__(128) k_reconstruct_done(state st, uint32_t const* list, uint32_t n) {
  constexpr auto kGroups = 4 / NW;
  __shared__ recon_smem<NW> sm[kGroups];
  auto const grp = threadIdx.x / (NW * 32u);
  for (auto i = blockIdx.x * kGroups + grp; i < n; i += gridDim.x * kGroups) {
    auto const e = list[i];
    auto const s = e >> 16, ji = e & 0xFFFFu;
    auto const& sl = st.slots[s];
    if (!sl.recon_defer || ji >= sl.n_journeys) continue;
    if (!recon_wanted(sl, st.journeys[static_cast<size_t>(s) * st.max_j + ji])) continue;
    reconstruct_one<NW>(st, sm[grp], s, ji);
  }
}

// early termination (search.h:477-492) and seeding of the next start-time
// group: next_start_time + add_start (raptor.h:179-203) + the
// time_at_dest bound of execute (raptor.h:211-214).  A warp; labels are
// combined with atomicMin (an older generation's word has a larger tag), so
// the lanes take the group's starts in any order.
__device__ void next_slot(state const& st, uint32_t* X, slot_t& sl, uint32_t s, uint32_t lane, bool collected) {
  auto const fwd = sl.fwd != 0;
  auto early = sl.early_term != 0;
  if (collected && sl.min_connection_count > 0 && !sl.one_to_all) {
    uint32_t n_in = 0;
    auto const* els = st.journeys + static_cast<size_t>(s) * st.max_j;
    for (auto i = lane; i < sl.n_journeys; i += 32u) {
      n_in += sl.ontrip ? 1u : ((sl.iv_from <= els[i].start_time && els[i].start_time < sl.iv_to) ? 1u : 0u);
    }
    n_in = __reduce_add_sync(kFull, n_in);
    if (n_in >= sl.min_connection_count &&
        ((fwd && sl.extend_earlier && !sl.extend_later) || (!fwd && !sl.extend_earlier && sl.extend_later))) {
      early = true;
      if (lane == 0u) {
        sl.early_term = 1;
        if (fwd) sl.iv_from = sl.cur_start_time;
        else sl.iv_to = sl.cur_start_time + 1;
      }
    }
  }
  if (lane == 0u && collected) sl.need_sweep = 1;
  auto const* starts = st.start_pool + sl.starts_off;
  auto const n_starts = sl.n_starts;
  auto const g0 = sl.next_start;
  if (early || g0 >= n_starts) {
    __syncwarp();
    if (lane == 0u) sl.state = S_DONE;
    return;
  }
  // next start-time group
  auto const tas = starts[g0].time_at_start;
  auto gen = sl.gen_group;
  __syncwarp();
  if (gen >= 0xFFFEu) {  // tag space exhausted: clear this slot's labels
    for (auto l = lane; l < st.tt.n_loc; l += 32u) {
      st.best[li(st, l, s)] = 0xFFFFFFFFu;
      st.tmp[li(st, l, s)] = 0xFFFFFFFFu;
    }
    gen = 0;
    __syncwarp();
  }
  ++gen;
  auto const gtag = tagcode(gen), qtag = tagcode(sl.gen_query);
  auto const g = s >> 5;
  auto const bit = 1u << (s & 31u);
  auto g1 = g0;
  while (g1 < n_starts) {
    auto const i = g1 + lane;
    auto const in = i < n_starts && starts[i].time_at_start == tas;
    auto const out = __ballot_sync(kFull, !in);
    auto const len = out == 0u ? 32u : static_cast<uint32_t>(__ffs(out) - 1);
    if (lane < len) {
      auto const l = starts[i].stop;
      auto const key = to_key(fwd, clamp16(starts[i].time_at_stop - sl.base_days * 1440));
      if (key != kKeyInv) {
        atomicMin(&st.best[li(st, l, s)], enc(gtag, key));
        atomicMin(&st.rt[rti(st, 0, l, s)], enc(qtag, key));
      }
      atomicOr(&X[l * st.G + g], bit);
    }
    g1 += len;
    if (len != 32u) break;
  }
  auto const worst = tas + (fwd ? static_cast<int>(sl.span) : -static_cast<int>(sl.span));
  auto const d_worst = to_key(fwd, clamp16(worst - sl.base_days * 1440));
  if (lane < kK && d_worst < sl.tad[lane]) sl.tad[lane] = static_cast<int16_t>(d_worst);
  __syncwarp();
  if (lane == 0u) {
    sl.gen_group = gen;
    sl.cur_start_time = tas;
    sl.next_start = g1;
    sl.k = 1;
    sl.state = S_RUN;
    ++sl.n_groups_run;
  }
}

// Round k of a slot whose last round marked no station, without a super-step
// of its own: all it does is to count, to sweep and to take the destination
// times (raptor.h:218-226) before it finds nothing marked (raptor.h:243-246),
// and of the swept labels only the destinations' are read again.
__device__ __forceinline__ void empty_round(state const& st, slot_t& sl, uint32_t s, uint32_t k, uint32_t lane) {
  if (!sl.one_to_all) {
    auto const gtag = tagcode(sl.gen_group), qtag = tagcode(sl.gen_query);
    int key = kKeyInv;
    auto const take = [&](uint32_t d) {
      key = min(key, min(dec(st.best[li(st, d, s)], gtag), dec(st.rt[rti(st, k, d, s)], qtag)));
    };
    if (sl.intermodal_dest) {
      take(B2R_SPECIAL_END);
    } else {
      for (auto i = lane; i < sl.n_dest; i += 32u) take(st.dest_pool[sl.dest_off + i].loc);
    }
    key = __reduce_min_sync(kFull, key);
    if (lane >= k && lane < kK && key < sl.tad[lane]) sl.tad[lane] = static_cast<int16_t>(key);
  }
  if (lane == 0u) ++sl.n_rounds;
}

// The end of a super-step, a warp per slot and a block per group of 32
// slots: the round's end (raptor.h:217), the next round at once if it would
// be empty (one step in six), collection when the group's rounds
// are over, the journeys to rebuild listed (the slot then waits one step in
// S_RECON; so does a failed one, whose round left marks that that step
// clears), the next start-time group seeded, and the slot's views for the
// next step (lane record, the group's run mask and, per round, its slots to
// sweep) and for the host
// (summary).  seed_only: admitted slots are seeded and the views renewed,
// nothing else (after an admission, so that a query's first super-step is
// its first round).
// A thread per slot walked destinations x rounds and the journey list one
// dependent load at a time.
__global__ void __launch_bounds__(1024, 1) k_end(state st, bool seed_only) {
  step_begin();
  __shared__ uint32_t run_bits, sweep_bits[kK];
  auto const lane = threadIdx.x & 31u;
  auto const g = blockIdx.x;
  auto const s = g * 32u + (threadIdx.x >> 5);
  if (threadIdx.x == 0u) run_bits = 0u;
  if (threadIdx.x < kK) sweep_bits[threadIdx.x] = 0u;
  __syncthreads();
  auto const par = st.counters[C_PAR];
  auto& sl = st.slots[s];
  auto state = sl.state;
  __syncwarp();
  if (seed_only) {
    if (state == S_START) next_slot(st, st.X[par], sl, s, lane, false);
  } else {
    auto const failed = sl.error != 0;
    if (state == S_START || (state == S_RECON && !failed)) {
      next_slot(st, st.X[par], sl, s, lane, state == S_RECON);
    } else if (state == S_RECON) {
      if (lane == 0u) sl.state = S_ERROR;
    } else {
      if (state == S_RUN) {
        auto const k = static_cast<uint8_t>(sl.k + 1u);
        __syncwarp();
        if (lane == 0u) sl.k = k;
        if (failed) {
          state = S_RECON;
        } else if (k >= sl.end_k) {
          state = S_COLLECT;
        } else if (((st.made_mask[g] >> (s & 31u)) & 1u) == 0u) {
          empty_round(st, sl, s, k, lane);
          state = S_COLLECT;
        }
      }
      if (state == S_COLLECT) {
        if (!sl.one_to_all && !collect_slot(st, sl, s, lane)) {
          state = S_ERROR;
          if (lane == 0u) sl.error = B2R_ERR_CAPACITY;
        } else if (!sl.one_to_all && !sl.recon_defer && list_recon(st, sl, s, lane, par)) {
          state = S_RECON;  // else rebuilt when the slot is done (k_reconstruct_done), or nothing to rebuild
        } else {
          next_slot(st, st.X[par], sl, s, lane, true);
        }
      }
      if ((state == S_ERROR || state == S_RECON) && lane == 0u) sl.state = state;
    }
  }
  __syncwarp();
  if (lane == 0u) {
    st.summary[s] = {sl.state, static_cast<uint8_t>(min(255u, sl.n_starts - sl.next_start)), {0, 0}, sl.n_journeys};
    st.lanes[s] = lane_of(sl);
    if (sl.state == S_RUN) {
      atomicOr(&run_bits, 1u << (s & 31u));
      if (sl.need_sweep) atomicOr(&sweep_bits[sl.k], 1u << (s & 31u));
    }
  }
  __syncthreads();
  if (threadIdx.x == 0u) {
    st.run_mask[g] = run_bits;
    st.any_mask[g] = 0u;
  }
  if (threadIdx.x < kK) st.sweep_k[g * kK + threadIdx.x] = sweep_bits[threadIdx.x];
}

// ------------------------------------------------------- lower bounds
// Dijkstra from the destinations over the lower-bound graph (dijkstra.cc:
// 18-67, dial.h), computed for all newly admitted queries at once as a
// frontier-driven Bellman-Ford: distances are shortest-path lengths capped
// below kMaxTravelTime + 1 = 7201 (the dial's bucket count), which no
// processing order changes (all weights are non-negative).
constexpr uint32_t kLbBuckets = B2R_MAX_TRAVEL_TIME_MIN + 1;

__global__ void k_lb_relax(state st, uint32_t p) {
  auto const lane = threadIdx.x & 31u;
  auto const warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  auto const n_warps = (gridDim.x * blockDim.x) >> 5;
  auto const n = st.counters[C_F0 + p];
  auto const& T = st.tt;
  for (auto w = warp; w < n; w += n_warps) {
    auto const e = st.flist[p][w];
    auto const g = e % st.G, l = e / st.G;
    auto const m = st.F[p][e];
    auto const s = g * 32u + lane;
    auto const& sl = st.slots[s];
    bool act = (m >> lane) & 1u;
    auto const qtag = tagcode(sl.gen_query);
    int d = kKeyInv;
    if (act) {
      d = dec(st.dist[li(st, l, s)], qtag);
      act = d != kKeyInv;
    }
    auto const fwd = sl.fwd != 0;
    auto const* gi = fwd ? T.lbg_fwd_idx : T.lbg_bwd_idx;
    auto const* gd = fwd ? T.lbg_fwd : T.lbg_bwd;
    auto const b = act ? gi[l] : 0u;
    auto const cnt = act ? gi[l + 1] - b : 0u;
    auto n_max = cnt;
    for (auto o = 16; o > 0; o >>= 1) n_max = max(n_max, __shfl_xor_sync(kFull, n_max, o));
    for (auto j = 0u; j != n_max; ++j) {
      bool improved = false;
      uint32_t tgt = 0;
      if (j < cnt) {
        auto const edge = gd[b + j];
        tgt = B2R_FP_TARGET(edge);
        auto const nd = static_cast<uint32_t>(d) + B2R_FP_DURATION(edge);
        if (nd < kLbBuckets) {
          auto const word = enc(qtag, static_cast<int>(nd));
          auto* dp = &st.dist[li(st, tgt, s)];
          if (word < *dp) improved = word < atomicMin(dp, word);
          if (improved && st.profile) atomicAdd(&st.prof[4], 1ull);
        }
      }
      mark_warp(st, st.F[1 - p], st.flist[1 - p], C_F0 + (1 - p), improved, tgt * st.G + g, lane);
    }
  }
}

__global__ void k_lb_clear(state st, uint32_t p) {
  auto const n = st.counters[C_F0 + p];
  for (auto i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    st.F[p][st.flist[p][i]] = 0u;
  }
}

__global__ void k_lb_reset(state st, uint32_t p) {
  if (blockIdx.x == 0 && threadIdx.x == 0) st.counters[C_F0 + p] = 0u;
}

// children inherit their parent's bound (dijkstra.cc:60-65), in location
// order per query
__global__ void k_lb_children(state st) {
  auto const s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= st.S || !((st.lb_mask[s >> 5] >> (s & 31)) & 1u)) return;
  auto const qtag = tagcode(st.slots[s].gen_query);
  auto const& T = st.tt;
  for (auto x = 0u; x != T.n_with_children; ++x) {
    auto const i = T.with_children[x];
    auto const lbw = st.dist[li(st, i, s)];
    for (auto c = T.children_idx[i]; c != T.children_idx[i + 1]; ++c) {
      auto* cw = &st.dist[li(st, T.children[c], s)];
      if (dec(lbw, qtag) < dec(*cw, qtag)) *cw = lbw;
    }
  }
}

// tagged distances -> the u16 lower-bound column (unreachable = 0xFFFF)
__global__ void k_lb_finish(state st) {
  auto const n = static_cast<size_t>(st.tt.n_loc) * st.S;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    auto const s = static_cast<uint32_t>(i % st.S);
    if (!((st.lb_mask[s >> 5] >> (s & 31)) & 1u)) continue;
    auto const d = dec(st.dist[i], tagcode(st.slots[s].gen_query));
    st.lb[i] = d == kKeyInv ? uint16_t{0xFFFFu} : static_cast<uint16_t>(d);
  }
}

}  // namespace b2r::dev
