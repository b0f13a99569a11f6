// One-to-all search of one query that allocates nothing
// (b2r_one_to_all_noalloc of include/b2r.h).
//
// routing::one_to_all (one_to_all.cc:25-92) for the static timetable: the
// starts of the query's offsets, then raptor::execute's rounds
// (raptor.h:218-387) without destinations and without lower bounds.  Its
// working state lives in g_noalloc_scratch, a fixed file-scope device array:
// the call issues no cudaMalloc / cudaFree and uses no engine, so callers
// whose device memory belongs to another allocator, or whose query path
// must not stall the device with cudaFree, can run one-to-all searches.
//
// A round is three kernels: stations mark routes, a warp per marked route
// scans it (lanes over the stops), stations relax transfers and footpaths.
// All rounds are launched at once; a round without a marked route returns at
// its first load.  What bounds it: on 40,000 stops the scans' dependent
// loads (0.66 ms a query; one cluster of 8 CTAs with a thread walking each
// route took 7.1 ms, the same cluster with this scan 3.5 ms on its eight
// SMs), on 1,000 stops the 45 launches (0.22 ms; the cluster 0.21 ms).
//
// The per-query rules are those of the batched engine's kernels (route
// scan, transfers, footpaths) for one query: labels are plain int keys
// (t forward, ~t backward, kKeyInv invalid) cleared at the start of every
// call, so the rows equal the rows b2r_search_batch returns.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <mutex>

#include "b2r.h"
#include "engine.cuh"
#include "errors.h"
#include "et_search.cuh"
#include "prep.h"
#include "timetable_image.h"

namespace b2r::noalloc {

constexpr uint32_t kRows = B2R_K;
constexpr uint32_t kMaxLoc = B2R_NOALLOC_MAX_LOCATIONS;
constexpr uint32_t kMaxRoutes = B2R_NOALLOC_MAX_ROUTES;
constexpr int kInv = dev::kKeyInv;

// scratch layout (byte offsets)
constexpr size_t kRtOff = 0;                                        // int [kRows][kMaxLoc]
constexpr size_t kBestOff = kRtOff + size_t{kRows} * kMaxLoc * 4;   // int [kMaxLoc]
constexpr size_t kTmpOff = kBestOff + size_t{kMaxLoc} * 4;          // int [kMaxLoc]
constexpr size_t kXOff = kTmpOff + size_t{kMaxLoc} * 4;             // station marks by round parity
constexpr size_t kYOff = kXOff + size_t{2} * kMaxLoc * 4;           // route-reached marks
constexpr size_t kROff = kYOff + size_t{kMaxLoc} * 4;               // route marks
constexpr size_t kOutOff = kROff + size_t{kMaxRoutes} * 4;          // int16 [rows][n_loc]
constexpr size_t kAnyOff = kOutOff + size_t{kRows} * kMaxLoc * 2;   // per round: a route is marked
constexpr size_t kBytes = B2R_NOALLOC_SCRATCH_BYTES;
static_assert(kAnyOff + size_t{kRows} * 4 <= kBytes, "scratch too small");

struct params {
  int32_t start_time;
  int32_t base_days;
  int32_t tad;  // worst time at destination (one_to_all.cc:44-46), as a key
  uint16_t base;
  uint8_t fwd;
  uint8_t mode;  // start match mode
  uint8_t end_k;
  uint32_t n_off;
  dev::tts_t tts;
  uint16_t claszes;  // allowed transport classes
  uint8_t req;       // required route flags
  uint8_t prf;       // footpath profile (query::prf_idx_)
  b2r_offset off[B2R_NOALLOC_MAX_OFFSETS];
};

}  // namespace b2r::noalloc

// The working state of every b2r_one_to_all_noalloc call on a device:
// round times, best / tmp labels, marks and the int16 result rows.  Calls
// that overlap on the GPU share it.
static __device__ __align__(256) uint8_t g_noalloc_scratch[b2r::noalloc::kBytes];

namespace b2r::noalloc {
namespace {

using dev::dtt;
using dev::kFull;

// the arrays of the scratch
struct arrays {
  int* rt;
  int* best;
  int* tmp;
  uint32_t* X;  // [2][kMaxLoc]
  uint32_t* Y;
  uint32_t* R;
  int16_t* out;
  uint32_t* any;
  __device__ explicit arrays(uint8_t* p)
      : rt{reinterpret_cast<int*>(p + kRtOff)}, best{reinterpret_cast<int*>(p + kBestOff)},
        tmp{reinterpret_cast<int*>(p + kTmpOff)}, X{reinterpret_cast<uint32_t*>(p + kXOff)},
        Y{reinterpret_cast<uint32_t*>(p + kYOff)}, R{reinterpret_cast<uint32_t*>(p + kROff)},
        out{reinterpret_cast<int16_t*>(p + kOutOff)}, any{reinterpret_cast<uint32_t*>(p + kAnyOff)} {}
};

// timetable::root (timetable.h:62-76) on the device image
__device__ uint32_t root_of(dtt const& T, uint32_t idx) {
  if (T.parent == nullptr) return idx;
  auto l = idx;
  for (auto i = 0;; ++i) {
    auto const par = T.parent[l];
    if (par == B2R_INVALID_IDX) break;
    if (par == idx || i > 20) {
      l = T.parent[idx];
      break;
    }
    l = par;
  }
  return l;
}

template <typename Fn>
__device__ void kids(dtt const& T, uint32_t l, Fn&& fn) {
  if (T.children_idx == nullptr) return;
  for (auto i = T.children_idx[l]; i != T.children_idx[l + 1]; ++i) fn(T.children[i]);
}

// for_each_meta (for_each_meta.h:8-45; the image has no equivalence lists)
template <typename Fn>
__device__ void metas(dtt const& T, uint8_t mode, uint32_t l, Fn&& fn) {
  switch (mode) {
    case B2R_MATCH_EXACT: fn(l); break;
    case B2R_MATCH_INTERMODAL:
      fn(l);
      kids(T, l, [&](uint32_t c) {
        if (T.loc_type != nullptr && T.loc_type[c] == B2R_LOC_GENERATED_TRACK) fn(c);
      });
      break;
    case B2R_MATCH_ONLY_CHILDREN:
      fn(l);
      kids(T, l, [&](uint32_t c) {
        fn(c);
        kids(T, c, fn);
      });
      break;
    default: {
      auto const r = root_of(T, l);
      fn(r);
      kids(T, r, [&](uint32_t c) {
        fn(c);
        kids(T, c, fn);
      });
    }
  }
}

// Labels that other blocks lower meanwhile are read through L2.
__device__ __forceinline__ int ldk(int const* p) { return __ldcg(p); }

// ---------------------------------------------------------------- phases
// Each phase is run by `n` threads (or warps), this one being number `i`.

// labels invalid, marks zero
__device__ void clear(arrays const& a, uint32_t nl, uint32_t nr, uint32_t rows, uint32_t i, uint32_t n) {
  for (auto k = 0u; k != rows; ++k) {
    for (auto l = i; l < nl; l += n) a.rt[k * kMaxLoc + l] = kInv;
  }
  for (auto l = i; l < nl; l += n) {
    a.best[l] = kInv;
    a.tmp[l] = kInv;
    a.X[l] = 0u;
    a.X[kMaxLoc + l] = 0u;
    a.Y[l] = 0u;
  }
  for (auto r = i; r < nr; r += n) a.R[r] = 0u;
  if (i < kRows) a.any[i] = 0u;
}

// starts in the order of the offsets (one_to_all.cc:30-39, add_start
// raptor.h:190-203): round 0 and best, station marked.  One thread.
__device__ void start(dtt const& T, params const& P, arrays const& a) {
  auto const fwd = P.fwd != 0;
  for (auto i = 0u; i != P.n_off; ++i) {
    auto const o = P.off[i];
    auto const t = fwd ? P.start_time + o.duration : P.start_time - o.duration;
    auto const key = dev::to_key(fwd, dev::clamp16(t - P.base_days * 1440));
    metas(T, P.mode, o.target, [&](uint32_t l) {
      if (key < ldk(&a.best[l])) a.best[l] = key;
      if (key < ldk(&a.rt[l])) a.rt[l] = key;
      a.X[l] = 1u;
    });
  }
}

// stations marked in round k - 1 mark their routes (raptor.h:228-241)
__device__ void mark_routes(dtt const& T, arrays const& a, uint32_t k, uint32_t i, uint32_t n) {
  auto const* X = a.X + ((k - 1u) & 1u) * kMaxLoc;
  for (auto l = i; l < T.n_loc; l += n) {
    if (X[l] == 0u) continue;
    auto const b = T.loc_routes_idx[l], e = T.loc_routes_idx[l + 1];
    if (b != e) a.any[k] = 1u;
    for (auto ri = b; ri != e; ++ri) a.R[T.loc_routes[ri]] = 1u;
  }
}

// the arrival-side label update of one stop (raptor.h:1242-1302)
__device__ __forceinline__ void arrive(arrays const& a, int tad, uint32_t l, int by) {
  if (by > tad) return;
  if (by < ldk(&a.tmp[l])) atomicMin(&a.tmp[l], by);
  a.Y[l] = 1u;
}

// The reference's sequential walk of a route whose trips keep no one order
// (raptor.h:1177-1349).  One lane.
__device__ void walk_route(dtt const& T, params const& P, arrays const& a, dev::route_rec const& R, uint32_t sec,
                           uint32_t k) {
  auto const* X = a.X + ((k - 1u) & 1u) * kMaxLoc;
  auto const fwd = P.fwd != 0;
  auto const wc = P.prf == B2R_PROFILE_WHEELCHAIR ? 1u : 0u;  // one_to_all.cc:69
  auto const* colbase = T.st + R.st;
  bool et_valid = false;
  uint32_t et_off = 0, n_ev = 0, n_days = 0;
  uint16_t et_day = 0;
  for (auto i = 0u; i != R.n; ++i) {
    auto const si = fwd ? i : R.n - 1u - i;
    auto const stp = T.route_stops[R.sb + si];
    auto const l = B2R_STOP_LOC(stp);
    auto const can_finish = fwd ? dev::stop_out_bit(stp, wc) : dev::stop_in_bit(stp, wc);
    auto const can_start = fwd ? dev::stop_in_bit(stp, wc) : dev::stop_out_bit(stp, wc);
    if (sec != 0u && i != 0u && !dev::section_ok(T, R.sb, fwd ? i - 1u : si, sec)) et_valid = false;
    bool arrival_ran = false;
    if (et_valid && can_finish) {
      arrival_ran = true;
      auto const ev = colbase[R.n_t * (si * 2u - (fwd ? 1u : 0u)) + et_off];
      arrive(a, P.tad, l, dev::to_delta_key(fwd, et_day, P.base, dev::delta_count(ev)));
    }
    if (i + 1u == R.n || !can_start || X[l] == 0u) continue;
    auto const board_col = R.n_t * (si * 2u - (fwd ? 0u : 1u));
    auto const et_time =
        et_valid ? dev::to_delta_key(fwd, et_day, P.base, dev::delta_count(colbase[board_col + et_off])) : kInv;
    auto const prt = ldk(&a.rt[(k - 1u) * kMaxLoc + l]);
    if (prt == kInv || prt > et_time) continue;
    auto const minutes = static_cast<int>(P.base) * 1440 + dev::from_key(fwd, prt);
    uint32_t nt = 0;
    uint16_t nd = 0;
    if (!dev::et_search(T, fwd, R, si, static_cast<uint16_t>(minutes / 1440), minutes % 1440, 0, P.tad, P.base, nt, nd,
                        n_ev, n_days)) {
      continue;
    }
    // current_best (raptor.h:1328-1329) is valid whenever the arrival part
    // ran or the station carries a label
    auto const cb_valid = arrival_ran || ldk(&a.best[l]) != kInv || ldk(&a.tmp[l]) != kInv;
    if (!cb_valid || dev::to_delta_key(fwd, nd, P.base, dev::delta_count(colbase[board_col + nt])) <= et_time) {
      et_valid = true;
      et_off = nt;
      et_day = nd;
    }
  }
}

// update_route (raptor.h:1177-1349), a warp per marked route, the lanes over
// its stops: every marked boardable stop searches its earliest trip, and on
// a route whose trips keep one order at every event (kRouteOrder) the trip a
// stop is reached by is the prefix minimum of the candidates before it, from
// the last section on that lacks a required flag.
__device__ void scan_routes(dtt const& T, params const& P, arrays const& a, uint32_t k, uint32_t lane, uint32_t i,
                            uint32_t n) {
  constexpr uint32_t kNone = 0xFFFFFFFFu;
  auto const* X = a.X + ((k - 1u) & 1u) * kMaxLoc;
  auto const fwd = P.fwd != 0;
  auto const wc = P.prf == B2R_PROFILE_WHEELCHAIR ? 1u : 0u;
  for (auto r = i; r < T.n_routes; r += n) {
    if (a.R[r] == 0u) continue;
    __syncwarp();
    if (lane == 0u) a.R[r] = 0u;
    auto const R = dev::load_route(T, r);
    uint32_t sec = 0u;  // required flags checked per section
    if ((P.claszes != 0xFFFFu || P.req != 0u) && !dev::filter_allowed(R.filter, P.claszes, P.req, sec)) continue;
    if ((R.flags & dev::kRouteOrder) == 0u) {
      if (lane == 0u) walk_route(T, P, a, R, sec, k);
      __syncwarp();
      continue;
    }
    uint32_t c_key = kNone, c_off = 0, c_day = 0;  // the trip carried into the chunk
    for (auto i0 = 0u; i0 < R.n; i0 += 32u) {
      auto const p = i0 + lane;
      auto const act = p < R.n;
      auto const si = fwd ? p : R.n - 1u - p;
      uint32_t l = 0, nt = 0, key = kNone;
      uint16_t nd = 0;
      bool finish = false, cut = false;
      if (act) {
        auto const stp = __ldg(T.route_stops + R.sb + si);
        l = B2R_STOP_LOC(stp);
        finish = (fwd ? dev::stop_out_bit(stp, wc) : dev::stop_in_bit(stp, wc)) != 0u;
        cut = sec != 0u && p != 0u && !dev::section_ok(T, R.sb, fwd ? p - 1u : si, sec);
        auto const board = p + 1u != R.n && (fwd ? dev::stop_in_bit(stp, wc) : dev::stop_out_bit(stp, wc)) != 0u;
        if (board && X[l] != 0u) {
          auto const prt = ldk(&a.rt[(k - 1u) * kMaxLoc + l]);
          auto const minutes = static_cast<int>(P.base) * 1440 + dev::from_key(fwd, prt);
          uint32_t n_ev = 0, n_days = 0;
          if (prt <= P.tad && prt != kInv &&
              dev::et_search(T, fwd, R, si, static_cast<uint16_t>(minutes / 1440), minutes % 1440, 0, P.tad, P.base, nt,
                             nd, n_ev, n_days)) {
            if ((R.flags & dev::kRouteOffsetOrder) != 0u) {  // the order key of the batched scan
              auto const x = static_cast<uint32_t>(static_cast<int>(nd) - static_cast<int>(P.base) + 64) * R.n_t + nt;
              key = fwd ? x : (1u << 21) - 1u - x;
            } else {
              auto const t =
                  (static_cast<int>(nd) - static_cast<int>(P.base)) * 1440 + dev::delta_count(__ldg(T.st + R.st + nt));
              key = static_cast<uint32_t>((fwd ? t : -t) + (1 << 20));
            }
          }
        }
      }
      auto const cuts = __ballot_sync(kFull, cut);
      if (__ballot_sync(kFull, key != kNone) == 0u && c_key == kNone) continue;
      auto v = key != kNone ? (key << 5) | lane : kNone;
      for (auto o = 1u; o < 32u; o <<= 1) {
        auto const y = __shfl_up_sync(kFull, v, o);
        if (lane >= o && ((cuts >> (lane + 1u - o)) & ((1u << o) - 1u)) == 0u) v = min(v, y);
      }
      auto const up = __shfl_up_sync(kFull, v, 1);
      auto const ex = lane == 0u || cut ? kNone : up;
      auto const x_off = __shfl_sync(kFull, nt, static_cast<int>(ex & 31u));
      auto const x_day = __shfl_sync(kFull, static_cast<uint32_t>(nd), static_cast<int>(ex & 31u));
      auto const carried = c_key != kNone && (cuts & ((2u << lane) - 1u)) == 0u;
      auto const use_x = ex != kNone && (!carried || (ex >> 5) <= c_key);
      if (act && finish && (use_x || carried)) {
        auto const off = use_x ? x_off : c_off;
        auto const day = static_cast<uint16_t>(use_x ? x_day : c_day);
        auto const ev = __ldg(T.st + (R.st + R.n_t * (si * 2u - (fwd ? 1u : 0u)) + off));
        arrive(a, P.tad, l, dev::to_delta_key(fwd, day, P.base, dev::delta_count(ev)));
      }
      auto const last = __shfl_sync(kFull, v, 31);
      auto const l_off = __shfl_sync(kFull, nt, static_cast<int>(last & 31u));
      auto const l_day = __shfl_sync(kFull, static_cast<uint32_t>(nd), static_cast<int>(last & 31u));
      if (cuts != 0u) c_key = kNone;
      if (last != kNone && (c_key == kNone || (last >> 5) <= c_key)) {
        c_key = last >> 5;
        c_off = l_off;
        c_day = l_day;
      }
    }
  }
}

// update_transfers and update_footpaths (raptor.h:680-845), a thread per
// station: the labels end at the minimum of the candidates whatever order
// they come in.  The marks the round has read are cleared on the way.
__device__ void relax(dtt const& T, params const& P, arrays const& a, uint32_t k, uint32_t i, uint32_t n) {
  auto const fwd = P.fwd != 0;
  auto* Xp = a.X + ((k - 1u) & 1u) * kMaxLoc;
  auto* X = a.X + (k & 1u) * kMaxLoc;
  auto const* idx = dev::fp_index(T, P.prf, fwd);
  auto const* dat = dev::fp_words(T, P.prf, fwd);
  auto const label = [&](uint32_t l, int key) {
    if (key >= ldk(&a.best[l])) return;
    atomicMin(&a.rt[k * kMaxLoc + l], key);
    if (key > P.tad) return;
    atomicMin(&a.best[l], key);
    X[l] = 1u;
  };
  for (auto l = i; l < T.n_loc; l += n) {
    Xp[l] = 0u;
    if (a.Y[l] == 0u) continue;
    a.Y[l] = 0u;
    auto const tk = ldk(&a.tmp[l]);
    if (tk == kInv) continue;
    label(l, dev::key_add(tk, dev::adjusted<int>(P.tts, static_cast<int>(T.transfer_time[l]))));
    for (auto j = idx[l], e = idx[l + 1]; j != e; ++j) {
      auto const w = dat[j];
      label(B2R_FP_TARGET(w), dev::key_add(tk, dev::adjusted<int>(P.tts, static_cast<int>(B2R_FP_DURATION(w)))));
    }
  }
}

// rows as deltas (kInvalidDelta<Dir> where unreached)
__device__ void rows_out(arrays const& a, uint32_t nl, uint32_t rows, bool fwd, uint32_t i, uint32_t n) {
  for (auto k = 0u; k != rows; ++k) {
    for (auto l = i; l < nl; l += n) {
      a.out[static_cast<size_t>(k) * nl + l] = static_cast<int16_t>(dev::from_key(fwd, ldk(&a.rt[k * kMaxLoc + l])));
    }
  }
}

// ---------------------------------------------------------------- kernels
__device__ __forceinline__ uint32_t grid_i() { return blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ uint32_t grid_n() { return gridDim.x * blockDim.x; }
__global__ void k_clear(dtt T, uint32_t rows, uint8_t* scratch) {
  clear(arrays{scratch}, T.n_loc, T.n_routes, rows, grid_i(), grid_n());
}
__global__ void k_start(dtt T, params P, uint8_t* scratch) {
  if (grid_i() == 0u) start(T, P, arrays{scratch});
}
__global__ void k_mark_routes(dtt T, uint8_t* scratch, uint32_t k) {
  mark_routes(T, arrays{scratch}, k, grid_i(), grid_n());
}
__global__ void __launch_bounds__(256) k_scan_routes(const __grid_constant__ dtt T, const __grid_constant__ params P,
                                                     uint8_t* scratch, uint32_t k) {
  arrays const a{scratch};
  if (a.any[k] == 0u) return;  // raptor.h:243-246
  scan_routes(T, P, a, k, threadIdx.x & 31u, grid_i() >> 5, grid_n() >> 5);
}
__global__ void k_relax_stations(const __grid_constant__ dtt T, const __grid_constant__ params P, uint8_t* scratch,
                                 uint32_t k) {
  arrays const a{scratch};
  if (a.any[k] == 0u) return;
  relax(T, P, a, k, grid_i(), grid_n());
}
__global__ void k_rows_out(dtt T, uint32_t rows, uint8_t fwd, uint8_t* scratch) {
  rows_out(arrays{scratch}, T.n_loc, rows, fwd != 0, grid_i(), grid_n());
}

cudaError_t search(b2r_timetable const& tt, params const& P, uint8_t* scratch, cudaStream_t s) {
  auto const& T = tt.d;
  auto const rows = static_cast<uint32_t>(P.end_k);
  auto const per_station = std::max(1u, (T.n_loc + 127u) / 128u);
  auto const per_route = std::max(1u, (T.n_routes + 7u) / 8u);  // a warp each
  k_clear<<<per_station, 128, 0, s>>>(T, rows, scratch);
  k_start<<<1, 32, 0, s>>>(T, P, scratch);
  for (uint32_t k = 1; k < rows; ++k) {
    k_mark_routes<<<per_station, 128, 0, s>>>(T, scratch, k);
    k_scan_routes<<<per_route, 256, 0, s>>>(T, P, scratch, k);
    k_relax_stations<<<per_station, 128, 0, s>>>(T, P, scratch, k);
  }
  k_rows_out<<<per_station, 128, 0, s>>>(T, rows, P.fwd, scratch);
  return cudaGetLastError();
}

// scratch address per device, looked up once with the device current
constexpr int kMaxDevices = 64;
std::mutex g_setup_mutex;
void* g_scratch[kMaxDevices] = {};

int scratch_on(int device, void** out) {
  std::lock_guard<std::mutex> lock{g_setup_mutex};
  if (g_scratch[device] == nullptr) {
    void* p = nullptr;
    auto const e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) {
      char msg[160];
      std::snprintf(msg, sizeof(msg), "b2r_one_to_all_noalloc: scratch address on device %d: %s",
                    device, cudaGetErrorString(e));
      return fail(B2R_ERR_CUDA, msg);
    }
    g_scratch[device] = p;
  }
  *out = g_scratch[device];
  return B2R_OK;
}

int run(b2r_timetable const* tt, b2r_query const* q, int16_t* round_times, uint64_t capacity,
        uint32_t* n_rows, int32_t* base_day, cudaStream_t stream) {
  char msg[192];
  if (tt == nullptr || q == nullptr || round_times == nullptr || n_rows == nullptr) {
    return fail(B2R_ERR_INVALID_ARGUMENT, "b2r_one_to_all_noalloc: null argument");
  }
  if (q->kind != B2R_ONE_TO_ALL || q->direction > B2R_BACKWARD ||
      q->start_match_mode > B2R_MATCH_INTERMODAL || (q->n_start != 0 && q->start == nullptr)) {
    return fail(B2R_ERR_INVALID_ARGUMENT,
                "b2r_one_to_all_noalloc: needs a one-to-all query with a valid direction, "
                "match mode and start offsets");
  }
  auto const nl = tt->d.n_loc, nr = tt->d.n_routes;
  if (nl > kMaxLoc || nr > kMaxRoutes) {
    std::snprintf(msg, sizeof(msg),
                  "b2r_one_to_all_noalloc: timetable has %u locations and %u routes; the "
                  "scratch array holds at most %u and %u",
                  nl, nr, kMaxLoc, kMaxRoutes);
    return fail(B2R_ERR_CAPACITY, msg);
  }
  if (q->n_start > B2R_NOALLOC_MAX_OFFSETS) {
    std::snprintf(msg, sizeof(msg),
                  "b2r_one_to_all_noalloc: query has %u start offsets; at most %u are supported",
                  q->n_start, B2R_NOALLOC_MAX_OFFSETS);
    return fail(B2R_ERR_CAPACITY, msg);
  }
  auto const end_k = static_cast<uint32_t>(std::min<int>(q->max_transfers, B2R_MAX_TRANSFERS) + 2);
  auto const need = static_cast<uint64_t>(end_k) * nl;
  if (capacity < need) {
    std::snprintf(msg, sizeof(msg),
                  "b2r_one_to_all_noalloc: round_times holds %llu values; %u rows of %u "
                  "locations need %llu",
                  static_cast<unsigned long long>(capacity), end_k, nl,
                  static_cast<unsigned long long>(need));
    return fail(B2R_ERR_CAPACITY, msg);
  }
  params P{};
  for (auto i = 0u; i != q->n_start; ++i) {
    if (q->start[i].target >= nl) {
      return fail(B2R_ERR_INVALID_ARGUMENT, "b2r_one_to_all_noalloc: start offset target out of range");
    }
    P.off[i] = q->start[i];
  }
  // one_to_all.cc:18-24 (make_base) and 44-46 (worst time at destination)
  auto const fwd = q->direction == B2R_FORWARD;
  P.n_off = q->n_start;
  P.fwd = fwd ? 1 : 0;
  P.mode = q->start_match_mode;
  P.end_k = static_cast<uint8_t>(end_k);
  P.start_time = q->start_time;
  P.base = static_cast<uint16_t>(round_to_days(q->start_time) - tt->d.internal_from_days);
  P.base_days = tt->d.internal_from_days + P.base;
  P.tts = {q->tts_default, q->tts_min_transfer_time, q->tts_additional_time, q->tts_factor};
  P.claszes = static_cast<uint16_t>(q->allowed_claszes & 0xFFFFu);
  if (q->prf_idx >= B2R_N_PROFILES) return fail(B2R_ERR_INVALID_ARGUMENT, "b2r_one_to_all_noalloc: prf_idx out of range");
  P.prf = q->prf_idx;
  P.req = static_cast<uint8_t>((q->require_bike_transport != 0 ? 1u << B2R_FLAG_BIKES : 0u) |
                               (q->require_car_transport != 0 ? 1u << B2R_FLAG_CARS : 0u) |
                               (q->prf_idx == B2R_PROFILE_WHEELCHAIR ? 1u << B2R_FLAG_WHEELCHAIR : 0u) |
                               (q->no_compulsory_reservation != 0 ? 1u << B2R_FLAG_RESERVATION_NOT_REQUIRED : 0u));
  auto const span = static_cast<int>(q->max_travel_time);
  auto const worst = std::clamp(q->start_time + (fwd ? span : -span) - P.base_days * 1440, -32768, 32767);
  P.tad = std::min(dev::kKeyInv, fwd ? worst : ~worst);

  int prev = 0;
  auto e = cudaGetDevice(&prev);
  if (e == cudaSuccess && prev != tt->device) e = cudaSetDevice(tt->device);
  if (e != cudaSuccess) {
    std::snprintf(msg, sizeof(msg), "b2r_one_to_all_noalloc: device %d: %s", tt->device,
                  cudaGetErrorString(e));
    return fail(B2R_ERR_CUDA, msg);
  }
  int status = B2R_OK;
  void* scratch = nullptr;
  if (tt->device < 0 || tt->device >= kMaxDevices) {
    status = fail(B2R_ERR_UNSUPPORTED, "b2r_one_to_all_noalloc: device index beyond 63");
  } else {
    status = scratch_on(tt->device, &scratch);
  }
  if (status == B2R_OK) {
    auto* base = static_cast<uint8_t*>(scratch);
    e = search(*tt, P, base, stream);
    if (e == cudaSuccess) {
      e = cudaMemcpyAsync(round_times, base + kOutOff, need * sizeof(int16_t), cudaMemcpyDeviceToHost,
                          stream);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) {
      std::snprintf(msg, sizeof(msg), "b2r_one_to_all_noalloc: %s", cudaGetErrorString(e));
      status = fail(B2R_ERR_CUDA, msg);
    } else {
      *n_rows = end_k;
      if (base_day != nullptr) *base_day = P.base_days;
    }
  }
  if (prev != tt->device) cudaSetDevice(prev);
  return status;
}

}  // namespace
}  // namespace b2r::noalloc

extern "C" int b2r_one_to_all_noalloc(const b2r_timetable* tt, const b2r_query* q, int16_t* round_times,
                                      uint64_t capacity, uint32_t* n_rows, int32_t* base_day,
                                      void* stream) {
  B2R_API_GUARD({
    return b2r::noalloc::run(tt, q, round_times, capacity, n_rows, base_day,
                             static_cast<cudaStream_t>(stream));
  });
}
