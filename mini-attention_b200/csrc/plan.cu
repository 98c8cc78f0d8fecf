// Host-side planner of balanced launches.
//
// The forward kernel runs one CTA per SM, so a launch of n work items (pairs of Q tiles of one
// (batch, head)) takes ceil(n / SMs) rounds when the items are equally heavy, and the last round
// may leave most SMs idle (256 items on 148 SMs: 2 rounds for 1.73 rounds of work).  The planner
// cuts the K/V range of some items into pieces that separate CTAs work on, so that every SM ends
// at about the same time; the CTAs of a cut item leave un-normalised partial results in scratch
// memory and the last one to arrive merges them (fwd_ws.cu).  The reference launches one CTA per
// (batch, head, Q block) and leaves the balance to the hardware scheduler
// (kernels/flash_attn/cuda/sm_120/kernel/flash_attention.cu:100-123).
//
// Model: a CTA covering s K/V tiles costs s + h steps (h = fixed cost of a CTA: set-up, first
// loads, epilogue); the hardware hands CTAs to SMs in index order as SMs become free.  Plan:
// walk the items heaviest first and give each to the least-loaded SM while it fits under the
// target time T; from the first item that does not fit, fill the SMs one after the other up to T,
// cutting an item where an SM's room ends and continuing it on the next SM (McNaughton's
// wrap-around rule, with a minimum piece length).  The resulting CTAs are launched
// longest first.  The plan is used only when its predicted makespan beats the plain launch.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <queue>
#include <utility>
#include <vector>

#include "common.cuh"

namespace ma {

namespace {

struct Piece {
  int item, t0, t1, part, nparts;
  int round;  // how many pieces the plan put on the same SM before this one (phase 2)
};

using SmLoad = std::pair<float, int>;  // (busy until, SM)
using MinHeap = std::priority_queue<SmLoad, std::vector<SmLoad>, std::greater<SmLoad>>;

MinHeap empty_sms(int sms) {
  std::vector<SmLoad> v;
  v.reserve(sms);
  for (int s = 0; s < sms; ++s) v.emplace_back(0.f, s);
  return MinHeap(std::greater<SmLoad>(), std::move(v));
}

// Makespan of CTAs with the given costs, handed out in order to the first free SM; `finish`
// (optional) receives the time each CTA ends.
float list_schedule(const std::vector<float>& cost, int sms, std::vector<float>* finish = nullptr) {
  MinHeap heap = empty_sms(sms);
  float end = 0.f;
  if (finish) finish->resize(cost.size());
  for (size_t i = 0; i < cost.size(); ++i) {
    SmLoad s = heap.top();
    heap.pop();
    s.first += cost[i];
    if (finish) (*finish)[i] = s.first;
    end = std::max(end, s.first);
    heap.push(s);
  }
  return end;
}

// K/V tiles; shorter pieces cost more than they balance.  A cut costs the same whatever the launch, so one
// that is short overall is better off with idle SMs (4-tile pieces: N = 1024, 2 x 8 heads 18.4 us against 15.3
// uncut; 777 against 3333 keys, 2 x 24/8 heads, 65.2 against 66.9 with 6-tile pieces; N = 4096 116.9 / 117.9).
int min_piece(float plain_steps) { return plain_steps >= 24.f ? 4 : 6; }
constexpr int kMaxParts = 64;      // pieces per item

// Cost model, in steps (one K/V tile of a two-Q-tile CTA, about 1.6 us at D = 128): fixed cost of
// a CTA, and what a piece of a cut item adds on average (publishing its partial takes about 0.6
// steps; the last piece to arrive also reads the others', about 2 steps).  The constants are from when a step took 2 us
// and have not been measured anew since.
float cta_cost(int D) { return D == 128 ? 2.0f : 3.0f; }
float grade_frac() { return 0.015f; }  // spread of the per-SM targets, as a fraction of T
float piece_cost() { return 1.3f; }

// Fill under the target time T.  Phase 1: items go whole to the least-loaded SM while they fit.
// Phase 2, from the first item that does not: the SMs are filled one after the other up to T
// (most room first); an item that crosses the end of an SM's room is cut there and continues on
// the next SM.  Returns false when an item would need too many pieces.
bool fill(const std::vector<int>& w, int sms, float T, float h, float fee, int least, std::vector<Piece>* out) {
  out->clear();
  const int n = static_cast<int>(w.size());
  MinHeap heap = empty_sms(sms);
  int i = 0;
  for (; i < n; ++i) {
    SmLoad s = heap.top();
    if (s.first + w[i] + h > T) break;
    heap.pop();
    out->push_back(Piece{i, 0, w[i], 0, 1, 0});
    s.first += w[i] + h;
    heap.push(s);
  }
  std::vector<float> load;
  load.reserve(sms);
  while (!heap.empty()) {
    load.push_back(heap.top().first);  // ascending: most room first
    heap.pop();
  }
  std::vector<int> placed(sms, 0);
  const float grade = grade_frac() * T;
  int si = 0;
  for (; i < n; ++i) {
    int t0 = 0;
    const size_t first = out->size();
    do {
      const int rem = w[i] - t0;
      int take, round;
      if (si >= sms) {
        // no SM has room left under T: the rest goes, in one piece, to the least-loaded SM
        const int s = static_cast<int>(std::min_element(load.begin(), load.end()) - load.begin());
        take = rem;
        load[s] += take + h + (t0 > 0 ? fee : 0.f);
        round = placed[s]++;
      } else {
        take = rem;
        // SMs do not run identical CTAs at identical speed (a few per cent apart), and CTAs are
        // handed out longest first to whichever SM is free first.  Grading the targets, more for
        // the SMs filled first, gives the SMs that come free early the longer pieces.
        const float Ts = T + grade * (1.f - 2.f * si / std::max(1, sms - 1));
        const bool whole_fits = (t0 == 0) && (load[si] + rem + h <= Ts);
        if (!whole_fits) {  // a piece of a cut item: it also pays the fee
          const int room = static_cast<int>(std::floor(Ts - load[si] - h - fee));
          if (room < rem) {
            if (room < least) {
              ++si;  // nothing useful fits here any more
              continue;
            }
            // both sides of a cut at least `least` long; a rest too short to cut stays whole
            // (and overruns this SM's target by less than that)
            if (rem >= 2 * least) take = std::min(room, rem - least);
          }
        }
        load[si] += take + h + (whole_fits ? 0.f : fee);
        round = placed[si]++;
        if (Ts - load[si] - h - fee < least) ++si;
      }
      out->push_back(Piece{i, t0, t0 + take, 0, 0, round});
      t0 += take;
    } while (t0 < w[i]);
    const int np = static_cast<int>(out->size() - first);
    if (np > kMaxParts) return false;
    for (int k = 0; k < np; ++k) {
      (*out)[first + k].part = k;
      (*out)[first + k].nparts = np;
    }
  }
  return true;
}

}  // namespace

// Many rounds balance themselves; the table holds every CTA from the first cut item on.
bool plan_considered(const FwdArgs& a, int sms) {
  const long long n_items = static_cast<long long>((a.n_q_tiles + 1) / 2) * a.Hq * a.B;
  return sms > 0 && n_items > 0 && n_items <= 16ll * sms && n_items <= 4096;
}

// Items in launch order (item_to_pair_bh): latest rows first within each group of heads.
void plan_fwd(const FwdArgs& a, int D, int sms, FwdPlan* plan) {
  plan->split = false;
  plan->n_whole = plan->n_table = plan->n_slots = plan->n_cut_items = 0;
  plan->est_plain = plan->est_balanced = 0.f;
  if (!plan_considered(a, sms)) return;
  const long long n_pairs = (a.n_q_tiles + 1) / 2;
  const int n = static_cast<int>(n_pairs * a.Hq * a.B);
  const float h = cta_cost(D);
  const float fee = piece_cost();

  std::vector<int> w(n);
  long long total = 0;
  for (int i = 0; i < n; ++i) {
    int pair, bh_i;
    item_to_pair_bh(a, static_cast<int>(n_pairs), i, &pair, &bh_i);
    const int q0 = pair * 2 * a.tpt;
    const int nt = (q0 + a.tpt < a.Nq) ? 2 : 1;
    w[i] = kv_tiles_of(a, q0, nt);
    if (w[i] > 65535) return;  // tile ranges travel as 16-bit numbers
    total += w[i];
  }
  std::vector<float> cost(n);
  for (int i = 0; i < n; ++i) cost[i] = w[i] + h;
  const float plain = list_schedule(cost, sms);
  plan->est_plain = plain;
  const float bound = (static_cast<float>(total) + h * n) / sms;
  if (plain <= 1.03f * bound) return;

  const int least = min_piece(plain);
  std::vector<Piece> best, cur;
  float best_t = plain;
  int best_whole = 0;
  // Targets tried: ten fine steps above the bound (several rounds of items: the answer is close
  // to it), then eight coarse ones up to about half the heaviest item (few, long items).
  const int w_max = *std::max_element(w.begin(), w.end());
  const float fine = std::max(0.5f, 0.004f * bound), coarse = std::max(fine, w_max / 16.f);
  for (int attempt = 0; attempt < 18; ++attempt) {
    const float up = attempt < 10 ? fine * attempt : fine * 9 + coarse * (attempt - 9);
    const float T = std::max(bound + 0.75f * (h + fee) + up, least + h + fee);
    if (!fill(w, sms, T, h, fee, least, &cur)) continue;
    int first_cut = n;
    for (const Piece& p : cur)
      if (p.nparts > 1) {
        first_cut = p.item;
        break;
      }
    if (first_cut == n) continue;  // nothing was cut
    // Launch order: the whole items before the first cut one, then everything else, either
    // longest first, or in the plan's rounds (first pieces of every SM, longest first, then the
    // second pieces, ...); whichever the dispatch model likes better.
    std::vector<Piece> tab;
    for (const Piece& p : cur)
      if (p.item >= first_cut) tab.push_back(p);
    if (static_cast<int>(tab.size()) > kPlanCap) continue;
    for (int order = 0; order < 2; ++order) {
      std::stable_sort(tab.begin(), tab.end(), [order](const Piece& x, const Piece& y) {
        if (order == 1 && x.round != y.round) return x.round < y.round;
        return (x.t1 - x.t0) > (y.t1 - y.t0);
      });
      // Every piece of a cut item publishes its partial; the one that ends last also merges.
      // Two passes: who ends last is read off a first schedule in which nobody pays the merge.
      const float fee_pub = 0.45f * fee, fee_last = 1.55f * fee;
      std::vector<float> c, fin;
      c.reserve(first_cut + tab.size());
      for (int i = 0; i < first_cut; ++i) c.push_back(w[i] + h);
      for (const Piece& p : tab) c.push_back((p.t1 - p.t0) + h + (p.nparts > 1 ? fee_pub : 0.f));
      list_schedule(c, sms, &fin);
      std::vector<int> last_of(n, -1);
      for (size_t k = 0; k < tab.size(); ++k) {
        const Piece& p = tab[k];
        if (p.nparts > 1 && (last_of[p.item] < 0 || fin[first_cut + k] > fin[first_cut + last_of[p.item]]))
          last_of[p.item] = static_cast<int>(k);
      }
      for (size_t k = 0; k < tab.size(); ++k)
        if (tab[k].nparts > 1 && last_of[tab[k].item] == static_cast<int>(k)) c[first_cut + k] += fee_last - fee_pub;
      const float t = list_schedule(c, sms);
      if (t < best_t) {
        best_t = t;
        best_whole = first_cut;
        best = tab;
      }
    }
  }
  plan->est_balanced = best_t;
  if (best.empty() || best_t > 0.97f * plain) return;

  // slots and counters: cut items in item order, pieces of an item on consecutive slots
  std::vector<int> slot0(n, -1), counter(n, -1);
  {
    std::vector<int> nparts(n, 0);
    for (const Piece& p : best) nparts[p.item] = p.nparts;
    int slots = 0, cuts = 0;
    for (int i = best_whole; i < n; ++i)
      if (nparts[i] > 1) {
        slot0[i] = slots;
        counter[i] = cuts++;
        slots += nparts[i];
      }
    if (slots > 65535) return;
    plan->n_slots = slots;
    plan->n_cut_items = cuts;
  }
  plan->split = true;
  plan->n_whole = best_whole;
  plan->n_table = static_cast<int>(best.size());
  for (int k = 0; k < plan->n_table; ++k) {
    const Piece& p = best[k];
    PlanEntry& e = plan->table.e[k];
    e.item = static_cast<uint32_t>(p.item);
    e.t0 = static_cast<uint16_t>(p.t0);
    e.t1 = static_cast<uint16_t>(p.t1);
    e.part = static_cast<uint8_t>(p.part);
    e.nparts = static_cast<uint8_t>(p.nparts);
    e.slot0 = static_cast<uint16_t>(p.nparts > 1 ? slot0[p.item] : 0);
    e.counter = static_cast<uint32_t>(p.nparts > 1 ? counter[p.item] : 0);
  }
}

// Calls with few query rows per KV head (fwd_decode.cu).  d->rg stays 0 where fwd_ws.cu is the faster one.
void plan_decode(int B, int Hq, int Hkv, int Nq, int Nk, int D, int causal, long long diag, int sms, bool cut,
                 DecodePlan* d) {
  *d = DecodePlan{};
  long long kv_end = Nk;
  if (causal) kv_end = std::min(kv_end, diag + Nq);
  const int G = Hq / Hkv;
  const long long rows = static_cast<long long>(G) * Nq;
  if (kv_end <= 0 || Nq > 64) return;
  const int rg = rows <= 16 ? 1 : rows <= 32 ? 2 : 4;
  const long long n_rb = (rows + 16 * rg - 1) / (16 * rg);
  const long long items = static_cast<long long>(B) * Hkv * n_rb;
  if (items > 0x3fffffffll) return;
  const int tiles = static_cast<int>((kv_end + 63) / 64);
  const long long total = items * tiles;
  const long long slots = 2ll * sms;  // two CTAs per SM
  // How the items are cut: pieces of at least four tiles, and no more of them than balances a tile's time against
  // what the CTA that folds them spends on each (in us: a round trip to L2 shared by eight, and the piece's rows at
  // what one SM reads).  An item of fewer than 12 tiles is left whole, of fewer than 10 where there are next to no
  // rows to fold: a cut costs 1 to 2 us (128 items of 8 tiles, D = 128: 16 rows 12.7 us cut in two, 10.6 whole, 1 row
  // 11.1 / 10.6; of 12 tiles 13.9 / 13.1 and 12.7 / 13.1; 36 items of 10 tiles, 1 row 10.5 / 11.3).
  const double t_tile = rg == 1 ? 0.5 : rg == 2 ? 0.8 : 1.5;
  const double t_fold = 0.02 + std::min<double>(rows, 16 * rg) * D * 4 / 55e3;
  const bool too_short = tiles < (rows <= 4 ? 10 : 12);
  const long long most =
      too_short ? 1 : std::max(1ll, std::min<long long>(tiles / 4, static_cast<long long>(std::sqrt(tiles * t_tile / t_fold))));
  // A CTA works on one item only wherever that leaves enough of them: one that ends a piece of one item and
  // begins the next pays for two ends (about 5 us of syncs, publishing and folding) and so does the launch.
  // 16 items of 563 tiles, D = 64: 39.3 us in 292 CTAs that straddle, 31.9 in 288 of one piece each, 30.0 in
  // 256; 128 items of 63 tiles, D = 128: 49.0 in 296, 46.6 in 256; 512 items of 16 tiles: 49.5 in 296, 46.0 in
  // 256 of two items each; 328 items of 2 tiles: 15.6 in 296, 11.9 in 328; 320 of 11 tiles, 32 rows: 33.5 in 296,
  // 37.1 in 320.  HBM is saturated by fewer CTAs than fit (208 to 272), and pieces cost; where the tiles are bound by
  // mma.sync (rg > 1) every slot counts: 400 items of 64 tiles, D = 64, 64 rows 138.8 in 200, 109.1 in 296.
  const long long room = rg == 1 ? slots * 7 / 8 : slots;
  long long n_ctas = items;
  if (cut && items <= room) {
    n_ctas = items * std::max(1ll, std::min(most, room / items));
  } else if (cut) {
    const long long enough = rg == 1 ? slots * 2 / 3 : slots * 9 / 10;
    long long j = (items + slots - 1) / slots;
    while (items % j != 0 && items / j >= enough) ++j;
    if (items / j >= enough) n_ctas = items / j;
    else if (tiles >= 10 || items >= 4 * slots) n_ctas = slots;
  }
  // Which kernel.  fwd_ws packs the query heads of a KV head into one Q tile (head_pack, api.cu), so that it too reads
  // K/V once; its tile of 128 rows takes 1.05 us for 128 keys whatever part of the rows is real, on one CTA per SM.
  // Measured on B200 (us, fwd_ws / this one, bf16, causal, the last Nq of Nk positions; balanced launches):
  //   up to 16 rows   two CTAs an SM, bound by HBM: 1 KV head, Nk=16384 45 / 18; 32 of 4096 keys 23 / 16; 128 of 2048
  //                   to 4096 within 5 % either way (27.4 / 28.2, 48.5 / 47.1), more items ahead (320 of 2048 69 / 58)
  //   17 to 32 rows   at D=64 ahead wherever an item is cut (72 of 2048 18.7 / 14.7, 128 of 1024 14.3 / 13.5) and whole
  //                   while it is short (512 keys 9.0 / 8.6, 16384 keys 137 / 143).  At D=128 a tile costs its warps
  //                   about what HBM takes to deliver it.  Ahead: more items than SMs (fwd_ws goes another round: 320 of
  //                   2048 71 / 67, of 512 whole 28 / 27); few items long enough to cut (1 of 4096 20.2 / 19.3, of 16384
  //                   45 / 30; 32 of 2048 20.3 / 19.3); more than half an SM each and long (128 of 8192 91.6 / 89.3).
  //                   Behind: 512 keys 9.4 / 12.3, 72 of 4096 34.5 / 35.6, 128 of 2048 27.9 / 32.4; all of them whole and
  //                   long (1 of 16384 167 / 229).  One query head (G=1): fwd_ws.
  //   more            bound by mma.sync, a block of 64 rows 1.5 us for 64 keys: behind where heads are packed (128 of
  //                   4096, D=128: 64 rows 49.6 / 80.7, 256 rows 64.7 / 260; 32 of 4096, D=64 24 / 44), but for one block
  //                   at D=64 in more items than SMs (320 of 1024 38.5 / 33.8, 192 of 300 16.4 / 12.3; 192 of 4096 whole
  //                   67 / 78), and level for one or two items of 20000 keys and more (1 of 40000: D=64 60 / 54, D=128
  //                   80 / 75; of 50000 50 / 57, 60 / 81).  More than 128 query heads to a KV head do not fit a Q
  //                   tile: ahead where there is work for every SM (192 heads, 4 of 1671 128 / 26).
  // A launch of one whole item per CTA needs no scratch, and a call without scratch can have no other: the line is the
  // same for both.
  const bool whole = n_ctas == items;
  if (rg == 2 && D == 64 && whole && items <= sms && tiles > 16) return;
  if (rg == 2 && D == 128) {
    const bool few = 4 * items <= sms, half = 2 * items > sms;
    if (G == 1) return;
    if (items <= sms && (whole || tiles < 16 || !(few || (half && tiles >= 128)))) return;
    if (items > slots && whole && !too_short) return;
  }
  if (rg == 4 && G <= kTileM && !(D == 64 && n_rb == 1 && items > sms && (tiles <= 16 || !whole))) return;
  if (rg == 4 && G > kTileM && (G < 2 * n_rb || G * total < 16 * slots)) return;
  d->rg = rg;
  d->n_rb = static_cast<int>(n_rb);
  d->tiles = tiles;
  d->total = total;
  d->n_ctas = static_cast<int>(n_ctas);
}

}  // namespace ma
