// Test-only host build of the device's Local_Alignment (csrc/align_warp.cuh),
// a call per warp on the lanes of warp_lanes.h, in any of its builds and with
// the table of shared extensions in host memory.  Requests and results as
// pga_local_alignment's.  Not part of the product library.
#include "warp_lanes.h"
#include "../../distributedpanga_b200/csrc/align_spec.h"
#include "../../distributedpanga_b200/csrc/align_warp.cuh"

using namespace pga::aln;

namespace pga {
namespace aln {
struct TaskChains {};
void scout_if_free(WarpWork &W) { W.task = nullptr; }
}  // namespace aln
}  // namespace pga

namespace {

// 2-bit copies as k_pack lays them out: forward, reversed, reverse complement, complement.
struct Packed {
  std::vector<uint32_t> w;
  int64_t nw;
  Packed(const uint8_t *s, int64_t n) : nw(2 * (n / 32 + 2)) {
    w.assign(4 * nw + 64, 0);
    for (int64_t i = 0; i < n; i++) {
      const uint32_t f = s[i], r = s[n - 1 - i], v[4] = {f, r, 3 - r, 3 - f};
      for (int c = 0; c < 4; c++) w[c * nw + (i >> 4)] |= v[c] << (30 - 2 * (i & 15));
    }
  }
};

struct Table {
  ShareTable X{};
  std::vector<unsigned long long> keys;
  std::vector<int> vals;
  std::vector<ShareEntry> entries;
  std::vector<ShareRec> recs;
  std::vector<uint32_t> list;
  unsigned counters[16] = {0};
  unsigned next_task = 0;
  unsigned long long nlist = 0;
  Table(int entry_cap, int rec_cap, int64_t list_cap)
      : keys(1 << 12), vals(1 << 12, -1), entries(entry_cap + 1), recs(rec_cap + 1), list(list_cap + 1) {
    X.keys = keys.data();
    X.vals = vals.data();
    X.mask = (1 << 12) - 1;
    X.entries = entries.data();
    X.recs = recs.data();
    X.list = list.data();
    X.entry_cap = entry_cap;
    X.rec_cap = rec_cap;
    X.list_cap = list_cap;
    X.nentry = counters;
    X.nrec = counters + 1;
    X.nlist = &nlist;
    X.joins = counters + 8;
    X.next_task = &next_task;
    X.ntasks = 1;
  }
};

}  // namespace

// seq: the contigs' bases (0..3) back to back, len: their lengths; req8: a b
// comp low hgh anti lbord hbord; path7: abpos aepos bbpos bepos diffs tlen err;
// trace: the results' trace values back to back (trace_cap of them at most).
// opt: {blocks, share, turns a call runs for before another may (0: to its
// end), the schedule's seed, entry_cap, rec_cap, list_cap, a call (not 0; -1:
// none) whose walk back fails: once it has waited for another extension that
// path crosses on another lane than it did, and the call's pebbles have lost
// their successors}.  A call has cells_each pebbles of its
// own, so that a pebble's number tells its call.  stat: {entries, records,
// entries by kind (none, head, pebble), pebbles named by an entry that are not
// from after its line, records by status (0 open, done, joined, failed)}.
extern "C" int warp_host(const uint8_t *seq, int ncontig, const int64_t *len, const float *freq, int64_t n,
                         const int32_t *req8, const int64_t *opt, int64_t cells_each, int32_t *path7, uint16_t *trace,
                         int64_t trace_cap, int64_t *stat) {
  AlignSpec spec;
  spec.trace_space = TSPACE;
  spec.reach = 0;
  spec.ave_path = align_params(freq, &spec.dscore);
  std::vector<Packed> pk;
  int64_t off = 0, maxctg = 0;
  for (int c = 0; c < ncontig; c++) {
    pk.emplace_back(seq + off, len[c]);
    off += len[c];
    maxctg = max(maxctg, len[c]);
  }
  Table share((int)opt[4], (int)opt[5], opt[6]);
  constexpr int VCAP = 8192;
  const int64_t room = 4 * (maxctg / TSPACE + 4) + 64;
  std::vector<Pebble> cells((size_t)(n * cells_each));
  struct Call {
    std::vector<int> wave = std::vector<int>(11 * VCAP);
    std::vector<uint16_t> points;
    unsigned long long next;
    alignas(16) int sm[128];
    Path P[32];
    int err[32];
    lanes::Warp w;
  };
  std::vector<std::unique_ptr<Call>> calls;
  for (int64_t i = 0; i < n; i++) {
    calls.emplace_back(new Call);
    Call &C = *calls.back();
    C.points.resize(room);
    C.next = (unsigned long long)(i * cells_each);
    C.w.body = [&, i] {
      const int32_t *q = req8 + 8 * i;
      const int lane = lanes::g_lane;
      Call &C = *calls[i];
      WarpWork W{};
      int *wb = (int *)(((uintptr_t)C.wave.data() + 15) & ~(uintptr_t)15);
      W.vcap = VCAP / 2;
      W.C[0] = (RingCell *)wb;
      W.C[1] = W.C[0] + W.vcap;
      W.V[0] = wb + 8 * W.vcap;
      W.V[1] = wb + 9 * W.vcap;
      W.NA = wb + 10 * W.vcap;
      W.points = C.points.data();
      W.point_cap = room;
      W.pool = PebblePool{cells.data(), &C.next, (i + 1) * cells_each};
      W.sm = C.sm;
      W.share = opt[1] ? &share.X : nullptr;
      W.pair = (unsigned)q[0] | (unsigned)q[1] << 15 | (unsigned)q[2] << 30;
      const Packed &a = pk[q[0]], &b = pk[q[1]];
      Seq A{nullptr, (int)len[q[0]]}, B{nullptr, (int)len[q[1]]};
      A.pf = a.w.data() + (q[2] ? 2 : 0) * a.nw;
      A.pr = a.w.data() + (q[2] ? 3 : 1) * a.nw;
      B.pf = b.w.data();
      B.pr = b.w.data() + b.nw;
      Path P{};
      int r;
      if (opt[0] && opt[1]) r = local_alignment_w<true, true>(W, spec, A, B, q[2] != 0, P, q[3], q[4], q[5], q[6], q[7]);
      else if (opt[0]) r = local_alignment_w<true, false>(W, spec, A, B, q[2] != 0, P, q[3], q[4], q[5], q[6], q[7]);
      else r = local_alignment_w<false, false>(W, spec, A, B, q[2] != 0, P, q[3], q[4], q[5], q[6], q[7]);
      C.P[lane] = P;
      C.err[lane] = r ? W.err | 0x100 : 0;
    };
  }
  bool cut = false;
  lanes::g_on_wake = [&] {
    const int64_t k = opt[7];
    if (cut || k < 0 || lanes::g_warp != &calls[k]->w) return;
    for (unsigned e = 0; e < share.counters[0]; e++) {
      ShareEntry &E = share.entries[e];
      if (E.mark / cells_each == k || E.kind != SHARE_PEBBLE || !share.recs[E.rec].status) continue;
      for (int l = 0, to = E.lane; l < 32; l++)
        if (E.HA[l] >= 0 && E.HA[l] != E.HA[to]) {
          E.lane = l;
          cut = true;
          break;
        }
    }
    if (cut)
      for (int64_t c = k * cells_each; c < (k + 1) * cells_each; c++) cells[c].ptr = min(cells[c].ptr, 0);
  };
  uint64_t rng = (uint64_t)opt[3] * 0x9e3779b97f4a7c15ull + 1;
  for (int64_t left = n, at = 0; left > 0;) {
    if (opt[2] > 0) {
      rng ^= rng << 13;
      rng ^= rng >> 7;
      rng ^= rng << 17;
      at = (int64_t)(rng % (uint64_t)n);
    }
    lanes::Warp &w = calls[at]->w;
    if (w.done) {
      at = (at + 1) % n;
      continue;
    }
    for (int64_t t = 0; !w.done && (opt[2] == 0 || t < opt[2]); t++) lanes::turn(w);
    if (w.done) left--;
  }
  lanes::g_on_wake = nullptr;
  int64_t nt = 0;
  for (int64_t i = 0; i < n; i++) {
    const Call &C = *calls[i];
    const Path &P = C.P[0];
    for (int l = 1; l < 32; l++)
      if (memcmp(&C.P[l], &P, sizeof(P)) != 0 || C.err[l] != C.err[0]) return 1;  // the lanes' results are one
    int32_t *o = path7 + 7 * i;
    o[0] = P.abpos; o[1] = P.aepos; o[2] = P.bbpos; o[3] = P.bepos; o[4] = P.diffs;
    o[5] = C.err[0] ? 0 : P.tlen;
    o[6] = C.err[0];
    if (nt + o[5] > trace_cap) return 2;
    memcpy(trace + nt, C.points.data() + P.trace_off, sizeof(uint16_t) * o[5]);
    nt += o[5];
  }
  for (int i = 0; i < 10; i++) stat[i] = 0;
  stat[0] = min((int64_t)share.counters[0], opt[4]);
  stat[1] = min((int64_t)share.counters[1], opt[5]);
  for (int64_t e = 0; e < stat[0]; e++) {
    const ShareEntry &E = share.entries[e];
    stat[2 + E.kind]++;
    if (E.kind != SHARE_PEBBLE) continue;
    bool found = false;
    for (int64_t c = E.mark; c < (E.mark / cells_each + 1) * cells_each; c++)
      found |= cells[c].diag == E.pdiag && cells[c].diff == E.pdiff && cells[c].mark == E.pmark;
    stat[5] += !found;
  }
  for (int64_t r = 0; r < stat[1]; r++) stat[6 + share.recs[r].status]++;
  return 0;
}
