// Test-only host build of the oracle's scalar Local_Alignment
// (oracle/scalar_align.cuh) on a list of requests over a contig set, in the
// request and result layout of pga_local_alignment.  Not part of the product
// library.
#include <cstdint>
#include <cstring>
#include <vector>
#include "../../distributedpanga_b200/csrc/align_core.cuh"
#include "../../distributedpanga_b200/csrc/align_spec.h"
#include "../../oracle/scalar_align.cuh"

using namespace pga::aln;

// seq: the contigs' bases (0..3) back to back, len: their lengths; req8: a b
// comp low hgh anti lbord hbord; path6: abpos aepos bbpos bepos diffs tlen;
// trace: the results' trace values back to back (trace_cap of them at most).
extern "C" int la_host(const uint8_t *seq, int ncontig, const int64_t *len, const float *freq, int64_t n,
                       const int32_t *req8, int32_t *path6, uint16_t *trace, int64_t trace_cap) {
  std::vector<int16_t> score(32768), table(32768);
  AlignSpec spec;
  spec.trace_space = 100;
  spec.reach = 0;
  spec.ave_path = build_align_spec(freq, score.data(), table.data());
  spec.score = score.data();
  spec.table = table.data();
  std::vector<std::vector<uint8_t>> fwd(ncontig), rc(ncontig);
  int64_t off = 0, maxctg = 0;
  for (int c = 0; c < ncontig; c++) {
    fwd[c].assign(len[c] + 2, 4);
    rc[c].assign(len[c] + 2, 4);
    for (int64_t i = 0; i < len[c]; i++) {
      fwd[c][i + 1] = seq[off + i];
      rc[c][len[c] - i] = 3 - seq[off + i];
    }
    off += len[c];
    maxctg = len[c] > maxctg ? len[c] : maxctg;
  }
  const int vcap = 1 << 14;
  const int64_t cell_cap = 40'000'000, pcap = 4 * (maxctg / 100 + 4) + 64;
  std::vector<int> V(vcap), M(vcap), HA(vcap), NA(vcap);
  std::vector<uint64_t> T(vcap);
  std::vector<Pebble> cells(cell_cap);
  std::vector<uint16_t> points(pcap);
  oracle::WaveWork W{};
  W.V = V.data(); W.M = M.data(); W.HA = HA.data(); W.NA = NA.data(); W.T = T.data();
  W.vcap = vcap; W.cells = cells.data(); W.cell_cap = cell_cap; W.points = points.data(); W.point_cap = pcap;
  int64_t nt = 0;
  for (int64_t i = 0; i < n; i++) {
    const int32_t *q = req8 + 8 * i;
    const Seq A{(q[2] ? rc[q[0]] : fwd[q[0]]).data() + 1, (int)len[q[0]]};
    const Seq B{fwd[q[1]].data() + 1, (int)len[q[1]]};
    Path P;
    memset(&P, 0, sizeof(P));
    W.err = 0;
    if (oracle::local_alignment(W, spec, A, B, q[2] != 0, P, q[3], q[4], q[5], q[6], q[7])) return 1;
    if (nt + P.tlen > trace_cap) return 2;
    int32_t *o = path6 + 6 * i;
    o[0] = P.abpos; o[1] = P.aepos; o[2] = P.bbpos; o[3] = P.bepos; o[4] = P.diffs; o[5] = P.tlen;
    memcpy(trace + nt, points.data() + P.trace_off, sizeof(uint16_t) * P.tlen);
    nt += P.tlen;
  }
  return 0;
}
