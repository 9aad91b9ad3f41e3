// Shared extensions: the table through which the calls of a launch take the
// rest of an extension from another call's (cross_line and extend,
// align_warp.cuh).
//
// The calls of one pair's band blocks keep extending the same alignment: a
// long one drifts through many blocks, each block's chain makes its own call,
// and each call grows the whole path again.  Two waves of one pair and
// direction with the same state -- window, furthest points, match histories,
// trace marks, best, last passing record -- have the same future, whatever
// wave number each is at: the wave after depends on nothing else.  Where a wave's best first crosses a line (a multiple of
// SHARE_LINE antidiagonals) its state is looked up in a table of the launch:
//   * not there: it is entered, and the extension goes on as its owner;
//   * there, with an equal state: the extension has joined the owner's and
//     stops.  Once the owner has stopped too -- it joined another extension
//     further along, or ended -- it is known on which diagonal the path crosses
//     the line, hence the joiner's own part of the trace; the tip and the rest
//     of the trace lie behind the owner, one part per extension on the way.
// A joiner waits only for an extension that is further along, and that started
// before, so waits never form a circle; a wait is bounded all the same, and
// whoever gives up goes on alone from its own state.  Either way the path and
// its trace are those of growing alone.
//
// A trace is kept as the intervals between its pebbles, last first.  What an
// owner has before a line differs from the joiner's; after it, only wave
// numbers differ, by a constant, and intervals hold differences.  The
// interval across the line starts at the joiner's own head pebble on the
// diagonal the owner's path crossed on; diagonals may have one head pebble in
// common, so which of them do is part of the state too: then any diagonal
// with the owner's head has the joiner's.
//
// Scouts.  A task's calls run one after the other, and the longest alignments
// are one warp's work from wherever their first call starts.  Once no task is
// left to start, a task that is about to make a call or crosses a line goes
// (once) over all its chains and queues, for the free warps: the first call
// of every other chain, whose result the task takes if it still makes that
// call with those inputs; and starts for extensions, in the chain's diagonal
// band at the midpoints between lines, grown both ways at once, each until it
// joins the next.  Either only saves time: a call nobody ran is made by its
// task, a start off the path serves nobody.  (Queued from the launch's first
// task on they took warps from tasks: 17 genomes of 2.5 Mbp 55 ms of pair
// phase against 15.)
#pragma once
#include <stdint.h>

namespace pga {
namespace aln {

// Antidiagonals between lines: a line costs an extension about 4 us, the
// waves between two at 0.5 % divergence about 30 us.
constexpr int SHARE_LINE = 16384;
constexpr int SHARE_MIN = 2048;    // antidiagonals an extension has behind it at its first line
constexpr int SHARE_PROBES = 64;   // table slots looked at
constexpr int SHARE_POLLS = 1 << 19;  // bound of a wait (a poll takes a microsecond or so)

enum : int { SHARE_NONE = 0, SHARE_HEAD = 1, SHARE_PEBBLE = 2 };      // ShareEntry::kind
enum : int { SHARE_DONE = 1, SHARE_JOINED = 2, SHARE_FAILED = 3 };  // ShareRec::status

// An owner's wave at a line.  Lane l holds the diagonal that is l mod 32.
struct ShareEntry {
  int rec, prev;           // its extension; that extension's entry before (-1: none)
  int low, hgh, besta, bestx, lasta, dif;
  int mark;                // pebbles numbered below are from before the line
  // how the finished path crosses the line: the tip's own head pebble is from
  // before it (HEAD), or `p` is the first pebble after it, `after` intervals
  // follow p; the head before the line is lane `lane`'s
  int kind, lane, after;
  int pdiag, pmark, pdiff;
  unsigned way;            // the pair, orientation and direction
  int V[32], HA[32], HM[32], NA[32], pat[32];
  uint64_t T[32];
};

// An extension that stopped: its own intervals, `own` of them at list + off,
// from its tip (DONE) or from its head pebble at the wave, number dif, where it
// joined the owner of `entry` (JOINED).
struct ShareRec {
  int status;
  int tipx, tipy, tipd;
  int entry, dif;
  int hdiag, hmark, hdiff;
  int own;
  int64_t off;
};

// A queued call, or a start to grow from: contigs, orientation, diagonal
// band, antidiagonal; a call's result (path, trace intervals at list + off).
struct Scout {
  int a, b, comp, low, hgh, anti;
  int call;   // a call (else a start)
  int state;  // SCOUT_*
  int abpos, aepos, bbpos, bepos, diffs, tlen;
  int64_t off;
};

enum : int { SCOUT_UNWRITTEN = 0, SCOUT_READY = 1, SCOUT_RUNS = 2, SCOUT_DONE = 3, SCOUT_VOID = 4 };

struct ShareTable {
  unsigned long long *keys;  // 0: free
  int *vals;                 // entry, -1 not yet written, -2 none
  unsigned mask;             // slots - 1
  ShareEntry *entries;
  ShareRec *recs;
  uint32_t *list;
  int entry_cap, rec_cap;
  int64_t list_cap;
  unsigned *nentry, *nrec;        // counters, zero at launch
  unsigned long long *nlist;
  // joins whose path goes on past the next trace mark [0], ends before it [1]
  // or at the line [2]; calls taken from a scout [3]
  unsigned *joins;
  // the scouts' queue: queued [0, min(qtail, qcap)), taken below qhead; tasks
  // that have ended
  Scout *scouts;
  unsigned long long *ckeys;  // the queued calls by their inputs, as keys and vals
  int *cvals;
  unsigned cmask;
  int qcap;
  unsigned *qhead, *qtail, *ended;
  // the launch's task counter and its tasks: past them, warps are free
  const unsigned *next_task;
  unsigned ntasks;
};

}  // namespace aln
}  // namespace pga
