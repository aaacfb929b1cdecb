// The reference profiles' face passes of a step and their split into launches.
#pragma once
#include <algorithm>

namespace cflbm {

struct FaceOp {
  int kind;  // 0 copy (inlet), 1 extrapolate (outlet), 2 bounce (wall)
  int axis;  // 0 x, 1 y, 2 z
  int side;  // 0 low, 1 high
  int trim;  // 1: the pass skips the two ghost ends of its tangential range
  int ndir;  // the populations the pass writes (filled by launch_ref_boundary),
  unsigned long long dirs;  // 5 bits each, the k-th at bit 5k
};

// The passes of a step in their order, and what one launch does of each: threads
// start[p] .. start[p + 1], from its population first[p] on.
struct FaceOps {
  int n;
  int start[7];
  int first[6];
  FaceOp op[6];
};

// Threads of one launch: its indices are 32-bit.  Every source is resolved to a value
// that no launch of the step writes, so any split gives the same ghosts; all but boxes
// whose faces hold more than 1.2e8 cells fit one launch.
constexpr long long FACE_THREADS = 1LL << 30;

// Fills start and first of the launch that begins at population k of pass p, as many
// whole (pass, population) planes as `limit` allows (cells[q]: face cells of pass q),
// and moves (p, k) to the next.  False when a plane alone is beyond the limit.
inline bool next_faces(FaceOps &ops, const long long *cells, long long limit, int &p, int &k) {
  long long total = 0;
  for (int q = 0; q < ops.n; ++q) {
    ops.start[q] = (int)total;
    ops.first[q] = 0;
    if (q != p) continue;
    const int take = (int)std::min<long long>((limit - total) / cells[q], ops.op[q].ndir - k);
    ops.first[q] = k;
    total += take * cells[q];
    k += take;
    if (k == ops.op[q].ndir) {
      ++p;
      k = 0;
    }
  }
  ops.start[ops.n] = (int)total;
  return total > 0 || ops.n == 0;
}

}  // namespace cflbm
