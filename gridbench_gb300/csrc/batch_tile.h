// The cut of an instance's slices into tiles for a batch's split (host code, no CUDA).
#pragma once

namespace gbdw {

// Slices per tile: the largest split <= the batch's that cuts a site's LsE = Ls*nrhs slices into whole slice
// groups of spt, with whole right-hand sides in a tile (a multiple of Ls: they lie one after the other) or
// a whole part of one's slices (a divisor of Ls); LsE where none does.
inline int batch_tile(int LsE, int Ls, int spt, int split) {
  for (int sp = split; sp > 1; sp >>= 1) {
    if (LsE % sp) continue;
    const int TE = LsE / sp;
    if (TE % spt == 0 && (TE % Ls == 0 || Ls % TE == 0)) return TE;
  }
  return LsE;
}

}  // namespace gbdw
