// The far kernel's cut of the source groups (far_parts): the partials of every
// ensemble the allocation-free evaluation takes fit its scratch, no part is
// below 8 sources, and the parts cover a group.  Exit status 1 otherwise.
#include <cstdio>

#include "../../quest_b200/csrc/qg_internal.h"

int main()
{
  int bad = 0;
  for(int nT = 1; nT <= qg::kNoAllocMaxTiles; ++nT)
    for(int g = 1; g <= nT; ++g) {
      const int parts = qg::far_parts(nT, g), unit = (g * qg::kTile + parts - 1) / parts;
      const long long slots = (long long)((nT + g - 1) / g) * parts * nT * qg::kTile;
      bool ok = parts >= 1 && unit >= 8 && parts * unit >= g * qg::kTile;
      if(g == (nT < qg::kTileGroup ? nT : qg::kTileGroup))
        ok = ok && slots <= (long long)qg::kNoAllocMaxGroups * qg::kNoAllocMaxDots;
      if(!ok) std::printf("mismatch: %d tiles, group %d\n", nT, g), ++bad;
    }
  std::printf("mismatches %d\n", bad);
  return bad != 0;
}
