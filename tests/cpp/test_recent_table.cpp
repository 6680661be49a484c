// RecentTable (recent_table.h): more keys than places, the last used stay.
#include <cstdio>

#include "recent_table.h"

int main() {
  opfc::RecentTable<int, int, 8> t;
  int bad = 0;
  const int *first = nullptr;
  for (int i = 0; i < 100; ++i) {
    if (t.find(i)) bad = 1;
    const int *p = t.keep(i, 10 * i);
    if (!p || *p != 10 * i) bad = 2;
    if (i == 0) first = p;
    // the keys of one launch: 0 and the seven newest are all there, and stay where they are
    for (int k = i < 7 ? 1 : i - 6; k <= i; ++k) {
      const int *q = t.find(k);
      if (!q || *q != 10 * k) bad = 4;
    }
    if (t.find(0) != first || *first != 0) bad = 3;
    if (i > 8 && t.find(i - 7)) bad = 5;
  }
  if (bad) std::printf("check %d failed\n", bad);
  return bad;
}
