// Prints the tile (tY tZ) of every ticket of a grid of tiles.
#include <stdio.h>
#include <stdlib.h>

#include "../poremaps_gb300/csrc/pm_wave.h"

int main(int argc, char** argv) {
  if (argc != 3) return 2;
  const int ty = atoi(argv[1]), tz = atoi(argv[2]);
  for (int t = 0; t < ty * tz; ++t) {
    int y = -1, z = -1;
    pm::wave_tile(t, ty, tz, y, z);
    printf("%d %d\n", y, z);
  }
  return 0;
}
