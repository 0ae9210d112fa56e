// Order of the reference-order sweep's tiles (pm_wave.cu).
#pragma once

#include <math.h>

namespace pm {

#ifdef __CUDACC__
#define PM_HD __host__ __device__
#else
#define PM_HD
#endif

// Tile (tY, tZ) of a ticket: tiles in order of tY + tZ, within one diagonal in
// order of tZ.  The tiles a tile waits for, (tY - 1, tZ) and (tY, tZ - 1), lie
// on the diagonal before, and tiles of one diagonal do not wait for each other,
// so those resident at a time run abreast.  (In order of rows a row's tiles
// follow each other four hyperplanes apart, and where fewer rows are resident
// than it takes to keep them all busy, the rest of the device waits: 16x512x512
// takes 2.05 ms a sweep and 11.8 in rows, 2x1000x1000 3.64 and 63.2, 256^3
// 3.52 and 5.10, 48x48x64, whose tiles are all resident, 0.20 and 0.20.)
PM_HD inline void wave_tile(int ticket, int tiles_y, int tiles_z, int& tY, int& tZ) {
  const int m = tiles_y < tiles_z ? tiles_y : tiles_z;
  const long long n = (long long)tiles_y * tiles_z, tri = (long long)m * (m - 1) / 2;
  const bool mirrored = ticket >= n - tri;  // the last diagonals, from the far corner
  const long long t = mirrored ? n - 1 - ticket : ticket;
  long long s, i;  // diagonal and place on it
  if (t < tri) {
    s = (long long)((sqrt(8.0 * (double)t + 1.0) - 1.0) / 2.0);
    while (s * (s + 1) / 2 > t) --s;
    while ((s + 1) * (s + 2) / 2 <= t) ++s;
    i = t - s * (s + 1) / 2;
  } else {
    s = m - 1 + (t - tri) / m;
    i = (t - tri) % m;
  }
  tZ = (int)((s > tiles_y - 1 ? s - (tiles_y - 1) : 0) + i);
  tY = (int)(s - tZ);
  if (mirrored) {
    tY = tiles_y - 1 - tY;
    tZ = tiles_z - 1 - tZ;
  }
}

}  // namespace pm
