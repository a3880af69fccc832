// Launch shape of the marching kernels (atm_march.cuh, atm_adj_march.cuh).
#pragma once

#include <cuda_runtime.h>

namespace atm {

// Strips of `out` columns and `rows` rows over w x h points of L layers: grid
// (x, y, layer) of blocks of threads / 32 independent warps, a strip a warp.
struct StripPlan {
  dim3 grid;
  int threads, rows;
};

// Warps a block: those of 4, 3, 2, 1 that leave the fewest of a row of blocks
// without a strip (a block's registers are held until its last warp ends).
// Rows: the height, of equal strips, at which the launch should end first.  A
// strip takes its rows and `warm` more to fill its windows; a row takes a time
// that grows with the warps an SM holds, about as 16 + warps (B200, per row
// of the FP64 C mass sweep: 0.91 us with 4, 1.28 us with 12 warps an SM); full
// waves are followed by one that is only as crowded as what is left.  most: the
// largest height; the least is 3 (strips of a height of about 4 share the rows
// evenly), 4 on domains of more than 512 rows.
// Measured on B200, mixed form at 150x130x48 (us, C mass / C momentum / D mass
// / D momentum): powers of two and a wave's cost independent of its size, 49 /
// 54 / 47 / 58; over all heights from 4 to 128 the best is 33 / 33 / 34 / 37
// and the heights chosen here are within 4% of it, as at 64x64x20 to 512x512x32.
inline StripPlan plan_strips(int w, int h, int L, int out, int warm, int warps_sm, int most = 128) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    sms = 148;
  const int nsx = (w + out - 1) / out;
  int wpb = 4;
  for (int q = 3; q > 0; --q)
    if ((nsx + q - 1) / q * q < (nsx + wpb - 1) / wpb * wpb) wpb = q;
  const long long slots = (long long)sms * (warps_sm / wpb * wpb);
  int best = 4;
  long long cost = -1;
  // every number of strips, or on tall domains every height: at most 128 candidates
  const bool tall = h > 512;
  const int c0 = tall ? 4 : (h + most - 1) / most, c1 = tall ? most : (h + 3) / 4;
  for (int c = c0; c <= c1; ++c) {
    const int ns = tall ? (h + c - 1) / c : c;
    const int rows = (h + ns - 1) / ns;
    const long long n = (long long)nsx * ((h + rows - 1) / rows) * L, full = n / slots, rem = n % slots;
    long long t = full * (16 + warps_sm);
    if (rem) t += 16 + (rem + (long long)sms * wpb - 1) / ((long long)sms * wpb) * wpb;
    t *= rows + warm;
    if (cost < 0 || t < cost) {
      cost = t;
      best = rows;
    }
  }
  StripPlan p;
  p.grid = dim3((nsx + wpb - 1) / wpb, (h + best - 1) / best, L);
  p.threads = 32 * wpb;
  p.rows = best;
  return p;
}

}  // namespace atm
