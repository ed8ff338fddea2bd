// Divisions and updates of one elimination level by index lists (lu.cu, lutree.cu).
#pragma once

__device__ __forceinline__ void lu_divide(int2 dv, double *mx) { mx[dv.x] = mx[dv.x] / mx[dv.y]; }

// A destination's updates with the level's L factors already stored (after its division step).
// ds = (destination, L(i, k), U(k, j), U(k, k)) for one update; (destination, first pair, count,
// -1) for more, pairs (L(i, k), U(k, j), U(k, k), 0) in increasing k.
__device__ __forceinline__ void lu_update(int4 ds, const int4 *__restrict__ pairs, double *mx) {
  double acc = mx[ds.x];
  if (ds.w >= 0) {
    acc = acc - mx[ds.y] * mx[ds.z];
  } else {
    for (int p = ds.y; p < ds.y + ds.z; ++p) {
      const int4 lu = pairs[p];
      acc = acc - mx[lu.x] * mx[lu.y];
    }
  }
  mx[ds.x] = acc;
}

// The same updates before the level's divisions: each L factor formed on the spot from the
// undivided column entry and the pivot, the division the division step makes, so the same value.
__device__ __forceinline__ void lu_update_divide(int4 ds, const int4 *__restrict__ pairs, double *mx) {
  double acc = mx[ds.x];
  if (ds.w >= 0) {
    acc = acc - (mx[ds.y] / mx[ds.w]) * mx[ds.z];
  } else {
    for (int p = ds.y; p < ds.y + ds.z; ++p) {
      const int4 lu = pairs[p];
      acc = acc - (mx[lu.x] / mx[lu.z]) * mx[lu.y];
    }
  }
  mx[ds.x] = acc;
}
