// Warp reductions shared by the solvers.
#pragma once

// Sums of N values over a warp: lane l returns the sum of v[l] (l < N), N <= 32.  At each of
// the five steps a lane passes on the half of its values that the other lane keeps.
template <int N> __device__ __forceinline__ double warp_sums(double (&v)[N])
{
  const int lane = threadIdx.x & 31;
  int cnt = N;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
  {
    const bool hi = lane & o;
#pragma unroll
    for (int j = 0; j < 16; j++)
    {
      if (j >= o || j >= cnt) continue;
      if (j + o < cnt)
      {
        const double keep = hi ? v[j + o < N ? j + o : j] : v[j], give = hi ? v[j] : v[j + o < N ? j + o : j];
        v[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
      else
      {
        const double other = __shfl_xor_sync(0xffffffffu, v[j], o);
        v[j] = hi ? 0.0 : v[j] + other;
      }
    }
    cnt = cnt < o ? cnt : o;
  }
  return v[0];
}
