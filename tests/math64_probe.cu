// The FP64 elementary functions of the sample loops on arrays, for
// tests/test_math64.py.  f: the function; a: arguments, b: a second argument.
#include "hxg_math64.cuh"

__global__ void eval(int f, int n, const double *a, const double *b, double *out, double *out2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = a[i];
  double r = 0., s = 0.;
  switch (f) {
    case 0: r = hxg::exp64<true>(x); break;
    case 1: r = hxg::exp64<false>(x); break;
    case 2: r = hxg::rsqrt64(x); break;
    case 3: r = hxg::sqrt64(x, s); break;
    case 4: r = hxg::rcp64(x); break;
    case 5: hxg::sincos_quarter(x, r, s); break;
    case 6: r = hxg::pow_k(x, b[i]); break;
    case 8: hxg::dot2_64(x, b[i], a[n - 1 - i], b[n - 1 - i], r, s); break;
    case 7: r = hxg::sqrt_pos(x); break;
  }
  out[i] = r;
  out2[i] = s;
}

extern "C" int probe(int f, int n, const double *a, const double *b, double *out, double *out2) {
  eval<<<(n + 255) / 256, 256>>>(f, n, a, b, out, out2);
  return (int)cudaDeviceSynchronize();
}
