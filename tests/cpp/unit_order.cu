// The choice and move of a vertex scanned by one lane with unit weights, in a build of any flags: a list of labels
// whose heaviest is known must move its vertex there, under both tie rules. Exit code: 0, or the case that failed.
#include <cstdio>

#include "rak_lpa.cuh"

using namespace rak;

__device__ int scan(const LpaArgs &a, const uint32_t *labels, int count, uint32_t d, int it) {
  UnitSketch<8> us;
  unit_clear(us);
  for (int i = 0; i < count; ++i) unit_acc(us, labels[i]);
  Sketch<8> sk;
  sk_clear<8>(sk);
  unit_to_sketch<8, true>(us, sk);
  const uint32_t u = 0;
  uint32_t vout[1] = {d};
  uint8_t fin[1] = {1}, fout[1] = {0};
  Counters cnt{0, 0, 0, 0};
  lane_close<8, MODE_SPLIT, true, false, RULE_CPU>(a, sk, u, d, 0, 0, count, it, false, vout, fin, fout, cnt, Phase{});
  return int(vout[0]);
}

__global__ void run(LpaArgs a, const uint32_t *labels, int *out) {
  out[0] = scan(a, labels, 12, 99, 0);       // hashed ties: 5 six times, others fewer
  out[1] = scan(a, labels, 12, 99, 1);       // the reference's tie rule
  out[2] = scan(a, labels, 0, 99, 1);        // nothing: stays
  out[3] = scan(a, labels, 1, 99, 1);        // one edge
}

int main() {
  const uint32_t labels[12] = {7, 5, 5, 3, 5, 7, 5, 2, 5, 7, 5, 3};
  uint32_t *d;
  int *o, out[4] = {-1, -1, -1, -1};
  if (cudaMalloc(&d, sizeof labels) != cudaSuccess || cudaMalloc(&o, sizeof out) != cudaSuccess) return 100;
  cudaMemcpy(d, labels, sizeof labels, cudaMemcpyHostToDevice);
  LpaArgs a{};
  a.tie_until = 1;
  run<<<1, 1>>>(a, d, o);
  if (cudaMemcpy(out, o, sizeof out, cudaMemcpyDeviceToHost) != cudaSuccess) return 101;
  const int want[4] = {5, 5, 99, 7};
  for (int i = 0; i < 4; ++i)
    if (out[i] != want[i]) { std::printf("case %d: %d, not %d\n", i, out[i], want[i]); return i + 1; }
  return 0;
}
