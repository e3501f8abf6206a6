// ordered_walk over small hand-made trees: prints the entries listed and the
// device error of (a) a cell with one particle, (b) a cell that is its own
// child, (c) a child outside the tree.  The walk bounds all three by itself.
#include <cmath>
#include <cstdio>
#include <cstring>

#include "walk_list.cuh"

using namespace nbb;

__global__ void __launch_bounds__(32) walk_kernel(Workspace ws, int m, int *entries) {
  __shared__ Frontier walk;
  __shared__ ListBuffer<64> buffer;
  ListBuffer<64> *list = &buffer;
  unsigned tests = 0;
  set_target_box(walk, make_double4(0.0, 0.0, 0.0, 1.0), 1.0);
  ordered_walk(ws, m, 0, 1.0, walk, list, tests, [&](int count, bool) {
    if (threadIdx.x == 0) *entries += count;
    return 0;
  });
}

template <typename T>
static T *managed(size_t n) {
  T *p = nullptr;
  if (cudaMallocManaged(&p, n * sizeof(T)) != cudaSuccess) return nullptr;
  memset(p, 0, n * sizeof(T));
  return p;
}

int main() {
  constexpr int m = 2;
  Workspace ws;
  ws.n = 1;
  ws.node_a = managed<double4>(m);
  ws.node_b = managed<double4>(m);
  ws.node_c = managed<double4>(m);
  ws.node_meta = managed<int4>(m);
  ws.node_kids = managed<int>(8 * m);
  ws.pm4 = managed<double4>(1);
  ws.sc = managed<DevScalars>(1);
  int *entries = managed<int>(1);
  if (!ws.node_a || !ws.node_b || !ws.node_c || !ws.node_meta || !ws.node_kids || !ws.pm4 || !ws.sc || !entries) return 1;
  for (int test = 0; test < 3; ++test) {
    for (int k = 0; k < m; ++k) {
      ws.node_a[k] = make_double4(0.5, 0.5, 0.5, 1.0);
      ws.node_c[k] = make_double4(INFINITY, INFINITY, INFINITY, INFINITY);  // every target opens it
      ws.node_meta[k] = make_int4(m, -1, 0, 1);
      for (int j = 0; j < 8; ++j) ws.node_kids[8 * k + j] = -1;
      ws.node_kids[8 * k] = 1;
    }
    if (test == 0) ws.node_meta[1] = make_int4(m, 0, 1, 0);
    if (test == 2) ws.node_kids[0] = m + 3;
    memset(ws.sc, 0, sizeof(DevScalars));
    *entries = 0;
    walk_kernel<<<1, 32>>>(ws, m, entries);
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    printf("%d %d\n", *entries, ws.sc->error);
  }
  return 0;
}
