// Host build of the 16-bit collision's backward y and z passes for the CPU tests: the packed ones
// the kernels run (psl_collision_g.cuh) and the same passes line by line in scalar operations.
#include "psl_collision_g.cuh"

// two lines (m0, m1, m2)
extern "C" void passes_pair(float* m, float u, float wpm, float w0, int weights) {
  const psl::BwdAxis2 k((psl::BwdAxis<float>(u)));
  psl::GPair a = psl::gpair(m[0], m[3]), b = psl::gpair(m[1], m[4]), c = psl::gpair(m[2], m[5]);
  if (weights) psl::bwd_full_w2(a, b, c, k, wpm, w0);
  else psl::bwd_full2(a, b, c, k);
  m[0] = a.x, m[1] = b.x, m[2] = c.x;
  m[3] = a.y, m[4] = b.y, m[5] = c.y;
}

extern "C" void passes_scalar(float* m, float u, float wpm, float w0, int weights) {
  const psl::BwdAxis<float> k(u);
  for (int i = 0; i < 2; ++i) {
    if (weights) psl::bwd_full_w(m[3 * i], m[3 * i + 1], m[3 * i + 2], k, wpm, w0);
    else psl::bwd_full(m[3 * i], m[3 * i + 1], m[3 * i + 2], k);
  }
}

// 27 moments after the x pass -> 27 populations
extern "C" void backward_pair(const float* moments, float uy, float uz, float* out) {
  float G[3][3][3], g[27];
  for (int i = 0; i < 27; ++i) G[i / 9][i / 3 % 3][i % 3] = moments[i];
  psl::backward_yz_g(G, psl::BwdAxis<float>(uy), psl::BwdAxis<float>(uz), g);
  for (int q = 0; q < 27; ++q) out[q] = g[q];
}

extern "C" void backward_scalar(const float* moments, float uy, float uz, float* out) {
  const psl::BwdAxis<float> by(uy), bz(uz);
  for (int i = 0; i < 3; ++i) {
    float line[3][3];  // [y slot][z order]
    for (int j = 0; j < 3; ++j)
      for (int k = 0; k < 3; ++k) line[j][k] = moments[9 * i + 3 * j + k];
    for (int k = 0; k < 3; ++k) psl::bwd_full(line[0][k], line[1][k], line[2][k], by);
    for (int j = 0; j < 3; ++j) {
      psl::bwd_full_w(line[j][0], line[j][1], line[j][2], bz, psl::lattice_weight(psl::slot(i, j, 0)),
                      psl::lattice_weight(psl::slot(i, j, 1)));
      for (int k = 0; k < 3; ++k) out[psl::slot(i, j, k)] = line[j][k];
    }
  }
}
