// Host build of csrc/pair_float.cuh for the CPU tests: reads m groups of four
// float32 planes (16 floats each) and writes, per group, whether pair_vertex
// accepts the first three, the vertex, and pair_side's sign for the fourth
// (five float32).
//
//   pair_float_host <rows.f32> <m> <out.f32>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "pair_float.cuh"

using namespace vgb;

int main(int argc, char** argv) {
  if (argc != 4) return 2;
  const int m = std::atoi(argv[2]);
  std::vector<float> v((size_t)m * 16), out((size_t)m * 5);
  FILE* f = std::fopen(argv[1], "rb");
  if (!f || std::fread(v.data(), sizeof(float), v.size(), f) != v.size()) return 3;
  std::fclose(f);
  for (int g = 0; g < m; ++g) {
    float4 r[4];
    for (int i = 0; i < 4; ++i) {
      const float* p = &v[(size_t)g * 16 + 4 * i];
      r[i] = make_float4(p[0], p[1], p[2], p[3]);
    }
    float3 x = make_float3(0.f, 0.f, 0.f);
    float* o = &out[(size_t)g * 5];
    o[0] = pair_vertex(r[0], r[1], r[2], x) ? 1.f : 0.f;
    o[1] = x.x;
    o[2] = x.y;
    o[3] = x.z;
    o[4] = (float)pair_side(r[0], r[1], r[2], r[3]);
  }
  f = std::fopen(argv[3], "wb");
  if (!f || std::fwrite(out.data(), sizeof(float), out.size(), f) != out.size()) return 4;
  std::fclose(f);
  return 0;
}
