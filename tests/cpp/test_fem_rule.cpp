// The rule between the two forms of the row assembly (fem_rule.h) against
// measured times of both, 152 SMs of 228 KB.
#include <cstdio>

#include "fem_rule.h"

int main() {
  const struct {
    int nv, len;
    double smem, global;  // ms, the whole call
  } measured[] = {
      {348480, 15, 3.382, 4.844}, {348480, 18, 3.606, 4.844},  {348480, 22, 4.138, 4.844},
      {348480, 24, 5.397, 4.844}, {348480, 32, 7.830, 4.844},  {348480, 56, 15.28, 4.844},
      {140544, 15, 1.415, 2.085}, {140544, 22, 1.745, 2.085},  {140544, 24, 2.263, 2.085},
      {140544, 40, 3.247, 2.085}, {17856, 15, 0.271, 0.380},   {17856, 22, 0.273, 0.380},
      {17856, 24, 0.470, 0.380},  {17856, 56, 0.874, 0.380},   {1700, 15, 0.239, 0.315},
      {1700, 32, 0.235, 0.315},   {1700, 80, 0.237, 0.315},    {85184, 52, 7.219, 2.821},
      {13824, 53, 1.614, 1.248},  {27000, 47, 2.796, 1.468},   {1000, 33, 0.628, 0.756},
  };
  int fails = 0;
  for (const auto &m : measured)
    if (mprgp::rows_in_smem(m.len, m.nv, 152, 228 * 1024) != (m.smem < m.global)) {
      std::printf("%d vertices, %d blocks\n", m.nv, m.len);
      ++fails;
    }
  // the widest row that shared memory holds, and lengths past any
  if (!mprgp::rows_in_smem(89, 89, 152, 228 * 1024)) ++fails;
  for (int len : {90, 1024, 1 << 20, 2147483647})
    if (mprgp::rows_in_smem(len, len, 152, 228 * 1024)) ++fails;
  std::printf(fails ? "FAILED\n" : "OK\n");
  return fails != 0;
}
