// The launch shape rules (cato_shape.h) as C functions for the tests.
#include "../fvleg_2d_gb300/csrc/cato_shape.h"

static void put(const cato::StageShape& s, int* out) {
  const int v[6] = {s.width, s.threads, s.rows, s.block, s.warps, s.variant};
  for (int k = 0; k < 6; ++k) out[k] = v[k];
}

extern "C" {
void default_shape(int sms, int ni, int nj, int ng, int precision, int* out) {
  put(cato::default_shape(sms, ni, nj, ng, precision), out);
}
// the register budget the kernel is launched with, and whether it is the split one
void launched_form(int sms, int ni, int nj, int ng, int precision, int width, int rows, int variant,
                   int* out) {
  cato::StageShape s = cato::plan_shape(sms, ni, nj, ng, precision, width, rows);
  s.variant = variant;
  const cato::StageForm f = cato::stage_form(s, precision);
  out[0] = f.variant;
  out[1] = f.split;
}
void plan_shape(int sms, int ni, int nj, int ng, int precision, int width, int rows, int* out) {
  put(cato::plan_shape(sms, ni, nj, ng, precision, width, rows), out);
}
int tune_shapes(int sms, int ni, int nj, int ng, int precision, int width, int rows, int* out) {
  const auto c = cato::tune_shapes(
      sms, ni, nj, ng, precision, cato::plan_shape(sms, ni, nj, ng, precision, width, rows));
  for (const auto& s : c) {
    put(s, out);
    out += 6;
  }
  return (int)c.size();
}
int batch_rows(int sms, int precision, int plan_rows, int n, int W, const int* ni, const int* nj) {
  std::vector<cato::BatchGrid> g;
  for (int k = 0; k < n; ++k) g.push_back({ni[k], nj[k], W});
  return cato::batch_rows(sms, precision, plan_rows, g);
}
}
