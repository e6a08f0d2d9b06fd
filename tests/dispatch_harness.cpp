// The rules of csrc/tcec_dispatch.h behind C names, for tests/test_dispatch.py.
#include "../wmma_extension_b200/csrc/tcec_dispatch.h"

using namespace tcec_host;

extern "C" {
int fused_pays_c(int m, int n, int k, int batch, int promo, int ec, int sms, int stores) {
  return fused_pays(m, n, k, batch, (k + 31) / 32, promo, ec != 0, sms, m > 128 && pairs_pay(m, n, k, batch, ec != 0),
                    static_cast<FusedStores>(stores));
}
int direct_pays_c(int m, int n, int nkb, int batch, int tf32, int sms) {
  return direct_pays(m, n, nkb, batch, tf32 != 0, sms);
}
int pairs_pay_c(int m, int n, int k, int batch, int ec) { return pairs_pay(m, n, k, batch, ec != 0); }
int pace_pays_c(int m, int n, int batch, int nkb, int images, int pairs) {
  return pace_pays(static_cast<int>(ceil_div(m, 256)), static_cast<int>(ceil_div(n, 256)), batch, nkb, images, pairs);
}
int draws_pay_c(int m, int n, int k, int ec, int pairs) {
  return draws_pay(m, n, k, 1, ec != 0, ceil_div(m, 256) * ceil_div(n, 256), pairs);
}
int divide_k_c(int m, int n, int k, int batch, int nkb, int ec, const int* slots, int forced) {
  const int s[3] = {slots[0], slots[1], slots[2]};
  return divide_k(m, n, k, batch, nkb, ec != 0, s, forced);
}
int batch_overlap_c(const Extent* c, const Extent* x, int batch) {
  const Overlap o = batch_overlap(*c, *x, batch);
  return (o.own ? 1 : 0) | (o.across ? 2 : 0);
}
int matrices_may_overlap_c(const Extent* c, const Extent* x) {
  return matrices_may_overlap(reinterpret_cast<unsigned long long>(c->base), c->ld, c->inner, c->outer,
                              reinterpret_cast<unsigned long long>(x->base), x->ld, x->inner, x->outer);
}
}
