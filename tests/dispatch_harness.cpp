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
}
