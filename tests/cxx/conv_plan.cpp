// C entries of the convolution kernels' plans (csrc/conv_plan.cuh) for the test.
#include "conv_plan.cuh"
using namespace xbg::nn;
extern "C" {
int rows_stages(int bn, int wc, int W, int cin) { return conv_rows_stages(bn, wc, W, cin); }
int rows_smem(int bn, int wc, int cin, int nst) { return conv_rows_smem(bn, wc, cin, nst); }
int rows_cols(int bn) { return conv_rows_cols(bn); }
int rows_pays(int bn, int cin, int W, int pixels, int sms) { return conv_rows_pays(bn, cin, W, pixels, sms); }
int rows_run(int S, int H, int sms, int extra, int* lohi) {   // CTAs; [lo, hi) of each
    const RowsRun r = conv_rows_run(S, H, sms, extra != 0);
    const int n = conv_rows_ctas(r, S, H);
    for (int k = 0; lohi && k < n; k++) {
        lohi[2 * k] = conv_rows_lo(r, H, k);
        lohi[2 * k + 1] = conv_rows_hi(r, S, H, k);
    }
    return n;
}
int wgrad_slots(int bn, int wc, int nseg) { return wgrad_rows_slots(bn, wc, nseg); }
int wgrad_smem(int bn, int wc, int nx) { return wgrad_rows_smem(bn, wc, nx); }
int wgrad_cols(int bn) { return wgrad_rows_cols(bn); }
}
