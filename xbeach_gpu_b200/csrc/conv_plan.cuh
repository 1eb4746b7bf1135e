// Shared memory and tensor memory of the box-fed convolution and weight-gradient
// kernels (nn_gemm.cu), as plain functions of the shape.
#pragma once

#ifdef __CUDACC__
#define XBG_PLAN __host__ __device__ constexpr
#else
#define XBG_PLAN constexpr
#endif

namespace xbg {
namespace nn {

constexpr int PLAN_GM = 128;               // pixels of a strip
constexpr int CR_MAXST = 18;               // input stages of k_conv_rows at most
constexpr int CR_SMEM = 225 * 1024;        // its dynamic shared memory at most
constexpr int WR_P = 64;                   // pixels of a chunk of k_wgrad_rows
constexpr int WR_MX = 24;                  // its input slots at most
constexpr int WR_ND = 3;                   // its dz slots
constexpr int WR_SMEM = 226 * 1024;

// Where a CTA asks for more than half of an SM's 512 tensor memory columns it takes
// more than half of the shared memory too: a second CTA of the launch would be
// placed there only to wait for columns.
constexpr int HALF_TCOLS = 256, HALF_SMEM = 115 * 1024;
XBG_PLAN int at_least(int a, int b) { return a > b ? a : b; }

// ---- k_conv_rows
// accumulator slots of `stride` columns: three rows under way, at least one being stored
XBG_PLAN int conv_rows_stride(int bn) { return bn <= 32 ? 32 : (bn <= 64 ? 64 : 128); }
XBG_PLAN int conv_rows_slots(int bn) { return bn <= 64 ? 8 : 4; }
XBG_PLAN int conv_rows_cols(int bn) { return conv_rows_slots(bn) * conv_rows_stride(bn); }
// stages, weights and alignment
XBG_PLAN int conv_rows_bytes(int bn, int wc, int cin, int nst) {
    return 1024 + nst * PLAN_GM * wc * 2 + 9 * cin * bn * 2;
}
XBG_PLAN int conv_rows_smem(int bn, int wc, int cin, int nst) {
    return at_least(conv_rows_bytes(bn, wc, cin, nst), conv_rows_cols(bn) > HALF_TCOLS ? HALF_SMEM : 0);
}
// stages that fit beside the weights of a layer (0: k_conv_rows does not apply)
XBG_PLAN int conv_rows_stages(int bn, int wc, int W, int cin) {
    // the last strip of a row may be ragged; strips of which over a third lies outside the image are not worth it
    const int strips = (W + PLAN_GM - 1) / PLAN_GM;
    if (bn > 128 || W < PLAN_GM || 2 * strips * PLAN_GM > 3 * W) return 0;
    // 16-channel boxes with more output channels (beyond 32) than input channels are
    // left to the other kernels: 16 -> 128 and 48 -> 96 faulted before whole warps
    // waited, and it is not shown that those waits were all that was wrong there
    if (wc == 16 && bn > 32 && bn > cin) return 0;
    const int nb = 3 * (cin / wc);   // an input row's boxes are waited for together; two rows' worth, or nearly
    if (nb > 30) return 0;
    const int room = CR_SMEM - conv_rows_bytes(bn, wc, cin, 0), box = PLAN_GM * wc * 2;
    const int n = room < 0 ? 0 : room / box;
    if (n < nb + (nb + 1) / 2) return 0;
    const int nst = n > CR_MAXST ? CR_MAXST : n;
    if (nst < nb) return 0;
    return nst;
}
// 16-channel boxes (32 bytes a pixel, so three times the boxes of a 48-channel input)
// pay only where a CTA has rows enough; below, k_conv_tma's and k_conv_tc's blocks,
// two and more to an SM, end first.  From three rows a CTA on for 16 -> 32 channels
// (256 x 256 pixels 10.5 us there, 10.2 here; 512 x 1024 50.9, 32.8), from seven for
// 16 -> 16 (256 x 512 12.3, 12.7; 4 x 192 x 192 17.9, 16.3), from six for 48 and 80
// channels (48 -> 48 at 304 x 300 23.4, 27.1; at 256 x 512 32.2, 27.2), not at all
// for these with 16 outputs (256 x 512 22.2, 26.5; 512 x 1024 74.4, 72.0), nor where
// more than a fifth of their strips lies outside the image (48 -> 32 at 4 x 192 x 192
// 31.6, 34.8).  Wider boxes are the faster at every size.
XBG_PLAN bool conv_rows_pays(int bn, int cin, int W, long long pixels, int sms) {
    if (cin % 32 == 0) return true;
    if (cin > 16 && (bn == 16 || 4 * ((W + PLAN_GM - 1) / PLAN_GM) * PLAN_GM > 5 * W)) return false;
    const long long rows = cin > 16 ? 6 : (bn == 16 ? 7 : 3);
    return pixels >= rows * PLAN_GM * sms;
}
// A CTA's run: `per` consecutive output rows of the S = images x strips strips of H
// rows, `cps` CTAs to a strip, or runs on end across strips (cps 0).  A run of n
// rows in one strip reads n + 2 input rows, one that crosses into the next strip
// n + 4, so runs keep to a strip where that makes them no longer, or one row longer
// in a layer whose time is its copies (extra).  With waits by single lanes 48 -> 48 channels at 160 x 176 pixels
// 19.9 us with runs across strips, 14.7 without; 32 -> 32 at 2 x 256 x 256 13.0, 11.1
// (7 rows either way); 96 -> 32 at 240 x 1016 36.7, 34.4 (13 rows, 14); where products
// bound the layer 14 rows for 13 lose: 64 -> 128 there 36.7, 38.2.
struct RowsRun { int per, cps; };
XBG_PLAN RowsRun conv_rows_run(int S, int H, int sms, bool extra) {
    const int per = (int)(((long long)S * H + sms - 1) / sms);
    if (H % per != 0 && S <= sms) {
        const int c = sms / S, p = (H + c - 1) / c;
        if (p <= per + (extra ? 1 : 0)) return RowsRun{p, (H + p - 1) / p};
    }
    return RowsRun{per, 0};
}
XBG_PLAN int conv_rows_ctas(RowsRun r, int S, int H) {
    return r.cps ? S * r.cps : (int)(((long long)S * H + r.per - 1) / r.per);
}
// first and last (exclusive) row of a CTA's run
XBG_PLAN int conv_rows_lo(RowsRun r, int H, int cta) { return r.cps ? cta / r.cps * H + cta % r.cps * r.per : cta * r.per; }
XBG_PLAN int conv_rows_hi(RowsRun r, int S, int H, int cta) {
    const int hi = conv_rows_lo(r, H, cta) + r.per, end = r.cps ? (cta / r.cps + 1) * H : S * H;
    return hi < end ? hi : end;
}

// ---- k_wgrad_rows
XBG_PLAN int wgrad_rows_cols(int bn) { return bn <= 16 ? 64 : (bn <= 32 ? 128 : (bn <= 64 ? 256 : 512)); }
// the dz slots, alignment, and the slot's worth that the last products of 16-channel boxes read beyond the slots
XBG_PLAN int wgrad_rows_fixed(int bn, int wc) { return 1024 + (wc == 16 ? 4 * WR_P * wc * 2 : 0) + WR_ND * WR_P * bn * 2; }
XBG_PLAN int wgrad_rows_bytes(int bn, int wc, int nx) { return wgrad_rows_fixed(bn, wc) + nx * 4 * WR_P * wc * 2; }
XBG_PLAN int wgrad_rows_smem(int bn, int wc, int nx) {
    return at_least(wgrad_rows_bytes(bn, wc, nx), wgrad_rows_cols(bn) > HALF_TCOLS ? HALF_SMEM : 0);
}
// input slots of rows of nseg chunks: the resident chunks and two to four copies
// ahead (0: k_wgrad_rows does not apply)
XBG_PLAN int wgrad_rows_slots(int bn, int wc, int nseg) {
    int nx = (WR_SMEM - wgrad_rows_fixed(bn, wc)) / (4 * WR_P * wc * 2);
    if (nx > 2 * nseg + 5) nx = 2 * nseg + 5;
    if (nx > WR_MX) nx = WR_MX;
    if (nx < 2 * nseg + 3) return 0;
    return nx;
}
// Where it pays: 32-channel boxes; 16-channel boxes for 16 input channels, and for
// more (a block each, with its own copy of the gradient's chunks) where the rows
// around a run are short: 48 -> 16 channels at 4 x 96 x 128 pixels 18.4 us by
// k_wgrad_tc, 14.7 here, but at 1 x 256 x 256 21.5 and 31.2, 48 -> 48 there 27.8 and
// 34.0.  Slices of under eight chunks are images of a few rows (128 -> 128 at 3 x 128
// pixels 12.1 there, 13.5 here).
XBG_PLAN bool wgrad_rows_pays(int cin, int nseg, int chunks_per_slice) {
    return (cin % 32 == 0 || cin == 16 || nseg <= 2) && chunks_per_slice >= 8;
}

}  // namespace nn
}  // namespace xbg
