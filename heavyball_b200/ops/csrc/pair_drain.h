// Bookkeeping for the teardown of a pair of CTAs that gave up on a wait (device code, and a CPU test of the protocol).
//
// A ring fill of the pair is one phase of the even CTA's barrier for its stage: one arrival, by the even producer, that announces
// the bytes of both CTAs' loads, and those bytes as they land.  When the producers stop at different fills, the phase of a fill
// that only one of them issued cannot complete by itself: the even CTA then supplies what is missing and waits for the rest.
#pragma once

#ifdef __CUDACC__
#define HB_HOST_DEVICE __host__ __device__
#else
#define HB_HOST_DEVICE
#endif

namespace hb {

enum PairFill : int {
  kFillBoth = 0,      // loads and announcement complete the phase
  kFillEvenOnly = 1,  // announced for both: the odd CTA's bytes have to be counted off
  kFillOddOnly = 2    // not announced: an arrival that expects the odd CTA's bytes is missing
};

// The first fill that may still be landing, from the numbers of fills that the two producers issued: a stage is filled again only
// after a product has read it, so everything before the last `stages` fills has landed.
HB_HOST_DEVICE inline int pair_drain_first(int fills_even, int fills_odd, int stages) {
  const int top = fills_even > fills_odd ? fills_even : fills_odd;
  return top > stages ? top - stages : 0;
}
HB_HOST_DEVICE inline int pair_fill_kind(int fill, int fills_even, int fills_odd) {
  return fill >= fills_even ? kFillOddOnly : fill >= fills_odd ? kFillEvenOnly : kFillBoth;
}

}  // namespace hb
