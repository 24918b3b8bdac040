// Host check of the exchange slots of colore_gb300/csrc/fft.cuh: for every
// column and row plan of fft_plans.h, padded, pad_at splits each exchange access into
// base and offset without changing the slot p + (p >> sh), the slots are
// distinct and below pad_len, and stage 0's writes by 16 consecutive threads
// of one column fall into 16 different float2 bank pairs.
#include <cstdio>
#include <set>

#include "fft.cuh"
#include "fft_plans.h"

template <int L, int R, int r0, int r1, int r2>
static int check_plan()
{
  constexpr int SH = cgfft::pad_shift(r0), P = L / R;
  int bad = 0;
  auto slot = [](int p) { return p + (p >> SH); };
  std::set<int> seen;
  for (int p = 0; p < L; p++) {
    seen.insert(slot(p));
    bad += slot(p) >= cgfft::pad_len(L, SH);
  }
  bad += (int)seen.size() != L;
  for (int t = 0; t < P; t++) {
    for (int i = 0; i < R / r0; i++)
      for (int q = 0; q < r0; q++)
        bad += cgfft::pad_at<SH>((t + P * i) * r0, q, true) != slot(cgfft::out_pos<L, R, r0, 1>(t, i, q));
    for (int i = 0; i < R / r1; i++)
      for (int q = 0; q < r1; q++) {
        bad += cgfft::pad_at<SH>(t, P * i + q * (L / r1), false) != slot(cgfft::in_pos<L, R, r1>(t, i, q));
        if (r2 > 1)
          bad += cgfft::pad_at<SH>(cgfft::out_pos<L, R, r1, r0>(t, i, 0), q * r0, false) !=
                 slot(cgfft::out_pos<L, R, r1, r0>(t, i, q));
      }
    for (int i = 0; r2 > 1 && i < R / r2; i++)
      for (int q = 0; q < r2; q++)
        bad += cgfft::pad_at<SH>(t, P * i + q * (L / r2), false) != slot(cgfft::in_pos<L, R, r2>(t, i, q));
  }
  std::set<int> banks;
  for (int t = 0; t < 16; t++) banks.insert(cgfft::pad_at<SH>(t * r0, 0, true) % 16);
  return bad + (banks.size() != 16);
}

template <int N>
static void check_size()
{
  using PL = Plan<N>;
  printf("%d %d\n", N,
         check_plan<N, PL::CR, PL::C0, PL::C1, PL::C2>() + check_plan<N, PL::FR, PL::F0, PL::F1, PL::F2>() +
             check_plan<N / 2, PL::RR, PL::R0, PL::R1, PL::R2>());
}

int main()
{
  check_size<64>();
  check_size<96>();
  check_size<128>();
  check_size<192>();
  check_size<256>();
  check_size<384>();
  check_size<512>();
  check_size<1024>();
  check_size<2048>();
  return 0;
}
