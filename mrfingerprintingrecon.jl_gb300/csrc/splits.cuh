// Line lengths with compiled two-step register kernels, L = R1 * R2 (fft4.cuh): X(L, R1, R2).
// Every even 2, 3, 5-smooth length from 64 to 768 whose factors the register transforms have
// (486 and 648 would need 27 points), and 1024; R1 even, so that the zero-padded half of a line
// is the first R1 / 2 inputs of a step-A task.  Other lengths run the generic shared-memory
// kernels (fft.cuh), whose stages are divisions, barriers and two buffers (half the CTAs an SM):
// 180 x 150, 12 coils, complex K = 3, an apply takes 152 us there and 48 us here.  Factors that are
// products without a common factor are taken where there are such, as their DFTs need no twiddles:
// 288 as 12 * 24 has an error of 2.07e-7 (Cartesian 288^2; generic kernels 2.29e-7), as 16 * 18
// 2.42e-7, and takes 51.9 against 55.4 us (zero-padded 144^2 35.8 against 33.0).  Zero-padded 60^2,
// 8 coils: 120 as 8 * 15 has an error of 7.0e-8, as 10 * 12 8.2e-8; 160^2: 320 as 20 * 16 8.6e-8 and
// 30.8 us, as 16 * 20 9.5e-8 and 33.2 us.  In groups, one
// translation unit per group and kernel family.
#pragma once

#define MRSR_SPLITS_0(X) X(64, 8, 8) X(128, 8, 16) X(256, 16, 16) X(384, 12, 32) X(512, 16, 32) X(768, 24, 32) X(1024, 32, 32)
#define MRSR_SPLITS_1(X) X(72, 6, 12) X(80, 8, 10) X(90, 6, 15) X(96, 8, 12) X(100, 10, 10) X(108, 6, 18) X(120, 8, 15)
#define MRSR_SPLITS_2(X) X(144, 12, 12) X(150, 10, 15) X(160, 8, 20) X(162, 18, 9) X(180, 12, 15) X(192, 12, 16) X(200, 10, 20)
#define MRSR_SPLITS_3(X) X(216, 12, 18) X(240, 16, 15) X(250, 10, 25) X(270, 18, 15) X(288, 12, 24) X(300, 20, 15) X(320, 20, 16)
#define MRSR_SPLITS_4(X) X(324, 18, 18) X(360, 18, 20) X(400, 20, 20) X(432, 18, 24) X(450, 18, 25) X(480, 20, 24) X(500, 20, 25)
#define MRSR_SPLITS_5(X) X(540, 18, 30) X(576, 24, 24) X(600, 24, 25) X(640, 20, 32) X(720, 24, 30) X(750, 30, 25)
#define MRSR_SPLITS(X) MRSR_SPLITS_0(X) MRSR_SPLITS_1(X) MRSR_SPLITS_2(X) MRSR_SPLITS_3(X) MRSR_SPLITS_4(X) MRSR_SPLITS_5(X)

namespace mrsr {
// R1 of the compiled split of L, 0 if none
inline int split_r1(int L) {
  switch (L) {
#define MRSR_CASE(L_, R1_, R2_) case L_: return R1_;
    MRSR_SPLITS(MRSR_CASE)
#undef MRSR_CASE
    default: return 0;
  }
}
inline bool split_length(int L) { return split_r1(L) != 0; }
}  // namespace mrsr
