// The axis lengths with register passes, N = A * B (A a multiple of 4, both at
// most 32), in groups of about equal compile time (one translation unit
// each).  In: the lengths from 16 to 768 with prime factors up to 7 that split so
// (20, 28 and 36 aside), and 800, 896, 960 and 1024.  784, 840 and 864 would split
// too and are not built; lengths with factors 11 and 13 (176, 208, 352, 416) have
// no sub-transforms here: they run the direct DFT, as all but 2^k and 3 * 2^k did.
// Against the shared-memory passes (sum of the passes of a forward and an adjoint,
// us, twofold oversampling): 16^3 x 8 coils 45 / 46, 32^3 x 16 50 / 53, 48^3 x 8 49
// / 55, 512^2 x 12 64 / 125, 768^2 x 8 84 / 126, 1024^2 x 4 80 / 178; 96 to 192
// points: shared_pass_faster in mlg_fft.cu.
//
// X(N, A, B, MAIN): MAIN lengths have kernels specialised for twofold
// oversampling and, with sub-transforms of up to 16 points, two columns per thread
// too, for three times the kernels: the grids of the matrix sizes most in use (32
// to 64 in steps of 8, 72 to 256; no rule on the length's factors).  What
// the others lose in 3-D, ps per grid value over the six passes, 8 coils: 108 13.5,
// 168 9.3, 180 9.1, 200 12.0, 216 10.8 beside 112 11.1, 160 8.3, 192 7.2, 224 6.6;
// long sub-transforms more (140 15.8, 196 20.3, 252 14.4).  In 2-D nothing to 5 %
// (a launch's latency each: 336^2 x 8 coils 52.7, 320^2 52.6, 420^2 38.2, 400^2 36.1).
#pragma once

#define MLG_REG_GROUP_0(X) \
  X(84, 12, 7, false) \
  X(280, 20, 14, false) \
  X(448, 28, 16, false) \
  X(512, 16, 32, true) \
  X(600, 24, 25, false)
#define MLG_REG_GROUP_1(X) \
  X(32, 8, 4, false) \
  X(108, 12, 9, false) \
  X(120, 12, 10, true) \
  X(300, 20, 15, false) \
  X(480, 20, 24, true) \
  X(672, 24, 28, false)
#define MLG_REG_GROUP_2(X) \
  X(56, 8, 7, false) \
  X(80, 8, 10, true) \
  X(100, 20, 5, false) \
  X(160, 16, 10, true) \
  X(384, 24, 16, true) \
  X(500, 20, 25, false)
#define MLG_REG_GROUP_3(X) \
  X(48, 8, 6, false) \
  X(168, 12, 14, false) \
  X(196, 28, 7, false) \
  X(400, 20, 20, true) \
  X(504, 24, 21, false) \
  X(640, 20, 32, false)
#define MLG_REG_GROUP_4(X) \
  X(112, 16, 7, true) \
  X(252, 12, 21, false) \
  X(320, 20, 16, true) \
  X(336, 16, 21, false) \
  X(720, 24, 30, false)
#define MLG_REG_GROUP_5(X) \
  X(16, 4, 4, false) \
  X(64, 8, 8, true) \
  X(288, 16, 18, true) \
  X(360, 20, 18, false) \
  X(540, 20, 27, false) \
  X(768, 24, 32, false)
#define MLG_REG_GROUP_6(X) \
  X(24, 4, 6, false) \
  X(144, 12, 12, true) \
  X(216, 12, 18, false) \
  X(256, 16, 16, true) \
  X(420, 20, 21, false) \
  X(800, 32, 25, false)
#define MLG_REG_GROUP_7(X) \
  X(60, 12, 5, false) \
  X(128, 16, 8, true) \
  X(140, 20, 7, false) \
  X(192, 16, 12, true) \
  X(432, 24, 18, false) \
  X(1024, 32, 32, false)
#define MLG_REG_GROUP_8(X) \
  X(72, 8, 9, false) \
  X(96, 12, 8, true) \
  X(180, 12, 15, false) \
  X(224, 16, 14, true) \
  X(240, 16, 15, true) \
  X(560, 20, 28, false)
#define MLG_REG_GROUP_9(X) \
  X(40, 8, 5, false) \
  X(200, 20, 10, false) \
  X(324, 12, 27, false) \
  X(576, 24, 24, false) \
  X(896, 28, 32, false) \
  X(960, 32, 30, false)
#define MLG_REG_GROUP_10(X) \
  X(392, 28, 14, false) \
  X(588, 28, 21, false) \
  X(648, 24, 27, false) \
  X(700, 28, 25, false) \
  X(756, 28, 27, false)
#define MLG_REG_ALL(X) \
  MLG_REG_GROUP_0(X) MLG_REG_GROUP_1(X) MLG_REG_GROUP_2(X) MLG_REG_GROUP_3(X) MLG_REG_GROUP_4(X) MLG_REG_GROUP_5(X) MLG_REG_GROUP_6(X) MLG_REG_GROUP_7(X) MLG_REG_GROUP_8(X) MLG_REG_GROUP_9(X) MLG_REG_GROUP_10(X)
