// The axis lengths with register passes, N = A * B (A a multiple of 4, both at
// most 32), in groups of about equal compile time (one translation unit
// each).  X(N, A, B, MAIN): MAIN lengths have kernels specialised for twofold
// oversampling too.
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
