// Line lengths of the two-pass stage: X(m, R1, R2) with m = R1 R2, the most
// even split into codelet lengths.  DFFT_FLEX_PLAIN_*: lengths transformed as
// they are; DFFT_FLEX_CHIRP_*: convolution lengths of the chirp-z form, those
// flex_chirp_length picks for some line (steps of about 7 % in the upper 3/8 of
// every octave).  In groups, one translation unit each per precision: the
// first use of a kernel loads the image of its group (10 ms for 19 lengths), so
// the lengths that have register kernels too, which plans of those try at
// creation, are one group (PLAIN_0); the others are of similar compile time.
#pragma once

#define DFFT_FLEX_PLAIN_0(X) \
  X(16, 4, 4) X(24, 6, 4) X(32, 8, 4) X(48, 8, 6) X(64, 8, 8) X(96, 12, 8) X(128, 16, 8) X(192, 16, 12) \
  X(256, 16, 16) X(384, 24, 16) X(512, 32, 16) X(768, 32, 24) X(1024, 32, 32)
#define DFFT_FLEX_PLAIN_1(X) \
  X(12, 4, 3) X(20, 5, 4) X(22, 11, 2) X(27, 9, 3) X(55, 11, 5) X(77, 11, 7) X(84, 12, 7) X(117, 13, 9) \
  X(130, 13, 10) X(135, 15, 9) X(165, 15, 11) X(198, 18, 11) X(200, 20, 10) X(320, 20, 16) X(405, 27, 15) \
  X(420, 21, 20) X(448, 28, 16) X(450, 25, 18) X(960, 32, 30)
#define DFFT_FLEX_PLAIN_2(X) \
  X(10, 5, 2) X(15, 5, 3) X(45, 9, 5) X(49, 7, 7) X(66, 11, 6) X(78, 13, 6) X(80, 10, 8) X(104, 13, 8) \
  X(125, 25, 5) X(126, 14, 9) X(156, 13, 12) X(182, 14, 13) X(216, 18, 12) X(252, 18, 14) X(336, 21, 16) \
  X(504, 24, 21) X(540, 27, 20) X(625, 25, 25) X(864, 32, 27)
#define DFFT_FLEX_PLAIN_3(X) \
  X(4, 2, 2) X(28, 7, 4) X(30, 6, 5) X(44, 11, 4) X(63, 9, 7) X(88, 11, 8) X(98, 14, 7) X(100, 10, 10) \
  X(112, 14, 8) X(154, 14, 11) X(176, 16, 11) X(210, 15, 14) X(250, 25, 10) X(280, 20, 14) X(324, 18, 18) \
  X(375, 25, 15) X(600, 25, 24) X(648, 27, 24) X(800, 32, 25)
#define DFFT_FLEX_PLAIN_4(X) \
  X(6, 3, 2) X(21, 7, 3) X(36, 6, 6) X(39, 13, 3) X(50, 10, 5) X(72, 9, 8) X(75, 15, 5) X(99, 11, 9) \
  X(132, 12, 11) X(147, 21, 7) X(150, 15, 10) X(160, 16, 10) X(224, 16, 14) X(360, 20, 18) X(378, 21, 18) \
  X(480, 24, 20) X(486, 27, 18) X(675, 27, 25) X(900, 30, 30)
#define DFFT_FLEX_PLAIN_5(X) \
  X(9, 3, 3) X(18, 6, 3) X(40, 8, 5) X(56, 8, 7) X(70, 10, 7) X(90, 10, 9) X(110, 11, 10) X(121, 11, 11) \
  X(143, 13, 11) X(169, 13, 13) X(189, 21, 9) X(195, 15, 13) X(225, 15, 15) X(243, 27, 9) X(300, 20, 15) \
  X(392, 28, 14) X(441, 21, 21) X(700, 28, 25) X(840, 30, 28)
#define DFFT_FLEX_PLAIN_6(X) \
  X(25, 5, 5) X(26, 13, 2) X(42, 7, 6) X(54, 9, 6) X(81, 9, 9) X(91, 13, 7) X(108, 12, 9) X(144, 12, 12) \
  X(162, 18, 9) X(168, 14, 12) X(175, 25, 7) X(180, 15, 12) X(288, 18, 16) X(294, 21, 14) X(350, 25, 14) \
  X(576, 24, 24) X(640, 32, 20) X(720, 30, 24)
#define DFFT_FLEX_PLAIN_7(X) \
  X(8, 4, 2) X(14, 7, 2) X(33, 11, 3) X(35, 7, 5) X(52, 13, 4) X(60, 10, 6) X(65, 13, 5) X(105, 15, 7) \
  X(120, 12, 10) X(140, 14, 10) X(196, 14, 14) X(240, 16, 15) X(270, 18, 15) X(315, 21, 15) X(400, 20, 20) \
  X(432, 24, 18) X(500, 25, 20) X(750, 30, 25) X(810, 30, 27)
#define DFFT_FLEX_CHIRP_0(X) \
  X(48, 8, 6) X(112, 14, 8) X(200, 20, 10) X(256, 16, 16) X(400, 20, 20) X(480, 24, 20) X(1024, 32, 32)
#define DFFT_FLEX_CHIRP_1(X) \
  X(60, 10, 6) X(120, 12, 10) X(210, 15, 14) X(320, 20, 16) X(420, 21, 20) X(512, 32, 16) X(960, 32, 30)
#define DFFT_FLEX_CHIRP_2(X) \
  X(64, 8, 8) X(128, 16, 8) X(224, 16, 14) X(336, 24, 14) X(448, 28, 16) X(784, 28, 28) X(900, 30, 30)
#define DFFT_FLEX_CHIRP_3(X) \
  X(96, 12, 8) X(192, 16, 12) X(240, 16, 15) X(360, 24, 15) X(720, 30, 24) X(840, 30, 28)
