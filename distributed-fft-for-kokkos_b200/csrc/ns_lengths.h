// Axis lengths of the Navier-Stokes line kernels: X(n, R1, R2) with n = R1 R2,
// the most even split into codelet lengths.  46 2^a 3^b 5^c lengths up to 512; a
// grid with another length on any axis runs on the plan's transforms (2.6 times
// slower at 192^3 complex64).  In groups of similar compile time,
// one translation unit each per precision.
#pragma once

#define DFFT_NS_LENGTHS_0(X) \
  X(8, 4, 2) X(12, 4, 3) X(30, 6, 5) X(36, 6, 6) X(54, 9, 6) X(96, 12, 8) X(100, 10, 10) X(160, 16, 10) \
  X(240, 16, 15) X(256, 16, 16) X(320, 20, 16) X(512, 32, 16)
#define DFFT_NS_LENGTHS_1(X) \
  X(15, 5, 3) X(24, 6, 4) X(32, 8, 4) X(64, 8, 8) X(90, 10, 9) X(108, 12, 9) X(150, 15, 10) X(216, 18, 12) \
  X(300, 20, 15) X(360, 20, 18) X(500, 25, 20)
#define DFFT_NS_LENGTHS_2(X) \
  X(16, 4, 4) X(20, 5, 4) X(48, 8, 6) X(50, 10, 5) X(72, 9, 8) X(128, 16, 8) X(144, 12, 12) X(200, 20, 10) \
  X(288, 18, 16) X(400, 20, 20) X(480, 24, 20)
#define DFFT_NS_LENGTHS_3(X) \
  X(9, 3, 3) X(10, 5, 2) X(25, 5, 5) X(40, 8, 5) X(60, 10, 6) X(80, 10, 8) X(120, 12, 10) X(180, 15, 12) \
  X(192, 16, 12) X(250, 25, 10) X(384, 24, 16) X(432, 24, 18)
