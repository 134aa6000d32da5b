// K = R1 R2 of the two-factor transforms: every 2^a 3^b 5^c from 16 to 256, with the pair
// of smallest larger factor (fewest registers, most threads).
#pragma once

#define SPME_FFT_LIST(X)                                                                    \
    X(4, 4) X(6, 3) X(5, 4) X(6, 4) X(5, 5) X(9, 3) X(6, 5) X(8, 4) X(6, 6) X(8, 5) X(9, 5)   \
    X(8, 6) X(10, 5) X(9, 6) X(10, 6) X(8, 8) X(9, 8) X(15, 5) X(10, 8) X(9, 9) X(10, 9)      \
    X(12, 8) X(10, 10) X(12, 9) X(12, 10) X(25, 5) X(16, 8) X(15, 9) X(12, 12) X(15, 10)     \
    X(16, 10) X(18, 9) X(15, 12) X(16, 12) X(20, 10) X(18, 12) X(15, 15) X(16, 15) X(27, 9)  \
    X(25, 10) X(16, 16)
