// The randomized CholeskyQR kernels on clusters of 4 CTAs per matrix.
#define CQ_CS 4
#include "k_rcholqr.cu"
