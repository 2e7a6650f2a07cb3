// The randomized CholeskyQR kernels on clusters of 2 CTAs per matrix.
#define CQ_CS 2
#include "k_rcholqr.cu"
