// Prefill products (qgemm.cu) and their kernel on CTA pairs (qgemm_pair.cu).
#pragma once

#include "common.cuh"

// RMSNorm of the rows in front of a product: (x + res) / rms * w (res may be null; rows contiguous, of the product's K)
struct fb200_row_norm {
  const float *res, *w;
  float eps;
};
// whether fb200_qgemm takes a product of these rows (the epilogue aside)
bool fb200_qgemm_covers(const fb200_qmatrix* w, const float* x, size_t m, const fb200_row_norm* norm = nullptr);
int fb200_qgemm(fb200_device* dev, const fb200_qmatrix* w, const float* x, size_t m, float* y, bool r1_is_bias, const float* r1,
                const float* r2, int swiglu, const fb200_row_norm* norm = nullptr);
int fb200_qgemm_group(fb200_device* dev, const fb200_qmatrix* const* ws, float* const* ys, int n, const float* x, size_t m,
                      const fb200_row_norm* norm = nullptr);

struct PairArgs {
  const uint8_t* w;      // tiled weights
  const __half* xh;      // fp16 activations, [x_halves][K / 64] tiles of 128 rows in the operand layout
  const float* xscale;   // [M] power-of-two scale of each row
  float* y;              // [M, N]; with splits > 1 the partial product of range z goes to y + z M N
  const float* r1;       // optional residuals [M, N], or one bias row [N] when r1_stride is 0
  const float* r2;
  int r1_stride;
  int M, N;
  int ngroups, ntiles;   // K groups per row-tile, 16-row tiles of W
  int pair_tiles;        // SwiGLU: up rows lie this many row-tiles behind their gate rows, y is [M, N / 2]; 0: plain product
  int m_tiles, n_tiles;  // tiles of 256 activation rows and of nw weight rows (SwiGLU: nw / 2 outputs)
  int splits, kg_per;    // K ranges, K groups per range (every range holds at least one)
  int x_halves;          // 128-row tiles in xh
  int vec;               // rows of y and of the residuals are 8-byte aligned
  int* status;
};

// Launches the product with nw = 128 or 256 weight rows per tile; 1 when the type has no kernel. `early`: it may start while the
// kernel in front on the stream (which packs its activations) still runs.
int fb200_qgemm_pair(fb200_device* dev, int nw, uint32_t type, const PairArgs& a, bool early);
