// tmpl_spectra.cuh — per-angle FP32 template spectra in two kernels (tmpl_spectra.cu).
#pragma once

#include "common.cuh"

namespace gisspa {

struct TmplSpectra {
  const float* src;      // prepared templates, [.][l][l]
  int nt, na;            // templates, angles: image v = a nt + t is template t at angle a
  const int* list;       // device list of n_list pairs (g: images 2 g, 2 g + 1), or null: all
  int n_list;
  float cose, sine;      // the angle (na = 1), unless st holds the na angles in device memory
  const AngleState* st;
  const float* pre;      // tmpl_prescale, by template
  const float* mask;     // mask_table
  const float2* twL;     // twiddles of length l
  float2* F;             // scratch, [pairs][l][l]
  double* sums;          // [pairs][4]: both templates' sum and sum of squares
  bool paired;           // out: interleaved pairs (corr_pair.cu), or one half spectrum per template
  void* out;             // at each image's own index
};
bool tmpl_spectra_supported(int l);
void tmpl_spectra(int l, const TmplSpectra& p, cudaStream_t s);
// The templates' power-of-two scales (p: src, nt, mask, twL and the scratch buffers).
void tmpl_prescale(int l, TmplSpectra p, float* pre, cudaStream_t s);

}  // namespace gisspa
