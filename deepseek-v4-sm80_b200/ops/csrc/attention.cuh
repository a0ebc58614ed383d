// What the sparse latent attention kernels (attention.cu, attention_mma.cu) are given.
#pragma once
#include "common.cuh"
#include "rope.cuh"

struct AttnArgs {
  const __nv_bfloat16* q;
  __nv_bfloat16* o;
  const int* slots;
  const int* pos;
  const int* page_table;
  int ld_pt;
  const __nv_bfloat16* swa;
  const int* swa_map;
  const __nv_bfloat16* comp;
  const int* topk_idx;
  const int* topk_len;
  int topk_width;
  int mode;   // 0: window only, 1: compressed entries from topk_idx, 2: all compressed entries
  int ratio;
  const float* sink;
  float scale;
  int ps;
  int window;
  const int* num_valid;
  int out_rope;   // != 0: rotate the last rp.rotary_dim dims of every output head row by -position (the inverse
  RopeParams rp;  //       RoPE the output projection expects), on the bf16-rounded values, in the epilogue
  int nsplit;        // CTAs per token (grid.y); > 1 needs the three buffers below
  float* part_acc;   // [t][nsplit][HL][512] unnormalised accumulators
  float* part_ml;    // [t][nsplit][HL][2]   running max and sum
  int* counters;     // [t] zero between launches (attention.cu)
};

int launch_attn_mma(const AttnArgs& a, int t, cudaStream_t st);   // 64 heads
