// The gated delta rule in chunks: what its kernels (delta_chunks.cu) and the rows of a chunk (linear_chunks.cu) share.
#pragma once
#include "common.cuh"

struct DeltaChunkArgs {
  const float* rows;           // [T, row_stride]: q of group g at g d, k at k_col + g d, v of head h at v_col + h dv
  long long row_stride;
  int k_col, v_col;
  const float* beta;           // [T, H]
  const float* decay;          // [T, H]
  float* state;                // [slots, H, dv, d]
  float* scratch;              // [tiles][H][dv][d]: the state before a tile
  float* factor;               // [2 tiles][H]: a chunk's whole decay
  float* w;                    // [2 tiles][H][64 D]
  float* k;                    // [2 tiles][G][64 D]
  float* tail;                 // [T, H]: what a chunk's end leaves of the token's write
  float* o_raw;                // [T, H dv]: V', then U, then the result
  const int* tile_seq;         // tiles of 128 tokens: sequence and first token of its portion; a sequence's side by side in their order
  const int* tile_q0;
  int tiles;
  const int* cu_q_lens;
  const int* context_lens;
  const int* state_slots;
  int T, B, G, H, d, dv, heads;   // heads: of one block of delta_solve (they share k)
  int* status;
};

// linear_chunks.cu: the rows of every tile from the states and U; the result takes U's place.
bool delta_rows_supported(const DeltaChunkArgs& p);
int delta_rows(const DeltaChunkArgs& p, cudaStream_t stream);
