// Shared by the chunkwise kernel (mlstm_chunkwise.cu) and the kernels that split long documents into parts
// (mlstm_parts.cu): tensor maps, chunk constants, the description of a split and small device helpers.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace xl {

constexpr int CW_L = 64;         // tokens per chunk
constexpr int CW_DV = 128;       // value columns per CTA (UMMA M)
constexpr int CW_BOX_BYTES = 64 * 128;  // one TMA box: 64 rows x 64 bf16

struct CwMaps {
  CUtensorMap q, k, v;
  // position (1..3) of the token / head / batch coordinate in each map; the outer dimensions are ordered by
  // ascending stride, which differs between a contiguous (B,NH,S,D) tensor and a transposed (B,S,NH,D) view
  int pos[3][3];  // [q|k|v][token|head|batch]
};

// The three outer coordinates of token `tk` in map `t` (selects: arrays indexed by pos would live in local memory, and the
// issuing thread's latency is on the path of every stage)
__device__ __forceinline__ int cw_coord(const CwMaps& maps, int t, int i, int tk, int head, int b) {
  return maps.pos[t][0] == i ? tk : (maps.pos[t][1] == i ? head : b);
}

// A document walked by ONE thread block per (head, value slice) is a serial chain of chunks.  Where there are too few
// chains for the machine, documents are cut into parts of whole chunks that run side by side: `mlstm_part_state_kernel`
// first forms the state every part but the last adds on its own (C_loc = sum_l w_l k_l v_l^T over the part, n_loc, and in
// log space the part's decay g and stabiliser), and the chunkwise kernel starts part j from the initial state folded with
// the parts in front of it.
constexpr int CW_MAX_PARTS = 32;
constexpr int CW_MAX_PART_CHUNKS = 128;   // (the part state kernel keeps the weight of every token in shared memory)

struct CwItem {   // one part of a document
  int doc, part, parts, first_chunk, chunks;
  int slot0;      // slot of the document's first part in c_loc / n_loc / gm (part j < parts - 1: slot0 + j)
};

struct CwSplit {
  const int* counts;      // packed batches: {items, slots} the plan kernel found; NULL: rows of equal length
  const CwItem* items;    // longest first
  const CwItem* slots;    // the part behind every slot
  int after_states;       // the launch in front is mlstm_part_state_kernel: only parts behind a document's first wait for it
  int parts, part_chunks; // equal rows: parts per row (1 = no split) and chunks per part
  float* c_loc;           // [slot][NH][value slice][DHQK / 4][128][4]: what a tensor-memory lane (value column) holds, in 16-byte pieces
  float* n_loc;           // [slot][NH][DHQK]
  float2* gm;             // [slot][NH]: (sum of log f, stabiliser of the part's own state)
};

__device__ __forceinline__ float fast_log_sigmoid(float x) { return fminf(x, 0.f) - __logf(1.f + __expf(-fabsf(x))); }

// 16 bytes of bf16 times a bf16x2 splat, rounded once per product
__device__ __forceinline__ uint4 scale_bf16x8(uint4 raw, __nv_bfloat162 s) {
  __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&raw);
  p[0] = __hmul2(p[0], s);
  p[1] = __hmul2(p[1], s);
  p[2] = __hmul2(p[2], s);
  p[3] = __hmul2(p[3], s);
  return raw;
}

__device__ __forceinline__ CwItem cw_load_item(const CwItem* p) {
  const int* w = reinterpret_cast<const int*>(p);
  return {__ldcg(w), __ldcg(w + 1), __ldcg(w + 2), __ldcg(w + 3), __ldcg(w + 4), __ldcg(w + 5)};
}

// offset, in 16-byte pieces, of the (slot, head, value slice) block of c_loc
template <int DHQK>
__device__ __forceinline__ long long cw_c_loc_offset(const xl_mlstm_seq_params& p, int slot, int head, int slice) {
  return (((long long)slot * p.NH + head) * (p.DHV / CW_DV) + slice) * (DHQK / 4 * CW_DV);
}

// Document `doc` -> (batch row, first token, length)
__device__ __forceinline__ void cw_document(const xl_mlstm_seq_params& p, int doc, int& b, long long& tok0, long long& len) {
  if (p.cu_seqlens) {
    const long long s = __ldcg(p.cu_seqlens + doc), e = __ldcg(p.cu_seqlens + doc + 1);
    b = (int)(s / p.S);
    tok0 = s - (long long)b * p.S;
    len = e - s;
  } else {
    b = doc; tok0 = 0; len = p.S;
  }
}

// mlstm_parts.cu
int64_t cw_split_scratch_bytes(const xl_mlstm_seq_params* p);
int cw_prepare_split(const CwMaps& maps, const xl_mlstm_seq_params* p, void* scratch, int64_t scratch_bytes, CwSplit* split, unsigned* grid_z,
                     cudaStream_t st);

}  // namespace xl
