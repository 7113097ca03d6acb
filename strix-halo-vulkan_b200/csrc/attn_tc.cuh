// Causal attention of a many-row pass of one sequence on the tensor cores (prefill). See attn_tc.cu.
#pragma once
#include "kernels.cuh"
#include "tgemm.cuh"

namespace b200 {

// query rows [rows][Hq][hd] and a layer's caches [slots * n_kv][Hkv][hd]
struct AttnTcMaps { TMap q, k, v; };
bool attn_tc_shape(int Hq, int Hkv, int hd);
inline bool attn_tc_fits(const AttnParams& p) { return attn_tc_shape(p.Hq, p.Hkv, p.hd) && p.M >= 16; }
int make_attn_maps(const __half* q16, int64_t rows, int Hq, const __half* kcache, const __half* vcache, int64_t cells, int Hkv, int hd, AttnTcMaps* out);
// Rows [0, p.M) sit at consecutive positions of one slot, the last at `last_pos`. partial_floats: room behind p.partial; where the query
// tiles leave SMs idle the keys are cut into as many parts as fit there, and p.split_cells / p.nsplit come back as launch_attn_merge
// wants them. p.nsplit comes back 0 when the rows are finished.
int launch_attn_tc(AttnParams& p, const AttnTcMaps& maps, int last_pos, int64_t partial_floats, bool pdl, cudaStream_t st);

}  // namespace b200
