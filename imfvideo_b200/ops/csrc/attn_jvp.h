// Host-side interface of the head_dim-64 attention forward with tangent (attn_jvp.cu); the public
// entry point imf_attn_fwd (attn_fwd.cu) dispatches here when tangents are given.
#pragma once
#include "attn_fwd128.h"

namespace imf {

typedef Fwd128Args JvpArgs;      // the same arguments; tensors (B, L, H, 64), dq, dk, dv and dout given

long attn_jvp_scratch_bytes(int B, int L, int H);
int attn_jvp_launch(const JvpArgs& a);

}  // namespace imf
