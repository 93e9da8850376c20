// What a captured decode step does around the model, one launch in front of it and one behind: cache slots, context lengths
// and embedding rows of the batch, then the new tokens into the batch state and the output ring.  A few hundred bytes per
// request: the launches are what counts (as tensor operations they were twenty, 1.2 us and a launch gap each).
#include "host_utils.h"

namespace gkds {
using namespace gk;

struct BeginParams {
  const long long* tokens;   // [B]
  const int* pos;            // [B]
  const unsigned char* active;
  const int* limit;          // positions below it have cache reserved
  const int* table;          // [B, max_blocks]
  const int* state;          // [B] or null
  const uint4* embed;        // [vocab, row_vec] or null
  int* slots;                // [B] cache row, -1 without one
  int* ctx;                  // [B] tokens seen with this one, 0 for a row that rests
  int* state_out;            // [B] with `state`: -1 for a row that rests
  long long* sink_slots;     // [B] or null: slots, `sink` where there is none
  uint4* x;                  // [B, row_vec] with `embed`
  long long vocab, sink;
  int max_blocks, block, row_vec;
};

__global__ void __launch_bounds__(128) decode_begin_kernel(const BeginParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x;
  if (threadIdx.x == 0) {
    // a request at its length limit has no cache behind it: the rest of the interval is discarded, nothing is stored
    const int pos = p.pos[b];
    const bool live = p.active[b] && pos < p.limit[b];
    int k = pos / p.block;
    if (k > p.max_blocks - 1) k = p.max_blocks - 1;
    const int slot = live ? p.table[static_cast<long long>(b) * p.max_blocks + k] * p.block + pos % p.block : -1;
    p.slots[b] = slot;
    p.ctx[b] = live ? pos + 1 : 0;
    if (p.state) p.state_out[b] = live ? p.state[b] : -1;
    if (p.sink_slots) p.sink_slots[b] = slot >= 0 ? slot : p.sink;
  }
  if (p.embed) {
    const long long t = p.tokens[b];
    const bool known = t >= 0 && t < p.vocab;
    for (int c = threadIdx.x; c < p.row_vec; c += blockDim.x)
      p.x[static_cast<long long>(b) * p.row_vec + c] = known ? p.embed[t * p.row_vec + c] : make_uint4(0, 0, 0, 0);
  }
}

struct EndParams {
  const long long* tok;   // [B] drawn
  const float* lp;
  const unsigned char* active;
  long long* tokens;      // [B] batch state
  int* pos;
  int* steps;
  long long* ring_idx;    // [1]
  long long* ring_tok;    // [R, B]
  float* ring_lp;
  int B, R;
};

__global__ void __launch_bounds__(256) decode_end_kernel(const EndParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const long long at = *p.ring_idx % p.R * p.B;
  for (int b = threadIdx.x; b < p.B; b += blockDim.x) {
    const long long t = p.tok[b];
    p.tokens[b] = t;
    p.ring_tok[at + b] = t;
    p.ring_lp[at + b] = p.lp[b];
    p.pos[b] += p.active[b] ? 1 : 0;
    p.steps[b] += 1;
  }
  __syncthreads();   // every thread has read the index
  if (threadIdx.x == 0) *p.ring_idx += 1;
}

}  // namespace gkds

using namespace gkds;

// ptrs: {tokens, pos, active, limit, table, state, embed, slots, ctx, state_out, sink_slots, x} (state with state_out, embed
// with x, sink_slots: optional); dims: {B, max_blocks, block, bytes of an embedding row (a multiple of 16), vocab, sink}
GK_EXPORT int gk_decode_begin(void* const* ptrs, const long long* dims, void* stream) {
  if (dims[0] == 0) return 0;
  if (dims[0] < 0 || dims[1] < 1 || dims[2] < 1 || dims[3] % 16) return -1;
  BeginParams p;
  p.tokens = static_cast<const long long*>(ptrs[0]); p.pos = static_cast<const int*>(ptrs[1]);
  p.active = static_cast<const unsigned char*>(ptrs[2]); p.limit = static_cast<const int*>(ptrs[3]);
  p.table = static_cast<const int*>(ptrs[4]); p.state = static_cast<const int*>(ptrs[5]);
  p.embed = static_cast<const uint4*>(ptrs[6]); p.slots = static_cast<int*>(ptrs[7]); p.ctx = static_cast<int*>(ptrs[8]);
  p.state_out = static_cast<int*>(ptrs[9]); p.sink_slots = static_cast<long long*>(ptrs[10]); p.x = static_cast<uint4*>(ptrs[11]);
  p.max_blocks = static_cast<int>(dims[1]); p.block = static_cast<int>(dims[2]); p.row_vec = static_cast<int>(dims[3] / 16);
  p.vocab = dims[4]; p.sink = dims[5];
  launch_k(decode_begin_kernel, dim3(static_cast<unsigned>(dims[0])), dim3(128), 0, reinterpret_cast<cudaStream_t>(stream), p);
  return launch_status();
}

// ptrs: {tok, lp, active, tokens, pos, steps, ring_idx, ring_tok, ring_lp}
GK_EXPORT int gk_decode_end(void* const* ptrs, int B, int R, void* stream) {
  if (B < 1 || R < 1) return -1;
  EndParams p;
  p.tok = static_cast<const long long*>(ptrs[0]); p.lp = static_cast<const float*>(ptrs[1]);
  p.active = static_cast<const unsigned char*>(ptrs[2]); p.tokens = static_cast<long long*>(ptrs[3]);
  p.pos = static_cast<int*>(ptrs[4]); p.steps = static_cast<int*>(ptrs[5]); p.ring_idx = static_cast<long long*>(ptrs[6]);
  p.ring_tok = static_cast<long long*>(ptrs[7]); p.ring_lp = static_cast<float*>(ptrs[8]);
  p.B = B; p.R = R;
  launch_k(decode_end_kernel, dim3(1), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream), p);
  return launch_status();
}
