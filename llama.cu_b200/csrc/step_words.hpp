// Token and error word of a step, on their way from the GPU's last kernel to the host: one 64-bit word of pinned memory, written by one
// store and read by one load.  Two words of 32 bits have no order between them, in one vector store either, and the host could
// take the token of the step before for the one whose error word it has just seen.  The token is the lower half: the two words lie in
// memory as they do in the GPU's state, so that a copy of 8 bytes gives the same.
#pragma once
#include <cstdint>

namespace lcu {

constexpr int NOT_BACK = -1;  // in place of an error word, which is 0 or positive: nothing has come yet
struct step_words {
  int token = 0, code = NOT_BACK;
  bool came() const { return code != NOT_BACK; }
};

#ifdef __CUDACC__
__host__ __device__
#endif
constexpr uint64_t packed_words(int token, int code) {
  return (uint64_t)(uint32_t)code << 32 | (uint32_t)token;
}
inline void clear_words(uint64_t* at) { __atomic_store_n(at, packed_words(0, NOT_BACK), __ATOMIC_RELEASE); }
inline step_words read_words(const uint64_t* at) {  // what was written before the words is seen behind them
  const uint64_t v = __atomic_load_n(at, __ATOMIC_ACQUIRE);
  step_words w;
  w.token = (int)(uint32_t)v;
  w.code = (int)(uint32_t)(v >> 32);
  return w;
}

}  // namespace lcu
