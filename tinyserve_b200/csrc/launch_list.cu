// Runs the launches of many layers that differ in nothing but their tensors: a step that is not replayed from a recording
// spends 14 to 17 us of the host's time on each of some 230 launches in the interpreter (2,048 tokens of 28 dense layers:
// 3.9 ms for 3.4 ms of work on the device); a launch run from here takes what the CUDA runtime takes for it.
//
// The caller has made the launches of two neighbouring layers (two, because layers work in the two halves of the scratch
// memory in turn) and hands over what it passed; every further layer is one of the two with each pointer that lies in one
// of that layer's own tensors moved to the same place of the further layer's.
#include "common.cuh"
#include "launch_list.cuh"

namespace ts {

struct ListEntry {
  const char* name;
  ListCall call;
  const char* kinds;
  int args;
};
constexpr int LIST_MAX_ENTRIES = 64;
struct ListTable {
  ListEntry entries[LIST_MAX_ENTRIES];
  int count = 0;
};
static ListTable& list_table() {      // (entries register themselves while the library is being loaded, in any order of files)
  static ListTable table;
  return table;
}
int list_register(const char* name, ListCall call, const char* kinds) {
  ListTable& t = list_table();
  if (t.count == LIST_MAX_ENTRIES) return -1;
  t.entries[t.count] = {name, call, kinds, (int)strlen(kinds)};
  return t.count++;
}

// The vendor library's product, for the shapes that go there: out[M, N] = x[M, K] * w[N, K]^T, bf16 with 32-bit sums, as
// torch.mm asks for it. The function and its handle (made for the stream the call is for) come from the caller.
typedef int (*BlasGemmEx)(void* handle, int transa, int transb, int m, int n, int k, const void* alpha, const void* a, int a_type, int lda,
                          const void* b, int b_type, int ldb, const void* beta, void* c, int c_type, int ldc, int compute_type, int algo);

}  // namespace ts

using namespace ts;

extern "C" int ts_library_gemm(const void* x, const void* w, void* out, int M, int N, int K, int out_dtype, const void* gemm_ex,
                               void* handle) {
  constexpr int OP_N = 0, OP_T = 1, R_32F = 0, R_16BF = 14, COMPUTE_32F = 68, GEMM_DEFAULT_TENSOR_OP = 99;
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || gemm_ex == nullptr || handle == nullptr) return TS_ERR_BAD_ARGUMENT;
  const float one = 1.f, zero = 0.f;
  const int status = reinterpret_cast<BlasGemmEx>(const_cast<void*>(gemm_ex))(
      handle, OP_T, OP_N, N, M, K, &one, w, R_16BF, K, x, R_16BF, K, &zero, out, out_dtype == TS_DTYPE_F32 ? R_32F : R_16BF, N,
      COMPUTE_32F, GEMM_DEFAULT_TENSOR_OP);
  return status == 0 ? 0 : TS_ERR_UNSUPPORTED;
}
TS_LIST_ENTRY(ts_library_gemm);

// The number of an entry point that lists may name, or -1; *args receives how many arguments it takes and kinds (room for
// 65 characters) their kinds.
extern "C" int ts_list_entry(const char* name, int* args, char* kinds) {
  const ListTable& t = list_table();
  for (int i = 0; i < t.count; ++i)
    if (strcmp(t.entries[i].name, name) == 0) {
      *args = t.entries[i].args;
      strncpy(kinds, t.entries[i].kinds, 65);
      return i;
    }
  return -1;
}

// Two lists of calls: list t has calls first[t] .. first[t + 1], call c is entries[c] with its arguments at words, one call
// after the other. places[l][r], bytes[r]: the tensors of a layer; layers 0 and 1 made the two lists, layer 2 + l runs list
// l % 2. at: the layer and the call that failed. Nothing is launched if a layer's tensors lie differently to the 16-byte
// grid than layer 0's (TS_ERR_UNLIKE) or if the lists are too long.
constexpr int TS_ERR_UNLIKE = -4;
extern "C" int ts_list_run(const int* entries, const int* first, const uint64_t* words, const uint64_t* places, const uint64_t* bytes,
                           int tensors, int layers, int* at) {
  constexpr int MOST_WORDS = 4096, MOST_MOVES = 1024;
  struct Move { int word, tensor; };
  const ListTable& t = list_table();
  static thread_local uint64_t mine[MOST_WORDS];
  static thread_local Move moves[MOST_MOVES];
  for (int l = 1; l < 2 + layers; ++l)
    for (int r = 0; r < tensors; ++r)
      if ((places[(size_t)l * tensors + r] ^ places[r]) & 15) return TS_ERR_UNLIKE;
  int move_first[3] = {0, 0, 0}, word_of_list[3] = {0, 0, 0}, word = 0, num_moves = 0;
  for (int list = 0; list < 2; ++list) {
    word_of_list[list] = word;
    for (int c = first[list]; c < first[list + 1]; ++c) {
      if (entries[c] < 0 || entries[c] >= t.count) return TS_ERR_BAD_ARGUMENT;
      const ListEntry& e = t.entries[entries[c]];
      if (word + e.args > MOST_WORDS) return TS_ERR_UNSUPPORTED;
      for (int i = 0; i < e.args; ++i, ++word) {
        mine[word] = words[word];
        if (e.kinds[i] != 'p') continue;
        for (int r = 0; r < tensors; ++r)
          if (words[word] - places[list * tensors + r] < bytes[r]) {
            if (num_moves == MOST_MOVES) return TS_ERR_UNSUPPORTED;
            moves[num_moves++] = {word, r};
            break;
          }
      }
    }
    move_first[list + 1] = num_moves;
  }
  for (int l = 0; l < layers; ++l) {
    const int list = l & 1;
    for (int i = move_first[list]; i < move_first[list + 1]; ++i)
      mine[moves[i].word] = words[moves[i].word] - places[list * tensors + moves[i].tensor] + places[(size_t)(2 + l) * tensors + moves[i].tensor];
    const uint64_t* args = mine + word_of_list[list];
    for (int c = first[list]; c < first[list + 1]; ++c) {
      const ListEntry& e = t.entries[entries[c]];
      const int status = e.call(args);
      if (status != 0) {
        at[0] = l;
        at[1] = c;
        return status;
      }
      args += e.args;
    }
  }
  return 0;
}
