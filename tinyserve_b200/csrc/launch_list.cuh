// Calls of this library's own entry points as data, so that a list of them can be run without the interpreter between
// them (launch_list.cu). An argument is a word of 64 bits: a pointer, an integer (sign-extended), a double, or a float in
// the low half. TS_LIST_ENTRY(f), once per entry point and beside its definition, makes f known by its name; the types of
// the arguments come from its declaration.
#pragma once
#include <stdint.h>
#include <string.h>

#include <type_traits>
#include <utility>

namespace ts {

typedef int (*ListCall)(const uint64_t* args);

template <typename A>
inline A list_argument(uint64_t word) {
  if constexpr (std::is_pointer<A>::value) {
    return reinterpret_cast<A>(word);
  } else if constexpr (std::is_floating_point<A>::value) {
    A value;
    memcpy(&value, &word, sizeof(A));
    return value;
  } else {
    return static_cast<A>(static_cast<int64_t>(word));
  }
}

template <auto F>
struct ListThunk;
template <typename... A, int (*F)(A...)>
struct ListThunk<F> {
  template <size_t... I>
  static int run(const uint64_t* words, std::index_sequence<I...>) { return F(list_argument<A>(words[I])...); }
  static int call(const uint64_t* words) { return run(words, std::index_sequence_for<A...>()); }
  // a letter per argument: p(ointer), f(loat), d(ouble), i(nteger) or l(ong)
  static const char* kinds() {
    static const char letters[] = {(std::is_pointer<A>::value ? 'p' : std::is_same<A, float>::value ? 'f'
                                    : std::is_same<A, double>::value ? 'd' : sizeof(A) == 8 ? 'l' : 'i')..., 0};
    return letters;
  }
};

int list_register(const char* name, ListCall call, const char* kinds);

}  // namespace ts

#define TS_LIST_ENTRY(f) \
  [[maybe_unused]] static const int list_entry_of_##f = ts::list_register(#f, &ts::ListThunk<&f>::call, ts::ListThunk<&f>::kinds())
