// Host-side helpers shared by all launchers: TMA descriptor encoding through the driver entry
// point (no link-time dependency on libcuda), launch-error capture, device properties.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <tuple>
#include <type_traits>

namespace ra {

// Error codes returned by every extern "C" launcher (0 = ok).
enum HostError : int {
  kHostOk = 0,
  kHostBadArg = -1,
  kHostTmapFail = -2,
  kHostLaunchFail = -3,
  kHostNoDriver = -4,
  kHostTooLarge = -5,
};

// rank-`rank` bf16 tensor map with 128-byte swizzle and zero fill for out-of-range elements.
// dims[0] is the innermost (contiguous) extent; strides_bytes has rank-1 entries (dims 1..).
int make_tmap_bf16_sw128(CUtensorMap* out, const void* base, int rank, const uint64_t* dims,
                         const uint64_t* strides_bytes, const uint32_t* box);

// Same, element type fp32 (box inner extent 32 elements = 128 bytes).
int make_tmap_f32_sw128(CUtensorMap* out, const void* base, int rank, const uint64_t* dims,
                        const uint64_t* strides_bytes, const uint32_t* box);

int sm_count();                 // SM count of the current device (cached per device)
int check_launch(const char*);  // cudaGetLastError -> HostError, message kept for ra_last_error
void set_error(const char* msg);

// A launcher's arguments as one block of memory, each at its natural alignment, as Python's struct module packs them: RA_PACKED(fn) adds
// fn_packed(block) and fn_packed_format(), the block's format ('P' pointer, 'i' int, 'q' long long, 'f' float ...). ctypes converts arguments
// one by one: 17 of them take 6.7 us, more than the launch, packed they take 1.1.
template <typename T> constexpr char pack_code() {
  static_assert(std::is_pointer<T>::value, "no code for this type");
  return 'P';
}
template <> constexpr char pack_code<int>() { return 'i'; }
template <> constexpr char pack_code<unsigned int>() { return 'I'; }
template <> constexpr char pack_code<long long>() { return 'q'; }
template <> constexpr char pack_code<unsigned long long>() { return 'Q'; }
template <> constexpr char pack_code<float>() { return 'f'; }
template <typename T>
T unpack_next(const unsigned char* block, size_t& at) {
  at = (at + alignof(T) - 1) / alignof(T) * alignof(T);
  T v;
  memcpy(&v, block + at, sizeof(T));
  at += sizeof(T);
  return v;
}
template <typename... A>
int call_packed(int (*fn)(A...), const void* block) {
  size_t at = 0;
  std::tuple<A...> args{unpack_next<A>(static_cast<const unsigned char*>(block), at)...};  // in order: a braced list
  return std::apply(fn, args);
}
template <typename... A>
const char* packed_format(int (*)(A...)) {
  static const char text[] = {pack_code<A>()..., 0};
  return text;
}
#define RA_PACKED(fn)                                                                    \
  extern "C" int fn##_packed(const void* block) { return ra::call_packed(fn, block); } \
  extern "C" const char* fn##_packed_format() { return ra::packed_format(fn); }

}  // namespace ra

extern "C" const char* ra_last_error();
