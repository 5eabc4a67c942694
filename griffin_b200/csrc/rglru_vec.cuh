// Vector loads and stores of the streaming kernels (conv, column sums, decode).
#pragma once

#include "rglru_device.cuh"

namespace rglru {

constexpr int CONV_TAPS = 4;

template <int BYTES> struct RawWord { using type = uint32_t; };
template <> struct RawWord<8> { using type = uint2; };
template <> struct RawWord<16> { using type = uint4; };

// VEC channels of IO as one aligned 8- or 16-byte access (VEC == 1: scalar fallback for odd widths).  The
// raw form is what a thread keeps in registers while several loads are in flight.
template <typename IO, int VEC>
struct Vec {
  static constexpr int BYTES = VEC * static_cast<int>(sizeof(IO));
  static_assert(VEC == 1 || BYTES == 8 || BYTES == 16, "one 8- or 16-byte access per thread and row");
  using Raw = typename RawWord<VEC == 1 ? 4 : BYTES>::type;

  static __device__ __forceinline__ Raw load_raw(const IO* p) {
    if constexpr (VEC == 1) {
      if constexpr (sizeof(IO) == 4) return __float_as_uint(p[0]);
      else return static_cast<uint32_t>(*reinterpret_cast<const unsigned short*>(p)) << 16;
    } else {
      return *reinterpret_cast<const Raw*>(p);
    }
  }
  static __device__ __forceinline__ void unpack(const Raw& r, float (&v)[VEC]) {
    if constexpr (VEC == 1) {
      v[0] = __uint_as_float(r);
    } else {
      constexpr int NW = BYTES / 4;
      uint32_t w[NW];
      if constexpr (NW == 2) { w[0] = r.x; w[1] = r.y; }
      else { w[0] = r.x; w[1] = r.y; w[2] = r.z; w[3] = r.w; }
      if constexpr (sizeof(IO) == 4) {
#pragma unroll
        for (int k = 0; k < NW; ++k) v[k] = __uint_as_float(w[k]);
      } else {
#pragma unroll
        for (int k = 0; k < NW; ++k) {
          v[2 * k] = __uint_as_float(w[k] << 16);
          v[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
        }
      }
    }
  }
  static __device__ __forceinline__ void load(const IO* p, float (&v)[VEC]) { unpack(load_raw(p), v); }
  static __device__ __forceinline__ void store(IO* p, const float (&v)[VEC]) {
    if constexpr (VEC == 1) {
      p[0] = Pack<IO>::from_float(v[0]);
    } else {
      constexpr int NW = BYTES / 4;
      uint32_t w[NW];
      if constexpr (sizeof(IO) == 4) {
#pragma unroll
        for (int k = 0; k < NW; ++k) w[k] = __float_as_uint(v[k]);
      } else {
#pragma unroll
        for (int k = 0; k < NW; ++k) {
          __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
          w[k] = *reinterpret_cast<uint32_t*>(&h);
        }
      }
      if constexpr (NW == 2) *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
      else *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
};

template <typename IO>
__host__ __device__ constexpr int vec_width() { return 16 / sizeof(IO); }

}  // namespace rglru
