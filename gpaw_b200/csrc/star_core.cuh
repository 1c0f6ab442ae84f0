// The arithmetic of the axis-aligned FD stencil shared by the marching
// kernels: a thread owns R1 x R2 neighbouring points of a plane, holds the
// last 2H + 1 planes of them in a register queue (axis 0) and reads the
// in-plane neighbours of the centre plane through the callables it is given.
// The order of the terms is the reference's: centre, axis 0, axis 2, axis 1,
// offsets ascending.
//
// FP32 enters every tap as a difference, c (x_p - x_c) plus (sum c) x_c, so
// that the operator annihilates constants exactly after the coefficients are
// rounded (otherwise every eigenvalue shifts by ~|c0| 2^-24); symmetric pairs
// as c ((x+ + x-) - 2 x_c), antisymmetric ones as c (x+ - x-).
#pragma once
#include <type_traits>
#include "internal.cuh"

namespace gb {

// A value the compiler must keep in a register.  sm_100 arithmetic takes
// constants through the uniform registers, and the FP64 and packed FP32
// instructions need them moved to ordinary ones first: re-read from the
// parameter bank the 19-point FP64 kernel spent a seventh of its instructions
// on such moves.
__device__ __forceinline__ double in_register(double v) {
  asm volatile("" : "+d"(v));
  return v;
}
__device__ __forceinline__ float in_register(float v) {
  asm volatile("" : "+f"(v));
  return v;
}

// Stencil coefficients.  SYM = 1: equal on both sides of every axis (the
// Laplacian), one value per axis and distance, held in registers;
// SYM = -1 (opposite on the two sides: first derivatives) and SYM = 0
// (anything): read from the kernel parameters.
template <typename R, int H, int SYM>
struct StarCoef {
  R c0, c[3][H];
  template <class A>
  __device__ __forceinline__ void init(const A& a) {
    c0 = in_register(sizeof(R) == 4 ? (R)a.c0diff : (R)a.c0);
#pragma unroll
    for (int ax = 0; ax < 3; ++ax)
#pragma unroll
      for (int k = 0; k < H; ++k) c[ax][k] = in_register((R)a.a[ax][HMAX + 1 + k]);
  }
  template <class A>
  __device__ __forceinline__ R at(const A& a, int ax, int m) const {   // offset m != 0
    if constexpr (SYM == 1) return c[ax][(m < 0 ? -m : m) - 1];
    else return (R)a.a[ax][HMAX + m];
  }
};

template <int SYM>
__device__ __forceinline__ float2 tap2(float2 acc, float cp, float cm, float2 vp, float2 vm, float2 xc) {
  const float2 m1 = make_float2(-1.f, -1.f);
  if constexpr (SYM == 1) {
    const float2 d = __ffma2_rn(make_float2(-2.f, -2.f), xc, __fadd2_rn(vp, vm));
    return __ffma2_rn(make_float2(cp, cp), d, acc);
  } else if constexpr (SYM == -1) {
    return __ffma2_rn(make_float2(cp, cp), __ffma2_rn(vm, m1, vp), acc);
  } else {
    acc = __ffma2_rn(make_float2(cp, cp), __ffma2_rn(xc, m1, vp), acc);
    return __ffma2_rn(make_float2(cm, cm), __ffma2_rn(xc, m1, vm), acc);
  }
}

// acc = S(x) at the centre plane.  q[(u + 1 + m) % NQ] is the plane at offset
// m - H from it; left / right(r, v): the HZ points beside the thread's row r;
// rowv(rr, v): its R2 points of row rr outside the own rows.
template <typename T, int H, int R1, int R2, int HZ, int SYM, class A, class L, class Rt, class Rw, class Own>
__device__ __forceinline__ void star_points(T (&acc)[R1][R2], const T (&q)[2 * H + 1][R1][R2], int u,
                                            const StarCoef<typename Elem<T>::R, H, SYM>& k, const A& a, L left,
                                            Rt right, Rw rowv, Own ownfix) {
  using R = typename Elem<T>::R;
  constexpr int NQ = 2 * H + 1;
  constexpr bool DIFF = sizeof(R) == 4;
  const int cu = (u + NQ - H) % NQ;
  if constexpr (std::is_same<T, float>::value && R2 % 2 == 0) {
    // two points per instruction (packed f32x2), pairs of columns
    float2 acc2[R1][R2 / 2];
#pragma unroll
    for (int r = 0; r < R1; ++r)
#pragma unroll
      for (int p = 0; p < R2 / 2; ++p) {
        const float2 xc = make_float2(q[cu][r][2 * p], q[cu][r][2 * p + 1]);
        const R cc = SYM == 1 ? k.c0 : (R)a.c0diff;
        float2 x = __fmul2_rn(make_float2(cc, cc), xc);
#pragma unroll
        for (int d = 1; d <= H; ++d) {
          const int mp = (u + 1 + H + d) % NQ, mm = (u + 1 + H - d) % NQ;
          x = tap2<SYM>(x, k.at(a, 0, d), k.at(a, 0, -d), make_float2(q[mp][r][2 * p], q[mp][r][2 * p + 1]),
                        make_float2(q[mm][r][2 * p], q[mm][r][2 * p + 1]), xc);
        }
        acc2[r][p] = x;
      }
#pragma unroll
    for (int r = 0; r < R1; ++r) {
      float w[HZ + R2 + HZ];
      float t[HZ];
      left(r, t);
#pragma unroll
      for (int v = 0; v < HZ; ++v) w[v] = t[v];
      right(r, t);
#pragma unroll
      for (int v = 0; v < HZ; ++v) w[HZ + R2 + v] = t[v];
#pragma unroll
      for (int c = 0; c < R2; ++c) w[HZ + c] = q[cu][r][c];
#pragma unroll
      for (int p = 0; p < R2 / 2; ++p) {
        const int c = HZ + 2 * p;
        const float2 xc = make_float2(w[c], w[c + 1]);
        float2 x = acc2[r][p];
#pragma unroll
        for (int d = 1; d <= H; ++d)
          x = tap2<SYM>(x, k.at(a, 2, d), k.at(a, 2, -d), make_float2(w[c + d], w[c + 1 + d]),
                        make_float2(w[c - d], w[c + 1 - d]), xc);
        acc2[r][p] = x;
      }
    }
#pragma unroll
    for (int rr = -H; rr < R1 + H; ++rr) {
      T v[R2];
      if (rr >= 0 && rr < R1) {
#pragma unroll
        for (int c = 0; c < R2; ++c) v[c] = q[cu][rr][c];
      } else {
        rowv(rr, v);
      }
#pragma unroll
      for (int r = 0; r < R1; ++r) {
        const int d = rr - r;
        if (d < -H || d > H || d == 0) continue;
        const float cc = k.at(a, 1, d);
#pragma unroll
        for (int p = 0; p < R2 / 2; ++p) {
          const float2 xc = make_float2(q[cu][r][2 * p], q[cu][r][2 * p + 1]);
          const float2 dv = __ffma2_rn(xc, make_float2(-1.f, -1.f), make_float2(v[2 * p], v[2 * p + 1]));
          acc2[r][p] = __ffma2_rn(make_float2(cc, cc), dv, acc2[r][p]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R1; ++r)
#pragma unroll
      for (int p = 0; p < R2 / 2; ++p) {
        acc[r][2 * p] = acc2[r][p].x;
        acc[r][2 * p + 1] = acc2[r][p].y;
      }
  } else {
#pragma unroll
    for (int r = 0; r < R1; ++r)
#pragma unroll
      for (int c = 0; c < R2; ++c) {
        const T xc = q[cu][r][c];
        T x = scale(SYM == 1 ? k.c0 : DIFF ? (R)a.c0diff : (R)a.c0, xc);
#pragma unroll
        for (int m = -H; m <= H; ++m) {
          if (m == 0) continue;
          const T v = q[(u + 1 + m + H) % NQ][r][c];
          x = fmadd(x, k.at(a, 0, m), DIFF ? sub(v, xc) : v);
        }
        acc[r][c] = x;
      }
#pragma unroll
    for (int r = 0; r < R1; ++r) {
      T wl[HZ], wr[HZ];
      left(r, wl);
      right(r, wr);
#pragma unroll
      for (int c = 0; c < R2; ++c) {
        const T xc = q[cu][r][c];
#pragma unroll
        for (int m = -H; m <= H; ++m) {
          if (m == 0) continue;
          const int cc = c + m;
          const T v = cc < 0 ? wl[HZ + cc] : (cc >= R2 ? wr[cc - R2] : ownfix(r, cc, q[cu][r][cc]));
          acc[r][c] = fmadd(acc[r][c], k.at(a, 2, m), DIFF ? sub(v, xc) : v);
        }
      }
    }
#pragma unroll
    for (int rr = -H; rr < R1 + H; ++rr) {
      T v[R2];
      if (rr >= 0 && rr < R1) {
#pragma unroll
        for (int c = 0; c < R2; ++c) v[c] = q[cu][rr][c];
      }
      rowv(rr, v);
#pragma unroll
      for (int r = 0; r < R1; ++r) {
        const int m = rr - r;
        if (m < -H || m > H || m == 0) continue;
#pragma unroll
        for (int c = 0; c < R2; ++c)
          acc[r][c] = fmadd(acc[r][c], k.at(a, 1, m), DIFF ? sub(v[c], q[cu][r][c]) : v[c]);
      }
    }
  }
}

// predicated stores, loads and copies (no branch around them); the loads are
// volatile so that they stay where they are written, ahead of the arithmetic
// that hides their latency
__device__ __forceinline__ double ld_if(const double* p, bool on) {
  double v;
  asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %2, 0;\nmov.f64 %0, 0d0000000000000000;\n@p ld.global.nc.f64 %0, [%1];\n}\n"
               : "=d"(v) : "l"(p), "r"((int)on));
  return v;
}
__device__ __forceinline__ float ld_if(const float* p, bool on) {
  float v;
  asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %2, 0;\nmov.f32 %0, 0f00000000;\n@p ld.global.nc.f32 %0, [%1];\n}\n"
               : "=f"(v) : "l"(p), "r"((int)on));
  return v;
}
__device__ __forceinline__ double2 ld_if(const double2* p, bool on) {
  double2 v;
  asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %3, 0;\nmov.f64 %0, 0d0000000000000000;\nmov.f64 %1, %0;\n@p ld.global.nc.v2.f64 {%0, %1}, [%2];\n}\n"
               : "=d"(v.x), "=d"(v.y) : "l"(p), "r"((int)on));
  return v;
}
__device__ __forceinline__ float2 ld_if(const float2* p, bool on) {
  float2 v;
  asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %3, 0;\nmov.f32 %0, 0f00000000;\nmov.f32 %1, %0;\n@p ld.global.nc.v2.f32 {%0, %1}, [%2];\n}\n"
               : "=f"(v.x), "=f"(v.y) : "l"(p), "r"((int)on));
  return v;
}
__device__ __forceinline__ float4 ld4_if(const void* p, bool on) {
  float4 v;
  asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %5, 0;\nmov.f32 %0, 0f00000000;\nmov.f32 %1, %0;\nmov.f32 %2, %0;\nmov.f32 %3, %0;\n"
               "@p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n}\n"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p), "r"((int)on));
  return v;
}
__device__ __forceinline__ void st_cs_if(double* p, double v, bool on) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %2, 0;\n@p st.global.cs.f64 [%0], %1;\n}\n" ::"l"(p), "d"(v), "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void st_cs_if(float* p, float v, bool on) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %2, 0;\n@p st.global.cs.f32 [%0], %1;\n}\n" ::"l"(p), "f"(v), "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void st_cs_if(double2* p, double2 v, bool on) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %3, 0;\n@p st.global.cs.v2.f64 [%0], {%1, %2};\n}\n" ::"l"(p), "d"(v.x),
               "d"(v.y), "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void st_cs_if(float2* p, float2 v, bool on) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %3, 0;\n@p st.global.cs.v2.f32 [%0], {%1, %2};\n}\n" ::"l"(p), "f"(v.x),
               "f"(v.y), "r"((int)on)
               : "memory");
}
template <typename T>
__device__ __forceinline__ void cp_async_elem_if(T* sdst, const T* gsrc, bool on) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %3, 0;\n@p cp.async.ca.shared.global [%0], [%1], %2;\n}\n" ::"r"(
                   smem_u32(sdst)),
               "l"(gsrc), "n"(sizeof(T)), "r"((int)on)
               : "memory");
}

}  // namespace gb
