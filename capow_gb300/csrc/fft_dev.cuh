// FP32 complex transforms in registers, forward sign, natural order in and out: DFTs of 2 to 32 points by one
// thread, and a row of N = 16 .. 1024 points by N / R1 lanes of one warp (RowFft).
#pragma once
#include <cuda_runtime.h>

// Packed FP32 additions: one instruction per complex sum, rounded as the scalar ones are.
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmul_mi(float2 a) { return make_float2(a.y, -a.x); }  // a * (-i)

__device__ __forceinline__ void dft8(float2 *a) {
  const float h = 0.70710678118654752f;
  float2 b0 = cadd(a[0], a[4]), b4 = csub(a[0], a[4]);
  float2 b1 = cadd(a[1], a[5]), t5 = csub(a[1], a[5]);
  float2 b2 = cadd(a[2], a[6]), t6 = csub(a[2], a[6]);
  float2 b3 = cadd(a[3], a[7]), t7 = csub(a[3], a[7]);
  const float2 b5 = make_float2((t5.x + t5.y) * h, (t5.y - t5.x) * h);    // * e^{-i pi/4}
  const float2 b6 = cmul_mi(t6);                                           // * e^{-i pi/2}
  const float2 b7 = make_float2((t7.y - t7.x) * h, -(t7.x + t7.y) * h);   // * e^{-3i pi/4}
  const float2 c0 = cadd(b0, b2), c2 = csub(b0, b2), c1 = cadd(b1, b3), c3 = cmul_mi(csub(b1, b3));
  const float2 c4 = cadd(b4, b6), c6 = csub(b4, b6), c5 = cadd(b5, b7), c7 = cmul_mi(csub(b5, b7));
  a[0] = cadd(c0, c1);
  a[4] = csub(c0, c1);
  a[2] = cadd(c2, c3);
  a[6] = csub(c2, c3);
  a[1] = cadd(c4, c5);
  a[5] = csub(c4, c5);
  a[3] = cadd(c6, c7);
  a[7] = csub(c6, c7);
}

__device__ __forceinline__ void dft4(float2 *a) {
  const float2 b0 = cadd(a[0], a[2]), b2 = csub(a[0], a[2]), b1 = cadd(a[1], a[3]), b3 = cmul_mi(csub(a[1], a[3]));
  a[0] = cadd(b0, b1);
  a[2] = csub(b0, b1);
  a[1] = cadd(b2, b3);
  a[3] = csub(b2, b3);
}

// v * exp(-2 pi i k / 32), k known at compile time (after unrolling)
__device__ __forceinline__ float2 mul_w32(float2 v, int k) {
  const float h = 0.70710678118654752f, c1 = 0.98078528040323044f, s1 = 0.19509032201612827f,
              c2 = 0.92387953251128676f, s2 = 0.38268343236508977f, c3 = 0.83146961230254524f,
              s3 = 0.55557023301960222f;
  switch (k & 31) {
    case 0: return v;
    case 1: return cmulf(v, make_float2(c1, -s1));
    case 2: return cmulf(v, make_float2(c2, -s2));
    case 3: return cmulf(v, make_float2(c3, -s3));
    case 4: return make_float2((v.x + v.y) * h, (v.y - v.x) * h);
    case 5: return cmulf(v, make_float2(s3, -c3));
    case 6: return cmulf(v, make_float2(s2, -c2));
    case 7: return cmulf(v, make_float2(s1, -c1));
    case 8: return cmul_mi(v);
    case 9: return cmulf(v, make_float2(-s1, -c1));
    case 10: return cmulf(v, make_float2(-s2, -c2));
    case 11: return cmulf(v, make_float2(-s3, -c3));
    case 12: return make_float2((v.y - v.x) * h, -(v.x + v.y) * h);
    case 13: return cmulf(v, make_float2(-c3, -s3));
    case 14: return cmulf(v, make_float2(-c2, -s2));
    case 15: return cmulf(v, make_float2(-c1, -s1));
    case 18: return cmulf(v, make_float2(-c2, s2));
    case 21: return cmulf(v, make_float2(-s3, c3));
    default: return v;  // no other power occurs in the DFTs below
  }
}

// R-point DFT by one thread.
template <int R>
__device__ __forceinline__ void dft(float2 *a) {
  if constexpr (R == 4) {
    dft4(a);
  } else if constexpr (R == 8) {
    dft8(a);
  } else {  // 16 = 4 x 4, 32 = 4 x 8
    constexpr int C = R / 4;
    static_assert(R == 16 || R == 32, "radix");
    float2 b[C][4];
#pragma unroll
    for (int j = 0; j < C; j++) {
#pragma unroll
      for (int q = 0; q < 4; q++) b[j][q] = a[j + C * q];
      dft4(b[j]);
#pragma unroll
      for (int p = 1; p < 4; p++) b[j][p] = mul_w32(b[j][p], j * p * (32 / R));
    }
#pragma unroll
    for (int p = 0; p < 4; p++) {
      float2 c[C];
#pragma unroll
      for (int j = 0; j < C; j++) c[j] = b[j][p];
      dft<C>(c);
#pragma unroll
      for (int r = 0; r < C; r++) a[p + 4 * r] = c[r];
    }
  }
}

// A row of N = 2^LOGN complex values by T lanes of one warp: lane t holds x[t + T q], q < R1, R1 = N / T. An R1-point
// DFT per lane, twiddles, one exchange through the row's shared buffer, then R1 DFTs of T points, R1 / T per lane
// (for N = 512, where 16 values a lane leave T = 32 > R1, half of one: two lanes take the even and the odd outputs
// of one, 16 points each after a first radix-2 step). Output j of lane t is frequency freq(t, j). Against three radix-8 stages a row crosses
// shared memory once instead of twice, and the lanes of one warp exchange without a block barrier. 16 values a lane
// fit 64 registers, 32 (N = 1024) 128.
template <int LOGN>
struct RowFft {
  static constexpr int N = 1 << LOGN;
  static constexpr int R1 = LOGN == 10 ? 32 : (LOGN >= 7 ? 16 : (LOGN >= 5 ? 8 : 4));
  static constexpr int T = N / R1;
  static constexpr int BUF = R1 * (T + 1);  // values of the exchange buffer
  static_assert(LOGN >= 4 && LOGN <= 10 && T <= 32, "row length");

  __device__ static __forceinline__ int freq(int t, int j) {
    if constexpr (T > R1) return (t & (R1 - 1)) + R1 * (2 * j + t / R1);
    else return t + T * (j / T) + R1 * (j % T);
  }

  // tw[p * T + t] = exp(-2 pi i t p / N) (shared memory); buf: the row's BUF values, free on entry and exit
  __device__ static __forceinline__ void run(float2 *v, float2 *buf, const float2 *tw, int t) {
    dft<R1>(v);
#pragma unroll
    for (int p = 1; p < R1; p++) v[p] = cmulf(v[p], tw[p * T + t]);
#pragma unroll
    for (int p = 0; p < R1; p++) buf[p * (T + 1) + t] = v[p];
    __syncwarp();
    if constexpr (T > R1) {  // N = 512: DFT p by lanes p and p + 16: outputs 2 r + h, h = 0 or 1
      static_assert(T == 32 && R1 == 16, "split second stage");
      const int p = t & 15, h = t >> 4;
      const float sg = h ? -1.0f : 1.0f;
#pragma unroll
      for (int r = 0; r < 16; r++) {
        const float2 lo = buf[p * 33 + r], hi = buf[p * 33 + r + 16];
        const float2 d = __ffma2_rn(hi, make_float2(sg, sg), lo);
        v[r] = r == 0 ? d : (h ? mul_w32(d, r) : d);
      }
      __syncwarp();
      dft<16>(v);
    } else {
      constexpr int G = R1 / T;
#pragma unroll
      for (int u = 0; u < G; u++)
#pragma unroll
        for (int r = 0; r < T; r++) v[u * T + r] = buf[(t + T * u) * (T + 1) + r];
      __syncwarp();
#pragma unroll
      for (int u = 0; u < G; u++) dft<T>(v + u * T);
    }
  }

  // the twiddle table from a table of exp(-2 pi i q / N), q < N
  __device__ static __forceinline__ void load_twiddles(float2 *tw, const float2 *w) {
    for (int e = threadIdx.x; e < N; e += blockDim.x) tw[e] = w[((e / T) * (e % T)) & (N - 1)];
  }
};
