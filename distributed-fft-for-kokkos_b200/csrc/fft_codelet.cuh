// DFT codelets of small length on registers: Dft<T, R>::run(v) transforms
// v[0..R-1] in place, X_q = sum_r v_r exp(-2 pi i r q / R).
// Only the forward direction exists: an inverse transform swaps the real and
// imaginary parts of its inputs and outputs, or reads its outputs in reverse
// (X_{R-q}).
//
// Prime lengths 2, 3, 5, 7, 11 and 13 are written out, 4 and 8 as radix-2
// trees; prime powers 9, 16, 25, 27 and 32 split as A x B with compile-time
// twiddles; products of coprime factors use the prime-factor index maps
// (n = B n1 + A n2 mod R in, k = k1 mod A = k2 mod B out), which need no
// twiddles at all.  Every index is a constant after unrolling, so a codelet
// costs its arithmetic and registers only.
#pragma once

#include "fft_radix.cuh"

namespace dfft {
namespace dev {
namespace codelet {

// cos and sin of 2 pi k / R for the k a codelet of length R uses
template <int R>
struct Root;
template <>
struct Root<5> {
  static __device__ __forceinline__ constexpr double c(int k) {
    switch (k) {
      case 1: return 0.309016994374947424102293417182819059;
      case 2: return -0.809016994374947424102293417182819059;
      default: return 1.0;
    }
  }
  static __device__ __forceinline__ constexpr double s(int k) {
    switch (k) {
      case 1: return 0.951056516295153572116439333379382143;
      case 2: return 0.587785252292473129168705954639072769;
      default: return 0.0;
    }
  }
};
template <>
struct Root<7> {
  static __device__ __forceinline__ constexpr double c(int k) {
    switch (k) {
      case 1: return 0.623489801858733530525004884004239811;
      case 2: return -0.222520933956314404288902564496794759;
      case 3: return -0.900968867902419126236102319507445051;
      default: return 1.0;
    }
  }
  static __device__ __forceinline__ constexpr double s(int k) {
    switch (k) {
      case 1: return 0.781831482468029808708444526674057750;
      case 2: return 0.974927912181823607018131682993931217;
      case 3: return 0.433883739117558120475768332848358755;
      default: return 0.0;
    }
  }
};
template <>
struct Root<9> {
  static __device__ __forceinline__ constexpr double c(int k) {
    switch (k) {
      case 1: return 0.766044443118978035202392650555416674;
      case 2: return 0.173648177666930348851716626769314796;
      case 4: return -0.939692620785908384054109277324731470;
      default: return 1.0;
    }
  }
  static __device__ __forceinline__ constexpr double s(int k) {
    switch (k) {
      case 1: return 0.642787609686539326322643409907263433;
      case 2: return 0.984807753012208059366743024589523014;
      case 4: return 0.342020143325668733044099614682259581;
      default: return 0.0;
    }
  }
};
template <>
struct Root<11> {
  static __device__ __forceinline__ constexpr double c(int k) {
    switch (k) {
      case 1: return 0.841253532831181168861811648919367718;
      case 2: return 0.415415013001886425529274149229623204;
      case 3: return -0.142314838273285140443792668616369669;
      case 4: return -0.654860733945285064056925072466293553;
      case 5: return -0.959492973614497389890368057066327699;
      default: return 1.0;
    }
  }
  static __device__ __forceinline__ constexpr double s(int k) {
    switch (k) {
      case 1: return 0.540640817455597582107635954318691695;
      case 2: return 0.909631995354518371411715383079028460;
      case 3: return 0.989821441880932732376092037776718787;
      case 4: return 0.755749574354258283774035843972344420;
      case 5: return 0.281732556841429697711417915346616899;
      default: return 0.0;
    }
  }
};
template <>
struct Root<13> {
  static __device__ __forceinline__ constexpr double c(int k) {
    switch (k) {
      case 1: return 0.885456025653209895900375522015098879;
      case 2: return 0.568064746731155802511807559127516625;
      case 3: return 0.120536680255323053349067687452543582;
      case 4: return -0.354604887042535625969637892600018474;
      case 5: return -0.748510748171101098634630599701351384;
      case 6: return -0.970941817426052027156982276293789227;
      default: return 1.0;
    }
  }
  static __device__ __forceinline__ constexpr double s(int k) {
    switch (k) {
      case 1: return 0.464723172043768545656015335133104778;
      case 2: return 0.822983865893656394579617423439381991;
      case 3: return 0.992708874098053992800751649492520179;
      case 4: return 0.935016242685414823439784599837830729;
      case 5: return 0.663122658240795202376785492666766280;
      case 6: return 0.239315664287557767148753726260211895;
      default: return 0.0;
    }
  }
};
template <>
struct Root<16> {
  static __device__ __forceinline__ constexpr double c(int k) {
    switch (k) {
      case 1: return 0.923879532511286756128183189396788287;
      case 2: return 0.707106781186547524400844362104849039;
      case 3: return 0.382683432365089771728459984030398867;
      case 4: return 0.0;
      case 6: return -0.707106781186547524400844362104849039;
      case 9: return -0.923879532511286756128183189396788287;
      default: return 1.0;
    }
  }
  static __device__ __forceinline__ constexpr double s(int k) {
    switch (k) {
      case 1: return 0.382683432365089771728459984030398867;
      case 2: return 0.707106781186547524400844362104849039;
      case 3: return 0.923879532511286756128183189396788287;
      case 4: return 1.0;
      case 6: return 0.707106781186547524400844362104849039;
      case 9: return -0.382683432365089771728459984030398867;
      default: return 0.0;
    }
  }
};
template <>
struct Root<25> {
  static __device__ __forceinline__ constexpr double c(int k) {
    switch (k) {
      case 1: return 0.968583161128631119490168375464735814;
      case 2: return 0.876306680043863587308115903922062583;
      case 3: return 0.728968627421411523146730319055259111;
      case 4: return 0.535826794978996618271308767867639978;
      case 6: return 0.062790519529313376076178224565631133;
      case 8: return -0.425779291565072648862502445744251704;
      case 9: return -0.637423989748689710176712811676016195;
      case 12: return -0.992114701314477831049793042785778521;
      case 16: return -0.637423989748689710176712811676016195;
      default: return 1.0;
    }
  }
  static __device__ __forceinline__ constexpr double s(int k) {
    switch (k) {
      case 1: return 0.248689887164854788242283746006447968;
      case 2: return 0.481753674101715274987191502872129654;
      case 3: return 0.684547105928688673732283357621209270;
      case 4: return 0.844327925502015078548558063966681505;
      case 6: return 0.998026728428271561952336806863450553;
      case 8: return 0.904827052466019527713668647932697594;
      case 9: return 0.770513242775789230803009636396177847;
      case 12: return 0.125333233564304245373118759816508794;
      case 16: return -0.770513242775789230803009636396177847;
      default: return 0.0;
    }
  }
};
template <>
struct Root<27> {
  static __device__ __forceinline__ constexpr double c(int k) {
    switch (k) {
      case 1: return 0.973044870579823838832885172784695920;
      case 2: return 0.893632640323412248192574186866655117;
      case 3: return 0.766044443118978035202392650555416674;
      case 4: return 0.597158591702786164851852160583959773;
      case 5: return 0.396079766039156823696043391609744568;
      case 6: return 0.173648177666930348851716626769314796;
      case 7: return -0.058144828910475828538748016847071524;
      case 8: return -0.286803232711090253103280173167157937;
      case 10: return -0.686241637868733585729604999617537983;
      case 12: return -0.939692620785908384054109277324731470;
      case 14: return -0.993238357741942988547895552193704340;
      case 16: return -0.835487811412936419653826170019583594;
      default: return 1.0;
    }
  }
  static __device__ __forceinline__ constexpr double s(int k) {
    switch (k) {
      case 1: return 0.230615870742440178450198349292939102;
      case 2: return 0.448799180200462172785040334733143616;
      case 3: return 0.642787609686539326322643409907263433;
      case 4: return 0.802123192755043785083294891933925134;
      case 5: return 0.918216106880274014758961415314636602;
      case 6: return 0.984807753012208059366743024589523014;
      case 7: return 0.998308158271268208047820708783277533;
      case 8: return 0.957989512315488874437374766956754624;
      case 10: return 0.727373641573048695987176417663815522;
      case 12: return 0.342020143325668733044099614682259581;
      case 14: return -0.116092914125230229675666523380711469;
      case 16: return -0.549508978070806035262780374050133917;
      default: return 0.0;
    }
  }
};
template <>
struct Root<32> {
  static __device__ __forceinline__ constexpr double c(int k) {
    switch (k) {
      case 1: return 0.980785280403230449126182236134239037;
      case 2: return 0.923879532511286756128183189396788287;
      case 3: return 0.831469612302545237078788377617905757;
      case 4: return 0.707106781186547524400844362104849039;
      case 5: return 0.555570233019602224742830813948532874;
      case 6: return 0.382683432365089771728459984030398867;
      case 7: return 0.195090322016128267848284868477022241;
      case 8: return 0.0;
      case 9: return -0.195090322016128267848284868477022241;
      case 10: return -0.382683432365089771728459984030398867;
      case 12: return -0.707106781186547524400844362104849039;
      case 14: return -0.923879532511286756128183189396788287;
      case 15: return -0.980785280403230449126182236134239037;
      case 18: return -0.923879532511286756128183189396788287;
      case 21: return -0.555570233019602224742830813948532874;
      default: return 1.0;
    }
  }
  static __device__ __forceinline__ constexpr double s(int k) {
    switch (k) {
      case 1: return 0.195090322016128267848284868477022241;
      case 2: return 0.382683432365089771728459984030398867;
      case 3: return 0.555570233019602224742830813948532874;
      case 4: return 0.707106781186547524400844362104849039;
      case 5: return 0.831469612302545237078788377617905757;
      case 6: return 0.923879532511286756128183189396788287;
      case 7: return 0.980785280403230449126182236134239037;
      case 8: return 1.0;
      case 9: return 0.980785280403230449126182236134239037;
      case 10: return 0.923879532511286756128183189396788287;
      case 12: return 0.707106781186547524400844362104849039;
      case 14: return 0.382683432365089771728459984030398867;
      case 15: return 0.195090322016128267848284868477022241;
      case 18: return -0.382683432365089771728459984030398867;
      case 21: return -0.831469612302545237078788377617905757;
      default: return 0.0;
    }
  }
};

template <typename T, int R>
struct Dft;

template <typename T>
struct Dft<T, 1> {
  static __device__ __forceinline__ void run(cplx<T>*) {}
};
template <typename T>
struct Dft<T, 2> {
  static __device__ __forceinline__ void run(cplx<T>* v) { radix::dftR<T, false, 2>(v); }
};
template <typename T>
struct Dft<T, 3> {
  static __device__ __forceinline__ void run(cplx<T>* v) { radix::r3<T, false>(v); }
};
template <typename T>
struct Dft<T, 4> {
  static __device__ __forceinline__ void run(cplx<T>* v) { radix::r4<false>(v[0], v[1], v[2], v[3]); }
};
template <typename T>
struct Dft<T, 8> {
  static __device__ __forceinline__ void run(cplx<T>* v) { radix::r8<T, false>(v); }
};

// odd prime R: with t_m = v_m + v_{R-m} and d_m = v_m - v_{R-m},
// X_q, X_{R-q} = v_0 + sum_m t_m cos(2 pi m q / R) -+ i sum_m d_m sin(2 pi m q / R)
template <typename T, int R>
struct DftOdd {
  static __device__ __forceinline__ void run(cplx<T>* v) {
    using C = cplx<T>;
    constexpr int H = (R - 1) / 2;
    C t[H], d[H];
#pragma unroll
    for (int m = 1; m <= H; ++m) {
      t[m - 1] = cadd(v[m], v[R - m]);
      d[m - 1] = csub(v[m], v[R - m]);
    }
    const C v0 = v[0];
#pragma unroll
    for (int m = 0; m < H; ++m) v[0] = cadd(v[0], t[m]);
#pragma unroll
    for (int q = 1; q <= H; ++q) {
      C re = v0, im;
#pragma unroll
      for (int m = 1; m <= H; ++m) {
        const int e = (m * q) % R, f = e <= H ? e : R - e;
        const T c = T(Root<R>::c(f)), s = e <= H ? T(Root<R>::s(f)) : T(-Root<R>::s(f));
        re = cfma(t[m - 1], c, re);
        im = m == 1 ? cscale(d[0], s) : cfma(d[m - 1], s, im);
      }
      v[q] = cadd_rot<false>(re, im);
      v[R - q] = csub_rot<false>(re, im);
    }
  }
};
template <typename T>
struct Dft<T, 5> : DftOdd<T, 5> {};
template <typename T>
struct Dft<T, 7> : DftOdd<T, 7> {};
template <typename T>
struct Dft<T, 11> : DftOdd<T, 11> {};
template <typename T>
struct Dft<T, 13> : DftOdd<T, 13> {};

// R = A B: A-point DFTs over n1 (n = B n1 + n2), twiddles w_R^(n2 k1), B-point
// DFTs over n2, k = k1 + A k2
template <typename T, int A, int B>
struct DftSplit {
  static __device__ __forceinline__ void run(cplx<T>* v) {
    using C = cplx<T>;
    constexpr int R = A * B;
    C y[B][A];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) y[n2][n1] = v[B * n1 + n2];
      Dft<T, A>::run(y[n2]);
#pragma unroll
      for (int k1 = 1; k1 < A; ++k1)
        if (n2 > 0) {
          const int e = n2 * k1;
          const C w = mk<T>(T(Root<R>::c(e)), T(-Root<R>::s(e)));
          y[n2][k1] = cmul(y[n2][k1], w);
        }
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      C z[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) z[n2] = y[n2][k1];
      Dft<T, B>::run(z);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = z[k2];
    }
  }
};
template <typename T>
struct Dft<T, 9> : DftSplit<T, 3, 3> {};
template <typename T>
struct Dft<T, 16> : DftSplit<T, 4, 4> {};
template <typename T>
struct Dft<T, 25> : DftSplit<T, 5, 5> {};
template <typename T>
struct Dft<T, 27> : DftSplit<T, 3, 9> {};
template <typename T>
struct Dft<T, 32> : DftSplit<T, 8, 4> {};

// the k with k mod A = k1 and k mod B = k2
template <int A, int B>
__host__ __device__ constexpr int crt(int k1, int k2) {
  for (int k = k1; k < A * B; k += A)
    if (k % B == k2) return k;
  return 0;
}

// R = A B with coprime A and B
template <typename T, int A, int B>
struct DftCoprime {
  static __device__ __forceinline__ void run(cplx<T>* v) {
    using C = cplx<T>;
    constexpr int R = A * B, E1 = crt<A, B>(1, 0), E2 = crt<A, B>(0, 1);
    C y[B][A];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) y[n2][n1] = v[(B * n1 + A * n2) % R];
      Dft<T, A>::run(y[n2]);
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      C z[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) z[n2] = y[n2][k1];
      Dft<T, B>::run(z);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[(k1 * E1 + k2 * E2) % R] = z[k2];
    }
  }
};
template <typename T>
struct Dft<T, 6> : DftCoprime<T, 2, 3> {};
template <typename T>
struct Dft<T, 10> : DftCoprime<T, 2, 5> {};
template <typename T>
struct Dft<T, 12> : DftCoprime<T, 4, 3> {};
template <typename T>
struct Dft<T, 14> : DftCoprime<T, 2, 7> {};
template <typename T>
struct Dft<T, 15> : DftCoprime<T, 3, 5> {};
template <typename T>
struct Dft<T, 18> : DftCoprime<T, 2, 9> {};
template <typename T>
struct Dft<T, 20> : DftCoprime<T, 4, 5> {};
template <typename T>
struct Dft<T, 21> : DftCoprime<T, 3, 7> {};
template <typename T>
struct Dft<T, 24> : DftCoprime<T, 8, 3> {};
template <typename T>
struct Dft<T, 28> : DftCoprime<T, 4, 7> {};
template <typename T>
struct Dft<T, 30> : DftCoprime<T, 5, 6> {};

}  // namespace codelet
}  // namespace dev
}  // namespace dfft
