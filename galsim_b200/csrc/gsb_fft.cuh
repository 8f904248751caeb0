// Per-warp Stockham FFT in shared memory for N = 2^a or 3 * 2^a (N <= 1024).
//
// One warp owns one length-N transform held in a shared-memory buffer.  Each pass of radix
// R (3 first when N has a factor 3, then 4, then a final 2 if needed) reads R inputs per
// butterfly, applies the twiddles, does the R-point DFT in registers and, after a
// __syncwarp, writes the outputs back in Stockham (self-sorting) order, so the result is
// in natural order with no bit reversal.  Twiddles come from a per-block table
// tw[m] = exp(+2 pi i m / N) built in FP64.  SIGN = +1 is the unnormalised inverse DFT
// (FFTW_BACKWARD), SIGN = -1 the forward DFT.
#pragma once

#include <cuda_runtime.h>
#include <type_traits>

namespace gsb {

template <typename T> struct CxT;
template <> struct CxT<float>  { using type = float2; };
template <> struct CxT<double> { using type = double2; };
template <typename T> using Cx = typename CxT<T>::type;

template <typename T> __device__ __forceinline__ Cx<T> cx(T x, T y) { Cx<T> r; r.x = x; r.y = y; return r; }
template <typename T> __device__ __forceinline__ Cx<T> cadd(Cx<T> a, Cx<T> b) { return cx<T>(a.x + b.x, a.y + b.y); }
template <typename T> __device__ __forceinline__ Cx<T> csub(Cx<T> a, Cx<T> b) { return cx<T>(a.x - b.x, a.y - b.y); }
// Multiply-adds and additions whose rounding is stated rather than left to the compiler, which contracts
// a sum of products by its surroundings: what the fused and the split draw kernels share gives the same
// bits in both.
__device__ __forceinline__ float mul_add(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double mul_add(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
template <typename T> __device__ __forceinline__ Cx<T> cmul(Cx<T> a, Cx<T> b)
{ return cx<T>(mul_add(a.x, b.x, -mul_rn(a.y, b.y)), mul_add(a.x, b.y, mul_rn(a.y, b.x))); }
// The same with the imaginary part's other product rounded (the k-space products of the program).
template <typename T> __device__ __forceinline__ Cx<T> cmul_yx(Cx<T> a, Cx<T> b)
{ return cx<T>(mul_add(a.x, b.x, -mul_rn(a.y, b.y)), mul_add(a.y, b.x, mul_rn(a.x, b.y))); }
template <typename T> __device__ __forceinline__ Cx<T> cconj(Cx<T> a) { return cx<T>(a.x, -a.y); }
template <typename T> __device__ __forceinline__ Cx<T> cscale(Cx<T> a, T s) { return cx<T>(a.x * s, a.y * s); }
// multiply by SIGN * i
template <typename T, int SIGN> __device__ __forceinline__ Cx<T> cmul_si(Cx<T> a)
{ return SIGN > 0 ? cx<T>(-a.y, a.x) : cx<T>(a.y, -a.x); }

template <typename T, int R, int SIGN>
__device__ __forceinline__ void dft_small(Cx<T>* v)
{
    if constexpr (R == 2) {
        const Cx<T> a = v[0], b = v[1];
        v[0] = cadd<T>(a, b);
        v[1] = csub<T>(a, b);
    } else if constexpr (R == 3) {
        const Cx<T> a = v[0], b = v[1], c = v[2];
        const Cx<T> t1 = cadd<T>(b, c);
        const Cx<T> t2 = csub<T>(a, cscale<T>(t1, T(0.5)));
        const Cx<T> t3 = cmul_si<T, SIGN>(cscale<T>(csub<T>(b, c), T(0.86602540378443864676)));
        v[0] = cadd<T>(a, t1);
        v[1] = cadd<T>(t2, t3);
        v[2] = csub<T>(t2, t3);
    } else if constexpr (R == 4) {
        const Cx<T> a = v[0], b = v[1], c = v[2], d = v[3];
        const Cx<T> s0 = cadd<T>(a, c), s1 = csub<T>(a, c);
        const Cx<T> s2 = cadd<T>(b, d), s3 = cmul_si<T, SIGN>(csub<T>(b, d));
        v[0] = cadd<T>(s0, s2);
        v[1] = cadd<T>(s1, s3);
        v[2] = csub<T>(s0, s2);
        v[3] = csub<T>(s1, s3);
    } else if constexpr (R == 8) {
        // two 4-point transforms of the even and odd inputs, joined by the 8th roots of unity
        Cx<T> e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        dft_small<T, 4, SIGN>(e);
        dft_small<T, 4, SIGN>(o);
        const T h = T(0.70710678118654752440);
        const Cx<T> i1 = cmul_si<T, SIGN>(o[1]), i3 = cmul_si<T, SIGN>(o[3]);
        o[1] = cscale<T>(cadd<T>(o[1], i1), h);
        o[2] = cmul_si<T, SIGN>(o[2]);
        o[3] = cscale<T>(csub<T>(i3, o[3]), h);
#pragma unroll
        for (int r = 0; r < 4; ++r) { v[r] = cadd<T>(e[r], o[r]); v[r + 4] = csub<T>(e[r], o[r]); }
    }
}

// Where value i of a warp's buffer lies: bits 4-5 of the index are folded into bits 0-1 and 2-3, so
// that 16 lanes storing with stride 1, 4 or 16 values (the radix-4 passes' outputs), or loading
// consecutive ones, touch 16 different bank pairs (without it the first two passes' stores take
// four times as long).
__device__ __forceinline__ int fft_slot(int i) { return i ^ (((i >> 4) & 3) * 5); }

// One pass of the warp transform.  The first takes its inputs from load(i), the last hands its
// outputs to store(i, value); between passes the values are in buf (fft_slot).  LOAD_BUF / STORE_BUF:
// load / store address buf, so the warp waits between reading and writing.
template <typename T, int N, int R, int NS, int SIGN, bool LOAD_BUF, bool STORE_BUF, class Load, class Store>
__device__ __forceinline__ void stockham_pass(Cx<T>* buf, const Cx<T>* tw, int lane, const Load& load, const Store& store)
{
    constexpr int NB = N / R;
    constexpr int PER = (NB + 31) / 32;
    constexpr int TSTEP = N / (NS * R);
    constexpr bool FIRST = NS == 1, LAST = NS * R == N;
    Cx<T> v[PER][R];
#pragma unroll
    for (int t = 0; t < PER; ++t) {
        const int b = lane + 32 * t;
        if (NB % 32 == 0 || b < NB) {
            const int k = b % NS;
#pragma unroll
            for (int r = 0; r < R; ++r) v[t][r] = FIRST ? load(b + r * NB) : buf[fft_slot(b + r * NB)];
#pragma unroll
            for (int r = 1; r < R && NS > 1; ++r) {      // (the first pass's twiddles are 1)
                // r k TSTEP <= (R - 1)(NS - 1) N / (NS R) < N: no reduction mod N needed
                const int idx = r * k * TSTEP;
                Cx<T> w = tw[idx];
                if (SIGN < 0) w.y = -w.y;
                v[t][r] = cmul<T>(v[t][r], w);
            }
            dft_small<T, R, SIGN>(v[t]);
        }
    }
    if ((!FIRST || LOAD_BUF) && (!LAST || STORE_BUF)) __syncwarp();
#pragma unroll
    for (int t = 0; t < PER; ++t) {
        const int b = lane + 32 * t;
        if (NB % 32 == 0 || b < NB) {
            const int k = b % NS;
            const int base = (b / NS) * NS * R + k;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (LAST) store(base + r * NS, v[t][r]);
                else buf[fft_slot(base + r * NS)] = v[t][r];
            }
        }
    }
    __syncwarp();
}

template <typename T, int N, int NS, int SIGN, bool LOAD_BUF, bool STORE_BUF, class Load, class Store>
__device__ __forceinline__ void fft_passes(Cx<T>* buf, const Cx<T>* tw, int lane, const Load& load, const Store& store)
{
    if constexpr (NS < N) {
        constexpr int rem = N / NS;
        constexpr int R = (NS == 1 && (N % 3) == 0) ? 3 : ((rem % 4) == 0 ? 4 : 2);
        stockham_pass<T, N, R, NS, SIGN, LOAD_BUF, STORE_BUF>(buf, tw, lane, load, store);
        fft_passes<T, N, NS * R, SIGN, LOAD_BUF, STORE_BUF>(buf, tw, lane, load, store);
    }
}

// Length-N DFT by the calling warp (all 32 lanes call) from load(i) to store(i, value); buf holds N
// values of working space.  LOAD_BUF / STORE_BUF: load / store address buf[fft_slot(i)].
template <typename T, int N, int SIGN, bool LOAD_BUF, bool STORE_BUF, class Load, class Store>
__device__ __forceinline__ void warp_fft_io(Cx<T>* buf, const Cx<T>* tw, const Load& load, const Store& store)
{
    fft_passes<T, N, 1, SIGN, LOAD_BUF, STORE_BUF>(buf, tw, threadIdx.x & 31, load, store);
}

// tw[m] = exp(+2 pi i m / N), filled by the whole block.
template <typename T>
__device__ inline void fill_twiddles(Cx<T>* tw, int N)
{
    for (int m = threadIdx.x; m < N; m += blockDim.x) {
        double s, c;
        sincospi(2.0 * m / N, &s, &c);
        tw[m] = cx<T>(T(c), T(s));
    }
}

// Block-wide length-N DFT (N = 2^a or 3 * 2^a) in shared memory, Stockham order, N and the thread
// count known at compile time so that every index is a shift or a constant: radix 8 (4 and 2 for the
// rest of the power of two), the factor 3 last.  Up to N = 1024, where a bucket may also run the fused
// kernel, warp_fft_io's radix plan and twiddles, so that both give the same bits.  The first pass takes
// its inputs from load(i) and the last hands its outputs to store(i, value), so that a caller can read from
// or write to memory without a trip through the buffer.  tw: exp(+2 pi i m / N), m < N, in T (global).  A
// radix-8 butterfly reads all seven twiddles: three read and the others multiplied from them are 8 % faster
// (six stamps of N = 4096 .. 8192: device time 5.7 ms against 6.2) but half as exact again (float).  As it is
// the transform is as exact as the radix-4 plan: rms error of a float transform 1.17e-7 .. 1.28e-7 of its rms
// at N = 2048 .. 8192, against 1.15e-7 .. 1.26e-7 (emulated, random and decaying inputs).
// Between passes the values lie padded by one in 16 (8 in double), which spreads a radix-8 butterfly's
// adjacent outputs over the banks (16 lanes would share one otherwise): buf holds fft_buf_len values.
// LOAD_BUF / STORE_BUF: load / store address `buf` itself (their pass then waits for the block
// between reading and writing).  All threads call; on return the last pass's reads of buf are done
// by this thread only (sync before reusing it).
template <typename T>
__host__ __device__ constexpr bool fft_padded(int N) { return sizeof(Cx<T>) * size_t(N) <= 128 * 1024; }
template <typename T>
__host__ __device__ constexpr size_t fft_buf_len(int N)
{ return size_t(N) + (fft_padded<T>(N) ? size_t(N) >> (sizeof(T) == 4 ? 4 : 3) : 0); }

template <typename T, int N, int THREADS, int NS, int SIGN, bool LOAD_BUF, bool STORE_BUF, class Load, class Store>
__device__ __forceinline__ void block_fft_pass(Cx<T>* buf, const Cx<T>* __restrict__ tw, const Load& load,
                                               const Store& store)
{
    constexpr int REM = N / NS;
    constexpr int P2 = REM % 3 == 0 ? REM / 3 : REM;      // what is left of the power of two
    constexpr int R = N <= 1024 ? (NS == 1 && N % 3 == 0 ? 3 : REM % 4 == 0 ? 4 : 2)
                                : P2 == 1 ? 3 : P2 == 2 ? 2 : (P2 == 4 || P2 == 16) ? 4 : 8;
    constexpr int NB = N / R;
    constexpr int PER = (NB + THREADS - 1) / THREADS;
    constexpr int TSTEP = N / (NS * R);
    constexpr bool FIRST = NS == 1, LAST = NS * R == N;
    auto at = [](int i) { return fft_padded<T>(N) ? i + (i >> (sizeof(T) == 4 ? 4 : 3)) : i; };
    Cx<T> v[PER][R];
#pragma unroll
    for (int t = 0; t < PER; ++t) {
        const int b = int(threadIdx.x) + t * THREADS;
        if (NB % THREADS == 0 || b < NB) {
#pragma unroll
            for (int r = 0; r < R; ++r) v[t][r] = FIRST ? load(b + r * NB) : buf[at(b + r * NB)];
            if (NS > 1) {
                const int k = b % NS;
                auto w = [&](int r) {
                    Cx<T> z = tw[r * k * TSTEP];
                    if (SIGN < 0) z.y = -z.y;
                    return z;
                };
#pragma unroll
                for (int r = 1; r < R; ++r) v[t][r] = cmul<T>(v[t][r], w(r));
            }
            dft_small<T, R, SIGN>(v[t]);
        }
    }
    if ((!FIRST || LOAD_BUF) && (!LAST || STORE_BUF)) __syncthreads();
#pragma unroll
    for (int t = 0; t < PER; ++t) {
        const int b = int(threadIdx.x) + t * THREADS;
        if (NB % THREADS == 0 || b < NB) {
            const int k = b % NS, base = (b / NS) * (NS * R) + k;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (LAST) store(base + r * NS, v[t][r]);
                else buf[at(base + r * NS)] = v[t][r];
            }
        }
    }
    if constexpr (!LAST) {
        __syncthreads();
        block_fft_pass<T, N, THREADS, NS * R, SIGN, LOAD_BUF, STORE_BUF>(buf, tw, load, store);
    }
}

// In place: buf -> buf, synchronised on return.
template <typename T, int N, int THREADS>
__device__ __noinline__ void block_fft_n(Cx<T>* buf, const Cx<T>* __restrict__ tw)
{
    block_fft_pass<T, N, THREADS, 1, +1, true, true>(buf, tw, [&](int i) { return buf[i]; },
                                                     [&](int i, Cx<T> z) { buf[i] = z; });
    __syncthreads();
}

// buf -> out[0 .. N) (global), synchronised on return.
template <typename T, int N, int THREADS>
__device__ __noinline__ void block_fft_out(Cx<T>* buf, const Cx<T>* __restrict__ tw, Cx<T>* __restrict__ out)
{
    block_fft_pass<T, N, THREADS, 1, +1, true, false>(buf, tw, [&](int i) { return buf[i]; },
                                                      [&](int i, Cx<T> z) { out[i] = z; });
    __syncthreads();
}

// Whether block_fft_any transforms length N with that many threads (asked on the host before a launch).
__host__ __device__ constexpr bool block_fft_has(int N, int threads)
{
    int m = N;
    while (m > 1 && m % 2 == 0) m /= 2;
    if (m != 1 && m != 3) return false;
    return threads == 256 ? N >= 192 && N <= 1024 : threads == 512 ? N >= 1536 && N <= 8192 : threads == 1024 && N >= 1536 && N <= 16384;
}

// The sizes of the split path, one instantiation each (N uniform over the block).  OUT: to `out`.
template <typename T, int THREADS, bool OUT>
__device__ __forceinline__ void block_fft_any(Cx<T>* buf, int N, const Cx<T>* __restrict__ tw, Cx<T>* out = nullptr)
{
    auto run = [&](auto n) {
        constexpr int M = decltype(n)::value;
        if constexpr (M <= 32 * THREADS) {
            if constexpr (OUT) block_fft_out<T, M, THREADS>(buf, tw, out);
            else block_fft_n<T, M, THREADS>(buf, tw);
        }
    };
    if constexpr (THREADS == 256) {
        switch (N) {
          case 192: run(std::integral_constant<int, 192>{}); return;
          case 256: run(std::integral_constant<int, 256>{}); return;
          case 384: run(std::integral_constant<int, 384>{}); return;
          case 512: run(std::integral_constant<int, 512>{}); return;
          case 768: run(std::integral_constant<int, 768>{}); return;
          case 1024: run(std::integral_constant<int, 1024>{}); return;
        }
    }
    if constexpr (THREADS >= 512) {
        switch (N) {
          case 1536: run(std::integral_constant<int, 1536>{}); return;
          case 2048: run(std::integral_constant<int, 2048>{}); return;
          case 3072: run(std::integral_constant<int, 3072>{}); return;
          case 4096: run(std::integral_constant<int, 4096>{}); return;
          case 6144: run(std::integral_constant<int, 6144>{}); return;
          case 8192: run(std::integral_constant<int, 8192>{}); return;
        }
    }
    if constexpr (THREADS >= 1024) {
        switch (N) {
          case 12288: run(std::integral_constant<int, 12288>{}); return;
          case 16384: run(std::integral_constant<int, 16384>{}); return;
        }
    }
}

// Block-wide in-place Stockham FFT of length N (2^a or 3 * 2^a, N / R <= PER blockDim.x) in shared
// memory with warp_fft_io's radix plan; all threads of the block must call.  tw: exp(+2 pi i m / N) for
// m < N (global, FP64).
template <typename T, int SIGN, int PER = 4>
__device__ void block_fft(Cx<T>* buf, int N, const double2* __restrict__ tw)
{
    int NS = 1;
    while (NS < N) {
        const int rem = N / NS;
        const int R = (NS == 1 && N % 3 == 0) ? 3 : ((rem % 4) == 0 ? 4 : 2);
        const int NB = N / R;
        const int tstep = N / (NS * R);
        Cx<T> v[PER][4];
#pragma unroll
        for (int t = 0; t < PER; ++t) {
            const int b = threadIdx.x + t * blockDim.x;
            if (b < NB) {
                const int k = b % NS;
                for (int r = 0; r < R; ++r) v[t][r] = buf[b + r * NB];
                for (int r = 1; r < R; ++r) {
                    // r k tstep <= (R - 1)(NS - 1) N / (NS R) < N
                    const double2 w = __ldg(&tw[r * k * tstep]);
                    v[t][r] = cmul<T>(v[t][r], cx<T>(T(w.x), SIGN > 0 ? T(w.y) : T(-w.y)));
                }
                if (R == 4) dft_small<T, 4, SIGN>(v[t]);
                else if (R == 3) dft_small<T, 3, SIGN>(v[t]);
                else dft_small<T, 2, SIGN>(v[t]);
            }
        }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < PER; ++t) {
            const int b = threadIdx.x + t * blockDim.x;
            if (b < NB) {
                const int k = b % NS;
                const int base = (b / NS) * NS * R + k;
                for (int r = 0; r < R; ++r) buf[base + r * NS] = v[t][r];
            }
        }
        __syncthreads();
        NS *= R;
    }
}

}  // namespace gsb
