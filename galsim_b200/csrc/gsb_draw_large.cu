// Large-FFT drawing path (1024 < N <= 16384): two kernels per chunk of stamps.
//
//   large_col_kernel: one CTA per (column group, stamp).  For each column kx = 0..N/2 it
//     builds the wrapped k-values of all N rows (alias sums of the program, as in the fused
//     kernel), inverse-transforms them with a block-wide Stockham FFT in shared memory and
//     stores the column into the stamp's slab W (column-major, coalesced).
//   large_row_kernel: one CTA per (row pair, stamp).  It gathers two image rows of W,
//     packs them as one complex row (row1 + i row2, Hermitian-extended in kx), transforms it,
//     writes the pixels inside the stamp scaled by 1/N^2 and adds the compensated flux sum.
// The slab W is the only HBM round trip; the chunk size keeps it inside the workspace.
#include <algorithm>
#include <map>
#include <mutex>

#include "gsb_draw.cuh"

namespace gsb {

static __global__ void twiddle_kernel(double2* tw, int N)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= N) return;
    double s, c;
    sincospi(2.0 * m / N, &s, &c);
    tw[m] = make_double2(c, s);
    reinterpret_cast<float2*>(tw + N)[m] = make_float2(float(c), float(s));
}

static std::map<int, double2*>& twiddle_cache()
{
    static std::map<int, double2*> cache[64];
    int dev = 0;
    cudaGetDevice(&dev);
    return cache[dev & 63];
}

// exp(+2 pi i m / N), m < N, in FP64 and after it rounded to FP32: built once per (device, N) and kept
// for the process.
int fft_twiddles(int N, cudaStream_t stream, const double2** out)
{
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    auto& c = twiddle_cache();
    auto it = c.find(N);
    if (it != c.end()) { *out = it->second; return GSB_OK; }
    double2* tw = nullptr;
    GSB_CUDA_CHECK(cudaMalloc(&tw, (sizeof(double2) + sizeof(float2)) * N));
    twiddle_kernel<<<(N + 255) / 256, 256, 0, stream>>>(tw, N);
    GSB_CUDA_CHECK(cudaGetLastError());
    GSB_CUDA_CHECK(cudaStreamSynchronize(stream));
    c[N] = tw;
    *out = tw;
    return GSB_OK;
}

namespace {

template <typename T> __device__ __forceinline__ const Cx<T>* twiddles(const double2* tw, int N);
template <> __device__ __forceinline__ const double2* twiddles<double>(const double2* tw, int) { return tw; }
template <> __device__ __forceinline__ const float2* twiddles<float>(const double2* tw, int N)
{ return reinterpret_cast<const float2*>(tw + N); }

struct LargeArgs {
    DrawArgs a;          // leaves/phases/scales/stamps already offset to the chunk
    int N;
    const double2* tw;
    void* W;             // n_stamps slabs of (N/2+1) x N complex
    int cache_bytes;     // shared memory for the per-stamp caches (factored program)
};

// Float arithmetic drawn into a double image takes the fused kernels' radix plan above N = 1024 too, with
// the general forms of the profiles (set_leaf_const): what such an image holds does not depend on its FFT
// size.  One object at a time is what is mostly drawn so, where the FFTs are little of the call (a 150 x 150
// image 0.86 ms); a batch of large stamps is slower by it (six of N = 4096 .. 8192: 11.7 ms against 6.8).
// PER: radix 2 at N = 8192 has 8 butterflies a thread.
template <int THREADS>
__device__ __noinline__ void block_fft_mixed(float2* buf, int N, const double2* tw)
{ block_fft<float, +1, (THREADS >= 1024 ? 4 : 8)>(buf, N, tw); }
template <int THREADS>
__device__ __forceinline__ void block_fft_mixed(double2*, int, const double2*) {}

// 256 threads for N <= 1024 (two CTAs an SM), 512 up to 8192, 1024 above: up to 128 registers but for
// the last, so that four wave vectors a thread and a radix-8 butterfly stay in them.
template <typename T, int THREADS, bool II>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? 2 : 1) large_col_kernel(const __grid_constant__ LargeArgs la)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    StampSmem& S = *reinterpret_cast<StampSmem*>(smem_raw);
    Cx<T>* buf = reinterpret_cast<Cx<T>*>(smem_raw + ((sizeof(StampSmem) + 15) & ~size_t(15)));
    const DrawArgs& a = la.a;
    const int N = la.N, H = N / 2 + 1;
    unsigned char* cache = reinterpret_cast<unsigned char*>(buf + ((fft_buf_len<T>(N) + 1) & ~size_t(1)));
    const int s = blockIdx.y;
    const double dk = 2. * kPi / N;
    load_stamp(S, a.tpl, s, a.leaves, a.phases, a.scales, a.stamps, a.sersic_header, a.sersic_node,
               a.sersic_stride, 1. / N);
    __syncthreads();
    const int Nk = S.geom.Nk, hk = Nk / 2;
    if (threadIdx.x == 0)
        plan_caches<T, II>(S, a.tpl, a.fac, Nk, 0u, N <= 1024 ? form_budget<T>(N) : la.cache_bytes, la.cache_bytes);
    __syncthreads();
    fill_caches<T, II>(S, a.tpl, cache, dk, Nk, sizeof(T) == 4 && a.out_dtype == GSB_F64);
    __syncthreads();
    Cx<T>* W = reinterpret_cast<Cx<T>*>(la.W) + (size_t)s * H * N;
    for (int c = blockIdx.x; c < H; c += gridDim.x) {
        const int kx0 = c + ceil_div(-hk - c, N) * N;
        if (sizeof(T) == 4 && N % THREADS == 0) {
            // the column's rows ky = -hk .. hk in order over the threads: a thread's slots s, s + NS, ...
            // are the aliases of one wrapped row, V slots at a time (as in draw_fused_kernel)
            constexpr int V = 4;
            const int NS = N / THREADS;
            for (int s0 = 0; s0 < NS; s0 += V) {
                const int nv = min(V, NS - s0);
                Cx<T> acc[V], comp[V];
#pragma unroll
                for (int v = 0; v < V; ++v) acc[v] = comp[v] = cx<T>(T(0), T(0));
                for (int kx = kx0; kx <= hk; kx += N) {
                    const bool pos = kx >= 0;
                    const int ii = pos ? kx : -kx;
                    for (int e0 = -hk + THREADS * s0; e0 <= hk; e0 += N) {
                        const int ky = e0 + int(threadIdx.x);
                        if (nv == V && e0 + THREADS * V - 1 <= hk) {
                            eval_any<T, II, V, false>(
                                a.tpl, S, cache, ii, pos ? ky : -ky, pos ? THREADS : -THREADS, hk, dk,
                                [&](int v, Cx<T> z, T r) { kahan_add<T>(acc[v], comp[v], z, r, pos); });
                        } else {
#pragma unroll 1
                            for (int u = 0; u < nv; ++u) {
                                const int ku = ky + THREADS * u;
                                if (ku > hk) break;
                                const Values<T, 1> z = eval_point<T, II>(a.tpl, S, cache, ii, pos ? ku : -ku, hk, dk);
#pragma unroll
                                for (int v = 0; v < V; ++v)
                                    if (v == u) kahan_add<T>(acc[v], comp[v], z.v[0], z.r[0], pos);
                            }
                        }
                    }
                }
#pragma unroll
                for (int v = 0; v < V; ++v)
                    if (v < nv) buf[pmod(-hk + THREADS * (s0 + v) + int(threadIdx.x), N)] = acc[v];
            }
        } else {
            // (double: one point at a time, compiled in place -- 1024 threads leave 64 registers, which
            // a call's saved registers would spill: 9.2 ms in place, 13.7 as calls, two stamps of 8192)
            for (int r = threadIdx.x; r < N; r += blockDim.x) {
                const int kyc = r < N / 2 ? r : r - N;
                Cx<T> acc = cx<T>(T(0), T(0)), comp = acc;     // Kahan-compensated fold
                for (int kx = kx0; kx <= hk; kx += N) {
                    const bool pos = kx >= 0;
                    for (int ky = kyc + ceil_div(-hk - kyc, N) * N; ky <= hk; ky += N) {
                        const Values<T, 1> z = eval_point<T, II, sizeof(T) == 8>(a.tpl, S, cache, pos ? kx : -kx, pos ? ky : -ky, hk, dk);
                        kahan_add<T>(acc, comp, z.v[0], z.r[0], pos);
                    }
                }
                buf[r] = acc;
            }
        }
        __syncthreads();
        if (sizeof(T) == 4 && a.out_dtype == GSB_F64 && N > 1024) {
            block_fft_mixed<THREADS>(buf, N, la.tw);
            for (int r = threadIdx.x; r < N; r += blockDim.x) W[(size_t)c * N + r] = buf[r];
            __syncthreads();
        } else {
            block_fft_any<T, THREADS, true>(buf, N, twiddles<T>(la.tw, N), W + (size_t)c * N);
        }
    }
}

// Threads of the row kernel: a radix-8 butterfly each, 512 at most (1024 above N = 8192).
__host__ __device__ constexpr int row_threads(int N)
{
    return N > 8192 ? 1024 : N >= 4096 ? 512 : N >= 2048 ? 256 : N >= 1024 ? 128 : 64;
}

// The rows' FFT reads its inputs straight from the slab and writes the stamp's pixels from its last
// pass, two image rows a transform.  Bound by the slab's reads (two of a 32-byte sector's values a
// row pair, the neighbouring pair's in L2) and the shared-memory passes between.
template <typename T, int N>
__global__ void __launch_bounds__(row_threads(N)) large_row_kernel(const __grid_constant__ LargeArgs la)
{
    constexpr int THREADS = row_threads(N);
    constexpr int H = N / 2 + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Cx<T>* buf = reinterpret_cast<Cx<T>*>(smem_raw);
    __shared__ gsb_stamp geom;
    const DrawArgs& a = la.a;
    const int s = blockIdx.y;
    if (threadIdx.x == 0) geom = a.stamps[s];
    __syncthreads();
    const gsb_stamp G = geom;
    const Cx<T>* tw = twiddles<T>(la.tw, N);
    const Cx<T>* W = reinterpret_cast<const Cx<T>*>(la.W) + (size_t)s * H * N;
    const T inv_n2 = T(1) / (T(N) * T(N));
    const int npairs = (G.ny + 1) / 2;
    double fsum = 0., fcomp = 0.;
    for (int p = blockIdx.x; p < npairs; p += gridDim.x) {
        const int py1 = G.ymin + 2 * p;
        const bool two = 2 * p + 1 < G.ny;
        const int y1 = pmod(py1, N), y2 = pmod(py1 + 1, N);
        const long long row1 = G.out_offset + (long long)(2 * p) * G.nx;
        auto load = [&](int kx) {
            const bool up = kx < H;
            const Cx<T>* w = W + (size_t)(up ? kx : N - kx) * N;
            Cx<T> a1 = w[y1], a2 = two ? w[y2] : cx<T>(T(0), T(0));
            if (!up) { a1 = cconj<T>(a1); a2 = cconj<T>(a2); }
            return cx<T>(a1.x - a2.y, a1.y + a2.x);
        };
        auto add = [&](double x) {        // Neumaier's compensated sum in FP64
            const double t = fsum + x;
            fcomp += fabs(fsum) >= fabs(x) ? (fsum - t) + x : (x - t) + fsum;
            fsum = t;
        };
        auto store = [&](int x, Cx<T> v) {
            int i = x - G.xmin % N;
            if (i >= N) i -= N;
            if (i < 0) i += N;
            for (; i < G.nx; i += N) {
                const T v1 = v.x * inv_n2;
                store_pixel<T>(a.out, a.out_dtype, a.add, row1 + i, v1);
                add(double(v1));
                if (two) {
                    const T v2 = v.y * inv_n2;
                    store_pixel<T>(a.out, a.out_dtype, a.add, row1 + G.nx + i, v2);
                    add(double(v2));
                }
            }
        };
        if (sizeof(T) == 4 && N > 1024 && a.out_dtype == GSB_F64) {
            for (int kx = threadIdx.x; kx < N; kx += THREADS) buf[kx] = load(kx);
            __syncthreads();
            block_fft_mixed<THREADS>(buf, N, la.tw);
            for (int x = threadIdx.x; x < N; x += THREADS) store(x, buf[x]);
        } else {
            block_fft_pass<T, N, THREADS, 1, +1, false, false>(buf, tw, load, store);
        }
        __syncthreads();
    }
    if (a.added_flux) {
        double v = fsum + fcomp;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        __shared__ double part[THREADS / 32];
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            double tot = 0.;
            for (int w = 0; w < THREADS / 32; ++w) tot += part[w];
            atomicAdd(&a.added_flux[s], tot);
        }
    }
}

template <typename T>
size_t slab_bytes(int N) { return sizeof(Cx<T>) * (size_t)(N / 2 + 1) * N; }

template <typename T>
size_t large_smem() { return ((sizeof(StampSmem) + 15) & ~size_t(15)); }

template <typename T, int N>
int launch_rows_n(const LargeArgs& la, dim3 grid, cudaStream_t stream)
{
    constexpr size_t sm = sizeof(Cx<T>) * fft_buf_len<T>(N);
    GSB_CUDA_CHECK(cudaFuncSetAttribute(large_row_kernel<T, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm)));
    large_row_kernel<T, N><<<grid, row_threads(N), sm, stream>>>(la);
    GSB_CUDA_CHECK(cudaGetLastError());
    return GSB_OK;
}

template <typename T>
int launch_rows(const LargeArgs& la, int N, dim3 grid, cudaStream_t stream)
{
    switch (N) {
      case 192: return launch_rows_n<T, 192>(la, grid, stream);
      case 256: return launch_rows_n<T, 256>(la, grid, stream);
      case 384: return launch_rows_n<T, 384>(la, grid, stream);
      case 512: return launch_rows_n<T, 512>(la, grid, stream);
      case 768: return launch_rows_n<T, 768>(la, grid, stream);
      case 1024: return launch_rows_n<T, 1024>(la, grid, stream);
      case 1536: return launch_rows_n<T, 1536>(la, grid, stream);
      case 2048: return launch_rows_n<T, 2048>(la, grid, stream);
      case 3072: return launch_rows_n<T, 3072>(la, grid, stream);
      case 4096: return launch_rows_n<T, 4096>(la, grid, stream);
      case 6144: return launch_rows_n<T, 6144>(la, grid, stream);
      case 8192: return launch_rows_n<T, 8192>(la, grid, stream);
      case 12288: return launch_rows_n<T, 12288>(la, grid, stream);
      case 16384: if constexpr (sizeof(T) == 4) return launch_rows_n<T, 16384>(la, grid, stream);
    }
    return set_error(GSB_ERR_UNSUPPORTED, "FFT size too large for this precision");
}

template <typename T, int THREADS>
int launch_large_t(const DrawArgs& args, int N, void* work, size_t work_bytes, cudaStream_t stream)
{
    if (!block_fft_has(N, THREADS)) return set_error(GSB_ERR_UNSUPPORTED, "FFT size not built");
    const size_t slab = slab_bytes<T>(N);
    if (!work || work_bytes < slab) return set_error(GSB_ERR_INVALID, "draw workspace too small");
    const size_t base = large_smem<T>() + sizeof(Cx<T>) * ((fft_buf_len<T>(N) + 1) & ~size_t(1));
    if (base > kSmemLimit) return set_error(GSB_ERR_UNSUPPORTED, "FFT size too large for this precision");
    // the rest of shared memory (up to 192 KB) holds the per-stamp caches of the column kernel; for
    // N <= 1024 as much as two CTAs an SM leave (the fused kernels' budget, and image taps)
    const size_t room = kSmemLimit - base > 1024 ? kSmemLimit - base - 1024 : 0;
    const size_t want = THREADS == 256 ? std::min<size_t>(28 * 1024 + 64 * sizeof(T) / 4 * N, 112 * 1024 - base)
                                       : size_t(192) * 1024;
    if (THREADS == 256 && std::min(room, want) < size_t(form_budget<T>(N)))
        return set_error(GSB_ERR_UNSUPPORTED, "FFT size too large for this precision");
    const int cache_bytes = int(std::min<size_t>(room, want) & ~size_t(15));
    const size_t sm = base + cache_bytes;
    const double2* tw = nullptr;
    int rc = fft_twiddles(N, stream, &tw);
    if (rc) return rc;
    // programs without image leaves run the column kernel compiled without their code
    const bool ii = has_image_leaves(args.tpl);
    if (ii)
        GSB_CUDA_CHECK(cudaFuncSetAttribute(large_col_kernel<T, THREADS, true>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm)));
    else
        GSB_CUDA_CHECK(cudaFuncSetAttribute(large_col_kernel<T, THREADS, false>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm)));
    const int chunk = int(std::max<size_t>(1, std::min<size_t>(work_bytes / slab, 65535)));
    DeviceState* st = device_state();
    if (args.added_flux)
        GSB_CUDA_CHECK(cudaMemsetAsync(args.added_flux, 0, sizeof(double) * args.n_stamps, stream));
    for (int s0 = 0; s0 < args.n_stamps; s0 += chunk) {
        const int n = std::min(chunk, args.n_stamps - s0);
        LargeArgs la;
        la.a = args;
        la.a.n_stamps = n;
        la.a.leaves = args.leaves + (size_t)s0 * args.tpl.n_leaves;
        la.a.phases = args.phases ? args.phases + (size_t)s0 * args.tpl.n_phases : nullptr;
        la.a.scales = args.scales ? args.scales + (size_t)s0 * args.tpl.n_scales : nullptr;
        la.a.stamps = args.stamps + s0;
        la.a.added_flux = args.added_flux ? args.added_flux + s0 : nullptr;
        la.N = N;
        la.tw = tw;
        la.W = work;
        la.cache_bytes = cache_bytes;
        const int cols = N / 2 + 1;
        const int gx = std::max(1, std::min(cols, (2 * st->sm_count + n - 1) / n));
        if (ii) large_col_kernel<T, THREADS, true><<<dim3(gx, n), THREADS, sm, stream>>>(la);
        else large_col_kernel<T, THREADS, false><<<dim3(gx, n), THREADS, sm, stream>>>(la);
        GSB_CUDA_CHECK(cudaGetLastError());
        // (as many row CTAs as are resident at once)
        const int per_sm = std::max(1, std::min(int(kSmemLimit / (sizeof(Cx<T>) * fft_buf_len<T>(N) + 1024)), 1024 / row_threads(N)));
        const int gr = std::max(1, std::min(N / 2, (per_sm * st->sm_count + n - 1) / n));
        const int rr = launch_rows<T>(la, N, dim3(gr, n), stream);
        if (rr) return rr;
    }
    return GSB_OK;
}

template <typename T>
int launch_large(const DrawArgs& args, int N, void* work, size_t work_bytes, cudaStream_t stream)
{
    if (N <= 1024) return launch_large_t<T, 256>(args, N, work, work_bytes, stream);
    if (N <= 8192) return launch_large_t<T, 512>(args, N, work, work_bytes, stream);
    return launch_large_t<T, 1024>(args, N, work, work_bytes, stream);
}

}  // namespace

bool is_large_fft(int N) { return N > 1024 && N <= 16384; }

size_t large_workspace_size(int N, int n_stamps, int precision)
{
    const size_t slab = precision == GSB_F64 ? slab_bytes<double>(N) : slab_bytes<float>(N);
    // up to 8 GiB of slabs per chunk, at least one stamp
    const size_t budget = size_t(8) << 30;
    const size_t k = std::max<size_t>(1, std::min<size_t>((size_t)n_stamps, budget / slab));
    return k * slab;
}

int draw_large(const DrawArgs& args, int N, int precision, void* work, size_t work_bytes,
               cudaStream_t stream)
{
    return precision == GSB_F64 ? launch_large<double>(args, N, work, work_bytes, stream)
                                : launch_large<float>(args, N, work, work_bytes, stream);
}

}  // namespace gsb
