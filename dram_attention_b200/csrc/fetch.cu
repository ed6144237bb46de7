// Miss-page fetch (gather-copy DRAM -> HBM slots, driven by the device-side miss
// list) and the cache construction pass (pagination, page summaries, warm start).

#include "da_common.cuh"

namespace da {

constexpr int kFetchThreads = 256;
constexpr int kFetchCtasPerHead = 64;

// One CTA per page in flight; each thread moves 16 bytes per load.  The source
// may be pinned host memory mapped into the device address space: many CTAs with
// several independent 128-bit loads each keep the host link busy.
__global__ void __launch_bounds__(kFetchThreads)
fetch_pages_kernel(const uint4 *__restrict__ dram, uint4 *__restrict__ slots,
                   const int32_t *__restrict__ miss_pages, const int32_t *__restrict__ miss_slots,
                   const int32_t *__restrict__ n_miss, int list_len, int n_dram_pages, int n_slots,
                   int page_vecs) {
    const int h = blockIdx.y;
    const int n = min(n_miss[h], list_len);
    for (int j = blockIdx.x; j < n; j += gridDim.x) {
        const int p = miss_pages[(size_t)h * list_len + j];
        const int v = miss_slots[(size_t)h * list_len + j];
        if (p < 0 || p >= n_dram_pages || v < 0 || v >= n_slots) continue;
        const uint4 *src = dram + ((size_t)h * n_dram_pages + p) * page_vecs;
        uint4 *dst = slots + ((size_t)h * n_slots + v) * page_vecs;
        for (int i0 = threadIdx.x; i0 < page_vecs; i0 += kFetchThreads * 4) {
            uint4 r[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = i0 + u * kFetchThreads;
                if (i < page_vecs) r[u] = __ldcs(src + i);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = i0 + u * kFetchThreads;
                if (i < page_vecs) dst[i] = r[u];
            }
        }
    }
}

__global__ void __launch_bounds__(kFetchThreads)
fetch_pages_bytes_kernel(const unsigned char *__restrict__ dram, unsigned char *__restrict__ slots,
                         const int32_t *__restrict__ miss_pages, const int32_t *__restrict__ miss_slots,
                         const int32_t *__restrict__ n_miss, int list_len, int n_dram_pages, int n_slots,
                         size_t page_bytes) {
    const int h = blockIdx.y;
    const int n = min(n_miss[h], list_len);
    for (int j = blockIdx.x; j < n; j += gridDim.x) {
        const int p = miss_pages[(size_t)h * list_len + j];
        const int v = miss_slots[(size_t)h * list_len + j];
        if (p < 0 || p >= n_dram_pages || v < 0 || v >= n_slots) continue;
        const unsigned char *src = dram + ((size_t)h * n_dram_pages + p) * page_bytes;
        unsigned char *dst = slots + ((size_t)h * n_slots + v) * page_bytes;
        for (size_t i = threadIdx.x; i < page_bytes; i += kFetchThreads) dst[i] = src[i];
    }
}

// Cache construction: CTA (page, head), thread = channel.  Reads K and V rows of
// the page's tokens, writes the page payload (token-major, key then value), the
// per-channel min/max summary, and the slot copy for the pages that start out
// resident.
template <typename T>
__global__ void build_pages_kernel(const T *__restrict__ k, const T *__restrict__ v, long long tok_stride,
                                   long long head_stride, T *__restrict__ dram, T *__restrict__ summaries,
                                   T *__restrict__ slots, int n_pages, int n_slots, int page_size,
                                   int head_dim) {
    const int page = blockIdx.x;
    const int h = blockIdx.y;
    const int first_resident = n_pages - n_slots;
    for (int d = threadIdx.x; d < head_dim; d += blockDim.x) {
        float mn = 0.f, mx = 0.f;
        T tmn = T(), tmx = T();
        for (int t = 0; t < page_size; ++t) {
            const size_t src = (size_t)(page * (long long)page_size + t) * tok_stride + (size_t)h * head_stride + d;
            const T kv = k[src];
            const T vv = v[src];
            const float kf = to_float(kv);
            if (t == 0 || kf < mn) { mn = kf; tmn = kv; }
            if (t == 0 || kf > mx) { mx = kf; tmx = kv; }
            const size_t off = ((size_t)t * 2) * head_dim + d;
            if (dram) {
                T *pg = dram + ((size_t)h * n_pages + page) * page_size * 2 * head_dim;
                pg[off] = kv;
                pg[off + head_dim] = vv;
            }
            if (slots && page >= first_resident) {
                T *sl = slots + ((size_t)h * n_slots + (page - first_resident)) * page_size * 2 * head_dim;
                sl[off] = kv;
                sl[off + head_dim] = vv;
            }
        }
        if (summaries) {
            T *sm = summaries + ((size_t)h * n_pages + page) * 2 * head_dim;
            sm[d] = tmn;
            sm[head_dim + d] = tmx;
        }
    }
}

// The same pass with 16 bytes per thread and load: 2 * chunks consecutive threads take one page of one head
// (chunks = 16-byte pieces of a row), thread c the c-th piece of its key row, then value row, of every token, so that
// a token leaves as one contiguous run of both rows and a thread sees all the keys of its channels (no exchange for
// the summaries).  For rows of whole 16-byte pieces, at most 1 KB long, on 16-byte boundaries.  Neighbouring groups take
// the heads of a page, whose rows are neighbours in the prompt's keys.
constexpr int kBuildThreads = 128;
constexpr int kBuildUnroll = 4;
constexpr int kBuildSms = 148;
// With pages in host memory the link is the bound, and a few CTAs keep it busy: 117 MB in 2269, 2254, 2255 us with
// 8, 24, 148 CTAs (52 GB/s; two bytes per thread and a CTA per page: 2678).  A CTA here takes 10 000 registers, more than two
// prefill CTAs leave of an SM: beside the prompt's attention each of the 24 keeps one prefill CTA off for the transfer.
// Pages in device memory take the whole chip.
constexpr int kBuildLinkCtas = 24;

// Per element of a 32-bit word: the smaller (larger) one as it lies in memory, the one that was there first when they
// do not compare (zeros of either sign, NaN).
template <typename T> __device__ __forceinline__ void keep_extremes(uint32_t w, uint32_t &mn, uint32_t &mx) {
    if constexpr (sizeof(T) == 4) {
        const float f = __uint_as_float(w);
        if (f < __uint_as_float(mn)) mn = w;
        if (f > __uint_as_float(mx)) mx = w;
    } else {
        float f0, f1, a0, a1, b0, b1;
        unpack2<T>(w, f0, f1);
        unpack2<T>(mn, a0, a1);
        unpack2<T>(mx, b0, b1);
        mn = (f0 < a0 ? w & 0xffffu : mn & 0xffffu) | (f1 < a1 ? w & 0xffff0000u : mn & 0xffff0000u);
        mx = (f0 > b0 ? w & 0xffffu : mx & 0xffffu) | (f1 > b1 ? w & 0xffff0000u : mx & 0xffff0000u);
    }
}

template <typename T>
__global__ void __launch_bounds__(kBuildThreads)
build_pages_vec_kernel(const unsigned char *__restrict__ k, const unsigned char *__restrict__ v, long long tok_stride,
                       long long head_stride, uint4 *__restrict__ dram, uint4 *__restrict__ summaries,
                       uint4 *__restrict__ slots, int n_kv_heads, int n_pages, int n_slots, int page_size, int chunks) {
    const int lanes = 2 * chunks;
    const int groups = kBuildThreads / lanes;
    const int g = threadIdx.x / lanes;
    if (g >= groups) return;
    const int c = threadIdx.x - g * lanes;
    const bool is_key = c < chunks;
    if (!is_key && !dram && !slots) return;   // summaries alone
    const unsigned char *rows = (is_key ? k : v) + (size_t)(is_key ? c : c - chunks) * 16;
    const int first_resident = n_pages - n_slots;
    const long long page_vecs = (long long)page_size * lanes;
    const unsigned items = (unsigned)n_pages * (unsigned)n_kv_heads;
    for (unsigned item = blockIdx.x * groups + g; item < items; item += gridDim.x * groups) {
        const int page = (int)(item / (unsigned)n_kv_heads);
        const int h = (int)(item % (unsigned)n_kv_heads);
        const unsigned char *src = rows + (long long)page * page_size * tok_stride + (long long)h * head_stride;
        uint4 *pg = dram ? dram + ((long long)h * n_pages + page) * page_vecs + c : nullptr;
        uint4 *sl = slots && page >= first_resident
                        ? slots + ((long long)h * n_slots + (page - first_resident)) * page_vecs + c : nullptr;
        uint32_t mn[4] = {0, 0, 0, 0}, mx[4] = {0, 0, 0, 0};
#pragma unroll 1
        for (int t0 = 0; t0 < page_size; t0 += kBuildUnroll) {
            const int n = page_size - t0;
            uint4 r[kBuildUnroll];
#pragma unroll
            for (int u = 0; u < kBuildUnroll; ++u) {
                if (u < n) r[u] = *reinterpret_cast<const uint4 *>(src);
                src += tok_stride;
            }
            if (pg) {
#pragma unroll
                for (int u = 0; u < kBuildUnroll; ++u) {
                    if (u < n) *pg = r[u];
                    pg += lanes;
                }
            }
            if (sl) {
#pragma unroll
                for (int u = 0; u < kBuildUnroll; ++u) {
                    if (u < n) *sl = r[u];
                    sl += lanes;
                }
            }
            if (!summaries || !is_key) continue;
#pragma unroll
            for (int u = 0; u < kBuildUnroll; ++u) {
                if (u >= n) break;
                const uint32_t w[4] = {r[u].x, r[u].y, r[u].z, r[u].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (u == 0 && t0 == 0) mn[i] = mx[i] = w[i];
                    keep_extremes<T>(w[i], mn[i], mx[i]);
                }
            }
        }
        if (summaries && is_key) {
            uint4 *sm = summaries + ((long long)h * n_pages + page) * lanes + c;
            sm[0] = make_uint4(mn[0], mn[1], mn[2], mn[3]);
            sm[chunks] = make_uint4(mx[0], mx[1], mx[2], mx[3]);
        }
    }
}

static bool in_device_memory(const void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) == cudaSuccess) return a.type == cudaMemoryTypeDevice;
    (void)cudaGetLastError();
    return false;
}

template <typename T>
static cudaError_t launch_build(const void *k, const void *v, long long tok_stride, long long head_stride,
                                void *dram, void *summaries, void *slots, int n_kv_heads, int n_pages,
                                int n_slots, int page_size, int head_dim, cudaStream_t stream) {
    constexpr long long E = (long long)sizeof(T);
    const int chunks = (int)(head_dim * E / 16);
    const uintptr_t all = (uintptr_t)k | (uintptr_t)v | (uintptr_t)dram | (uintptr_t)summaries | (uintptr_t)slots |
                          (uintptr_t)(tok_stride * E) | (uintptr_t)(head_stride * E) | (uintptr_t)(head_dim * E);
    if ((all & 15) == 0 && 2 * chunks <= kBuildThreads && (long long)n_pages * n_kv_heads <= 0x7fffffffll) {
        const long long groups = kBuildThreads / (2 * chunks);
        long long ctas = ((long long)n_pages * n_kv_heads + groups - 1) / groups;
        const long long most = dram && !in_device_memory(dram) ? kBuildLinkCtas : 12 * kBuildSms;
        if (ctas > most) ctas = most;
        build_pages_vec_kernel<T><<<(unsigned)ctas, kBuildThreads, 0, stream>>>(
            static_cast<const unsigned char *>(k), static_cast<const unsigned char *>(v), tok_stride * E,
            head_stride * E, static_cast<uint4 *>(dram), static_cast<uint4 *>(summaries), static_cast<uint4 *>(slots),
            n_kv_heads, n_pages, n_slots, page_size, chunks);
        return cudaGetLastError();
    }
    int threads = head_dim < 32 ? 32 : (head_dim > 256 ? 256 : (head_dim + 31) / 32 * 32);
    dim3 grid(n_pages, n_kv_heads);
    build_pages_kernel<T><<<grid, threads, 0, stream>>>(
        static_cast<const T *>(k), static_cast<const T *>(v), tok_stride, head_stride, static_cast<T *>(dram),
        static_cast<T *>(summaries), static_cast<T *>(slots), n_pages, n_slots, page_size, head_dim);
    return cudaGetLastError();
}

}  // namespace da

extern "C" int da_fetch_pages(const void *dram_pages, void *slots, const int32_t *miss_pages,
                              const int32_t *miss_slots, const int32_t *n_miss, int list_len, int n_kv_heads,
                              int n_dram_pages, int n_slots, size_t page_bytes, da_stream_t stream) {
    if (!dram_pages || !slots || !miss_pages || !miss_slots || !n_miss) return DA_ERR_NULL;
    if (list_len < 1 || n_kv_heads < 1 || n_dram_pages < 1 || n_slots < 1 || page_bytes < 1) return DA_ERR_SHAPE;
    if (n_kv_heads > 65535) return DA_ERR_UNSUPPORTED;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int gx = list_len < da::kFetchCtasPerHead ? list_len : da::kFetchCtasPerHead;
    dim3 grid(gx, n_kv_heads);
    const bool vec = (page_bytes % 16 == 0) && ((((uintptr_t)dram_pages | (uintptr_t)slots) & 15) == 0) &&
                     (page_bytes / 16 < (size_t)1 << 30);
    if (vec) {
        da::fetch_pages_kernel<<<grid, da::kFetchThreads, 0, s>>>(
            static_cast<const uint4 *>(dram_pages), static_cast<uint4 *>(slots), miss_pages, miss_slots, n_miss,
            list_len, n_dram_pages, n_slots, (int)(page_bytes / 16));
    } else {
        da::fetch_pages_bytes_kernel<<<grid, da::kFetchThreads, 0, s>>>(
            static_cast<const unsigned char *>(dram_pages), static_cast<unsigned char *>(slots), miss_pages,
            miss_slots, n_miss, list_len, n_dram_pages, n_slots, page_bytes);
    }
    return (int)cudaGetLastError();
}

extern "C" int da_build_pages(const void *k, const void *v, long long kv_token_stride, long long kv_head_stride,
                              void *dram_pages, void *summaries, void *slots, int n_kv_heads, int n_pages,
                              int n_slots, int page_size, int head_dim, int dtype, da_stream_t stream) {
    if (!k || !v) return DA_ERR_NULL;
    if (n_kv_heads < 1 || n_pages < 1 || page_size < 1 || head_dim < 1 || n_slots < 0 || n_slots > n_pages)
        return DA_ERR_SHAPE;
    if (n_kv_heads > 65535) return DA_ERR_UNSUPPORTED;
    if (slots && n_slots < 1) return DA_ERR_SHAPE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaError_t e;
    switch (dtype) {
    case DA_F32: e = da::launch_build<float>(k, v, kv_token_stride, kv_head_stride, dram_pages, summaries, slots, n_kv_heads, n_pages, n_slots, page_size, head_dim, s); break;
    case DA_F16: e = da::launch_build<__half>(k, v, kv_token_stride, kv_head_stride, dram_pages, summaries, slots, n_kv_heads, n_pages, n_slots, page_size, head_dim, s); break;
    case DA_BF16: e = da::launch_build<__nv_bfloat16>(k, v, kv_token_stride, kv_head_stride, dram_pages, summaries, slots, n_kv_heads, n_pages, n_slots, page_size, head_dim, s); break;
    default: return DA_ERR_DTYPE;
    }
    return (int)e;
}
