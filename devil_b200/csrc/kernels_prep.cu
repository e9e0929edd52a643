// Preparation kernels: count-matrix conversion, design staging, per-gene
// statistics, size factors (R/size_factors.R), theta_0
// (R/overdispersion.R:129-135), beta_0 (R/beta.R:13-20, R/main.R:404-406)
// and the CSR offsets of every cell segment.
#include "internal.h"

#include <type_traits>

namespace devil {

static inline unsigned nblk(int64_t m, int t) { return (unsigned)((m + t - 1) / t); }

// ------------------------------------------------------------------
// dense -> CSR (gene-major)
// ------------------------------------------------------------------
__global__ void dense_count_kernel(const void* Y, int is_f64, int cell_major, int64_t G, int64_t n,
                                   int64_t* rowcnt) {
    int64_t g = blockIdx.x;
    if (g >= G) return;
    int64_t cnt = 0;
    for (int64_t c = threadIdx.x; c < n; c += blockDim.x) {
        int64_t idx = cell_major ? c * G + g : g * n + c;
        double v = is_f64 ? ((const double*)Y)[idx] : (double)((const float*)Y)[idx];
        cnt += (v != 0.0);
    }
    cnt = warp_sum(cnt);
    __shared__ int64_t red[32];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t s = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
        rowcnt[g] = s;
    }
}

// one warp per gene walks its row in order and compacts the nonzeros
__global__ void dense_fill_kernel(const void* Y, int is_f64, int cell_major, int64_t G, int64_t n,
                                  const int64_t* rowptr, int32_t* col, float* val) {
    int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    if (g >= G) return;
    int64_t pos = rowptr[g];
    for (int64_t c0 = 0; c0 < n; c0 += 32) {
        int64_t c = c0 + lane;
        double v = 0.0;
        if (c < n) {
            int64_t idx = cell_major ? c * G + g : g * n + c;
            v = is_f64 ? ((const double*)Y)[idx] : (double)((const float*)Y)[idx];
        }
        unsigned m = __ballot_sync(0xffffffffu, v != 0.0);
        if (v != 0.0) {
            int r = __popc(m & ((1u << lane) - 1u));
            col[pos + r] = (int32_t)c;
            val[pos + r] = (float)v;
        }
        pos += __popc(m);
    }
}

cudaError_t launch_dense_count(const void* Y, int is_f64, int cell_major, int64_t G, int64_t n,
                               int64_t* rowcnt, cudaStream_t st) {
    if (G == 0) return cudaSuccess;
    dense_count_kernel<<<(unsigned)G, 256, 0, st>>>(Y, is_f64, cell_major, G, n, rowcnt);
    return cudaGetLastError();
}
cudaError_t launch_dense_fill(const void* Y, int is_f64, int cell_major, int64_t G, int64_t n,
                              const int64_t* rowptr, int32_t* col, float* val, cudaStream_t st) {
    if (G == 0) return cudaSuccess;
    dense_fill_kernel<<<nblk(G, 8), 256, 0, st>>>(Y, is_f64, cell_major, G, n, rowptr, col, val);
    return cudaGetLastError();
}

__global__ void f64_to_f32_kernel(const double* in, float* out, int64_t m) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
         i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (float)in[i];
}
cudaError_t launch_csr_f64_to_f32(const double* in, float* out, int64_t nnz, cudaStream_t st) {
    if (nnz == 0) return cudaSuccess;
    f64_to_f32_kernel<<<(unsigned)std::min<int64_t>(nblk(nnz, 256), 148 * 16), 256, 0, st>>>(in, out, nnz);
    return cudaGetLastError();
}
cudaError_t launch_double_to_float(const double* in, float* out, int64_t m, cudaStream_t st) {
    return launch_csr_f64_to_f32(in, out, m, st);
}

// CSC (cell-major) -> sortable (gene, cell) keys
// out-of-range gene indices or column pointers set bad[0] and produce key 0
__global__ void csc_keys_kernel(const int64_t* colptr, const int32_t* rowidx, int64_t n, int64_t G,
                                int64_t nnz, int64_t* keys, int32_t* bad) {
    int64_t c = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    if (c >= n) return;
    const int64_t e0 = colptr[c], e1 = colptr[c + 1];
    if (e0 < 0 || e1 < e0 || e1 > nnz) {
        if (lane == 0) atomicOr(bad, 1);
        return;
    }
    for (int64_t e = e0 + lane; e < e1; e += 32) {
        int32_t g = rowidx[e];
        if (g < 0 || g >= G) {
            atomicOr(bad, 1);
            keys[e] = 0;
        } else {
            keys[e] = (int64_t)g * n + c;
        }
    }
}
cudaError_t launch_csc_keys(const int64_t* colptr, const int32_t* rowidx, int64_t n, int64_t G,
                            int64_t nnz, int64_t* keys, int32_t* bad, cudaStream_t st) {
    if (n == 0 || nnz == 0) return cudaSuccess;
    csc_keys_kernel<<<nblk(n, 8), 256, 0, st>>>(colptr, rowidx, n, G, nnz, keys, bad);
    return cudaGetLastError();
}
__global__ void keys_to_csr_kernel(const int64_t* keys, int64_t nnz, int64_t n, int32_t* col,
                                   unsigned long long* rowcnt) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nnz;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t k = keys[i];
        int64_t g = k / n;
        col[i] = (int32_t)(k - g * n);
        atomicAdd(rowcnt + g, 1ull);
    }
}
cudaError_t launch_keys_to_csr(const int64_t* keys, int64_t nnz, int64_t n, int64_t G,
                               int32_t* col, int64_t* rowcnt, cudaStream_t st) {
    (void)G;
    if (nnz == 0) return cudaSuccess;
    keys_to_csr_kernel<<<(unsigned)std::min<int64_t>(nblk(nnz, 256), 148 * 16), 256, 0, st>>>(
        keys, nnz, n, col, reinterpret_cast<unsigned long long*>(rowcnt));
    return cudaGetLastError();
}

// ------------------------------------------------------------------
// design matrix: column-major doubles -> row-major padded floats
// ------------------------------------------------------------------
__global__ void x_rowmajor_kernel(const double* Xcm, int64_t n, int P, int xs, float* Xrm) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n * xs;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t c = i / xs;
        int j = (int)(i - c * xs);
        Xrm[i] = j < P ? (float)Xcm[(int64_t)j * n + c] : 0.f;
    }
}
cudaError_t launch_x_rowmajor(const double* Xcm, int64_t n, int P, int xs, float* Xrm,
                              cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    x_rowmajor_kernel<<<(unsigned)std::min<int64_t>(nblk(n * xs, 256), 148 * 16), 256, 0, st>>>(
        Xcm, n, P, xs, Xrm);
    return cudaGetLastError();
}

__global__ void x_rowmajor_d_kernel(const double* Xcm, int64_t n, int P, int xs, double* Xrm) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n * xs;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t c = i / xs;
        int j = (int)(i - c * xs);
        Xrm[i] = j < P ? Xcm[(int64_t)j * n + c] : 0.0;
    }
}
cudaError_t launch_x_rowmajor_d(const double* Xcm, int64_t n, int P, int xs, double* Xrm,
                                cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    x_rowmajor_d_kernel<<<(unsigned)std::min<int64_t>(nblk(n * xs, 256), 148 * 16), 256, 0, st>>>(
        Xcm, n, P, xs, Xrm);
    return cudaGetLastError();
}

// ------------------------------------------------------------------
// per-gene statistics, two passes over each row (warp per gene):
// stats[g*6 + 0..5] = mean, sample variance (n-1), sum y,
//                     sum (y-1) y, max y, nnz
// ------------------------------------------------------------------
// (order: the genes in the order the warps take them, largest first; null: gene
// order)
template <class VT>
__global__ void gene_stats_kernel(const int64_t* rowptr, const VT* val, int64_t G, int64_t n,
                                  double* stats, const int32_t* order) {
    int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    if (g >= G) return;
    if (order) g = order[g];
    const int64_t e0 = rowptr[g], e1 = rowptr[g + 1];
    // Counts that are whole numbers (always for uint16; checked for float): one
    // pass with exact integer sums of y and y^2 (below 2^64 for any int32 cell
    // count and counts below 2^16) and the variance from the exact numerator n sum
    // y^2 - (sum y)^2 in 128 bits, so a uint16 (here or in gene_sums_kernel) and a
    // float copy of the same counts give the same statistics.  Other counts: a second pass over the squared
    // deviations in FP64.
    unsigned long long s1 = 0, s2 = 0;
    double s = 0.0, mx = 0.0;
    bool whole = true;
    constexpr int U = 4;  // loads in flight per lane
    for (int64_t base = e0 + lane; base < e1; base += 32 * U) {
        VT raw[U];
#pragma unroll
        for (int u = 0; u < U; ++u) raw[u] = base + 32 * u < e1 ? __ldg(val + base + 32 * u) : VT(0);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const double y = (double)raw[u];
            mx = fmax(mx, y);
            if constexpr (std::is_same<VT, uint16_t>::value) {
                const unsigned long long v = (unsigned long long)raw[u];
                s1 += v;
                s2 += v * v;
            } else {
                s += y;
                const bool w = y >= 0.0 && y < 65536.0 && y == floor(y);
                whole = whole && w;
                if (w) {
                    const unsigned long long v = (unsigned long long)y;
                    s1 += v;
                    s2 += v * v;
                }
            }
        }
    }
    whole = __all_sync(0xffffffffu, whole);
    double* o = stats + g * 6;
    if (whole) {
#pragma unroll
        for (int sh = 16; sh > 0; sh >>= 1) {
            s1 += __shfl_xor_sync(0xffffffffu, s1, sh);
            s2 += __shfl_xor_sync(0xffffffffu, s2, sh);
        }
        mx = warp_max(mx);
        if (lane == 0) {
            const __int128 num = (__int128)n * (__int128)s2 - (__int128)s1 * (__int128)s1;
            o[0] = (double)s1 / (double)n;
            o[1] = (double)num / ((double)n * (double)(n - 1));
            o[2] = (double)s1;
            o[3] = (double)(s2 - s1);
            o[4] = mx;
            o[5] = (double)(e1 - e0);
        }
        return;
    }
    double sp = 0.0;
    for (int64_t e = e0 + lane; e < e1; e += 32) {
        const double y = (double)val[e];
        sp += (y - 1.0) * y;
    }
    s = warp_sum(s);
    sp = warp_sum(sp);
    mx = warp_max(mx);
    const double mean = s / (double)n;
    double ss = 0.0;
    for (int64_t e = e0 + lane; e < e1; e += 32) {
        const double d = (double)val[e] - mean;
        ss += d * d;
    }
    ss = warp_sum(ss);
    if (lane == 0) {
        ss += (double)(n - (e1 - e0)) * mean * mean;
        o[0] = mean;
        o[1] = ss / (double)(n - 1);
        o[2] = s;
        o[3] = sp;
        o[4] = mx;
        o[5] = (double)(e1 - e0);
    }
}
// The same statistics for uint16 counts, by spans of the value array instead
// of by rows: a warp takes `span` consecutive entries, cuts them at the row
// ends, and adds each row's exact integer sums and maximum to the gene's
// accumulators with atomics (integers: the order does not matter).  A warp
// per row took as long as the longest row (a gene seen in most of a million
// cells: 1,000 dependent rounds, 2.49 ms at 790 M entries); the spans read the
// array near the memory's rate (0.42 ms).  VEC: the array starts on a 16-byte
// boundary and is read as 16-byte pieces of eight counts (four in flight per
// lane), pieces that straddle a row's ends masked, the array's last piece
// (which may end past nnz) read count by count; otherwise count by count.
struct GeneSums {
    unsigned long long s1, s2;  // sum y, sum y^2
    unsigned mx, pad;
};
template <bool VEC>
__global__ void __launch_bounds__(256) gene_sums_kernel(const int64_t* rowptr, const uint16_t* val, int64_t G,
                                                        int64_t span, GeneSums* acc) {
    const int lane = threadIdx.x & 31;
    const int64_t w = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int64_t nnz = rowptr[G], pfull = nnz >> 3;
    int64_t a = max(w * span, rowptr[0]);
    const int64_t b = min((w + 1) * span, nnz);
    if (a >= b) return;
    int64_t g = 0, hi = G;  // the last row that starts at or before a
    while (hi - g > 1) {
        const int64_t mid = (g + hi) >> 1;
        if (rowptr[mid] <= a) g = mid; else hi = mid;
    }
    const uint4* v4 = reinterpret_cast<const uint4*>(val);
    for (; a < b; ++g) {
        const int64_t e0 = a, e1 = min(rowptr[g + 1], b);
        if (e1 <= e0) continue;
        a = e1;
        unsigned long long s1 = 0, s2 = 0;
        unsigned mx = 0, mx2 = 0;  // mx2: two 16-bit maxima
        constexpr int U = 4;
        if constexpr (VEC) {
            const int64_t p1 = (e1 + 7) >> 3;
            for (int64_t base = (e0 >> 3) + lane; base < p1; base += 32 * U) {
                uint4 pc[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int64_t pp = base + 32 * u;
                    pc[u] = make_uint4(0, 0, 0, 0);
                    if (pp < p1) {
                        if (pp < pfull) {
                            pc[u] = __ldg(v4 + pp);
                        } else {
                            uint16_t h[8];
#pragma unroll
                            for (int r = 0; r < 8; ++r) h[r] = pp * 8 + r < nnz ? val[pp * 8 + r] : (uint16_t)0;
                            pc[u] = make_uint4(h[0] | (unsigned)h[1] << 16, h[2] | (unsigned)h[3] << 16,
                                               h[4] | (unsigned)h[5] << 16, h[6] | (unsigned)h[7] << 16);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int64_t ea = (base + 32 * u) * 8;
                    if (ea >= e1) continue;
                    unsigned wd[4] = {pc[u].x, pc[u].y, pc[u].z, pc[u].w};
                    if (ea < e0 || ea + 8 > e1) {  // a piece across a row's end: zeros outside
#pragma unroll
                        for (int r = 0; r < 8; ++r)
                            if (ea + r < e0 || ea + r >= e1) wd[r >> 1] &= r & 1 ? 0xffffu : 0xffff0000u;
                    }
                    unsigned p = 0;
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const unsigned lo = wd[r] & 0xffffu, hi = wd[r] >> 16;
                        p += lo + hi;
                        asm("mad.wide.u32 %0, %1, %1, %0;" : "+l"(s2) : "r"(lo));
                        asm("mad.wide.u32 %0, %1, %1, %0;" : "+l"(s2) : "r"(hi));
                        mx2 = __vmaxu2(mx2, wd[r]);
                    }
                    s1 += p;
                }
            }
        } else {
            for (int64_t e = e0 + lane; e < e1; e += 32) {
                const unsigned y = val[e];
                s1 += y;
                s2 += (unsigned long long)(y * y);
                mx = max(mx, y);
            }
        }
        mx = max(mx, max(mx2 & 0xffffu, mx2 >> 16));
#pragma unroll
        for (int sh = 16; sh > 0; sh >>= 1) {
            s1 += __shfl_xor_sync(0xffffffffu, s1, sh);
            s2 += __shfl_xor_sync(0xffffffffu, s2, sh);
            mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, sh));
        }
        if (lane == 0) {
            atomicAdd(&acc[g].s1, s1);
            atomicAdd(&acc[g].s2, s2);
            atomicMax(&acc[g].mx, mx);
        }
    }
}
__global__ void gene_stats_from_sums_kernel(const int64_t* rowptr, const GeneSums* acc, int64_t G, int64_t n,
                                            double* stats) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G) return;
    const GeneSums a = acc[g];
    double* o = stats + g * 6;
    const __int128 num = (__int128)n * (__int128)a.s2 - (__int128)a.s1 * (__int128)a.s1;
    o[0] = (double)a.s1 / (double)n;
    o[1] = (double)num / ((double)n * (double)(n - 1));
    o[2] = (double)a.s1;
    o[3] = (double)(a.s2 - a.s1);
    o[4] = (double)a.mx;
    o[5] = (double)(rowptr[g + 1] - rowptr[g]);
}

size_t gene_sums_bytes(int64_t G) { return (size_t)G * sizeof(GeneSums); }

// Rows of at most kShortRows cells: a warp per row (20,000 genes x 500 cells, 15
// entries a row: 14 us, 34 by spans; 2,000 x 4,000, 600 entries: 15 us, 18; 2,000 x
// 8,000, 2,400 entries: 25, 17; 300 x 16,000: 43, 13).
constexpr int64_t kShortRows = 4096;
cudaError_t launch_gene_stats(const int64_t* rowptr, const void* val, int val_u16, int64_t G, int64_t nnz,
                              int64_t n, double* stats, void* sums, cudaStream_t st, const int32_t* order) {
    if (G == 0) return cudaSuccess;
    if (!val_u16) {
        gene_stats_kernel<float><<<nblk(G, 8), 256, 0, st>>>(rowptr, (const float*)val, G, n, stats, order);
        return cudaGetLastError();
    }
    if (n <= kShortRows) {
        gene_stats_kernel<uint16_t><<<nblk(G, 8), 256, 0, st>>>(rowptr, (const uint16_t*)val, G, n, stats, order);
        return cudaGetLastError();
    }
    GeneSums* acc = static_cast<GeneSums*>(sums);
    cudaError_t e = cudaMemsetAsync(acc, 0, gene_sums_bytes(G), st);
    if (e != cudaSuccess) return e;
    // about 64 warps per SM in flight, up to 16,384 entries each and no fewer than
    // two rows' or 1,024: a row costs a warp about a microsecond however short it
    // is (20,000 genes x 100,000 cells, 30 entries a row: 51 us with 1,024, 31 so)
    int64_t span = (nnz / (148 * 64) + 255) / 256 * 256;
    const int64_t least = std::max<int64_t>(32, std::min<int64_t>(1024, (2 * nnz / G + 7) / 8 * 8));
    span = std::max<int64_t>(least, std::min<int64_t>(16384, span));
    const unsigned b = nblk((nnz + span - 1) / span, 8);
    if (b > 0) {
        if ((reinterpret_cast<uintptr_t>(val) & 15) == 0)
            gene_sums_kernel<true><<<b, 256, 0, st>>>(rowptr, (const uint16_t*)val, G, span, acc);
        else
            gene_sums_kernel<false><<<b, 256, 0, st>>>(rowptr, (const uint16_t*)val, G, span, acc);
    }
    gene_stats_from_sums_kernel<<<nblk(G, 256), 256, 0, st>>>(rowptr, acc, G, n, stats);
    return cudaGetLastError();
}

// ------------------------------------------------------------------
// column statistics for size factors (atomics; integer-valued sums are
// exact in FP64 whatever the order)
// ------------------------------------------------------------------
template <class VT>
__global__ void colstats_kernel(const int32_t* col, const VT* val, int64_t nnz, double* colsum,
                                double* collog, int32_t* colcnt, int32_t* colmin_bits) {
    if (!collog) {
        // normed_sum: column sums only; four entries' loads in flight per thread
        constexpr int U = 4;
        const int64_t stride = (int64_t)gridDim.x * blockDim.x;
        for (int64_t e0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e0 < nnz; e0 += stride * U) {
            int c[U];
            float v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int64_t e = e0 + stride * u;
                c[u] = e < nnz ? __ldg(col + e) : -1;
                v[u] = e < nnz ? (float)val[e] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (c[u] >= 0) atomicAdd(colsum + c[u], (double)v[u]);
        }
        return;
    }
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nnz;
         e += (int64_t)gridDim.x * blockDim.x) {
        int c = col[e];
        float v = (float)val[e];
        atomicAdd(colsum + c, (double)v);
        if (collog) {
            atomicAdd(collog + c, log1p((double)v));
            atomicAdd(colcnt + c, 1);
            float l = (float)log1p((double)v);
            // log1p of counts is >= 0; int ordering of non-negative floats
            // matches float ordering
            atomicMin(colmin_bits + c, __float_as_int(fmaxf(l, 0.f)));
        }
    }
}
// normed_sum column sums of 16-bit counts as 32-bit integers (a column sum is
// at most G x 65535, below 2^32 for G <= 65537); colsum_from_u32_kernel turns
// them into FP64 (the same exact integers the FP64 atomics give).
//
// Columns with many entries: a block keeps kColTile columns' counters in
// shared memory and takes a share of the genes (blockIdx.y); a gene's entries
// of the columns are one run of its row (found by a search per lane, 32 genes
// at a time), read as 16-byte pieces of four cell indices and 8-byte pieces of
// their counts.  The counters are added to the global ones at the end.
// Bound by the read (6 B an entry) and the shared atomics' bank conflicts;
// one global atomic per entry ran at the L2's atomic rate (790 M entries:
// 2.51 -> 1.17 ms).  (Entries before rowptr[0], which no row holds, are
// counted too, as the per-entry kernels do.)
constexpr int kColTile = 49152;  // 192 KB of counters, one block per SM
__global__ void __launch_bounds__(1024, 1) colsum_tile_kernel(const int64_t* rowptr, const int32_t* col,
                                                              const uint16_t* val, int64_t G, int64_t n,
                                                              const int32_t* order, uint32_t* colsum) {
    extern __shared__ uint32_t ccnt[];
    const int c0 = blockIdx.x * kColTile;
    const int c1 = (int)(n - c0 < kColTile ? n : c0 + kColTile);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = blockDim.x >> 5;
    for (int i = t; i < c1 - c0; i += blockDim.x) ccnt[i] = 0;
    __syncthreads();
    const int64_t nnz = rowptr[G], pfull = nnz >> 2;
    const int4* c4 = reinterpret_cast<const int4*>(col);
    const uint2* v4 = reinterpret_cast<const uint2*>(val);
    if (blockIdx.y == 0)
        for (int64_t e = t; e < rowptr[0]; e += blockDim.x) {
            const int c = col[e];
            if (c >= c0 && c < c1) atomicAdd(&ccnt[c - c0], (uint32_t)val[e]);
        }
    // warp `w` of the column tile's gridDim.y blocks takes every W-th batch
    const int64_t W = (int64_t)gridDim.y * nw, w0 = (int64_t)warp * gridDim.y + blockIdx.y;
    // the genes of a batch are W apart in the list, so that every warp gets a
    // like share of a list in decreasing order of entries
    for (int64_t b = 0; b * 32 * W < G; ++b) {
        const int64_t k = (b * 32 + lane) * W + w0;
        int64_t lo = 0, hi = 0;
        if (k < G) {
            const int64_t g = order ? order[k] : k;
            const int64_t r0 = rowptr[g], r1 = rowptr[g + 1];
            auto first_at = [&](int key) {
                int64_t x = r0, y = r1;
                while (x < y) {
                    const int64_t m = (x + y) >> 1;
                    if (col[m] < key) x = m + 1; else y = m;
                }
                return x;
            };
            lo = c0 == 0 ? r0 : first_at(c0);
            hi = c1 >= n ? r1 : first_at(c1);
        }
        for (int q = 0; q < 32; ++q) {
            const int64_t e0 = __shfl_sync(0xffffffffu, lo, q), e1 = __shfl_sync(0xffffffffu, hi, q);
            const int64_t p1 = (e1 + 3) >> 2;
            constexpr int U = 4;
            for (int64_t base = (e0 >> 2) + lane; base < p1 && e0 < e1; base += 32 * U) {
                int4 c[U];
                uint2 v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int64_t pp = base + 32 * u;
                    if (pp < p1 && pp < pfull) {
                        c[u] = __ldg(c4 + pp);
                        v[u] = __ldg(v4 + pp);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int64_t pp = base + 32 * u;
                    if (pp >= p1) continue;
                    if (pp >= pfull) {  // the array's last piece
                        for (int64_t e = max(pp * 4, e0); e < e1; ++e) atomicAdd(&ccnt[col[e] - c0], (uint32_t)val[e]);
                        continue;
                    }
                    const int cc[4] = {c[u].x, c[u].y, c[u].z, c[u].w};
                    const unsigned vv[4] = {v[u].x & 0xffffu, v[u].x >> 16, v[u].y & 0xffffu, v[u].y >> 16};
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        if (pp * 4 + r >= e0 && pp * 4 + r < e1) atomicAdd(&ccnt[cc[r] - c0], vv[r]);
                }
            }
        }
    }
    __syncthreads();
    for (int i = t; i < c1 - c0; i += blockDim.x)
        if (ccnt[i]) atomicAdd(colsum + c0 + i, ccnt[i]);
}
// Otherwise: one global atomic per entry, four entries' loads in flight per
// thread
__global__ void colsum_u32_kernel(const int32_t* col, const uint16_t* val, int64_t nnz, uint32_t* colsum) {
    constexpr int U = 4;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e0 < nnz; e0 += stride * U) {
        int c[U];
        uint32_t v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t e = e0 + stride * u;
            c[u] = e < nnz ? __ldg(col + e) : -1;
            v[u] = e < nnz ? (uint32_t)__ldg(val + e) : 0u;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c[u] >= 0 && v[u]) atomicAdd(colsum + c[u], v[u]);
    }
}
__global__ void colsum_from_u32_kernel(const uint32_t* in, int64_t n, double* out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (double)in[i];
}

cudaError_t launch_colstats(const int64_t* rowptr, const int32_t* col, const void* val,
                            int val_u16, int64_t G, int64_t nnz, double* colsum,
                            double* collog, int32_t* colcnt, int32_t* colmin_bits,
                            cudaStream_t st, uint32_t* colsum_u32, int64_t n, const int32_t* order) {
    if (nnz == 0) return cudaSuccess;
    unsigned b = (unsigned)std::min<int64_t>(nblk(nnz, 256), 148 * 32);
    if (colsum_u32 && val_u16 && !collog && G <= 65537) {
        // the tiles add up to gy counters per column to the global ones: at
        // most one per eight entries, and a block's SM takes 0.22 ns an entry
        // against 3.2 ps for the per-entry kernel on the whole chip, so the
        // tiles pay from 69 blocks on (3.5 M entries in 20,000 columns allow 21
        // blocks: 71 us against 44 us)
        const int64_t tiles = (n + kColTile - 1) / kColTile;
        const int64_t gy = std::min<int64_t>(std::max<int64_t>(1, 148 / tiles), nnz / (8 * n));
        const bool aligned = (reinterpret_cast<uintptr_t>(col) & 15) == 0 && (reinterpret_cast<uintptr_t>(val) & 7) == 0;
        if (gy >= 1 && aligned && tiles * gy >= 96) {
            const size_t smem = (size_t)std::min<int64_t>(n, kColTile) * sizeof(uint32_t);
            cudaError_t e = raise_dyn_smem(colsum_tile_kernel, (size_t)kColTile * sizeof(uint32_t));
            if (e != cudaSuccess) return e;
            colsum_tile_kernel<<<dim3((unsigned)tiles, (unsigned)gy), 1024, smem, st>>>(
                rowptr, col, (const uint16_t*)val, G, n, order, colsum_u32);
        } else {
            colsum_u32_kernel<<<b, 256, 0, st>>>(col, (const uint16_t*)val, nnz, colsum_u32);
        }
        colsum_from_u32_kernel<<<(unsigned)std::min<int64_t>(nblk(n, 256), 1024), 256, 0, st>>>(colsum_u32, n,
                                                                                               colsum);
        return cudaGetLastError();
    }
    if (val_u16)
        colstats_kernel<uint16_t><<<b, 256, 0, st>>>(col, (const uint16_t*)val, nnz, colsum, collog, colcnt, colmin_bits);
    else
        colstats_kernel<float><<<b, 256, 0, st>>>(col, (const float*)val, nnz, colsum, collog, colcnt, colmin_bits);
    return cudaGetLastError();
}

// sum of f over c = t, t + T, ... (T threads), 16 loads in flight per thread
// and added in that order
template <class F>
DEV double strided_sum(int64_t n, F&& at) {
    constexpr int U = 16;
    const int64_t T = blockDim.x;
    double acc = 0.0;
    for (int64_t c = threadIdx.x; c < n; c += T * U) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = c + T * u < n ? at(c + T * u) : 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c + T * u < n) acc += v[u];
    }
    return acc;
}

// size factors from the column statistics.
// method 1 = normed_sum (R/size_factors.R:75-88), 2 = psinorm (:100-117).
// The logarithms on every SM, then one block for their sum (in a fixed order),
// then the division and the offsets on every SM: one block for all of it took
// 1.29 ms at a million cells, the three take 0.25 ms.  Up to kOneBlock cells one
// block does all three, with the same sums: there the launches cost more.
constexpr int64_t kOneBlock = 16384;
struct SfArgs {
    int method;
    int64_t G, n;
    const double *colsum, *collog;
    const int32_t *colcnt, *colmin_bits;
    double offset;
    double *sf, *off;  // (off holds the logarithms first)
    float* off_f;
    int32_t* err;
};
DEV void sf_logs(const SfArgs& a, int64_t first, int64_t step) {
    for (int64_t c = first; c < a.n; c += step) {
        double v;
        if (a.G <= 1) {
            v = 1.0;
        } else if (a.method == 1) {
            v = a.colsum[c];
            if (v == 0.0) *a.err = 1;
        } else {
            double m = a.colcnt[c] < a.G ? 0.0 : (double)__int_as_float(a.colmin_bits[c]);
            v = a.collog[c] / (double)a.G - m;
        }
        a.sf[c] = v;
        a.off[c] = log(v);
    }
}
// the geometric mean, by one block; valid in thread 0
DEV double sf_mean(const SfArgs& a, double* red, double* red2) {
    double cntv = 0.0;
    double acc = strided_sum(a.n, [&](int64_t c) {
        const double l = a.off[c];
        const bool ok = !isnan(l);
        cntv += ok ? 1.0 : 0.0;
        return ok ? l : 0.0;
    });
    acc = warp_sum(acc);
    cntv = warp_sum(cntv);
    if ((threadIdx.x & 31) == 0) { red[threadIdx.x >> 5] = acc; red2[threadIdx.x >> 5] = cntv; }
    __syncthreads();
    double s = 0.0, k = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { s += red[w]; k += red2[w]; }
    return a.G <= 1 ? 1.0 : exp(s / k);
}
DEV void sf_scale(const SfArgs& a, double gm, int64_t first, int64_t step) {
    for (int64_t c = first; c < a.n; c += step) {
        double v = (a.G <= 1) ? 1.0 : a.sf[c] / gm;
        a.sf[c] = v;
        double o = a.offset + log(v);
        a.off[c] = o;
        a.off_f[c] = (float)o;
    }
}
__global__ void sf_log_kernel(SfArgs a) {
    sf_logs(a, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}
__global__ void __launch_bounds__(1024) sf_mean_kernel(SfArgs a, double* gm) {
    __shared__ double red[32], red2[32];
    const double m = sf_mean(a, red, red2);
    if (threadIdx.x == 0) *gm = m;
}
__global__ void sf_scale_kernel(SfArgs a, const double* gm) {
    sf_scale(a, *gm, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}
__global__ void __launch_bounds__(1024) sf_block_kernel(SfArgs a) {
    __shared__ double red[32], red2[32], gm;
    if (threadIdx.x == 0) *a.err = 0;
    __syncthreads();
    sf_logs(a, threadIdx.x, blockDim.x);
    __syncthreads();
    const double m = sf_mean(a, red, red2);
    if (threadIdx.x == 0) gm = m;
    __syncthreads();
    sf_scale(a, gm, threadIdx.x, blockDim.x);
}
cudaError_t launch_sf_finalize(int method, int64_t G, int64_t n, const double* colsum,
                               const double* collog, const int32_t* colcnt,
                               const int32_t* colmin_bits, double offset, double* sf,
                               double* off, float* off_f, double* gm, int32_t* err, cudaStream_t st) {
    const SfArgs a{method, G, n, colsum, collog, colcnt, colmin_bits, offset, sf, off, off_f, err};
    if (n <= kOneBlock) {
        sf_block_kernel<<<1, 1024, 0, st>>>(a);
        return cudaGetLastError();
    }
    cudaError_t e = cudaMemsetAsync(err, 0, sizeof(int32_t), st);
    if (e != cudaSuccess) return e;
    const unsigned b = (unsigned)std::min<int64_t>(nblk(n, 256), 148 * 8);
    sf_log_kernel<<<b, 256, 0, st>>>(a);
    sf_mean_kernel<<<1, 1024, 0, st>>>(a, gm);
    sf_scale_kernel<<<b, 256, 0, st>>>(a, gm);
    return cudaGetLastError();
}

// offsets from given (or unit) size factors: compute_offset_vector
// (R/size_factors.R:172-184)
__global__ void sf_given_kernel(const double* sf_in, int64_t n, double offset, int use_sf,
                                double* sf, double* off, float* off_f) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
         c += (int64_t)gridDim.x * blockDim.x) {
        double s = use_sf ? sf_in[c] : 1.0;
        sf[c] = s;
        double o = use_sf ? offset + log(s) : offset;
        off[c] = o;
        off_f[c] = (float)o;
    }
}
cudaError_t launch_sf_given(const double* sf_in, int64_t n, double offset, int use_sf, double* sf,
                            double* off, float* off_f, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    sf_given_kernel<<<(unsigned)std::min<int64_t>(nblk(n, 256), 1024), 256, 0, st>>>(
        sf_in, n, offset, use_sf, sf, off, off_f);
    return cudaGetLastError();
}

// ------------------------------------------------------------------
// theta_0 = (var - mean / mean(exp(off))) / mean^2, NaN or < 0 -> 0.01
// (R/overdispersion.R:129-135); k = 1/theta_0 as the float beta_fit keeps
// (src/beta.cpp:25-28: theta_0 arrives as float, 1.0/k stored as float).
// ------------------------------------------------------------------
// eoff = exp(off), evaluated on every SM beforehand (this kernel's one block
// took 0.53 ms for a million cells, the two take 0.14 ms); up to kOneBlock cells
// null: evaluated here
__global__ void exp_off_kernel(const double* off, int64_t n, double* eoff) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
         c += (int64_t)gridDim.x * blockDim.x)
        eoff[c] = exp(off[c]);
}
__global__ void __launch_bounds__(1024) theta0_kernel(const double* stats, const double* off, const double* eoff,
                                                      int64_t G, int64_t n, int has_init, double init_value,
                                                      double* theta0, float* k) {
    __shared__ double red[32];
    __shared__ double moi_s;
    double acc = strided_sum(n, [&](int64_t c) { return eoff ? eoff[c] : exp(off[c]); });
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
        moi_s = 1.0 / (s / (double)n);
    }
    __syncthreads();
    const double moi = moi_s;
    for (int64_t g = threadIdx.x; g < G; g += blockDim.x) {
        double th;
        if (has_init) {
            th = init_value;
        } else {
            double mean = stats[g * 6 + 0], var = stats[g * 6 + 1];
            double d = (var - moi * mean) / (mean * mean);
            th = (isnan(d) || d < 0.0) ? 0.01 : d;
        }
        theta0[g] = th;
        float kf = (float)th;
        k[g] = (float)(1.0 / (double)kf);
    }
}
cudaError_t launch_theta0(const double* stats, const double* off, int64_t G, int64_t n,
                          int has_init, double init_value, double* eoff, double* theta0, float* k,
                          cudaStream_t st) {
    if (has_init) n = 0;  // theta_0 is given: no mean of exp(off)
    if (n <= kOneBlock)
        eoff = nullptr;
    else
        exp_off_kernel<<<(unsigned)std::min<int64_t>(nblk(n, 256), 148 * 8), 256, 0, st>>>(off, n, eoff);
    theta0_kernel<<<1, 1024, 0, st>>>(stats, off, eoff, G, n, has_init, init_value, theta0, k);
    return cudaGetLastError();
}

// ------------------------------------------------------------------
// (X'X)^-1 in FP64 (one block): the least-squares solve of init_beta
// ------------------------------------------------------------------
// partial X'X over the cells of one block (kXtxCells cells, staged in
// shared memory 256 at a time, row stride P+1); thread t of block y owns the
// packed pair 256 y + t (up to three blocks share a range of cells: one block
// whose threads owned three pairs each took 0.93 ms at p = 32 and a million
// cells, these take 0.65 ms)
constexpr int kXtxCells = 8192;
constexpr int kXtxStage = 256;
__global__ void __launch_bounds__(256) xtx_partial_kernel(const double* Xcm, int64_t n, int P,
                                                          double* part) {
    extern __shared__ double xs[];  // [kXtxStage][P + 1]
    const int NP = P * (P + 1) / 2;
    const int RS = P + 1;
    const int64_t c0 = (int64_t)blockIdx.x * kXtxCells;
    const int64_t c1 = c0 + kXtxCells < n ? c0 + kXtxCells : n;
    const int q = blockIdx.y * 256 + threadIdx.x;
    int j = 0;
    while ((j + 1) * (j + 2) / 2 <= q) ++j;
    const int pi = q < NP ? q - j * (j + 1) / 2 : 0, pj = q < NP ? j : 0;
    double acc = 0.0;
    for (int64_t cb = c0; cb < c1; cb += kXtxStage) {
        const int nc = (int)(c1 - cb < kXtxStage ? c1 - cb : kXtxStage);
        __syncthreads();
        for (int i = threadIdx.x; i < nc * P; i += blockDim.x) {
            const int col = i / nc, c = i - col * nc;  // coalesced along cells
            xs[c * RS + col] = Xcm[(int64_t)col * n + cb + c];
        }
        __syncthreads();
        if (q >= NP) continue;
        double s = 0.0;
        for (int c = 0; c < nc; ++c) s = fma(xs[c * RS + pi], xs[c * RS + pj], s);
        acc += s;
    }
    if (q < NP) part[(int64_t)blockIdx.x * NP + q] = acc;
}

// sum the partials in block order (deterministic), then invert by LU with
// partial pivoting: the row updates of a column over all threads, a thread per
// column of the inverse (one thread for everything took 0.97 ms at p = 32, this
// takes 0.13 ms);
// rank check on the pivots relative to the largest diagonal
__global__ void xtx_finish_kernel(const double* part, int nb, int P, double* ginv, int32_t* err) {
    extern __shared__ double sh[];
    double* Gm = sh;         // P*P
    double* W = sh + P * P;  // P*P
    int* piv = reinterpret_cast<int*>(W + P * P);
    __shared__ int ok_s;
    const int t = threadIdx.x, nt = blockDim.x;
    const int NP = P * (P + 1) / 2;
    for (int q = t; q < NP; q += nt) {
        int j = 0;
        while ((j + 1) * (j + 2) / 2 <= q) ++j;
        const int i = q - j * (j + 1) / 2;
        double s = 0.0;
        for (int b = 0; b < nb; ++b) s += part[(int64_t)b * NP + q];
        Gm[j * P + i] = s;
        Gm[i * P + j] = s;
    }
    __syncthreads();
    double dmax = 0.0;
    for (int i = 0; i < P; ++i) dmax = fmax(dmax, fabs(Gm[i * P + i]));
    if (t == 0) ok_s = 1;
    __syncthreads();
    for (int k = 0; k < P; ++k) {
        int mx = k;  // (every thread finds the same pivot)
        double mv = fabs(Gm[k * P + k]);
        for (int i = k + 1; i < P; ++i) {
            const double v = fabs(Gm[k * P + i]);
            if (v > mv) { mv = v; mx = i; }
        }
        __syncthreads();
        if (t == 0) piv[k] = mx;
        if (mx != k && t < P) {
            const double x = Gm[t * P + k];
            Gm[t * P + k] = Gm[t * P + mx];
            Gm[t * P + mx] = x;
        }
        __syncthreads();
        const double d = Gm[k * P + k];
        if (t == 0 && (!(d != 0.0) || !isfinite(d))) ok_s = 0;
        const double rd = 1.0 / d;
        for (int i = k + 1 + t; i < P; i += nt) Gm[k * P + i] *= rd;
        __syncthreads();
        const int r = P - k - 1;
        for (int q = t; q < r * r; q += nt) {
            const int j = k + 1 + q / r, i = k + 1 + q % r;
            Gm[j * P + i] -= Gm[k * P + i] * Gm[j * P + k];
        }
        __syncthreads();
    }
    if (t == 0)
        for (int i = 0; i < P; ++i)
            if (!(fabs(Gm[i * P + i]) > 1e-12 * dmax)) ok_s = 0;
    __syncthreads();
    const bool ok = ok_s != 0;
    if (ok && t < P) {
        double* x = W + t * P;
        for (int i = 0; i < P; ++i) x[i] = i == t ? 1.0 : 0.0;
        lu_solve(P, Gm, piv, x);
    }
    __syncthreads();
    for (int i = t; i < P * P; i += nt) ginv[i] = ok ? W[i] : NAN;
    if (t == 0) *err = ok ? 0 : 1;
}

int xtx_blocks(int64_t n) { return (int)((n + kXtxCells - 1) / kXtxCells); }

// (X'X)^-1 in FP64 for the least-squares solve of init_beta: partial
// sums over cell blocks on every SM, then one block sums and inverts
cudaError_t launch_xtx_inverse(const double* Xcm, int64_t n, int P, double* part, double* ginv,
                               int32_t* err, cudaStream_t st) {
    const int nb = xtx_blocks(n);
    const size_t sm1 = (size_t)kXtxStage * (P + 1) * sizeof(double);
    cudaError_t e = raise_dyn_smem(xtx_partial_kernel, sm1);
    if (e != cudaSuccess) return e;
    xtx_partial_kernel<<<dim3(nb, (P * (P + 1) / 2 + 255) / 256), 256, sm1, st>>>(Xcm, n, P, part);
    const size_t sm2 = (size_t)2 * P * P * 8 + (size_t)P * 4 + 16;
    xtx_finish_kernel<<<1, 256, sm2, st>>>(part, nb, P, ginv, err);
    return cudaGetLastError();
}
// beta_0 (warp per gene).  QR least squares of log1p(y / exp(off)) on X:
// the solution equals (X'X)^-1 X' z; z is zero wherever y is zero, so
// X' z is a sum over the nonzero entries of the row.  Rough init:
// beta_0 = (log1p(mean y), 0, ..., 0).  U entries a lane are in flight and are
// added in order; the genes with the most entries are taken first (one entry at
// a time, a gene seen in every cell held its warp for 3,000 dependent rounds:
// 10,000 x 100,000, p = 4: 3.59 -> 2.18 ms).  Up to kShortInit cells one entry a
// lane (SHORT): rows of a few rounds cost the deep loop its registers and masked
// loads (p = 4, short / deep: 20,000 x 500 24 / 69 us, 8,000 x 2,000 41 / 58, 6,000 x
// 3,000 55 / 61, 5,000 x 4,000 78 / 64; p = 12: 65 / 101, 78 / 91, 87 / 101, 114 / 108).
constexpr int64_t kShortInit = 3072;
template <class VT, int PMAX, bool SHORT>
__global__ void init_beta_kernel(const int64_t* rowptr, const int32_t* col, const VT* val,
                                 const double* Xrm, int xs, const double* inv_sf,
                                 const double* ginv, const double* stats, int64_t G, int64_t n,
                                 int P, int rough, double* beta, float* beta_f, const int32_t* order) {
    int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    if (g >= G) return;
    if (order) g = order[g];
    if (rough) {
        if (lane < P) {
            double b = lane == 0 ? log1p(stats[g * 6 + 0]) : 0.0;
            beta[g * P + lane] = b;
            beta_f[g * P + lane] = (float)b;
        }
        return;
    }
    double r[PMAX];
#pragma unroll
    for (int i = 0; i < PMAX; ++i) r[i] = 0.0;
    constexpr int U = SHORT ? 1 : (PMAX <= 8 ? 8 : 4);    // entries in flight
    constexpr int V = SHORT ? 1 : (PMAX <= 4 ? 8 : (PMAX <= 8 ? 4 : (PMAX <= 16 ? 2 : 1)));  // design rows in flight
    const int64_t e1 = rowptr[g + 1];
    int cn[U];
    VT vn[U];
    auto load_step = [&](int64_t eb) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t e = eb + 32 * u;
            cn[u] = e < e1 ? __ldg(col + e) : -1;
            vn[u] = e < e1 ? val[e] : VT(0);
        }
    };
    load_step(rowptr[g] + lane);
    for (int64_t eb = rowptr[g] + lane; eb < e1; eb += 32 * U) {
        int c[U];
        double z[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            c[u] = cn[u];
            z[u] = c[u] >= 0 ? (double)vn[u] * __ldg(inv_sf + c[u]) : 0.0;
        }
        load_step(eb + 32 * U);
#pragma unroll
        for (int u0 = 0; u0 < U; u0 += V) {
            double x[V][PMAX];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const double* xr = Xrm + (int64_t)(c[u0 + v] >= 0 ? c[u0 + v] : 0) * xs;
#pragma unroll
                for (int i = 0; i < PMAX; ++i) x[v][i] = i < P ? __ldg(xr + i) : 0.0;
            }
#pragma unroll
            for (int v = 0; v < V; ++v) {
                if (c[u0 + v] < 0) continue;
                const double l = log1p(z[u0 + v]);
#pragma unroll
                for (int i = 0; i < PMAX; ++i)
                    if (i < P) r[i] += x[v][i] * l;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < PMAX; ++i)
        if (i < P) r[i] = warp_sum(r[i]);
    if (lane < P) {
        double b = 0.0;
#pragma unroll
        for (int j = 0; j < PMAX; ++j)
            if (j < P) b += ginv[j * P + lane] * r[j];
        beta[g * P + lane] = b;
        beta_f[g * P + lane] = (float)b;
    }
}
__global__ void inv_exp_kernel(const double* off, int64_t n, double* out) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
         c += (int64_t)gridDim.x * blockDim.x)
        out[c] = exp(-off[c]);
}
// z = log1p(y / exp(off)) as in R/beta.R:18; y * exp(-off) differs from
// y / exp(off) by at most an ulp of the quotient
cudaError_t launch_init_beta(const int64_t* rowptr, const int32_t* col, const void* val,
                             int val_u16, const double* Xrm, int xs, const double* off,
                             double* inv_sf, const double* ginv, const double* stats, int64_t G,
                             int64_t n, int P, int rough, double* beta, float* beta_f,
                             cudaStream_t st, const int32_t* order) {
    if (G == 0) return cudaSuccess;
    if (!rough) {
        inv_exp_kernel<<<(unsigned)std::min<int64_t>(nblk(n, 256), 1024), 256, 0, st>>>(off, n, inv_sf);
    }
    const unsigned b = nblk(G, 8);
    auto go = [&](auto kern, auto* v) {
        kern<<<b, 256, 0, st>>>(rowptr, col, v, Xrm, xs, inv_sf, ginv, stats, G, n, P, rough, beta, beta_f, order);
    };
#define DEVIL_INIT(PM)                                                                            \
    if (val_u16)                                                                                  \
        go(n <= kShortInit ? init_beta_kernel<uint16_t, PM, true> : init_beta_kernel<uint16_t, PM, false>, \
           (const uint16_t*)val);                                                                 \
    else                                                                                          \
        go(n <= kShortInit ? init_beta_kernel<float, PM, true> : init_beta_kernel<float, PM, false>, \
           (const float*)val);
    if (P <= 4) {
        DEVIL_INIT(4)
    } else if (P <= 8) {
        DEVIL_INIT(8)
    } else if (P <= 16) {
        DEVIL_INIT(16)
    } else {
        DEVIL_INIT(32)
    }
#undef DEVIL_INIT
    return cudaGetLastError();
}

// ------------------------------------------------------------------
// segptr[g][b] = first CSR entry of row g with col >= bound[b]
// (warp per gene, lanes search boundaries in parallel)
// ------------------------------------------------------------------
__global__ void segptr_kernel(const int64_t* rowptr, const int32_t* col, int64_t G,
                              const int32_t* bound, int nbound, int64_t* segptr) {
    int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    if (g >= G) return;
    const int64_t e0 = rowptr[g], e1 = rowptr[g + 1];
    for (int b = lane; b < nbound; b += 32) {
        int32_t key = bound[b];
        int64_t lo = e0, hi = e1;
        while (lo < hi) {
            int64_t mid = (lo + hi) >> 1;
            if (col[mid] < key) lo = mid + 1; else hi = mid;
        }
        segptr[g * nbound + b] = lo;
    }
}
cudaError_t launch_segptr(const int64_t* rowptr, const int32_t* col, int64_t G,
                          const int32_t* bound, int nbound, int64_t* segptr, cudaStream_t st) {
    if (G == 0) return cudaSuccess;
    segptr_kernel<<<nblk(G, 8), 256, 0, st>>>(rowptr, col, G, bound, nbound, segptr);
    return cudaGetLastError();
}

// CSR sanity: row pointers non-decreasing and ending at nnz, cell indices in
// [0, n) and strictly increasing within each row.  *bad != 0 on failure.  The
// index array is scanned as one run: an index that does not exceed the one
// before it must start a row, which a search of the row pointers settles (one
// per row at most in valid input).  A warp per row took as long as the longest
// row (2.91 ms at 790 M entries); the scan takes 0.71 ms.
// VEC: the array starts on a 16-byte boundary and is read as 16-byte pieces of
// four indices, eight in flight per lane, the index before a piece taken from
// the lane before (lane 0 loads it); the array's last piece, which may end past
// nnz, is read index by index.
template <bool VEC>
__global__ void __launch_bounds__(256) validate_csr_kernel(const int64_t* rowptr, const int32_t* col, int64_t G,
                                                           int64_t n, int64_t nnz, int32_t* bad) {
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    int b = 0;
    for (int64_t g = tid; g < G; g += nt) {
        const int64_t e0 = rowptr[g], e1 = rowptr[g + 1];
        if (e0 < 0 || e1 < e0 || e1 > nnz || (g == G - 1 && e1 != nnz)) b = 1;
    }
    const int64_t first = max((int64_t)0, min(rowptr[0], nnz));
    auto starts_row = [&](int64_t e) {
        int64_t lo = 0, hi = G;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (rowptr[mid] < e) lo = mid + 1; else hi = mid;
        }
        return rowptr[lo] == e;
    };
    auto check = [&](int64_t e, int before, int c) {
        if (c < 0 || c >= n) b = 1;
        if (e > first && before >= c && !starts_row(e)) b = 1;
    };
    if constexpr (VEC) {
        const int64_t p0 = first >> 2, p1 = (nnz + 3) >> 2, pfull = nnz >> 2;
        const int4* c4 = reinterpret_cast<const int4*>(col);
        constexpr int U = 8;
        // (whole warps go round together: the shuffles need every lane)
        for (int64_t base = p0 + (tid - lane); base < p1; base += nt * U) {
            int4 pc[U];
            int before[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int64_t pp = base + nt * u + lane;
                pc[u] = make_int4(0, 0, 0, 0);
                before[u] = -1;
                if (pp < p1) {
                    if (pp < pfull) {
                        pc[u] = __ldg(c4 + pp);
                    } else {
                        int h[4];
#pragma unroll
                        for (int r = 0; r < 4; ++r) h[r] = pp * 4 + r < nnz ? col[pp * 4 + r] : 0;
                        pc[u] = make_int4(h[0], h[1], h[2], h[3]);
                    }
                    if (lane == 0 && pp > 0) before[u] = __ldg(col + pp * 4 - 1);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int64_t e = (base + nt * u + lane) * 4;
                const int up = __shfl_up_sync(0xffffffffu, pc[u].w, 1);
                if (lane > 0) before[u] = up;
                // a piece inside the scan that rises from the index before it
                // (0 or more) to below n is fine: one test for four entries
                if (before[u] >= 0 && e > first && pc[u].x > before[u] && pc[u].y > pc[u].x && pc[u].z > pc[u].y &&
                    pc[u].w > pc[u].z && pc[u].w < n)
                    continue;
                const int c[5] = {before[u], pc[u].x, pc[u].y, pc[u].z, pc[u].w};
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (e + r >= first && e + r < nnz) check(e + r, c[r], c[r + 1]);
            }
        }
    } else {
        for (int64_t e = first + tid; e < nnz; e += nt) check(e, e > first ? col[e - 1] : -1, col[e]);
    }
    if (b) atomicOr(bad, 1);
}
// The same check, a warp a row, for matrices of up to kShortRows cells: their rows
// end within a few rounds, where the scan searches the row pointers once a row and
// waits for each load of a search (rows / scan: 20,000 genes x 500 cells 9 / 22 us,
// 10,000 x 1,500 12 / 20, 6,000 x 3,000 15 / 19, 5,000 x 4,000 19 / 18).
__global__ void __launch_bounds__(256) validate_rows_kernel(const int64_t* rowptr, const int32_t* col, int64_t G,
                                                            int64_t n, int64_t nnz, int32_t* bad) {
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int lane = threadIdx.x & 31;
    int b = 0;
    for (int64_t g = warp; g < G; g += nw) {
        const int64_t e0 = rowptr[g], e1 = rowptr[g + 1];
        if (e0 < 0 || e1 < e0 || e1 > nnz || (g == G - 1 && e1 != nnz)) {
            b = 1;
            continue;
        }
        for (int64_t e = e0 + lane; e < e1; e += 32) {
            const int c = __ldg(col + e), before = e > e0 ? __ldg(col + e - 1) : -1;
            b |= (c < 0) | (c >= n) | (before >= c);
        }
    }
    if (b) atomicOr(bad, 1);
}
cudaError_t launch_validate_csr(const int64_t* rowptr, const int32_t* col, int64_t G, int64_t n,
                                int64_t nnz, int32_t* bad, cudaStream_t st) {
    if (G == 0) return cudaSuccess;
    if (n <= kShortRows) {
        validate_rows_kernel<<<(unsigned)std::min<int64_t>(nblk(G, 8), 148 * 8), 256, 0, st>>>(rowptr, col, G, n,
                                                                                              nnz, bad);
        return cudaGetLastError();
    }
    const bool vec = (reinterpret_cast<uintptr_t>(col) & 15) == 0;
    const unsigned b = (unsigned)std::max<int64_t>(1, std::min<int64_t>(nblk(std::max(nnz / 16, 4 * G), 256), 148 * 8));
    if (vec)
        validate_csr_kernel<true><<<b, 256, 0, st>>>(rowptr, col, G, n, nnz, bad);
    else
        validate_csr_kernel<false><<<b, 256, 0, st>>>(rowptr, col, G, n, nnz, bad);
    return cudaGetLastError();
}

// acc[0] += sum_g passes[g] * nnz_g, acc[1] += sum_g passes[g]
__global__ void pass_volume_kernel(const int64_t* rowptr, const int32_t* passes, int64_t G,
                                   long long* acc) {
    long long v = 0, w = 0;
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < G;
         g += (int64_t)gridDim.x * blockDim.x) {
        long long k = passes[g];
        v += k * (long long)(rowptr[g + 1] - rowptr[g]);
        w += k;
    }
    v = warp_sum(v);
    w = warp_sum(w);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(reinterpret_cast<unsigned long long*>(acc), (unsigned long long)v);
        atomicAdd(reinterpret_cast<unsigned long long*>(acc + 1), (unsigned long long)w);
    }
}
cudaError_t launch_pass_volume(const int64_t* rowptr, const int32_t* passes, int64_t G,
                               int64_t* acc, cudaStream_t st) {
    if (G == 0) return cudaSuccess;
    pass_volume_kernel<<<(unsigned)std::min<int64_t>(nblk(G, 256), 256), 256, 0, st>>>(
        rowptr, passes, G, reinterpret_cast<long long*>(acc));
    return cudaGetLastError();
}
__global__ void fill_i32_kernel(int32_t* a, int32_t v, int64_t m) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
         i += (int64_t)gridDim.x * blockDim.x)
        a[i] = v;
}
cudaError_t launch_fill_i32(int32_t* a, int32_t v, int64_t m, cudaStream_t st) {
    if (m == 0) return cudaSuccess;
    fill_i32_kernel<<<(unsigned)std::min<int64_t>(nblk(m, 256), 1024), 256, 0, st>>>(a, v, m);
    return cudaGetLastError();
}
// MLE passes per gene: 0 for all-zero genes, else the far-left evaluation
// plus the Newton evaluations
__global__ void mle_passes_kernel(const int32_t* it, const int32_t* phase, const double* stats,
                                  int64_t G, int32_t* out) {
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < G;
         g += (int64_t)gridDim.x * blockDim.x)
        out[g] = stats[g * 6 + 2] == 0.0 ? 0 : 1 + it[g];
}
cudaError_t launch_mle_passes(const int32_t* it, const int32_t* phase, const double* stats,
                              int64_t G, int32_t* out, cudaStream_t st) {
    if (G == 0) return cudaSuccess;
    mle_passes_kernel<<<(unsigned)std::min<int64_t>(nblk(G, 256), 1024), 256, 0, st>>>(it, phase, stats, G, out);
    return cudaGetLastError();
}

__global__ void iota_kernel(int32_t* a, int64_t m) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
         i += (int64_t)gridDim.x * blockDim.x)
        a[i] = (int32_t)i;
}
cudaError_t launch_iota(int32_t* a, int64_t m, cudaStream_t st) {
    if (m == 0) return cudaSuccess;
    iota_kernel<<<(unsigned)std::min<int64_t>(nblk(m, 256), 1024), 256, 0, st>>>(a, m);
    return cudaGetLastError();
}
// act_next = the genes of act[0, n) with keep[g] != 0, in their order in
// act; *n_next = their count.  Keeping the order keeps a list sorted by work
// sorted from one iteration to the next.  One block; per batch every thread
// loads kCompactR elements strided by the block size (coalesced, all loads
// in flight), the kept ones are placed by warp ballots and one scan of the
// (round, warp) totals.
constexpr int kCompactNT = 1024, kCompactR = 16;
__global__ void __launch_bounds__(kCompactNT) compact_kept_kernel(const int32_t* act, const int32_t* n_act,
                                                                  int64_t n_fixed, const int8_t* keep,
                                                                  int32_t* act_next, int32_t* n_next,
                                                                  const int32_t* wkey, int32_t thr,
                                                                  int32_t* n_heavy_next,
                                                                  volatile int32_t* mirror) {
    __shared__ int wtot[kCompactR][32];
    __shared__ int batch_total;
    grid_trigger();
    grid_wait();
    const int64_t n = n_act ? (int64_t)*n_act : n_fixed;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const unsigned lt = (1u << lane) - 1u;
    int base = 0, heavy = 0;
    for (int64_t c0 = 0; c0 < n; c0 += (int64_t)kCompactNT * kCompactR) {
        int32_t g[kCompactR];
        unsigned bal[kCompactR];
#pragma unroll
        for (int r = 0; r < kCompactR; ++r) {
            const int64_t i = c0 + (int64_t)r * kCompactNT + t;
            g[r] = i < n ? act[i] : -1;
        }
#pragma unroll
        for (int r = 0; r < kCompactR; ++r) {
            const bool f = g[r] >= 0 && keep[g[r]] != 0;
            bal[r] = __ballot_sync(0xffffffffu, f);
            if (f && wkey) heavy += wkey[g[r]] >= thr;
            if (lane == 0) wtot[r][w] = __popc(bal[r]);
        }
        __syncthreads();
        if (w == 0) {
            // lane r: the exclusive offsets of round r's warps, after the
            // rounds before it
            int v = 0;
            if (lane < kCompactR)
                for (int q = 0; q < 32; ++q) v += wtot[lane][q];
            int incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += x;
            }
            if (lane < kCompactR) {
                int run = incl - v;
                for (int q = 0; q < 32; ++q) {
                    const int c = wtot[lane][q];
                    wtot[lane][q] = run;
                    run += c;
                }
            }
            if (lane == 31) batch_total = incl;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kCompactR; ++r)
            if (bal[r] >> lane & 1u) act_next[base + wtot[r][w] + __popc(bal[r] & lt)] = g[r];
        base += batch_total;
        __syncthreads();  // wtot and batch_total are rewritten by the next batch
    }
    if (t == 0) {
        *n_next = base;
        if (mirror) *mirror = base;  // the host's copy (pinned, mapped)
    }
    if (wkey) {
        heavy = __reduce_add_sync(0xffffffffu, heavy);
        if (lane == 0) wtot[0][w] = heavy;
        __syncthreads();
        if (t == 0) {
            int h = 0;
            for (int q = 0; q < kCompactNT / 32; ++q) h += wtot[0][q];
            *n_heavy_next = h;
        }
    }
}
cudaError_t launch_compact_kept(const int32_t* act, const int32_t* n_act, int64_t n_fixed, const int8_t* keep,
                                int32_t* act_next, int32_t* n_next, cudaStream_t st, const int32_t* wkey,
                                int32_t thr, int32_t* n_heavy_next, volatile int32_t* mirror) {
    return launch_dependent(compact_kept_kernel, 1, kCompactNT, 0, st, act, n_act, n_fixed, keep, act_next, n_next, wkey,
                            thr, n_heavy_next, mirror);
}
// *out = the number of leading entries of key (descending) that are >= thr
__global__ void count_at_least_kernel(const int32_t* key, int64_t n, int32_t thr, int32_t* out) {
    int64_t lo = 0, hi = n;  // key[0, lo) >= thr, key[hi, n) < thr
    while (lo < hi) {
        const int64_t mid = (lo + hi) / 2;
        if (key[mid] >= thr) lo = mid + 1; else hi = mid;
    }
    *out = (int32_t)lo;
}
cudaError_t launch_count_at_least(const int32_t* key, int64_t n, int32_t thr, int32_t* out, cudaStream_t st) {
    count_at_least_kernel<<<1, 1, 0, st>>>(key, n, thr, out);
    return cudaGetLastError();
}
__global__ void set_i32_kernel(int32_t* a, int32_t v) { *a = v; }
cudaError_t launch_set_i32(int32_t* a, int32_t v, cudaStream_t st) {
    set_i32_kernel<<<1, 1, 0, st>>>(a, v);
    return cudaGetLastError();
}
}  // namespace devil
