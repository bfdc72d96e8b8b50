// CSR -> SELL-32 on the device, for the entry points that take a host CSR matrix and need no
// host copy of the pattern.
//
// On the host this took 3.3 of the 10.5 ms of a 60,680-row BiCGSTAB call (row lists with the
// diagonal first 1.05 ms, SELL positions 0.55, the sweeps' level schedules and uploads 1.2,
// values 0.5).  Here the CSR arrays go up as they are (20 to 30 us a megabyte) and two kernels
// form the same arrays, the host only adding up the slices' widths: 9.75 -> 6.8 ms a call with the
// solver's vectors in one allocation (now 5.7, 4.4 of it the solve's kernel).
#include "csr_device.hpp"

namespace sysu {

namespace {

struct CsrCheck {
    unsigned long long entries;  // diagonal-first row lists, without padding
    int bad;                     // a column out of range
};

// Width of each slice (warp a slice, lane a row): the longest row, counting its diagonal once
// whether it is stored or not.
__global__ void k_csr_widths(int n, int nslices, const int *__restrict__ rowptr, int base,
                             const int *__restrict__ col, int *__restrict__ sl_w, CsrCheck *chk) {
    const int s = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (s >= nslices) return;
    const int i = s * 32 + lane;
    int len = 0;
    bool bad = false;
    if (i < n) {
        len = 1;
        const int e = rowptr[i + 1] - base;
        for (int k = rowptr[i] - base; k < e; ++k) {
            const int c = col[k];
            bad = bad || c < 0 || c >= n;
            len += c != i;
        }
    }
    unsigned sum = (unsigned)len;
    int w = len;
    for (int o = 16; o > 0; o >>= 1) {
        w = max(w, __shfl_xor_sync(0xFFFFFFFFu, w, o));
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    }
    if (lane == 0) {
        sl_w[s] = w;
        atomicAdd(&chk->entries, (unsigned long long)sum);
    }
    if (bad) chk->bad = 1;
}

// Entries of a row in their CSR order behind the diagonal (repeated diagonal entries added up in
// order); padding holds 0 and the row itself, the last row in a slice's lanes past the end.
__global__ void k_csr_fill(int n, int nslices, const int *__restrict__ rowptr, int base, const int *__restrict__ col,
                           const double *__restrict__ val, const int *__restrict__ sl_ptr,
                           const int *__restrict__ sl_w, int *__restrict__ scol, double *__restrict__ sval) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nslices * 32) return;
    const size_t p = (size_t)sl_ptr[i >> 5] + (i & 31);
    const int w = sl_w[i >> 5], self = min(i, n - 1);
    double d = 0.0;
    int m = 0;
    if (i < n) {
        m = 1;
        const int e = rowptr[i + 1] - base;
        for (int k = rowptr[i] - base; k < e; ++k) {
            const int c = col[k];
            if (c == i) {
                d += val[k];
            } else {
                scol[p + 32 * (size_t)m] = c;
                sval[p + 32 * (size_t)m] = val[k];
                ++m;
            }
        }
        scol[p] = i;
        sval[p] = d;
    }
    for (; m < w; ++m) {
        scol[p + 32 * (size_t)m] = self;
        sval[p + 32 * (size_t)m] = 0.0;
    }
}

}  // namespace

void CsrDevice::load_on_device(int n, const int *rowptr, const int *col, const double *v, cudaStream_t st) {
    // the kernels index with rowptr: row lists that run backwards (and no rows) take the host path, which reads
    // such rows as empty
    bool ordered = n > 0 && rowptr[0] >= 0;
    for (int i = 0; i < n; ++i) ordered = ordered && rowptr[i] <= rowptr[i + 1];
    if (!ordered) return load(n, rowptr, col, v, st);
    const int base = rowptr[0], nslices = (n + 31) / 32;
    const size_t m = (size_t)(rowptr[n] - base);
    DevBuf<int> rp_d(n + 1), col_d(m);
    DevBuf<double> val_d(m);
    DevBuf<CsrCheck> chk(1);
    rp_d.upload(rowptr, n + 1, st);
    col_d.upload(col + base, m, st);
    val_d.upload(v + base, m, st);
    chk.zero(st);
    A.sl_w.alloc(nslices);
    k_csr_widths<<<(nslices * 32 + 255) / 256, 256, 0, st>>>(n, nslices, rp_d.get(), base, col_d.get(), A.sl_w.get(),
                                                             chk.get());
    ++g_launches;
    SYSU_CUDA(cudaGetLastError());
    std::vector<int> w(nslices), ptr(nslices + 1, 0);
    CsrCheck h;
    A.sl_w.download(w.data(), nslices, st);
    chk.download(&h, 1, st);
    SYSU_CUDA(cudaStreamSynchronize(st));
    if (h.bad) throw CaseError{"column index out of range"};
    long off = 0;
    int wmax = 0;
    for (int s = 0; s < nslices; ++s) {
        ptr[s] = (int)off;
        off += (long)w[s] * 32;
        wmax = std::max(wmax, w[s]);
        if (off > 0x7fffffffL) throw CaseError{"matrix too large for 32-bit positions"};
    }
    ptr[nslices] = (int)off;
    A.n = n;
    A.nslices = nslices;
    A.wmax = wmax;
    A.nnz = off;
    A.nnz_true = (long)h.entries;
    A.sl_ptr.upload(ptr, st);
    A.col.alloc(off);
    val.alloc(off);
    k_csr_fill<<<(nslices * 32 + 255) / 256, 256, 0, st>>>(n, nslices, rp_d.get(), base, col_d.get(), val_d.get(),
                                                           A.sl_ptr.get(), A.sl_w.get(), A.col.get(), val.get());
    ++g_launches;
    SYSU_CUDA(cudaGetLastError());
    SYSU_CUDA(cudaStreamSynchronize(st));
}

}  // namespace sysu
