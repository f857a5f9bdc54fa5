// OSCAR text of the hadron records on the GPU (FSSW::combine_samples_to_OSCAR,
// src/FSSW.cpp:365-494): every record becomes one fixed-width line
//   setw(10) ipart+1, "  ", setw(10) pid, then nine "%24.16e" fields
//   (px py pz E mass x y z t) separated by two spaces, and "\n",
// and every event with hadrons gets the sub-header
//   setw(10) iev, "  ", setw(10) n, "  ", setw(8) 0.0, "  ", setw(8) 0.0, "\n".
// The fields are formatted exactly (format_e.h), so the bytes equal those of
// the C library's printf.
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "format_e.h"
#include "kernels.h"

namespace iss {

namespace {

constexpr int kOscarHadrons = 32;                   // per block and step
constexpr int kOscarThreads = 9 * kOscarHadrons;    // a warp per floating field

// A block makes the text of 32 hadrons at a time in shared memory, warp k the
// k-th floating field of every line, and stores it in 16-byte words: the lines
// are contiguous in the file, with a sub-header before the first hadron of an
// event.  Bound by the formatting's integer instructions.  222,078 hadrons (57
// MB): 553 us with a thread per line writing bytes to memory, 76 us so (seven
// launches).
__global__ void __launch_bounds__(kOscarThreads)
oscar_lines_kernel(const HadronRec* __restrict__ had, int64_t h0, int64_t h1,
                   const int64_t* __restrict__ ev_off, const int64_t* __restrict__ ev_byte,
                   int e_lo, int e_hi, int64_t byte0, char* __restrict__ out) {
    __shared__ __align__(16) char s_text[16 + kOscarHadrons * (kOscarLine + kOscarSubHeader)];
    __shared__ int64_t s_line[kOscarHadrons];   // byte of each line, from the chunk's first
    const int lane = threadIdx.x & 31, field = threadIdx.x >> 5;
    const float* rec0 = reinterpret_cast<const float*>(had);
    constexpr int kRec = sizeof(HadronRec) / sizeof(float);
    // records hold pid, mass, E, px, py, pz, t, x, y, z
    constexpr int kColumn[9] = {3, 4, 5, 2, 1, 7, 8, 9, 6};
    int column = 0;
#pragma unroll
    for (int k = 0; k < 9; k++)
        if (field == k) column = kColumn[k];
    for (int64_t b0 = h0 + static_cast<int64_t>(blockIdx.x) * kOscarHadrons; b0 < h1;
         b0 += static_cast<int64_t>(gridDim.x) * kOscarHadrons) {
        const int64_t h = b0 + lane;
        const bool on = h < h1;
        int64_t ipart = 0, n_ev = 0;
        int event = 0;
        if (field < 2 && on) {
            // event of hadron h: the last e in [e_lo, e_hi) with ev_off[e] <= h
            int lo = e_lo, hi = e_hi - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (ev_off[mid] <= h) lo = mid; else hi = mid - 1;
            }
            event = lo;
            ipart = h - ev_off[lo];
            n_ev = ev_off[lo + 1] - ev_off[lo];
            if (field == 0) s_line[lane] = ev_byte[lo] - byte0 + kOscarSubHeader + ipart * kOscarLine;
        }
        if (field == 0 && lane == 0 && ipart == 0) s_line[0] -= kOscarSubHeader;   // the block's first byte
        __syncthreads();
        const int64_t begin = s_line[0];
        // the text sits at the same offset from a 16-byte boundary as its place
        const int pad = static_cast<int>(reinterpret_cast<uintptr_t>(out + begin) & 15);
        __syncthreads();
        if (field == 0 && lane == 0 && ipart == 0) s_line[0] += kOscarSubHeader;
        __syncthreads();
        if (on) {
            char* line = s_text + pad + static_cast<int>(s_line[lane] - begin);
            if (field == 0) {
                fmt::format_int(ipart + 1, 10, line);
                line[10] = ' ';
                line[11] = ' ';
                fmt::format_int(__float_as_int(rec0[h * kRec]), 10, line + 12);
                line[kOscarLine - 1] = '\n';
            } else if (field == 1 && ipart == 0) {
                char* sh = line - kOscarSubHeader;
                fmt::format_int(event, 10, sh);
                sh[10] = ' ';
                sh[11] = ' ';
                fmt::format_int(n_ev, 10, sh + 12);
                const char tail[] = "         0         0\n";   // "  " + setw(8) "0", twice
                for (int i = 0; i < 21; i++) sh[22 + i] = tail[i];
            }
            char* f = line + 22 + field * 26;
            f[0] = ' ';
            f[1] = ' ';
            fmt::format_e24_16(rec0[h * kRec + column], f + 2);
        }
        __syncthreads();
        const int last = static_cast<int>(min(static_cast<int64_t>(kOscarHadrons), h1 - b0)) - 1;
        const int end = pad + static_cast<int>(s_line[last] - begin) + kOscarLine;
        char* dst = out + begin - pad;   // 16-byte aligned
        const int w0 = (pad + 15) >> 4, w1 = end >> 4;
        for (int w = w0 + threadIdx.x; w < w1; w += kOscarThreads)
            reinterpret_cast<uint4*>(dst)[w] = reinterpret_cast<const uint4*>(s_text)[w];
        if (threadIdx.x < 16) {
            const int i = pad + threadIdx.x;             // before the first whole word
            if (i < min(16 * w0, end)) dst[i] = s_text[i];
            const int j = max(16 * w1, 16 * w0) + threadIdx.x;   // behind the last one
            if (j < end) dst[j] = s_text[j];
        }
        __syncthreads();
    }
}

}  // namespace

cudaError_t launch_oscar_lines(const HadronRec* had, int64_t h0, int64_t h1, const int64_t* ev_off,
                               const int64_t* ev_byte, int e_lo, int e_hi, int64_t byte0,
                               char* out, int num_sms, cudaStream_t stream) {
    if (h1 <= h0) return cudaSuccess;
    int64_t blocks = (h1 - h0 + kOscarHadrons - 1) / kOscarHadrons;
    const int64_t cap = static_cast<int64_t>(num_sms) * 32;
    if (blocks > cap) blocks = cap;
    oscar_lines_kernel<<<static_cast<unsigned>(blocks), kOscarThreads, 0, stream>>>(
        had, h0, h1, ev_off, ev_byte, e_lo, e_hi, byte0, out);
    return cudaGetLastError();
}

}  // namespace iss
