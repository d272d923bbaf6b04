// Preparation of a per-class-pair call (jk_build_class_pair and its
// non-allocating twin): what the class kernel reads of the bins, in one launch.
#pragma once
#include "jk_common.cuh"

// Block-wide inclusive scan of two counts (whole warps), with running carries.
__device__ __forceinline__ void jk_block_scan2(long long a, long long b, long long& ia, long long& ib,
                                               long long* wa, long long* wb, long long& carry_a,
                                               long long& carry_b) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        long long ya = __shfl_up_sync(0xffffffffu, a, o), yb = __shfl_up_sync(0xffffffffu, b, o);
        if (lane >= o) {
            a += ya;
            b += yb;
        }
    }
    if (lane == 31) {
        wa[warp] = a;
        wb[warp] = b;
    }
    __syncthreads();
    if (warp == 0) {
        long long x = (lane < (int)(blockDim.x >> 5)) ? wa[lane] : 0;
        long long y = (lane < (int)(blockDim.x >> 5)) ? wb[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            long long u = __shfl_up_sync(0xffffffffu, x, o), v = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) {
                x += u;
                y += v;
            }
        }
        wa[lane] = x;
        wb[lane] = y;
    }
    __syncthreads();
    ia = a + (warp ? wa[warp - 1] : 0) + carry_a;
    ib = b + (warp ? wb[warp - 1] : 0) + carry_b;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) {
        carry_a = ia;
        carry_b = ib;
    }
    __syncthreads();
}

// the segment of a call to the device (any block size)
__device__ __forceinline__ void jk_seg_copy(const JKSeg& sg, JKSeg* __restrict__ dst) {
    const int* a = reinterpret_cast<const int*>(&sg);
    int* d = reinterpret_cast<int*>(dst);
    for (int x = threadIdx.x; x < (int)(sizeof(JKSeg) / 4); x += blockDim.x) d[x] = a[x];
}

static inline int jk_pair_prep_threads(int nrun) { return nrun >= 1024 ? 1024 : (nrun + 31) / 32 * 32; }

// Run classes, one block: the ket end of every entry (cols(rank): columns the
// bins keep of a row), the items of every run, their exclusive prefix and
// total, and the segment itself.  The three launches that this replaces, and
// one for the segment, took 11.6 us of a call of 40 to 60 (13 atoms, TZVP);
// they stay for classes of more than JK_PAIR_PREP_ROWS bra pairs, which one
// block would walk for too long.
template <class Cols>
__global__ void __launch_bounds__(1024) jk_pair_prep_kernel(const __grid_constant__ Cols cols,
                                                            const __grid_constant__ JKSeg sg, JKSeg* dst,
                                                            const int* __restrict__ erank, int chunk,
                                                            int* __restrict__ ehi, long long* __restrict__ ioff,
                                                            long long* __restrict__ itm) {
    __shared__ long long carry, carry2;
    __shared__ long long wsum[32], wsum2[32];
    jk_seg_copy(sg, dst);
    if (threadIdx.x == 0) carry = carry2 = 0;
    __syncthreads();
    for (int base = 0; base < sg.nrun; base += blockDim.x) {
        const int r = base + threadIdx.x;
        int h = 0;
        if (r < sg.nrun) {
            const int e1 = sg.run0[r + 1];
            for (int e = sg.run0[r]; e < e1; e++) {
                const int c = cols(erank[e]);
                ehi[e] = c;
                h = max(h, c);
            }
        }
        const long long n = (jk_bucket_end(h, sg.bucket, sg.pst_kl) + chunk - 1) / chunk;
        long long incl, unused;
        jk_block_scan2(n, 0, incl, unused, wsum, wsum2, carry, carry2);
        if (r < sg.nrun) ioff[r] = incl - n;
    }
    if (threadIdx.x == 0) {
        itm[0] = 0;
        itm[1] = carry;
    }
}
