// jt_batch.cu -- the batch kernel (jt_batch.cuh).
#include "jt_batch.cuh"
#include "jt_batchmix.cuh"
#include "jt_fixmix.cuh"

namespace jt {

template <typename T> __device__ void elem_dispatch(const BOp &o, int64_t idx) {
    typedef typename V2<T>::t C2;
    const EArgs &e = o.e;
    switch (o.kind) {
        case EK_COPY_COMPLEX:
            copy_complex_body<T>((const C2 *)e.p[0], e.i[0], (C2 *)e.p[1], e.i[1], e.i[2], e.i[3], (T)e.d[0], e.f, idx);
            break;
        case EK_BLUE_PRE:
            if (o.sign < 0)
                bluestein_pre_body<-1, T>((const C2 *)e.p[0], e.i[0], (C2 *)e.p[1], (const C2 *)e.p[2], e.i[1], e.i[2], e.i[3], idx);
            else
                bluestein_pre_body<1, T>((const C2 *)e.p[0], e.i[0], (C2 *)e.p[1], (const C2 *)e.p[2], e.i[1], e.i[2], e.i[3], idx);
            break;
        case EK_BLUE_MUL:
            if (o.sign < 0) bluestein_mul_body<-1, T>((C2 *)e.p[0], (const C2 *)e.p[1], e.i[0], e.i[1], idx);
            else bluestein_mul_body<1, T>((C2 *)e.p[0], (const C2 *)e.p[1], e.i[0], e.i[1], idx);
            break;
        case EK_BLUE_POST:
            if (o.sign < 0)
                bluestein_post_body<-1, T>((C2 *)e.p[0], e.i[0], (const C2 *)e.p[1], (const C2 *)e.p[2], e.i[1], e.i[2], e.i[3],
                                           (T)e.d[0], idx);
            else
                bluestein_post_body<1, T>((C2 *)e.p[0], e.i[0], (const C2 *)e.p[1], (const C2 *)e.p[2], e.i[1], e.i[2], e.i[3],
                                          (T)e.d[0], idx);
            break;
        case EK_REAL_POST_PACKED:
            real_post_packed_body<T>((T *)e.p[0], e.i[0], e.i[1], e.i[2], (const C2 *)e.p[1], idx);
            break;
        case EK_REAL_POST_FULL:
            if (o.sign < 0)
                real_post_full_body<-1, T>((const T *)e.p[0], e.i[0], (T *)e.p[1], e.i[1], e.i[2], e.i[3], (const C2 *)e.p[2],
                                           (T)e.d[0], idx);
            else
                real_post_full_body<1, T>((const T *)e.p[0], e.i[0], (T *)e.p[1], e.i[1], e.i[2], e.i[3], (const C2 *)e.p[2],
                                          (T)e.d[0], idx);
            break;
        case EK_REAL_PRE_INV:
            real_pre_inverse_body<T>((T *)e.p[0], e.i[0], e.i[1], e.i[2], (const C2 *)e.p[1], (T)e.d[0], idx);
            break;
        case EK_R2C: real_to_complex_body<T>((const T *)e.p[0], e.i[0], (C2 *)e.p[1], e.i[1], e.i[2], idx); break;
        case EK_PACK_FULL: pack_from_full_body<T>((const C2 *)e.p[0], (T *)e.p[1], e.i[0], e.i[1], e.i[2], idx); break;
        case EK_UNPACK_FULL: unpack_to_full_body<T>((const T *)e.p[0], e.i[0], (C2 *)e.p[1], e.i[1], e.i[2], idx); break;
        case EK_REAL_PART: real_part_body<T>((const C2 *)e.p[0], (T *)e.p[1], e.i[0], e.i[1], e.i[2], (T)e.d[0], idx); break;
        case EK_DCT2_PRE:
            dct2_pre_body<T>((const T *)e.p[0], e.i[0], (T *)e.p[1], e.i[1], e.i[2], e.i[3], e.f, idx);
            break;
        case EK_DCT2_POST:
            dct2_post_body<T>((const T *)e.p[0], e.i[0], (T *)e.p[1], e.i[1], e.i[2], e.i[3], (const C2 *)e.p[2], (T)e.d[0],
                              (T)e.d[1], e.f, idx);
            break;
        case EK_DCT3_PRE:
            dct3_pre_body<T>((const T *)e.p[0], e.i[0], (T *)e.p[1], e.i[1], e.i[2], e.i[3], (const C2 *)e.p[2], (T)e.d[0],
                             (T)e.d[1], e.f, idx);
            break;
        case EK_DCT3_POST:
            dct3_post_body<T>((const T *)e.p[0], e.i[0], (T *)e.p[1], e.i[1], e.i[2], e.i[3], e.f, idx);
            break;
        case EK_DHT_POST:
            dht_post_body<T>((const T *)e.p[0], e.i[0], (T *)e.p[1], e.i[1], e.i[2], e.i[3], (T)e.d[0], idx);
            break;
        case EK_SCALE: scale_body<T>((T *)e.p[0], e.i[0], e.i[1], e.i[2], (T)e.d[0], idx); break;
        case EK_COPY_REAL: copy_real_body<T>((const T *)e.p[0], e.i[0], (T *)e.p[1], e.i[1], e.i[2], e.i[3], idx); break;
    }
}

template <typename T> __device__ void r2r_dispatch(const BOp &o, int idx, unsigned char *smem) {
    typedef typename V2<T>::t C2;
    const T *in = (const T *)o.in;
    T *out = (T *)o.out;
    const C2 *W = (const C2 *)o.W, *Wr = (const C2 *)o.Whi, *Wd = (const C2 *)o.Wlo;
    if (o.kind == R2R_DCT2) r2r_tile_body<R2R_DCT2, T>(in, out, o.rp, W, Wr, Wd, idx, smem);
    else if (o.kind == R2R_DCT3) r2r_tile_body<R2R_DCT3, T>(in, out, o.rp, W, Wr, Wd, idx, smem);
    else if (o.kind == R2R_DHT) r2r_tile_body<R2R_DHT, T>(in, out, o.rp, W, Wr, Wd, idx, smem);
    else if (o.kind == R2R_RFWD) r2r_tile_body<R2R_RFWD, T>(in, out, o.rp, W, Wr, Wd, idx, smem);
    else r2r_tile_body<R2R_RINV, T>(in, out, o.rp, W, Wr, Wd, idx, smem);
}

__device__ __forceinline__ int ld_acquire_gpu(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// wait_polls: polls of a dependency wait (64 ns apart) before it gives up;
// the library's default, 2^24, is about a second
template <typename T>
__global__ void __launch_bounds__(JT_BATCH_THREADS, sizeof(T) == 4 ? 3 : 2)
    batch_kernel(const BOp *__restrict__ ops, const BTask *__restrict__ tasks, int ntasks, int *head, int *done, int *err,
                 int wait_polls) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_task;
    __shared__ int s_ok;
    const int tid = threadIdx.x;
    for (;;) {
        if (tid == 0) s_task = atomicAdd(head, 1);
        __syncthreads();
        const int ti = s_task;
        if (ti >= ntasks) break;
        const BTask tk = tasks[ti];
        const BOp &o = ops[tk.op];
        if (tid == 0) {
            int ok = 1;
            if (o.dep >= 0) {
                const int need = ops[o.dep].ntasks;
                int it = 0;
                while (ld_acquire_gpu(&done[o.dep]) < need) {
                    if (++it > wait_polls) {
                        ok = 0;
                        atomicExch(err, 1);
                        break;
                    }
                    __nanosleep(64);
                }
            }
            s_ok = ok;
        }
        __syncthreads();
        if (s_ok) {
            typedef typename V2<T>::t C2;
            const C2 *in = (const C2 *)o.in, *W = (const C2 *)o.W, *Whi = (const C2 *)o.Whi, *Wlo = (const C2 *)o.Wlo;
            C2 *out = (C2 *)o.out;
            if (sizeof(T) == 4 && o.type == BOP_MIX) {
                if constexpr (sizeof(T) == 4) batch_mix_body(in, out, o.mp, Whi, Wlo, tk.idx, smem_raw);
            } else if (sizeof(T) == 8 && o.type == BOP_FIX) {
                if constexpr (sizeof(T) == 8) fixmix_body(in, out, o.fm, tk.idx, smem_raw);
            } else if (o.type == BOP_TILE) {
                if (o.sign < 0) tile_fft_body<-1, T>(in, out, o.tp, W, Whi, Wlo, tk.idx, smem_raw);
                else tile_fft_body<1, T>(in, out, o.tp, W, Whi, Wlo, tk.idx, smem_raw);
            } else if (o.type == BOP_BLUE) {
                if (o.sign < 0) blue_tile_body<-1, T>(in, out, o.bp, W, Whi, Wlo, tk.idx, smem_raw);
                else blue_tile_body<1, T>(in, out, o.bp, W, Whi, Wlo, tk.idx, smem_raw);
            } else if (o.type == BOP_R2R) {
                r2r_dispatch<T>(o, tk.idx, smem_raw);
            } else {
                const int64_t base = (int64_t)tk.idx * JT_BATCH_ELEMS_PER_TASK;
                for (int k = tid; k < JT_BATCH_ELEMS_PER_TASK; k += JT_BATCH_THREADS) {
                    const int64_t idx = base + k;
                    if (idx < o.total) elem_dispatch<T>(o, idx);
                }
            }
        }
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            atomicAdd(&done[tk.op], 1);
        }
    }
}

static const void *batch_function(int prec) {
    return prec == 0 ? (const void *)batch_kernel<float> : (const void *)batch_kernel<double>;
}
// Once per process: both kernels may take the most there is. (Set to what one
// batch needs, it was too little for another made before.)
cudaError_t batch_setup(int smem_optin) {
    for (int prec = 0; prec < 2; prec++) {
        const void *k = batch_function(prec);
        cudaFuncAttributes at;
        cudaError_t e = cudaFuncGetAttributes(&at, k);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin - (int)at.sharedSizeBytes);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}
// Blocks per SM of the kernel of prec (0: float, 1: double) with `smem` bytes each.
cudaError_t batch_occupancy(int prec, int smem, int *per_sm) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, batch_function(prec), JT_BATCH_THREADS, smem);
}

void batch_launch(int prec, const BOp *ops, const BTask *tasks, int ntasks, int *head, int *done, int *err, int wait_polls, int grid,
                  int smem, cudaStream_t s) {
    if (prec == 0) batch_kernel<float><<<grid, JT_BATCH_THREADS, smem, s>>>(ops, tasks, ntasks, head, done, err, wait_polls);
    else batch_kernel<double><<<grid, JT_BATCH_THREADS, smem, s>>>(ops, tasks, ntasks, head, done, err, wait_polls);
}

}  // namespace jt
