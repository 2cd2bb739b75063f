// Tensor memory (TMEM) used as a per-lane table: 128 lanes x 512 columns of 32 bits per SM. A warp reaches the 32
// lanes of its own quarter, (warp index mod 4), so warps w and w + 4 of a CTA see the same 32 x 512 words; lane l of
// the warp reads and writes row l. Reads do not go through the shared-memory data pipe.
#pragma once
#include "tma.cuh"

namespace gn {

// all 512 columns; one warp, all lanes; the base address lands in shared memory
__device__ __forceinline__ void tmem_alloc_all(unsigned *slot)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free_all(unsigned base)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(base));
}
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld4(unsigned a, float *r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3},[%4];" : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]) : "r"(a));
}
__device__ __forceinline__ void tmem_ld8(unsigned a, float *r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7},[%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
                 : "r"(a));
}
__device__ __forceinline__ void tmem_ld16(unsigned a, float *r)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15},[%16];"
        : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]),
          "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
        : "r"(a));
}
__device__ __forceinline__ void tmem_st4(unsigned a, const float *r)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%4],{%0,%1,%2,%3};" ::"f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]), "r"(a));
}
__device__ __forceinline__ void tmem_st8(unsigned a, const float *r)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8],{%0,%1,%2,%3,%4,%5,%6,%7};" ::"f"(r[0]), "f"(r[1]), "f"(r[2]),
                 "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]), "r"(a));
}
__device__ __forceinline__ void tmem_st16(unsigned a, const float *r)
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16],{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"f"(r[0]),
        "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]), "f"(r[8]), "f"(r[9]), "f"(r[10]),
        "f"(r[11]), "f"(r[12]), "f"(r[13]), "f"(r[14]), "f"(r[15]), "r"(a));
}
// mark registers of an earlier tmem_ld as ready, after a wait that named other registers
__device__ __forceinline__ void tmem_use8(float *r)
{
    asm volatile("" : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]));
}
__device__ __forceinline__ void tmem_use4(float *r) { asm volatile("" : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3])); }
__device__ __forceinline__ void tmem_use12(float *r)
{
    asm volatile("" : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]), "+f"(r[8]),
                 "+f"(r[9]), "+f"(r[10]), "+f"(r[11]));
}
__device__ __forceinline__ void tmem_use16(float *r)
{
    asm volatile("" : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]), "+f"(r[8]),
                 "+f"(r[9]), "+f"(r[10]), "+f"(r[11]), "+f"(r[12]), "+f"(r[13]), "+f"(r[14]), "+f"(r[15]));
}
// Waits for every earlier tmem_ld of this thread. The registers that those loads fill are operands, so that no use
// of them can move above the wait.
__device__ __forceinline__ void tmem_wait_ld16(float *r)
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]), "+f"(r[8]),
                   "+f"(r[9]), "+f"(r[10]), "+f"(r[11]), "+f"(r[12]), "+f"(r[13]), "+f"(r[14]), "+f"(r[15]));
}
__device__ __forceinline__ void tmem_wait_ld4(float *r)
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]));
}
__device__ __forceinline__ void tmem_wait_ld8(float *r)
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]));
}
__device__ __forceinline__ void tmem_wait_ld12(float *r)
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]), "+f"(r[8]),
                   "+f"(r[9]), "+f"(r[10]), "+f"(r[11]));
}

}  // namespace gn
