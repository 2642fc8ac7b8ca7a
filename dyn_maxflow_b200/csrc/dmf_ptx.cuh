// dmf_ptx.cuh -- the inline PTX of the solve kernel: loads, stores and atomics
// with a memory order, and special registers.  Everything else in the kernel is
// plain CUDA C++; the include guard lets the CPU tests put their own versions of
// these functions in this file's place and run the kernel on host threads.
#ifndef DMF_PTX_CUH
#define DMF_PTX_CUH

namespace dmfd {

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned atom_add_release_u32(unsigned *p, unsigned x) {
  unsigned v;
  asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "r"(x) : "memory");
  return v;
}
__device__ __forceinline__ unsigned atom_add_acqrel_u32(unsigned *p, unsigned x) {
  unsigned v;
  asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "r"(x) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sys_u32(unsigned *p, unsigned x) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(x) : "memory");
}
__device__ __forceinline__ int ld_rlx(const int *p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ long long ld_rlx(const long long *p) {
  long long v;
  asm volatile("ld.relaxed.gpu.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_rlx(const unsigned long long *p) {
  return (unsigned long long)ld_rlx((const long long *)p);
}
__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}
// Keeps a value that is computed only for its ordering.
__device__ __forceinline__ void keep_u64(unsigned long long x) { asm volatile("" ::"l"(x) : "memory"); }

}  // namespace dmfd

#endif
