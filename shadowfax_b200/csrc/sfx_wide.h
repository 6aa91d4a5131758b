/*
 * 32-byte global loads and stores (sm_100: one instruction moves a whole
 * 32-byte sector per lane).  A gather of a record costs the L1 one tag lookup
 * per lane and instruction whatever its width, so a record is read in the
 * fewest, widest loads.  Addresses are 32-byte aligned; loads take the
 * read-only path (nothing a kernel writes is read back through them).
 */
#ifndef SFX_WIDE_H
#define SFX_WIDE_H

__device__ __forceinline__ void sfx_load32(const float* p, float* v) {
    asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),
                   "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}

__device__ __forceinline__ void sfx_load32(const double* p, double* v) {
    asm volatile("ld.global.nc.v4.f64 {%0,%1,%2,%3}, [%4];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
                 : "l"(p));
}

__device__ __forceinline__ void sfx_store32(float* p, const float* v) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]),
                 "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

__device__ __forceinline__ void sfx_store32(double* p, const double* v) {
    asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(p), "d"(v[0]), "d"(v[1]),
                 "d"(v[2]), "d"(v[3])
                 : "memory");
}

#endif
