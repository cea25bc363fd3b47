// Device-side helpers shared by the multi-job kernels: a job list passed by
// value in kernel parameters, the job of the current block, 16-byte Z_q loads.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "dm_jobs.cuh"

namespace dm {
namespace jobkit {

template <class J>
struct JobList {
    J j[kMaxJobs];
    int n;
    bool beside;  // stage_open()
};

// Job of this block (jobs are sorted by cta0; at most kMaxJobs, uniform per block).
template <class J>
DM_D int find_job(const JobList<J>& L) {
    int k = 0;
    while (k + 1 < L.n && blockIdx.x >= L.j[k + 1].cta0) ++k;
    return k;
}

DM_D fq ldq(const uint4* p, uint64_t i) {
    const uint4 v = p[i];
    return fq{{v.x, v.y, v.z, v.w}};
}
DM_D fq ldq(PastL1<uint4> p, uint64_t i) {
    const uint4 v = p[i];
    return fq{{v.x, v.y, v.z, v.w}};
}
DM_D void stq(uint4* p, uint64_t i, const fq& a) { p[i] = make_uint4(a.w[0], a.w[1], a.w[2], a.w[3]); }

// A proof is a chain of short kernels, and at small rings a kernel's launch and
// drain take as long as its work.  These kernels are launched so that the next
// one's blocks may be set up while the last of this one's still run
// (launch_overlapped); each begins with stage_begin(), which lets the next kernel
// in and then waits until everything before this one has finished and is visible.
// Every thread passes it before any global access and before any return, so a
// kernel that has finished implies that all before it have.  (A launch without the
// attribute makes both instructions empty.)  Loads after it must not be of the
// read-only kind, which a compiler may move above it: no __ldg of what another
// kernel wrote.  Without / with it: a
// proof of 52 KB 633 / 522 us, of 1 MiB 1,300 / 1,089, of 16 MiB 4,180 / 3,918; five
// ring products at 2^6 24.5 / 20.9 us, 301 at 2^11 74.8 / 68.4.
DM_D void stage_begin() {
    asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
}
// Kernels of one stage that do not need one another's results (the file's hash, its
// unpacking and the generators; the finishes of two ring sizes; a verifier's transcript
// and the generators) run side by side the same way: the first one opens, letting the next in only after its own wait, and the
// others are launched "beside" it, start without a wait and make it at their end.
// One thread does, so that blocks come and go meanwhile; the kernel has finished only
// when those before it have, which is what the next wait relies on.  What a kernel
// beside another reads was finished before the first one's wait, but not waited for
// here: it is read past L1, which may hold what was there before (PastL1, and the
// finishes' partials by __ldcg).  A proof of 1 MiB went
// from 889 to 838 us, of 16 MiB from 3,711 to 3,621, 24 files of 50 KB to 16 MiB
// through the engine from 11.3 to 11.0 ms.
struct Beside {
    bool last;
    DM_D ~Beside() {
        if (last) asm volatile("griddepcontrol.wait;" ::: "memory");
    }
};
DM_D Beside stage_open(bool beside) {
    if (!beside) asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    return Beside{beside && blockIdx.x == 0 && threadIdx.x == 0};
}
template <class... P, class... A>
inline cudaError_t launch_stage(bool overlapped, void (*kernel)(P...), uint32_t grid, uint32_t block, size_t smem,
                                cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = overlapped ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
template <class... P, class... A>
inline cudaError_t launch_overlapped(void (*kernel)(P...), uint32_t grid, uint32_t block, size_t smem, cudaStream_t st,
                                     A&&... args) {
    return launch_stage(true, kernel, grid, block, smem, st, std::forward<A>(args)...);
}

// Numbers the blocks of each job consecutively and copies the jobs into L.
template <class J>
inline uint32_t assign_ctas(J* jobs, int n, JobList<J>& L, uint64_t (*ctas_of)(const J&), bool beside = false) {
    uint64_t total = 0;
    L.n = n;
    L.beside = beside;
    for (int i = 0; i < n; ++i) {
        jobs[i].cta0 = (uint32_t)total;
        L.j[i] = jobs[i];
        total += ctas_of(jobs[i]);
    }
    return (uint32_t)total;
}

}  // namespace jobkit
}  // namespace dm
