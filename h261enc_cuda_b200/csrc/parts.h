/* The encode kernels in parts: kernels.cu is compiled eight times, once for each
 * pair of arithmetics, of searches and of staging variants, so that each part
 * is a module of its own.  CUDA loads a module when a program first uses one of
 * its kernels, in a time that goes with all of the module's code and line
 * tables.  As one module the 69 kernels, of which a program uses a handful,
 * took 25 ms of a process's first engine (nvcc compresses an image of that
 * size; without that, 13 ms); a part takes about 2.  A new process up to the
 * 40th picture of one QCIF stream: 57 ms before, 35 so; of 64 mixed streams
 * 65 and 43.  launch.cu picks the part and the kernel of a launch. */
#pragma once

#include <cuda_runtime.h>

#include "h261b_device.h"

namespace h261b {

/* what a launch of the step kernel does per MB */
enum StepKind {
    KIND_FUSED = 0,    /* the phases the launch asks for, in one pass       */
    KIND_SEARCH = 1,   /* search, costs and mode decision (into md_out)     */
    KIND_ENCODE = 2,   /* MC ... reconstruction from md_in, after a search
                          launch (programmatic dependent launch: waits for
                          that grid before it reads anything)               */
    KIND_FULL = 3,     /* KIND_FUSED with every phase (search, mode decision,
                          encode): the engine's and the no-allocation
                          entry point's launch, compiled without the paths
                          of partial launches                               */
};

/* small launches: warps of the CTA that takes a macroblock */
constexpr int TEAM_WARPS = 4, TEAM_THREADS = 32 * TEAM_WARPS;

using StepFn = void (*)(const h261b_session_dev_t *, const uint32_t *, int32_t, int32_t, int32_t, int32_t *);
using TeamFn = void (*)(const h261b_session_dev_t *, const uint32_t *, int32_t);
using TeamPictureFn = void (*)(h261b_session_dev_t, int32_t);

struct KernelPart {
    StepFn (*step)(int kind, int abi, int code);      /* (KIND_ENCODE: the reference search's parts) */
    TeamFn (*team)(int code);                         /* the team kernels: cp.async parts            */
    TeamPictureFn (*team_picture)(int abi);
    int (*checks)(unsigned long long *n, int first[2]);   /* the checking build's violations, cleared */
    int (*timeouts)(unsigned int *n);                     /* bulk staging's, cleared                 */
    /* shared memory of a warp: search only, encode, encode and code; and of
     * a CTA that codes */
    size_t search_bytes, encode_bytes, code_bytes, table_bytes;
};
/* by fmad * 4 + exhaustive search * 2 + bulk staging */
extern const KernelPart kernel_part_0, kernel_part_1, kernel_part_2, kernel_part_3, kernel_part_4, kernel_part_5,
    kernel_part_6, kernel_part_7;

/* sum of |a_i - b_i| over the four bytes, added to acc: one instruction,
 * one ALU-pipe slot (2.1 cycles a warp on an SM quarter).  The accumulating
 * form is written in PTX because acc += __vsadu4(a, b) compiles to a
 * separate add (5.1 against 4.05 cycles a word with its funnel shift), and
 * __vabsdiffu4 + __dp4a issues two instructions for the same ALU time. */
__device__ __forceinline__ uint32_t sad4(uint32_t a, uint32_t b, uint32_t acc)
{
    uint32_t d;
    asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(acc));
    return d;
}

} // namespace h261b
