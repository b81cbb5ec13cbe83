// jt_batch.cuh -- one persistent launch per precision for a batch of
// transforms of mixed sizes and kinds.
//
// The host records each transform as a chain of steps (line passes of
// jt_batchmix.cuh, jt_fixmix.cuh and jt_device.cuh, one-step real, DCT and
// Bluestein lines, elementwise pre/post steps) into a table of ops.  Each op
// is split into tasks of one CTA's work; the queue holds them in the order of
// a schedule made beforehand.  batch_kernel's CTAs pull tasks with an atomic
// counter, wait (bounded) until the task's previous step in the same transform
// has finished, run it and count it done.  Because a step's tasks are all
// queued before any task of the next step, every awaited task is already held
// by a running CTA and the waits end.  Producer CTAs publish with a gpu-scope
// fence before the counter update; consumers read the counter with acquire
// semantics before their threads touch the data.
#pragma once

#include "jt_device.cuh"
#include "jt_stockham.cuh"
#include "jt_r2r.cuh"
#include "jt_chirp.cuh"
#include "jt_bluemix.cuh"
#include "jt_batchmix_params.cuh"
#include "jt_fixmix.cuh"

namespace jt {

enum BOpType { BOP_TILE = 0, BOP_MIX = 1, BOP_ELEM = 2, BOP_R2R = 3, BOP_BLUE = 4, BOP_FIX = 5 };

enum ElemKind {
    EK_COPY_COMPLEX = 0,
    EK_BLUE_PRE,
    EK_BLUE_MUL,
    EK_BLUE_POST,
    EK_REAL_POST_PACKED,
    EK_REAL_POST_FULL,
    EK_REAL_PRE_INV,
    EK_R2C,
    EK_PACK_FULL,
    EK_UNPACK_FULL,
    EK_REAL_PART,
    EK_DCT2_PRE,
    EK_DCT2_POST,
    EK_DCT3_PRE,
    EK_DCT3_POST,
    EK_DHT_POST,
    EK_SCALE,
    EK_COPY_REAL,
};

struct EArgs {
    const void *p[4];
    int64_t i[6];
    double d[3];
    int f;
};

struct BOp {
    int type, prec, sign, kind;
    int dep;     // op this one waits for (-1: none)
    int ntasks;  // CTA work units
    int64_t total;  // elementwise: number of indices
    // tile / stock
    union {
        TileParams tp;
        R2rParams rp;   // DCT/DST/DHT and packed real lines in one step (kind: the R2rOp)
        BlueParams bp;  // a Bluestein transform in one step (W, Whi, Wlo: roots, bk1, bk2)
        BatchMix mp;    // float lines and convolutions on register passes
        FixMixParams fm;  // double lines (jt_fixmix.cuh)
    };
    const void *in;
    void *out;
    const void *W, *Whi, *Wlo;
    int smem;  // shared memory the step needs (bytes)
    // elementwise
    EArgs e;
};

struct BTask {
    int op;
    int idx;
};

// A batch CTA has 256 threads and at most JT_BATCH_SMEM_CAP bytes of shared
// memory per task, so that three CTAs share an SM and their loads overlap one
// another's arithmetic (lines whose tile would need more are recorded as two
// passes of shorter lines).  Each precision has a kernel and a queue of its
// own: the double lines' fixed-point passes take 128 registers a thread (two
// CTAs per SM), the float ones 80.
#define JT_BATCH_THREADS 256
#define JT_BATCH_ELEMS_PER_TASK (JT_BATCH_THREADS * 8)
#define JT_BATCH_SMEM_CAP (72 * 1024)

}  // namespace jt
