/*
 * b200ng -- C ABI of the B200 backend for nGraph-Python graphs.
 *
 * Every entry point has C linkage, takes plain pointers and sizes, and returns an int status:
 * 0 on success, a negative B2_ERR_* code on failure (b2_last_error() then returns a
 * description owned by the library, valid until the next failing call on the same thread).
 * Device pointers are raw CUDA device addresses; `stream` is a cudaStream_t passed as void*.
 * Unless stated otherwise an entry point allocates no device memory: the caller owns every
 * buffer, including scratch.
 *
 * The reference drives its GPU through pycuda and has no C ABI of its own; each group below
 * names the reference interface (file:line in NervanaSystems/ngraph-python) whose job it takes
 * over.
 */
#ifndef B200NG_H
#define B200NG_H

#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

#define B2_OK 0
#define B2_ERR_INVALID (-1)     /* bad argument / unsupported program */
#define B2_ERR_CUDA (-2)        /* a CUDA runtime call failed */
#define B2_ERR_COMPILE (-3)     /* run-time kernel compilation failed */
#define B2_ERR_UNAVAILABLE (-4) /* a required system library could not be loaded */
#define B2_ERR_TIMEOUT (-5)     /* a bounded device-side wait ran out */
#define B2_ERR_COMM (-6)        /* NCCL reported an error */

const char* b2_last_error(void);
/* library version: major * 10000 + minor * 100 + patch */
int b2_version(void);
/* number of visible CUDA devices, or a negative error */
int b2_device_count(void);

/* ------------------------------------------------------------------------------------------
 * Fused elementwise + reduction kernels.
 * Replaces: ElementWiseKernel / CudaSourceFile / _get_compound_kernel / _generate_kernel_args
 * (ngraph/transformers/gputransform.py:86-345, ngraph/transformers/gpu/float_ew2.py:553-1653).
 * A program is a straight-line list of fp32 ops over up to 12 input tensors, with elementwise
 * outputs and at most one family of reductions, over an iteration space [A, B, C] (C innermost).
 * ------------------------------------------------------------------------------------------ */
#define B2_EW_MAX_IN 12
#define B2_EW_MAX_OUT 6   /* elementwise + reduction outputs together */
#define B2_EW_MAX_CONST 16
#define B2_EW_MAX_OPS 96

/* B2_FLEX16_PLANES (elementwise results only): the int16 mantissa is stored as two byte planes,
 * high bytes at the destination pointer and low bytes plane_bytes further -- the operand format
 * of the convolution entry points that take planes, so no separate split pass is needed. */
/* B2_F32_AT (inputs only): the pointer given at launch is the address of a device word that holds the
 * address of the values when the kernel runs, 16-byte aligned.  An fp32 result that is such an input's
 * register, laid out as the input, is not stored where that address is the result's own.
 * B2_FLEX16_AT (likewise): where that address is the result's own -- a B2_FLEX16 result with the input's
 * register, layout and slot, which there has to be -- it holds mantissas; elsewhere fp32 values, which
 * the program sees as b2_flex_host_quantize would store them (and that result stores so). */
enum b2_dtype { B2_F32 = 0, B2_FLEX16 = 1, B2_FLEX16_PLANES = 2, B2_F32_AT = 3, B2_FLEX16_AT = 4 };

/* op codes: one per template of float_ew2.py:31-68 */
enum b2_ew_opcode {
    B2_OP_ASSIGN = 0, B2_OP_NEG, B2_OP_ABS, B2_OP_SQRT, B2_OP_SQR, B2_OP_EXP, B2_OP_LOG,
    B2_OP_RCP, B2_OP_EXP2, B2_OP_LOG2, B2_OP_SIG, B2_OP_TANH, B2_OP_SAFELOG, B2_OP_SGN,
    B2_OP_SIN, B2_OP_COS,
    B2_OP_ADD = 32, B2_OP_SUB, B2_OP_MUL, B2_OP_DIV, B2_OP_INT_DIV, B2_OP_MOD, B2_OP_EQ,
    B2_OP_NE, B2_OP_LT, B2_OP_LE, B2_OP_GT, B2_OP_GE, B2_OP_POW, B2_OP_MINIMUM, B2_OP_MAXIMUM,
    B2_OP_ONEHOT, /* (index along the reduction-free axis B) == x */
    /* a: register, b: index k of an elementwise flex16 result of the same program.  The value
     * register a has after being stored as result k and read back: mantissa(a) * scale_k.  Lets
     * a kernel go on computing with a tensor it has just written, exactly as a later kernel would
     * see it.  In a probe launch results whose exponent is still to be chosen (bit k of the
     * launch's probe argument, counted from bit 1) pass through unchanged. */
    B2_OP_REQUANT
};

/* reduction codes: float_ew2.py:70-90 */
enum b2_ew_redop {
    B2_RED_SUM = 0, B2_RED_PROD, B2_RED_MAX, B2_RED_MIN, B2_RED_ARGMAX, B2_RED_ARGMIN
};

enum b2_ew_reduce_mode {
    B2_REDUCE_NONE = 0, /* elementwise only */
    B2_REDUCE_C = 1,    /* reduce the innermost axis: results have shape [A, B] */
    B2_REDUCE_B = 2     /* reduce the middle axis: results have shape [A, C] */
};

typedef struct b2_ew_tensor {
    int32_t dtype;       /* enum b2_dtype */
    int32_t flex_slot;   /* row of the flex table / stats array; -1 for fp32 */
    int64_t sa, sb, sc;  /* element strides along A, B, C; 0 broadcasts */
    int64_t plane_bytes; /* B2_FLEX16_PLANES: byte offset of the low plane (multiple of 8) */
} b2_ew_tensor;

/* registers: 0..n_in-1 inputs, n_in..n_in+n_const-1 constants, then one per op in order */
typedef struct b2_ew_op {
    int32_t opcode;
    int32_t a, b;        /* source registers (b ignored by unary ops) */
} b2_ew_op;

typedef struct b2_ew_result {
    int32_t reg;         /* register stored (elementwise) or reduced */
    int32_t redop;       /* enum b2_ew_redop; ignored for elementwise outputs */
    b2_ew_tensor t;      /* strides of the destination; the reduced axis has stride 0 */
} b2_ew_result;

typedef struct b2_ew_program {
    int64_t A, B, C;
    int32_t reduce_mode; /* enum b2_ew_reduce_mode */
    int32_t n_in, n_const, n_ops, n_out, n_red;
    b2_ew_tensor in[B2_EW_MAX_IN];
    b2_ew_op ops[B2_EW_MAX_OPS];
    b2_ew_result out[B2_EW_MAX_OUT]; /* n_out elementwise outputs, then n_red reductions */
} b2_ew_program;

typedef struct b2_flex_scale {
    float scale;      /* 2^-dec : readers multiply mantissas by it */
    float inv_scale;  /* 2^dec  : writers multiply values by it before rounding */
} b2_flex_scale;

typedef struct b2_ew_kernel b2_ew_kernel;

/* Compiles (or fetches from the in-process cache) the kernel for a program.
 * replaces CudaSourceFile.add_kernel + compile (float_ew2.py:1553-1623). */
int b2_ew_compile(const b2_ew_program* prog, b2_ew_kernel** out_kernel);
/* Generates and compiles the program for sm_100a without loading it (needs no GPU): the
 * build-time check of a program.  `vec` asks for the 128-bit variant where the program allows
 * it; the generated source is copied to `source` when given. */
int b2_ew_check(const b2_ew_program* prog, int vec, int probe, char* source, size_t source_cap);
/* The same for the form that shares a launch with others (b2_ew_launch_many). */
int b2_ew_check_joint(const b2_ew_program* prog, int vec, char* source, size_t source_cap);
/* Bytes of caller-provided scratch a launch needs (0 for most programs; reductions of a few
 * very long rows are split across CTAs and combined from scratch). */
int b2_ew_scratch_bytes(const b2_ew_kernel* k, size_t* bytes);
/* Launches.  `out` holds the n_out elementwise destinations followed by the n_red reduction
 * destinations.  `probe` != 0 runs the measuring variant used on a tensor's first write: nothing
 * is stored, and flex_stats[slot] receives the bit pattern of the largest |fp32 value| each
 * flex output would have been given (fmaxf order == integer order for non-negative floats).
 * Bits 1.. of `probe` name the results whose exponent is still to be chosen (bit 1 = result 0):
 * a B2_OP_REQUANT op that refers to such a result passes its value through unchanged.
 * `status` (device int32, may be NULL) is set to 1 if a bounded device-side wait ran out, in
 * which case the results of that launch are undefined.
 * replaces ElementWiseKernel.execute / bind_flex_scales (gputransform.py:277-345,
 * flexgputransform.py:56-64). */
int b2_ew_launch(b2_ew_kernel* k, const void* const* in, void* const* out, const float* consts,
                 const b2_flex_scale* flex_table, int32_t* flex_stats, void* scratch,
                 size_t scratch_bytes, int32_t* status, int probe, void* stream);
/* Compiles and loads what b2_ew_launch with these pointers (probe 0) runs, so that a launch inside a
 * stream capture compiles nothing. */
int b2_ew_prepare(b2_ew_kernel* k, const void* const* in, void* const* out);
/* Programs of one and the same non-empty b2_ew_joint_source (no reductions, one row) in as few launches
 * as their arguments take (one with pointers that are not 16-byte aligned goes by itself). */
typedef struct b2_ew_launch_job {
    b2_ew_kernel* kernel;
    const void* const* in;
    void* const* out;
    const float* consts;
} b2_ew_launch_job;
int b2_ew_joint_source(const b2_ew_kernel* k, const char** source);
int b2_ew_joint_prepare(b2_ew_kernel* first);   /* compiles what b2_ew_launch_many launches */
int b2_ew_launch_many(const b2_ew_launch_job* jobs, int32_t n, const b2_flex_scale* flex_table,
                      int32_t* flex_stats, int32_t* status, int32_t* launches, void* stream);
/* The same launch for callers that cannot allocate (no counterpart in the reference, which
 * always allocates through pycuda).  Meant for hosts that gave the whole device to their own
 * arena at start-up, and for execution loops that must never reach cudaMalloc because it
 * synchronises the device.  Scratch for split reductions comes from an array inside the library
 * (B2_EW_BUILTIN_SCRATCH_BYTES per device, held until the process exits); a launch that needs more
 * fails with B2_ERR_INVALID.  Calls no cudaMalloc/cudaFree and never compiles or loads a kernel:
 * the variant must already exist (b2_ew_compile builds the one for 16-byte-aligned pointers,
 * probe == 0).  The first call on a device resolves the array's address -- make it before any
 * stream capture.  All calls share the array: launches that overlap on the GPU race. */
#define B2_EW_BUILTIN_SCRATCH_BYTES (16 * 1024)
int b2_ew_launch_builtin_scratch(b2_ew_kernel* k, const void* const* in, void* const* out,
                                 const float* consts, const b2_flex_scale* flex_table,
                                 int32_t* flex_stats, int32_t* status, int probe, void* stream);
/* Generated CUDA source of a compiled kernel (for inspection / tests). */
const char* b2_ew_source(const b2_ew_kernel* k);
/* Number of kernel launches one b2_ew_launch issues (1, or 2 for split reductions). */
int b2_ew_launch_count(const b2_ew_kernel* k);
/* Directory searched first for libnvrtc.so.12 (optional; NULL keeps the default search). */
int b2_set_nvrtc_path(const char* path);

/* ------------------------------------------------------------------------------------------
 * Flex16 host<->device conversions, done on the device.
 * Replaces: FlexGPUDeviceTensor.get / __setitem__ (ngraph/transformers/flexgputransform.py:
 * 178-208), which convert on the host with numpy.
 * ------------------------------------------------------------------------------------------ */
/* dst[i] = (int16) trunc(clip(src[i] * table[slot].inv_scale, -32768, 32767));
 * stats[slot] = max(stats[slot], max |dst|). */
int b2_flex_host_quantize(const float* src, int16_t* dst, int64_t n, const b2_flex_scale* table,
                          int32_t slot, int32_t* stats, void* stream);
/* dst[i] = table[slot].scale * (float) src[i] */
int b2_flex_dequantize(const int16_t* src, float* dst, int64_t n, const b2_flex_scale* table,
                       int32_t slot, void* stream);
/* *out = max(*out, bit pattern of max |src[i]|) (NaN counts as 0); used to pick a first exponent
 * for data arriving from the host. */
int b2_absmax_bits_f32(const float* src, int64_t n, int32_t* out, void* stream);
/* End of a call in one launch: host_stats[i] = stats[i], stats[i] = 0 for i < n, and
 * *host_status = *status (both NULL to skip).  host_stats / host_status are pinned host memory
 * that the device can address (cudaHostAlloc memory under unified addressing); the values are
 * there once the stream has been synchronised.  Replaces the per-kernel synchronous statistics
 * read of the reference's flex transformer (manage_after_computation after every kernel,
 * ngraph/transformers/flexgputransform.py:347-371) by one read per call. */
int b2_flex_publish(int32_t* stats, int32_t n, const int32_t* status, int32_t* host_stats,
                    int32_t* host_status, void* stream);

/* ------------------------------------------------------------------------------------------
 * The two ends of a recorded step list, and the host work between calls.
 * b2_call_inputs launches the kernel that takes a call's arguments in: for every input k whose
 * address in the block is not NULL, dst[0..n) <- the fp32 values there (flex_slot >= 0: quantised
 * as b2_flex_host_quantize does, with the block's inv_scale, statistic in stats[flex_slot]).  The
 * block lies in pinned host memory that the device can address and is read when the kernel runs, so
 * one recorded launch serves every call; so may be the arguments.  table_rows > 0 copies that many
 * rows of the block's scale table to `table` first.
 * where, unless NULL: a device word that gets the address at which the values are to be read -- src for
 * an argument marked in_place, which is then not copied (its reader does that: B2_F32_AT,
 * B2_FLEX16_AT), else dst.
 * b2_call_take does the same in front of the step list instead of inside it: the block (any host memory)
 * is read by the call itself, and pageable[k], unless pageable or that is NULL, is host memory that is first copied
 * to the pinned block at arg[k].src, in pieces that the device reads while the next is copied.
 * *launches gets how many kernels that took (none where there is nothing to copy and no word or row to set).
 * holds, unless NULL: a host word with what `where` holds, kept by b2_call_take alone (NULL in it: not known); a
 * device word that holds its address already is not written again.
 * b2_call_outputs is b2_flex_publish with results: dst[k] (pinned host memory) <- bytes[k] bytes of
 * src[k], both 16-byte aligned.
 * b2_call_stage: the address at which the device can read `bytes` bytes of host memory at src:
 * src itself where it is page-locked, else `pinned`, to which they are copied; NULL where that is NULL.
 * b2_call_wait returns when all that was launched on the device's stream has ended.
 * Replace FlexGPUDeviceTensor.__setitem__ / get and the per-kernel statistics read of the reference
 * (ngraph/transformers/flexgputransform.py:178-208, 347-371).
 * ------------------------------------------------------------------------------------------ */
#define B2_CALL_MAX_INPUTS 16
#define B2_CALL_MAX_OUTPUTS 16
typedef struct b2_call_arg { const void* src; float inv_scale; int32_t in_place; } b2_call_arg;
typedef struct b2_call_block {
    const b2_flex_scale* table; int32_t table_rows; int32_t reserved;
    b2_call_arg arg[B2_CALL_MAX_INPUTS];
} b2_call_block;
typedef struct b2_call_input { void* dst; int64_t n; int32_t flex_slot; int32_t reserved; const void** where; const void** holds; } b2_call_input;
typedef struct b2_call_output { const void* src; void* dst; int64_t bytes; } b2_call_output;
int b2_call_inputs(const b2_call_input* inputs, int32_t n, const b2_call_block* block,
                   b2_flex_scale* table, int32_t* stats, void* stream);
int b2_call_take(const b2_call_input* inputs, int32_t n, const b2_call_block* block, const void* const* pageable,
                 b2_flex_scale* table, int32_t* stats, int32_t* launches, int32_t device, void* stream);
int b2_call_outputs(const b2_call_output* outputs, int32_t n, int32_t* stats, int32_t n_stats,
                    const int32_t* status, int32_t* host_stats, int32_t* host_status, void* stream);
int b2_call_wait(int32_t device, void* stream);
int b2_call_stage(const void* src, size_t bytes, void* pinned, const void** visible);
/* Exponent bookkeeping of a whole call over the state arrays of all entries (one row per entry; the
 * rule is ngraph_python_b200/flex.py's, FlexEntry.begin_write / end_write).
 *   begin: every initialised entry ids[k] adopts its pending exponent; row slot_write[k] of the host
 *          table gets it, row slot_read[k] (where it is another one) the exponent of the data stored
 *          so far.  uploaded[row] holds the exponent each row has; *changed tells whether any moved.
 *   end:   records maxima[slots[k]] (maxima[k] without slots) for ids[k], no id twice, and chooses
 *          the next exponents.  undecided[0..*n_undecided) lists the k whose choice lies so close to
 *          a boundary that it needs exactly rounded sums; *settled: every entry has seen the same
 *          maximum for longer than its history window and keeps its exponent.
 *   rows written: row slot_read[k] gets the exponent that ids[k] was written with, for calls that read it
 *          and do not write it.
 * Replace manage_before_computation / manage_after_computation (flexgputransform.py:347-371). */
#define B2_FLEX_HISTORY 16
typedef struct b2_flex_state {
    int64_t *dec, *pending; uint8_t* initialized; int64_t* overflows;
    double* hist; int64_t *hist_len, *hist_pos; double* run_value; int64_t *run_length, *run_choice;
} b2_flex_state;
int b2_flex_rows_written(const b2_flex_state* s, int32_t n, const int64_t* ids, const int64_t* slot_read,
                         int64_t* uploaded, b2_flex_scale* host_table, int32_t* changed);
int b2_flex_begin_call(const b2_flex_state* s, int32_t n, const int64_t* ids,
                       const int64_t* slot_write, const int64_t* slot_read, int64_t* uploaded,
                       b2_flex_scale* host_table, int32_t* changed);
int b2_flex_end_call(const b2_flex_state* s, int32_t n, const int64_t* ids, const int64_t* slots,
                     const int32_t* maxima, int32_t* undecided, int32_t* n_undecided,
                     int32_t* settled);

/* ------------------------------------------------------------------------------------------
 * Dense GEMM on tcgen05 tensor cores: C[M,N] = op(A)[M,K] * op(B)[K,N], C row-major (ldc).
 * Replaces: GEMMKernel and the sgemm / fgemm SASS kernels (ngraph/transformers/gpu/gemm.py:26-263,
 * gpu/kernels/sass/fgemm_common_128x128.sass).  op() is given by element strides, as the
 * reference derives nn/nt/tn from strides (gemm.py:95-110): element (m,k) of op(A) is
 * A[m*a_row_stride + k*a_k_stride], element (k,n) of op(B) is B[k*b_k_stride + n*b_col_stride];
 * one stride of each pair must be 1.  `scratch` (1024-byte aligned, b2_gemm_scratch_bytes) holds
 * the K-major operand planes the kernel streams with TMA.
 * ------------------------------------------------------------------------------------------ */
int b2_gemm_scratch_bytes(int32_t flex, int32_t M, int32_t N, int32_t K, size_t* bytes);
/* Kernels one product launches: 1 where its operands are converted on the way in, else the operand
 * planes and the tile kernel (K strides as below, operands dense along the other side). */
int b2_gemm_launches(int32_t flex, int64_t a_k_stride, int64_t b_k_stride, int32_t M, int32_t N,
                     int32_t K, int32_t* launches);
/* Which kernel that is, and how it cuts the product: tile_n columns to a tile, K in `slices` parts that
 * the CTAs or pairs of a cluster take, `waves` times as many clusters as the machine holds at once. */
enum b2_gemm_kernel { B2_GEMM_DIRECT = 0, B2_GEMM_PAIRS = 1, B2_GEMM_TILES = 2, B2_GEMM_STREAM = 3 };
typedef struct b2_gemm_plan_info { int32_t kernel, tile_n, slices, waves; } b2_gemm_plan_info;
int b2_gemm_plan(int32_t flex, int64_t a_k_stride, int64_t b_k_stride, int32_t M, int32_t N, int32_t K,
                 b2_gemm_plan_info* plan);
/* Both for strides as a product is called with (b2_gemm_plan has B2_GEMM_DIRECT for either kernel that takes one launch;
 * here B2_GEMM_STREAM is the one with A's planes in tensor memory). */
int b2_gemm_route(int32_t flex, int64_t a_row_stride, int64_t a_k_stride, int64_t b_k_stride, int64_t b_col_stride,
                  int32_t M, int32_t N, int32_t K, b2_gemm_plan_info* plan, int32_t* launches);
/* fp32 via 3xTF32 (relative error ~2^-21).  Sums of K in chains of 512 products; up to K = 4096 every
 * kernel adds the chains in order, so that a result does not depend on the number of rows and columns
 * computed beside it. */
int b2_gemm_f32(const float* A, int64_t a_row_stride, int64_t a_k_stride, const float* B,
                int64_t b_k_stride, int64_t b_col_stride, float* C, int64_t ldc, int32_t M,
                int32_t N, int32_t K, void* scratch, size_t scratch_bytes, int32_t* status,
                void* stream);
/* flex16: exact integer products (int8 hi/lo split, int32 accumulation), output rescaled by
 * 2^(decC - decA - decB) with round-to-nearest-even, saturated to int16; stats[slotC] receives
 * max |mantissa| (fgemm epilogue, fgemm_common_128x128.sass:29-97,331-420).  K above 32768 is
 * cut into slices of exact int32 sums that are added in 64-bit.
 * probe != 0: nothing is stored; *probe_out receives max |exact integer sum| (the caller
 * multiplies by 2^-(decA+decB) to get the unsaturated range of the result). */
int b2_gemm_flex16(const int16_t* A, int64_t a_row_stride, int64_t a_k_stride, const int16_t* B,
                   int64_t b_k_stride, int64_t b_col_stride, int16_t* C, int64_t ldc, int32_t M,
                   int32_t N, int32_t K, const b2_flex_scale* table, int32_t slotA, int32_t slotB,
                   int32_t slotC, int32_t* stats, void* scratch, size_t scratch_bytes,
                   uint64_t* probe_out, int32_t* status, int32_t probe, void* stream);

/* ------------------------------------------------------------------------------------------
 * Convolution forward and average pooling on C,D,H,W,N tensors (filters C,T,R,S,K, outputs
 * K,M,P,Q,N), the reference's layouts.
 * Replaces: ConvFpropKernel / FlexConvFpropKernel (ngraph/transformers/gpu/conv.py:24-100,
 * gpu/flex_conv.py:49-200) and PoolFpropKernel avg (gpu/pool.py:27-220).
 * The dims struct has the fields of the reference's conv_params plus the tensor extents
 * (ngraph/op_graph/convolution.py; ngraph/testing/conv_utils.py:ConvParams).
 * ------------------------------------------------------------------------------------------ */
typedef struct b2_conv_dims {
    int32_t C, D, H, W, N;        /* input */
    int32_t K, T, R, S;           /* filter */
    int32_t M, P, Q;              /* output */
    int32_t pad_d, pad_h, pad_w, str_d, str_h, str_w, dil_d, dil_h, dil_w;
} b2_conv_dims;
int b2_conv_fprop_scratch_bytes(int32_t flex, const b2_conv_dims* d, size_t* bytes);
/* fp32 (3xTF32 on the tensor cores). */
int b2_conv_fprop_f32(const float* I, const float* F, float* O, const b2_conv_dims* d,
                      void* scratch, size_t scratch_bytes, int32_t* status, void* stream);
/* Kernels that the scratch-based entry points launch for a pass (0 forward, 1 input gradient, 2 filter
 * gradient); 1: the operands are gathered and converted inside the product, no scratch needed. */
int b2_conv_launches(int32_t flex, const b2_conv_dims* d, int32_t pass, int32_t* launches);
/* With the layer's tail, where b2_conv_launches(0, d, 0) is 1: y = relu?(conv + bias[k] + residual);
 * bias (K values) and residual (the output's layout) may be NULL. */
int b2_conv_fprop_f32_fused(const float* I, const float* F, float* O, const b2_conv_dims* d,
                            const float* bias, const float* residual, int32_t relu, int32_t* status,
                            void* stream);
/* flex16: exact integer sums, rescale/saturate/statistic as b2_gemm_flex16; probe as there. */
int b2_conv_fprop_flex16(const int16_t* I, const int16_t* F, int16_t* O, const b2_conv_dims* d,
                         const b2_flex_scale* table, int32_t slotI, int32_t slotF, int32_t slotO,
                         int32_t* stats, void* scratch, size_t scratch_bytes, uint64_t* probe_out,
                         int32_t* status, int32_t probe, void* stream);
/* The flex16 convolution in parts, for callers that keep operand planes around: the tile kernel
 * reads its streamed tensor (pass 0: the activations I; pass 1, the input gradient of a
 * convolution: the error tensor E) and the filters as byte planes -- high and low
 * bytes of the int16 mantissas, the streamed tensor in its own C,H,W,N (K,P,Q,N) order, every row
 * of N images padded to a multiple of 16 bytes, the low plane after the high plane at the next
 * multiple of 1024 bytes, 1024-byte aligned; act_plane_bytes is the room to reserve for each.  A fused elementwise kernel
 * can emit such planes directly (B2_FLEX16_PLANES) and the filter planes of constant weights can
 * be built once, which leaves ONE launch per convolution.  `supported` is 0 where the plane path
 * does not apply (dilation, very large windows; pass 1: strides whose product exceeds 4, strides
 * with a batch that is no multiple of 128);
 * use b2_conv_fprop_flex16 / b2_conv_bprop_flex16 there.  `d` always describes the FORWARD
 * convolution.  No counterpart in the reference, whose kernels read int16 tensors directly. */
enum b2_conv_pass { B2_CONV_FPROP = 0, B2_CONV_BPROP = 1 };
int b2_conv_planes_info(const b2_conv_dims* d, int32_t pass, int32_t* supported,
                        size_t* act_plane_bytes, size_t* filter_planes_bytes);
int b2_conv_split_activations(const int16_t* X, const b2_conv_dims* d, int32_t pass, void* planes,
                              void* stream);
/* ... of any tensor of c x h x w x n mantissas. */
int b2_conv_split_planes(const int16_t* X, int32_t c, int32_t h, int32_t w, int32_t n, void* planes,
                         void* stream);
int b2_conv_filter_planes(const int16_t* F, const b2_conv_dims* d, int32_t pass, void* planes,
                          void* stream);
/* ... of several convolutions at once, in as few launches as their arguments take. */
typedef struct b2_conv_filter_job {
    const void* filters;
    void* planes;
    b2_conv_dims dims;
    int32_t pass;
} b2_conv_filter_job;
int b2_conv_filter_planes_many(const b2_conv_filter_job* jobs, int32_t n, int32_t* launches, void* stream);
/* fp32 convolutions (pass 0 forward, 1 input gradient) with the filters laid out beforehand, as the stages of
 * the kernel that gathers its operands hold them: bytes of that (0: this one takes none), the launches that
 * make it for several convolutions (job.filters: fp32; planes on 128-byte boundaries), and the pass with the
 * tails of b2_conv_fprop_f32_fused and b2_conv_bprop_f32_fused. */
int b2_conv_filter_tiles_info(const b2_conv_dims* d, int32_t pass, size_t* bytes);
/* How an fp32 pass gathers its operands, with filters as they lie or laid out (tiles): pixels to a row of the
 * product, columns to a tile, slices of K, its k-blocks of 32 columns and those that go into one sum; all zero
 * where it does not. */
typedef struct b2_conv_plan_info { int32_t tile_h, tile_w, tile_n, slices, blocks, in_one_sum; } b2_conv_plan_info;
int b2_conv_f32_plan(const b2_conv_dims* d, int32_t pass, int32_t tiles, b2_conv_plan_info* plan);
/* With filters laid out: which kernel that is (0: none; B2_CONV_GATHER keeps A's planes in tensor memory), the k-blocks
 * in one of its sums of large terms (hi x hi; in_one_sum) and in one of small terms, and what the sums lose to the tensor
 * core's rounding, in units that compare shapes of one layer and pass, beside the other kernel's shape for it (not less). */
enum { B2_CONV_DIRECT = 1, B2_CONV_GATHER = 2 };
typedef struct b2_conv_sums_info { int32_t kernel, large, small, reserved; double loss, other_loss; } b2_conv_sums_info;
int b2_conv_f32_sums(const b2_conv_dims* d, int32_t pass, b2_conv_sums_info* sums);
int b2_conv_filter_tiles(const b2_conv_filter_job* jobs, int32_t n, int32_t* launches, void* stream);
int b2_conv_f32_tiles(int32_t pass, const float* X, const void* filter_tiles, float* O, const b2_conv_dims* d,
                      const float* bias, const float* residual, int32_t relu, const float* mask, int32_t* status,
                      void* stream);
int b2_conv_flex16_planes(int32_t pass, const void* act_planes, const void* filter_planes,
                          int16_t* out, const b2_conv_dims* d, const b2_flex_scale* table,
                          int32_t slotX, int32_t slotF, int32_t slotOut, int32_t* stats,
                          uint64_t* probe_out, int32_t* status, int32_t probe, void* stream);
/* The same with the elementwise tail of a convolution layer folded into the tile kernel's
 * epilogue: y = relu?(conv + bias[k] + residual) evaluated in fp32 from the exact integer sums,
 * quantised ONCE with the output's exponent (slotOut), stored as int16 (write_int16) and / or as
 * the byte planes the next convolution reads (out_planes, low plane plane_bytes further).  bias:
 * int16 per output channel; residual: int16 tensor in the output's K,P,Q,N layout; NULL = absent.
 * probe != 0 stores nothing and leaves the bit pattern of max |y| (fp32) in *probe_out.
 * Replaces the bias / activation arguments the reference's convolution kernels carry
 * (ConvFpropKernel bsum / relu flags, ngraph/transformers/gpu/conv.py:48-100) and the
 * elementwise kernels it launches after them. */
typedef struct b2_conv_epilogue {
    const int16_t* bias;     int32_t slot_bias;
    const int16_t* residual; int32_t slot_residual;
    int32_t relu;
    int32_t write_int16;
    void* out_planes;        size_t plane_bytes;
    const int16_t* mask;     /* int16 tensor in the output's layout: y = mask > 0 ? y : 0 (the
                              * gradient of a ReLU, taken from its activation); NULL = absent */
} b2_conv_epilogue;
int b2_conv_flex16_planes_fused(int32_t pass, const void* act_planes, const void* filter_planes,
                                int16_t* out, const b2_conv_dims* d, const b2_flex_scale* table,
                                int32_t slotX, int32_t slotF, int32_t slotOut,
                                const b2_conv_epilogue* epilogue, int32_t* stats,
                                uint64_t* probe_out, int32_t* status, int32_t probe, void* stream);
/* A run of flex16 convolution layers in one launch, for networks whose images fit into shared memory:
 * layer l reads the chain's input (input = -1) or the result of layer `input`, adds bias and such a
 * tensor (residual) as b2_conv_flex16_planes_fused does, bit for bit, and may be stored as an int16 K,P,Q,N tensor (out; NULL: only layers of the chain read it).
 * Statistics go to slot_out of every layer.  The chain's input is an int16 C,H,W,N tensor (x) or, with
 * x = NULL, its byte planes; pooled (K x N, or NULL) receives the averages of the last layer's images as
 * b2_pool_avg_fprop makes them (up to 512 pixels).  b2_conv_chain_info says whether the layers can make a chain (strides of 1
 * and 2, no dilation, output channels in multiples of 16 up to 112, activations of at least one image
 * in shared memory, no tensor read at both strides) that is faster than launches of their own -- `out` of
 * every layer as it will be -- and gives the bytes of their filter planes, which
 * b2_conv_chain_filters writes (16-byte aligned; again whenever the filters have changed). */
#define B2_CONV_CHAIN_MAX 32
#define B2_CONV_CHAIN_NONE (-2)       /* no residual */
typedef struct b2_conv_chain_layer {
    b2_conv_dims dims;
    int32_t input, residual;
    int32_t relu;
    int32_t slot_in, slot_filters, slot_out, slot_bias, slot_residual;
    const int16_t* filters;
    const int16_t* bias;
    int16_t* out;
} b2_conv_chain_layer;
int b2_conv_chain_info(const b2_conv_chain_layer* layers, int32_t n, int32_t* supported, size_t* filter_bytes);
int b2_conv_chain_filters(const b2_conv_chain_layer* layers, int32_t n, void* filter_planes,
                          int32_t* launches, void* stream);
int b2_conv_chain_flex16(const b2_conv_chain_layer* layers, int32_t n, const int16_t* x, const void* x_planes,
                         size_t plane_bytes, const void* filter_planes, const b2_flex_scale* table,
                         int32_t* stats, int16_t* pooled, int32_t* status, void* stream);
/* The two training contractions of a convolution whose forward pass has the dimensions `d`
 * (d always describes the FORWARD convolution: I is C,D,H,W,N, F is C,T,R,S,K, E is K,M,P,Q,N).
 * Replace ConvBpropKernel / ConvUpdateKernel (ngraph/transformers/gpu/conv.py:121-312) and
 * FlexConvBpropKernel / FlexConvUpdateKernel (gpu/flex_conv.py:203-621); arithmetic as the
 * reference's CPU engine states it (ngraph/transformers/cpu/cpuengine.py:256-271, 395-418).
 *   bprop:  GI[C,D,H,W,N] = sum_{k,r,s} F[c,r,s,k] * E[k,p,q,n],  h = p*str - pad + r*dil
 *   update: U[C,T,R,S,K]  = sum_{p,q,n} I[c,h,w,n] * E[k,p,q,n]   (sums added in a fixed order)
 * flex16 variants: exact integer sums, rescale / saturate / statistic / probe as b2_gemm_flex16
 * with (slot of first operand, slot of second operand, slot of the result). */
int b2_conv_bprop_scratch_bytes(int32_t flex, const b2_conv_dims* d, size_t* bytes);
int b2_conv_bprop_f32(const float* E, const float* F, float* GI, const b2_conv_dims* d,
                      void* scratch, size_t scratch_bytes, int32_t* status, void* stream);
/* With the tail of back-propagation, where b2_conv_launches(0, d, 1) is 1: GI = conv + residual, times
 * (mask > 0); both in the input's layout, either may be NULL. */
int b2_conv_bprop_f32_fused(const float* E, const float* F, float* GI, const b2_conv_dims* d,
                            const float* residual, const float* mask, int32_t* status, void* stream);
int b2_conv_bprop_flex16(const int16_t* E, const int16_t* F, int16_t* GI, const b2_conv_dims* d,
                         const b2_flex_scale* table, int32_t slotE, int32_t slotF, int32_t slotGI,
                         int32_t* stats, void* scratch, size_t scratch_bytes, uint64_t* probe_out,
                         int32_t* status, int32_t probe, void* stream);
int b2_conv_update_scratch_bytes(int32_t flex, const b2_conv_dims* d, size_t* bytes);
int b2_conv_update_f32(const float* I, const float* E, float* U, const b2_conv_dims* d,
                       void* scratch, size_t scratch_bytes, int32_t* status, void* stream);
int b2_conv_update_flex16(const int16_t* I, const int16_t* E, int16_t* U, const b2_conv_dims* d,
                          const b2_flex_scale* table, int32_t slotI, int32_t slotE, int32_t slotU,
                          int32_t* stats, void* scratch, size_t scratch_bytes, uint64_t* probe_out,
                          int32_t* status, int32_t probe, void* stream);
/* The filter gradient from the byte planes of both tensors (laid out as b2_conv_planes_info says for
 * the activations of pass 0 and the error tensor of pass 1), with the sum of the error tensor over
 * (p,q,n) -- the bias gradient, quantised like an elementwise sum -- where bias_grad is not NULL.
 * workspace: workspace_bytes, 1024-byte aligned, zero before the first call and left zero by every
 * call.  probe: probe_out[0] for U, probe_out[1] for the bias (|sum of mantissas|). */
int b2_conv_update_planes_info(const b2_conv_dims* d, int32_t* supported, size_t* workspace_bytes);
int b2_conv_update_flex16_planes(const void* act_planes, const void* err_planes, int16_t* U,
                                 int16_t* bias_grad, const b2_conv_dims* d, const b2_flex_scale* table,
                                 int32_t slotI, int32_t slotE, int32_t slotU, int32_t slotB,
                                 int32_t* stats, void* workspace, uint64_t* probe_out, int32_t* status,
                                 int32_t probe, void* stream);
/* Average pooling over H,W windows.  flex != 0: int16 in and out sharing one exponent
 * (ngraph/transformers/passes/flexpass.py:40-48); *stats_slot = max(*stats_slot, max |out|). */
int b2_pool_avg_fprop(const void* I, void* O, int32_t flex, int32_t C, int32_t H, int32_t W,
                      int32_t N, int32_t P, int32_t Q, int32_t R, int32_t S, int32_t pad_h,
                      int32_t pad_w, int32_t str_h, int32_t str_w, int32_t* stats_slot,
                      void* stream);
/* Max pooling over the part of each window that lies inside the image (np.max of the same
 * slices, ngraph/transformers/cpu/cpuengine.py:297-300); flex as for the average. */
int b2_pool_max_fprop(const void* I, void* O, int32_t flex, int32_t C, int32_t H, int32_t W,
                      int32_t N, int32_t P, int32_t Q, int32_t R, int32_t S, int32_t pad_h,
                      int32_t pad_w, int32_t str_h, int32_t str_w, int32_t* stats_slot,
                      void* stream);
/* Gradient of pooling with respect to its input (BpropPoolOp; arithmetic and summation order of
 * ngraph/transformers/cpu/cpuengine.py:306-336).  avg: every element of a window receives
 * E / (elements of the window inside the image); max: the first maximum of the window (np.argmax
 * order) receives E, found again from the pooled tensor I (unused, may be NULL, for avg).
 * flex16: fp32 arithmetic, one quantisation with slotGI's exponent, statistic or probe (bit
 * pattern of max |fp32 result| into *probe_out) as for the other flex16 entry points. */
int b2_pool_bprop(const void* E, const void* I, void* GI, int32_t flex, int32_t is_max, int32_t C,
                  int32_t H, int32_t W, int32_t N, int32_t P, int32_t Q, int32_t R, int32_t S,
                  int32_t pad_h, int32_t pad_w, int32_t str_h, int32_t str_w,
                  const b2_flex_scale* table, int32_t slotE, int32_t slotGI, int32_t* stats,
                  uint64_t* probe_out, int32_t probe, void* stream);

/* ------------------------------------------------------------------------------------------
 * N-d strided copy / transpose between two tensors of the same extents.
 * Replaces: DimShuffleKernel and the generated copy-transpose kernels (ngraph/transformers/gpu/
 * tensor_ops.py:119-204, gpu/kernels/cuda/copy_transpose.py:78-282), which also implement AssignOp
 * between differently laid-out tensors (gputransform.py:393-395) and non-contiguous host I/O
 * (gputransform.py:873-909).  dst[sum_i idx_i * dst_strides[i]] = src[sum_i idx_i *
 * src_strides[i]] for every index tuple below `shape`; strides are in elements and non-negative
 * (a source stride of 0 broadcasts); the destination must not alias itself.  Where the axis that
 * is contiguous in the source differs from the one contiguous in the destination the copy goes
 * through 32 x 32 shared-memory tiles so that both sides move whole rows.
 * ------------------------------------------------------------------------------------------ */
#define B2_DIMSHUFFLE_MAX_RANK 8
int b2_dimshuffle(const void* src, void* dst, int32_t elem_bytes, int32_t rank,
                  const int64_t* shape, const int64_t* src_strides, const int64_t* dst_strides,
                  void* stream);

/* ------------------------------------------------------------------------------------------
 * Random fill: out[i] ~ U[a, b) (B2_RNG_UNIFORM: a = low, b = high) or N(a, b) (B2_RNG_NORMAL:
 * a = loc, b = scale), n elements, fp32 or flex16 (quantised with slot's exponent; statistic or
 * probe -- bit pattern of max |fp32 value| into *probe_out -- as for b2_pool_bprop).
 * Replaces RngFillKernel / FlexRngFillKernel (ngraph/transformers/gpu/tensor_ops.py:621-661,
 * 713-740).  Counter-based generator (Philox-4x32-10): (seed, offset) determines the tensor.
 * device_counter (may be NULL): a 64-bit device word added to `offset` and advanced by one after
 * a storing launch, so that launches replayed from a CUDA graph still draw fresh numbers.
 * ------------------------------------------------------------------------------------------ */
enum b2_rng_distribution { B2_RNG_UNIFORM = 0, B2_RNG_NORMAL = 1 };
int b2_rng_fill(void* out, int32_t flex, int64_t n, int32_t distribution, float a, float b,
                uint64_t seed, uint64_t offset, uint64_t* device_counter,
                const b2_flex_scale* table, int32_t slot, int32_t* stats, uint64_t* probe_out,
                int32_t probe, void* stream);

/* Lookup table (embedding).  lut_axis 0: lut [V][F], out / delta [n_idx][F], dW [V][F];
 * lut_axis 1: lut [F][V], out / delta [F][n_idx], dW [F][V].  Indices are values of the tensor
 * idx (fp32, or flex16 mantissas with the scale of slot_idx), rounded to the nearest integer.
 *   fprop:  out = lut.take(idx, axis)                (rows outside [0, V) read as zero);
 *           flex16: mantissas are copied, the result carries the table's exponent
 *   update: dW[w] = sum of the rows of delta whose index is w, in increasing position; the row
 *           pad_idx (pass -1 for none) and rows never looked up are zero
 * replaces LUTBpropKernel / fprop_lut / update_lut (ngraph/transformers/gpu/lut.py,
 * ngraph/transformers/cpu/cpuengine.py:421-435).  flex16 update: fp32 sums, one quantisation with
 * slot_dW's exponent, statistic or probe as for b2_pool_bprop. */
int b2_lut_fprop(const void* lut, const void* idx, void* out, int32_t flex, int32_t lut_axis,
                 int32_t V, int32_t F, int32_t n_idx, const b2_flex_scale* table,
                 int32_t slot_idx, void* stream);
int b2_lut_update(const void* delta, const void* idx, void* dW, int32_t flex, int32_t lut_axis,
                  int32_t V, int32_t F, int32_t n_idx, int32_t pad_idx, const b2_flex_scale* table,
                  int32_t slot_delta, int32_t slot_idx, int32_t slot_dW, int32_t* stats,
                  uint64_t* probe_out, int32_t probe, void* stream);

/* ------------------------------------------------------------------------------------------
 * Gradient allreduce over NCCL (NVLink / NVSwitch), one process per GPU.
 * Replaces: CudaAllReduceKernel and its reduction kernel (ngraph/transformers/gpu/tensor_ops.py:
 * 52-116, 416-618), which reduce one gradient tensor at a time with peer-to-peer copies, MPI
 * barriers and host synchronisations.  The caller reduces a whole bucket of fp32 gradients in
 * place, on the stream it names.  NCCL is loaded at run time (the copy already in the process if
 * there is one); without it these entry points return B2_ERR_UNAVAILABLE and the rest of the
 * library is unaffected.
 *   b2_comm_unique_id   one replica makes the 128-byte identifier and hands it to the others
 *                       (any channel: a file, a socket, torch.distributed's store)
 *   b2_comm_init        every replica joins (collective: returns once all have called it)
 *   b2_comm_allreduce_f32  buf[0..count) <- sum over replicas, / nranks when mean != 0; queued on
 *                       `stream`, returns at once
 *   b2_comm_poll_error  B2_OK, or B2_ERR_COMM once NCCL has reported an asynchronous failure (a
 *                       replica that died, a link fault); never blocks
 *   b2_comm_abort       ends the collectives in flight after a failure so that a stream
 *                       synchronisation returns; the handle can then only be destroyed
 * ------------------------------------------------------------------------------------------ */
#define B2_COMM_ID_BYTES 128
typedef struct b2_comm b2_comm;
int b2_set_nccl_path(const char* path);
int b2_comm_version(int32_t* version);
int b2_comm_unique_id(void* id_out);
int b2_comm_init(const void* id, int32_t rank, int32_t nranks, int32_t device, b2_comm** out);
int b2_comm_allreduce_f32(b2_comm* comm, float* buf, int64_t count, int32_t mean, void* stream);
int b2_comm_poll_error(b2_comm* comm);
int b2_comm_abort(b2_comm* comm);
int b2_comm_destroy(b2_comm* comm);

/* ------------------------------------------------------------------------------------------
 * Self-test of the bounded-wait path.  Every device-side wait of the tile kernels gives up after
 * a fixed number of polls, sets the caller's status word to 1 (the launching entry point's
 * `status` argument; the host then reports B2_ERR_TIMEOUT-class failure for that call) and lets
 * the kernel finish normally, tensor memory freed.  This entry point runs that path on purpose: a
 * one-block kernel waits, with the kernels' own wait routine, `poll_limit` polls (1..65536) on a
 * barrier nothing completes, then sets *status = 1, writes the polls it waited to *polls_waited
 * (may be NULL), frees its tensor memory and returns.  Harmless: no fault, no trap, the context
 * stays usable.  No counterpart in the reference (its kernels have no device-side waits).
 * ------------------------------------------------------------------------------------------ */
int b2_selftest_bounded_wait(int32_t poll_limit, int32_t* status, int32_t* polls_waited,
                             void* stream);

#ifdef __cplusplus
}
#endif
#endif /* B200NG_H */
