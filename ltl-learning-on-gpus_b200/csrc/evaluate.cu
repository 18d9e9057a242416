// Evaluation of arbitrary formula strings on traces, on the device: the checker the
// divide-and-conquer driver applies to every sub-formula (the reference's dc.py does it on
// the host with bitarray, code/dc.py:136-187).  The string is parsed the way dc.py's bitVec
// reads it (code/dc.py:136-183): "~(f)", "X(f)", "F(f)", "G(f)", "(f)&(g)", "(f)|(g)",
// "(f)U(g)", single letters; the postfix program then runs on every trace in parallel on words in
// natural order made from the step masks (unary_bits, until_bits; apply_op_kernel checks them against the
// enumerator's operators on row words).
#include <cuda_runtime.h>

#include <cstring>
#include <string>
#include <vector>

#include "ltl_kernels.cuh"
#include "ltlgpu.h"
#include "ops.cuh"
#include "traces.hpp"

namespace ltlg {
namespace {

struct Parser {
    const std::string &s;
    const std::string &alpha;
    std::vector<int> prog;  // (op, arg) pairs; arg of a letter: its bit in the step masks
    int depth = 0, max_depth = 0;

    void emit(int op, int arg, int push) {
        prog.push_back(op);
        prog.push_back(arg);
        depth += push;
        if (depth > max_depth) max_depth = depth;
    }

    // s[b, e) is one formula.
    bool parse(size_t b, size_t e) {
        if (b >= e) return false;
        size_t i = b;
        if (s[b] == '(') {  // skip the first parenthesised group: the operator follows it
            int p = 1;
            for (i = b + 1; i < e && p; ++i) p += s[i] == '(' ? 1 : s[i] == ')' ? -1 : 0;
            if (p) return false;
        }
        if (i >= e) return false;
        const char c = s[i];
        switch (c) {
        case '~':
        case 'X':
        case 'F':
        case 'G': {
            if (i != b || e - b < 4 || s[b + 1] != '(' || s[e - 1] != ')') return false;
            if (!parse(b + 2, e - 1)) return false;
            emit(c == '~' ? OP_NEG : c == 'X' ? OP_X : c == 'F' ? OP_F : OP_G, 0, 0);
            return true;
        }
        case '&':
        case '|':
        case 'U': {
            if (s[b] != '(' || i + 1 >= e || s[i + 1] != '(' || s[e - 1] != ')') return false;
            if (!parse(b + 1, i - 1) || !parse(i + 2, e - 1)) return false;
            emit(c == '&' ? OP_AND : c == '|' ? OP_OR : OP_U, 0, -1);
            return true;
        }
        default: {
            if (e - b != 1) return false;
            if (alpha.find(c) == std::string::npos) return false;
            emit(OP_ATOM, c - 'a', 1);
            return true;
        }
        }
    }
};

// A formula as a postfix program on every trace at once, one thread per trace: a letter's CS comes
// from the trace's step masks (bit k of the word is step k), the subformulas are on a stack, in
// shared memory laid out [depth][thread] up to SMEM_DEPTH and in global memory [depth][n] beyond.
//
// Bound by the copies of the step masks down and the words back: the kernel reads each mask once per
// letter of the formula, out of L1 after the first time.  Making the letters' words of all traces on the
// host took 12 of the 17 ms that 100,000 traces of 10 steps and a formula of 20 operators took.
constexpr int EVAL_THREADS = 128, SMEM_DEPTH = 32;
__global__ void __launch_bounds__(EVAL_THREADS)
    eval_traces_kernel(const int *__restrict__ prog, int len, const u32 *__restrict__ steps, const int *__restrict__ offs, int n,
                       u64 *__restrict__ deep, u64 *__restrict__ cs, unsigned char *__restrict__ holds) {
    extern __shared__ u64 stack_smem[];
    const int t = blockIdx.x * EVAL_THREADS + threadIdx.x;
    if (t >= n) return;
    const int a = offs[t], ln = offs[t + 1] - a;
    const u64 m = (1ull << ln) - 1ull;
    u64 *st = deep ? deep + t : stack_smem + threadIdx.x;
    const size_t row = deep ? (size_t)n : (size_t)EVAL_THREADS;
    int sp = 0;
    for (int k = 0; k < len; ++k) {
        const int op = prog[2 * k], arg = prog[2 * k + 1];
        u64 v = 0;
        if (op == OP_ATOM) {
            for (int q = 0; q < ln; ++q) v |= (u64)((steps[a + q] >> arg) & 1u) << q;
        } else if (op == OP_NEG || op == OP_X || op == OP_F || op == OP_G) {
            v = unary_bits(op, st[(size_t)--sp * row], m);
        } else {
            const u64 y = st[(size_t)(sp - 1) * row], x = st[(size_t)(sp - 2) * row];
            v = op == OP_U ? until_bits(x, y) : op == OP_AND ? (x & y) : (x | y);
            sp -= 2;
        }
        st[(size_t)sp++ * row] = v;
    }
    cs[t] = st[0];
    holds[t] = (unsigned char)(st[0] & 1ull);
}

}  // namespace
}  // namespace ltlg

using namespace ltlg;

extern "C" LTLG_API int ltlg_evaluate(const ltlg_traces *t, const char *formula, uint64_t *cs, uint8_t *holds) {
    if (!formula || !traces_well_formed(t)) return LTLG_BAD_ARGS;
    const int n = t->num_pos + t->num_neg;
    const std::string alpha = t->alphabet ? t->alphabet : "";
    const std::string f = formula;
    Parser P{f, alpha, {}};
    if (!P.parse(0, f.size())) return LTLG_BAD_ARGS;
    if (n == 0) return 0;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return LTLG_NO_DEVICE;
    for (int i = 0; i < n; ++i)
        if (t->offsets[i + 1] - t->offsets[i] > 63) return LTLG_INPUT_LIMITS;
    // one block of device memory: results, step masks, offsets, program, and a deep formula's stack
    const int len = (int)P.prog.size() / 2, base = t->offsets[0];
    const size_t nsteps = (size_t)(t->offsets[n] - base);
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const bool deep = P.max_depth > SMEM_DEPTH;
    const size_t at_cs = 0, at_holds = up((size_t)n * 8), at_steps = at_holds + up((size_t)n), at_offs = at_steps + up(nsteps * 4),
                 at_prog = at_offs + up((size_t)(n + 1) * 4), at_deep = at_prog + up(P.prog.size() * sizeof(int)),
                 bytes = at_deep + (deep ? (size_t)P.max_depth * n * 8 : 0);
    char *d = nullptr;
    // stream-ordered: the driver's pool keeps the block for the next call until something synchronises,
    // where mapping and unmapping it took 600 of the 660 us of a call on 40 traces
    cudaError_t err = cudaMallocAsync(&d, bytes, 0);
    if (err != cudaSuccess) return err == cudaErrorMemoryAllocation ? LTLG_NO_MEMORY : LTLG_CUDA_ERROR;
    // the masks as they are: a trace's steps start at its offset less the first one
    if (nsteps) err = cudaMemcpyAsync(d + at_steps, t->steps + base, nsteps * 4, cudaMemcpyHostToDevice, 0);
    if (err == cudaSuccess) err = cudaMemcpyAsync(d + at_offs, t->offsets, (size_t)(n + 1) * 4, cudaMemcpyHostToDevice, 0);
    if (err == cudaSuccess)
        err = cudaMemcpyAsync(d + at_prog, P.prog.data(), P.prog.size() * sizeof(int), cudaMemcpyHostToDevice, 0);
    if (err == cudaSuccess) {
        const size_t smem = deep ? 0 : (size_t)P.max_depth * EVAL_THREADS * 8;
        eval_traces_kernel<<<(n + EVAL_THREADS - 1) / EVAL_THREADS, EVAL_THREADS, smem>>>(
            (const int *)(d + at_prog), len, (const u32 *)(d + at_steps) - base, (const int *)(d + at_offs), n,
            deep ? (u64 *)(d + at_deep) : nullptr, (u64 *)(d + at_cs), (unsigned char *)(d + at_holds));
        err = cudaGetLastError();
    }
    if (err == cudaSuccess && cs) err = cudaMemcpy(cs, d + at_cs, (size_t)n * 8, cudaMemcpyDeviceToHost);
    if (err == cudaSuccess && holds) err = cudaMemcpy(holds, d + at_holds, (size_t)n, cudaMemcpyDeviceToHost);
    if (err == cudaSuccess && !cs && !holds) err = cudaStreamSynchronize(0);
    cudaFreeAsync(d, 0);
    if (err != cudaSuccess) return LTLG_CUDA_ERROR;
    return 0;
}
