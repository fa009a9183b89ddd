// The attention kernels with waits that give up at once, as a library of its own: no CTA sees its operands arrive.
#define NNCU_FAB_POLLS 1u // the adjoint's: one look, long before its first products can be done
#include <cstdarg>
#include <cstdio>

#include "common.cuh"
#include "gemm_tc.cuh"
namespace tc { // the others': none; what a kernel waits for before it leaves is waited for as usual
__device__ __forceinline__ bool expired_wait(uint32_t bar, uint32_t parity, volatile int *abort_s, int *err_flag, int code, uint32_t tries = 0)
{
    if (tries == DRAIN_TRIES)
        return mbar_wait(bar, parity, abort_s, err_flag, code, tries);
    *abort_s = 1;
    atomicExch(err_flag, code);
    return false;
}
} // namespace tc
#define mbar_wait expired_wait
#include "attention_bwd.cuh"

thread_local char g_nncu_err[512] = "";
unsigned long long g_nncu_launches = 0;
GemmProfiler *g_nncu_prof = nullptr;
thread_local int g_nncu_edges = 0;
int nncu_fail(int code, const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_nncu_err, sizeof(g_nncu_err), fmt, ap);
    va_end(ap);
    return code;
}

extern "C" const char *expired_error() { return g_nncu_err; }
extern "C" int expired_forward(const nncu_attn_shape *s, const void *q, const void *kv, const float *w_r, const void *w_r16, const float *b_r, void *out,
                               float *lse, int *flag)
{
    AttnArgs a = attn_args(s);
    a.q = q; a.kv = kv; a.w_r = w_r; a.w_r16 = w_r16; a.b_r = b_r; a.o = out; a.lse = lse; a.err_flag = flag;
    return fa::forward_dk<64>(a, 0);
}
extern "C" int expired_backward(const nncu_attn_shape *s, int sum, const void *q, const void *kv, const float *w_r, const float *b_r, const void *out,
                                const float *lse, const void *dout, void *dq, void *dkv, float *dwr_part, float *dbr_part, int *flag)
{
    AttnArgs a = attn_args(s);
    a.q = q; a.kv = kv; a.w_r = w_r; a.b_r = b_r; a.out = out; a.lse = const_cast<float *>(lse); a.dout = dout;
    a.dq = dq; a.dkv = dkv; a.dwr_part = dwr_part; a.dbr_part = dbr_part; a.sum = sum; a.err_flag = flag;
    return fab::backward(a, 0);
}
