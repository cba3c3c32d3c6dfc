// Context state behind the opaque Parament_Context_f32/_f64 handles.
//
// Mirrors what src/cuda/parament_context.hpp:26-78 keeps (dimension, norm
// bound, order control, quadrature settings, last error) with a new layout:
// one expansion stack [H0, H_k, commutators] instead of separate H0/H1
// buffers, grow-only work buffers, and a private non-blocking stream.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stddef.h>

#include <vector>

#include "parament.h"

namespace pgb {

bool fault_inject_alloc();
// Whether calls on `stream` go into a graph: nothing is allocated or waited for then.
bool capturing(cudaStream_t stream);

struct DevBuf {
    void *ptr = nullptr;
    size_t cap = 0;
    cudaError_t ensure(size_t bytes);
    void release();
};

struct Ctx {
    bool fp64 = false;
    int device = 0;
    int num_sms = 0;
    cudaStream_t stream = nullptr;
    Parament_ErrorCode last_error = PARAMENT_STATUS_SUCCESS;

    // Hamiltonian (src/cuda/parament_context.hpp:37-56)
    bool has_h = false;
    unsigned dim = 0, K = 0, Ke = 0;
    bool magnus = true;                          // defaults as src/cuda/parament.cpp:72-75
    int quad = PARAMENT_QUADRATURE_SIMPSON;
    double hnorm = 0.0;
    // The stack is held in units of 2^hexp, hexp = ilogb(hnorm): exact, and powers of
    // X and their coefficients stay within the range of FP32 for Hamiltonians in any
    // units (rad/s: with h = 1e-10 s, c_5 = h^5/5! is zero in FP32, and X^3
    // overflows from norms of 1e13 on).
    int hexp = 0;
    DevBuf stack;                                // (1+Ke) d x d, context precision
    double held_norm() const { return ldexp(hnorm, -hexp); }
    double held_step(double h) const { return ldexp(h, hexp); }

    // Chebyshev order control (src/cuda/parament_context.hpp:72-73)
    unsigned mmax = 11;
    bool manual = false;
    int last_M = 0;

    // Precision form (complex64 contexts)
    int precision = PARAMENT_PRECISION_PLAIN;
    DevBuf split_stack;                          // split form's stack (commutators from FP64)
    bool split_ready = false;
    bool split_herm = false;                     // split stack exactly (anti-)Hermitian per slot

    // Fixed-point form (fx.cu): the stack as integers, that of the split form,
    // and the workspace of a propagation.
    void *fx_stack = nullptr;  // behind the matrices of `stack`, in its allocation
    DevBuf fx_split, fx_ws;
    bool fx_ready = false, fx_split_ready = false;
    bool fx_ran = false;  // by the last equiprop

    // Instrumentation: CUDA events around the dominant kernel of the last call
    // and the number of kernels it launched.
    bool timing = false;
    cudaEvent_t ev_start = nullptr, ev_stop = nullptr;
    int launches = 0;

    // Work buffers (grow-only, like src/cuda/parament.cpp:418-474)
    DevBuf carr, out, chunks, work, X, B1, B2, aux, grad, wts, xplanes;
    DevBuf arrived;  // arrivals at the pairs of the small groups' tree (step_group.cu)
    unsigned group_turn = 0;  // of the last launch of small groups

    // Pinned memory that kernels reach directly: samples and result of small
    // host-buffer calls.
    void *h_stage = nullptr, *d_stage = nullptr;

    // Bounded-wait faults of this context's tensor-core kernels.  The kernels
    // add to a device counter (d_fault, zero at creation, never reset); after
    // each call that may run such a kernel the counter is copied into pinned
    // host memory (h_fault) on the call's stream and ev_fault is recorded
    // there.  A count above faults_seen is reported as
    // PARAMENT_STATUS_KERNEL_TIMEOUT by the call itself (host-buffer entry
    // points), by Parament_synchronize, or by the next device-buffer call on
    // the context.  Calls that go into a graph leave copy and events out; once
    // there was one (`captured`), Parament_synchronize copies the counter itself.
    int *d_fault = nullptr;
    int *h_fault = nullptr;
    int faults_seen = 0;
    cudaEvent_t ev_fault = nullptr;  // h_fault refreshed
    bool fault_recorded = false;
    cudaEvent_t ev_done = nullptr;   // end of the last call's work
    bool done_recorded = false;
    bool captured = false;

    size_t esize() const { return fp64 ? 16 : 8; }
    size_t device_bytes() const {
        return stack.cap + split_stack.cap + carr.cap + out.cap + chunks.cap + work.cap + X.cap + B1.cap + B2.cap +
               aux.cap + grad.cap + wts.cap + xplanes.cap + fx_split.cap + fx_ws.cap +
               arrived.cap;
    }
    void release_all() {
        stack.release();
        split_stack.release();
        carr.release();
        out.release();
        chunks.release();
        work.release();
        X.release();
        B1.release();
        B2.release();
        aux.release();
        grad.release();
        wts.release();
        xplanes.release();
        fx_split.release();
        fx_ws.release();
        arrived.release();
    }
};

// Marks the end of a call's work on `stream`; with tensor_kernels set, the
// fault counter is copied to the host there.  new_faults() reports whether a
// kernel gave up since the last report (wait: block until the last call's
// work is done; otherwise only look if it already is).
void note_call_end(Ctx *c, cudaStream_t stream, bool tensor_kernels);
bool new_faults(Ctx *c, bool wait);

double onenorm_host(const void *m, unsigned d, bool fp64);
int select_cycles(bool fp64, double hnorm, double dt);
void bessel_coeffs(int M, double x, double *J);
long long num_steps(int quad, bool magnus, unsigned pts);

// Split-precision form (complex64 contexts): order choice and propagation;
// run_split_large serves d > 64 (split_large.cu).
struct SplitArgs;
int split_order(double hnorm, double h, long long P);
Parament_ErrorCode run_split(Ctx *c, const void *d_carr, unsigned pts, unsigned amps, double h, int M, long long P,
                             void *d_out, cudaStream_t stream);
Parament_ErrorCode run_split_large(Ctx *c, const SplitArgs &a, double h, void *d_out, cudaStream_t stream);

// c0 = m_0 - 1 and mu_n = m_n / Hnorm^n of the regrouped polynomial (split.cu); here and
// below hnorm is the norm of the stack as it is held.
void power_coefficients(int M, double x, double hnorm, double *c0, std::vector<double> &mu);
// The same polynomial with the FP32 coefficients of the complex64 contexts;
// returns J_0, which c_0 = p(0) - J_0 leaves out.  Each c_n n >= 1 is a sum over orders
// and so no FP32 number itself.  Rounded to one, c_1 and c_2 would turn every step by the
// same angle (0.3 x 2^-24 of x on average, adding up along the steps, where the recurrence
// has the roundings of J_k only); kernels add the rests c - (float)c times X and X^2.
double plain_coefficients(int M, double x, double hnorm, std::vector<double> &c);
inline float low_part(double c) { return (float)(c - (double)(float)c); }

// Exact sliced products (fx.cu): fx_prepare / fx_prepare_split convert the stack
// (set_hamiltonian; the split form's first call), fx_ensure allocates the
// workspace of P steps (not into a capture: what is there has to do), run_fx propagates (x = Hnorm h).
struct WeightSpecHost;
enum class FxForm { kFp64, kPlain32, kSplit32 };
size_t fx_stack_bytes(const Ctx *c, unsigned dim, unsigned Ke);  // 0: none is kept
void fx_prepare(Ctx *c);
void fx_prepare_split(Ctx *c);
bool fx_applies(const Ctx *c, FxForm form, int M, double x, long long P);
bool fx_ensure(Ctx *c, long long P, cudaStream_t stream);
cudaError_t run_fx(Ctx *c, FxForm form, const void *d_carr, const WeightSpecHost &wh, double x, int M, long long P,
                   void *d_out, cudaStream_t stream);

// Adjoint: d/du_k[i] Re Tr(W^H U) for real samples, d <= adj_max_dim.
int adj_max_dim(bool fp64);
Parament_ErrorCode run_vjp(Ctx *c, const void *d_carr, double dt, unsigned pts, unsigned amps, const void *d_W,
                           void *d_grad, cudaStream_t stream);

}  // namespace pgb
