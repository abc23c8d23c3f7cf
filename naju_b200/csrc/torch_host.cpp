// Host path of the scan as a CPython extension over libtorch: what happens between a Python call
// (naju_scan, naju_scan_step) and the C ABI of libnaju_b200.so.
//
// The small calls are bound by this path, not by the GPU: a decode step is a 2 us kernel, and the
// argument checks, the descriptor and the ctypes call of a Python host layer took 48 us around it
// (measured, 24 layers, one sequence: 1150 us); a forward + backward of the smallest training call took
// 265 us of host time for 106 us of kernels.  So the checks, the workspaces and the autograd node are
// C++ here, scan() and step() are METH_FASTCALL functions, and the GIL is released around the launches.
//
// Semantics are those of the reference's scan entry (naju/scan.py:75-76) and of its autograd wrapper
// (naju/cuda/__init__.py:38-63): any of the supported types, strided views as they come, gradients in
// each input's type.
#include <torch/extension.h>

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/core/AutogradState.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cctype>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "naju_b200.h"

namespace {

using at::Tensor;
using torch::autograd::variable_list;

// ------------------------------------------------------------------------------ switches
// Read per call, as the Python layer did (os.environ assignments reach getenv).
bool env_on(const char* name) {
  const char* v = std::getenv(name);
  return v != nullptr && std::strcmp(v, "1") == 0;
}

int form_flags() {
  const char* v = std::getenv("NAJU_B200_FORM");
  if (v == nullptr) return 0;
  std::string f(v);
  for (auto& c : f) c = static_cast<char>(std::tolower(static_cast<unsigned char>(c)));
  if (f == "auto") return 0;
  if (f == "chunked") return NAJU_FLAG_CHUNKED_ONLY;
  TORCH_CHECK_VALUE(f == "recurrent", "NAJU_B200_FORM must be 'auto', 'chunked' or 'recurrent', got '", f, "'");
  return NAJU_FLAG_RECURRENT_ONLY;
}

int call_flags() { return form_flags() | (env_on("NAJU_B200_INJECT_TIMEOUT") ? NAJU_FLAG_INJECT_TIMEOUT : 0); }

int dtype_code(at::ScalarType t) {
  return t == at::kFloat ? NAJU_F32 : t == at::kBFloat16 ? NAJU_BF16 : t == at::kHalf ? NAJU_F16 : -1;
}

void check(int rc, const char* what) {
  TORCH_CHECK(rc == 0, what, " failed: ", naju_b200_strerror(rc), " (code ", rc, ")");
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// ------------------------------------------------------------------------------ arguments
// A [B,T,D] view of [B,D,T] memory (time stride 1, channels T or more apart) that the kernels can take
// as it is: what the mixer's depthwise convolution leaves behind (naju/mixer.py:115).  TMA wants the
// channel and batch strides to be multiples of 16 bytes.
bool time_contig(const Tensor& u) {
  if (u.dim() != 3 || u.size(1) < 2 || u.size(2) < 2) return false;
  const int64_t sb = u.stride(0), st = u.stride(1), sd = u.stride(2), es = u.element_size();
  return st == 1 && sd >= u.size(1) && sb >= 0 && reinterpret_cast<uintptr_t>(u.data_ptr()) % 16 == 0 &&
         (sd * es) % 16 == 0 && (sb * es) % 16 == 0 && (u.size(0) == 1 || sb >= sd * u.size(2));
}

// Tensors whose last stride is 1 and whose outer strides are non-negative pass through.
Tensor inner_contig(const Tensor& t) {
  bool ok = t.stride(-1) == 1 && reinterpret_cast<uintptr_t>(t.data_ptr()) % t.element_size() == 0;
  for (int64_t i = 0; ok && i < t.dim(); ++i) ok = t.stride(i) >= 0;
  if (ok && (t.dim() < 3 || t.stride(-2) >= t.size(-1))) return t;
  return t.contiguous();
}

Tensor as_type(const Tensor& t, at::ScalarType to) { return t.scalar_type() == to ? t : t.to(to); }

struct Args {
  Tensor u, fl, il, Bm, Cm, D;
};

// The types the kernels run in: logits in u's type or fp32 (autocast hands fp32 logits next to bf16
// activations), B and C in their common type or fp32, D_skip fp32.
at::ScalarType gate_type(const Tensor& u, const Tensor& fl, const Tensor& il) {
  return (fl.scalar_type() == u.scalar_type() && il.scalar_type() == u.scalar_type()) ? u.scalar_type() : at::kFloat;
}
at::ScalarType bc_type(const Tensor& Bm, const Tensor& Cm) {
  return (Bm.scalar_type() == Cm.scalar_type() && dtype_code(Bm.scalar_type()) >= 0) ? Bm.scalar_type() : at::kFloat;
}

Args prepare(const Tensor& u, const Tensor& fl, const Tensor& il, const Tensor& Bm, const Tensor& Cm, const Tensor& D) {
  TORCH_CHECK(u.is_cuda(), "naju_b200 scan needs CUDA tensors (there is no CPU fallback)");
  TORCH_CHECK_VALUE(u.dim() == 3 && fl.sizes() == u.sizes() && il.sizes() == u.sizes(),
                    "u, f_logit, i_logit must all be [B, T, D]");
  TORCH_CHECK_VALUE(Bm.dim() == 3 && Bm.sizes() == Cm.sizes() && Bm.size(0) == u.size(0) && Bm.size(1) == u.size(1),
                    "B and C must both be [B, T, N] matching u's batch and time");
  TORCH_CHECK_VALUE(D.dim() == 1 && D.size(0) == u.size(2), "D_skip must be [D]");
  TORCH_CHECK(Bm.size(2) >= 1 && Bm.size(2) <= 128, "d_state must be in 1..128");
  TORCH_CHECK(dtype_code(u.scalar_type()) >= 0, "unsupported dtype ", u.scalar_type());
  const auto gdt = gate_type(u, fl, il), bdt = bc_type(Bm, Cm);
  return {time_contig(u) ? u : inner_contig(u), inner_contig(as_type(fl, gdt)), inner_contig(as_type(il, gdt)),
          inner_contig(as_type(Bm, bdt)), inner_contig(as_type(Cm, bdt)), as_type(D, at::kFloat).contiguous()};
}

naju_scan_desc describe(const Args& a, int flags) {
  naju_scan_desc d{};
  d.B = static_cast<int32_t>(a.u.size(0));
  d.T = static_cast<int32_t>(a.u.size(1));
  d.D = static_cast<int32_t>(a.u.size(2));
  d.N = static_cast<int32_t>(a.Bm.size(2));
  d.act_dtype = dtype_code(a.u.scalar_type());
  d.gate_dtype = dtype_code(a.fl.scalar_type());
  d.bc_dtype = dtype_code(a.Bm.scalar_type());
  d.flags = flags;
  d.u_sb = a.u.stride(0); d.u_st = a.u.stride(1);
  d.u_sd = (a.u.stride(2) != 1 && a.u.stride(1) == 1) ? a.u.stride(2) : 1;
  d.fl_sb = a.fl.stride(0); d.fl_st = a.fl.stride(1);
  d.il_sb = a.il.stride(0); d.il_st = a.il.stride(1);
  d.bm_sb = a.Bm.stride(0); d.bm_st = a.Bm.stride(1);
  d.cm_sb = a.Cm.stride(0); d.cm_st = a.Cm.stride(1);
  if (d.T <= 1) {  // a size-1 dimension may carry any stride; give the kernel a legal one
    const int64_t D = d.D, N = d.N;
    d.u_st = std::max(d.u_st, D); d.fl_st = std::max(d.fl_st, D); d.il_st = std::max(d.il_st, D);
    d.bm_st = std::max(d.bm_st, N); d.cm_st = std::max(d.cm_st, N);
  }
  return d;
}

Tensor state_arg(const Tensor& h, int64_t B, int64_t D, int64_t N, const char* name) {
  if (!h.defined()) return h;
  TORCH_CHECK_VALUE(h.dim() == 3 && h.size(0) == B && h.size(1) == D && h.size(2) == N, name, " must be [B, D, N]");
  return as_type(h, at::kFloat).contiguous();
}

// ------------------------------------------------------------------------------ fewer than 16 states
// The tcgen05 kernels are built for 16 states; the recurrence (naju/scan.py:87-91) is diagonal in the
// state index and y only sums over it, so zero columns added to B and C (and to h0 / dhT) change
// nothing: N < 16 is padded up to 16 and the state-shaped results are sliced back.
constexpr int64_t kGroup = 16;
constexpr int64_t kPadMinWork = 1 << 20;  // B*T*D below which the recurrent kernels are as fast

bool pad_to_group(const Tensor& u, const Tensor& Bm, int flags) {
  if (Bm.size(-1) >= kGroup || (flags & NAJU_FLAG_RECURRENT_ONLY)) return false;
  if ((u.scalar_type() != at::kBFloat16 && u.scalar_type() != at::kHalf) || Bm.scalar_type() != at::kBFloat16) return false;
  return u.numel() >= kPadMinWork && u.size(1) >= 128;
}

Tensor pad_states(const Tensor& t) {
  if (!t.defined() || t.size(-1) == kGroup) return t;
  return at::constant_pad_nd(t, {0, kGroup - t.size(-1)});
}

// ------------------------------------------------------------------------------ workspaces
// Caller-owned workspaces of the library (torch's caching allocator returns 512-byte aligned blocks).
// With NAJU_B200_GUARD=1 every workspace sits between two canary bands that the Python layer's
// check_workspace_guards() verifies (a debug aid; off by default).
constexpr int64_t kGuard = 4096;
constexpr int kGuardByte = 0xA5;
std::mutex g_guard_mutex;
std::vector<std::pair<Tensor, int64_t>> g_guarded;  // (whole buffer, payload size) since the last check

Tensor workspace(size_t nbytes, at::Device dev) {
  const int64_t n = std::max<int64_t>(static_cast<int64_t>(nbytes), 256);
  const auto opt = at::TensorOptions().dtype(at::kByte).device(dev);
  if (!env_on("NAJU_B200_GUARD")) return at::empty({n}, opt);
  Tensor whole = at::full({kGuard + (n + 255) / 256 * 256 + kGuard}, kGuardByte, opt);
  {
    std::lock_guard<std::mutex> lock(g_guard_mutex);
    g_guarded.emplace_back(whole, n);
  }
  return whole.narrow(0, kGuard, n);
}

// Kernel family (NAJU_FORM_*) of the last forward / backward made with NAJU_B200_CHECK_STATUS=1
// (reading it synchronises the stream); -1 = none yet.
std::atomic<int> g_form_fwd{-1}, g_form_bwd{-1};

void check_status(const Tensor& scratch, void* stream, std::atomic<int>& form, const char* what) {
  const int st = naju_b200_read_status(scratch.data_ptr(), stream);
  form.store(naju_b200_read_form(scratch.data_ptr(), stream));
  TORCH_CHECK(st == 0, what, " device status ", st, " (bounded wait ran out)");
}

const void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
void* mptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
const float* fptr(const Tensor& t) { return static_cast<const float*>(ptr(t)); }
float* mfptr(const Tensor& t) { return static_cast<float*>(mptr(t)); }

// ------------------------------------------------------------------------------ forward / backward
struct FwdOut {
  Tensor y, hT, pT, ckpt;
  naju_scan_desc desc;   // of the call as it was made (states padded where the rule says so)
};

FwdOut naju_forward(const Args& in, const Tensor& h0_in, bool want_final, bool want_decay, int flags) {
  Args a = in;
  Tensor h0 = h0_in;
  const int64_t B = a.u.size(0), T = a.u.size(1), D = a.u.size(2), N = a.Bm.size(2);
  if (pad_to_group(a.u, a.Bm, flags)) {
    a.Bm = pad_states(a.Bm); a.Cm = pad_states(a.Cm); h0 = pad_states(h0);
  }
  const int64_t Np = a.Bm.size(2);
  const naju_scan_desc d = describe(a, flags);
  c10::cuda::CUDAGuard guard(a.u.device());
  const auto f32 = a.u.options().dtype(at::kFloat);
  FwdOut o;
  o.desc = d;
  o.y = at::empty({B, T, D}, a.u.options());
  if (want_final) o.hT = at::empty({B, D, Np}, f32);
  if (want_decay) o.pT = at::empty({B, D}, f32);
  o.ckpt = workspace(naju_b200_ckpt_bytes(&d), a.u.device());
  Tensor scratch = workspace(naju_b200_fwd_scratch_bytes(&d), a.u.device());
  void* st = stream_of(a.u);
  check(naju_b200_fwd(&d, ptr(a.u), ptr(a.fl), ptr(a.il), ptr(a.Bm), ptr(a.Cm), fptr(a.D), fptr(h0), mptr(o.y), mfptr(o.hT),
                      mfptr(o.pT), mptr(o.ckpt), mptr(scratch), st),
        "naju_b200_fwd");
  if (env_on("NAJU_B200_CHECK_STATUS") && a.u.numel() > 0) check_status(scratch, st, g_form_fwd, "naju_b200_fwd");
  if (want_final && Np != N) o.hT = o.hT.narrow(-1, 0, N).contiguous();
  return o;
}

struct BwdOut {
  Tensor du, dfl, dil, dB, dC, dD, dh0;
};

BwdOut naju_backward(const Args& in, const Tensor& h0_in, const Tensor& dy_in, const Tensor& dhT_in, const Tensor& ckpt,
                bool want_dh0, int flags) {
  Args a = in;
  Tensor h0 = h0_in, dhT = dhT_in;
  const int64_t B = a.u.size(0), T = a.u.size(1), D = a.u.size(2), N = a.Bm.size(2);
  if (pad_to_group(a.u, a.Bm, flags)) {
    a.Bm = pad_states(a.Bm); a.Cm = pad_states(a.Cm); h0 = pad_states(h0); dhT = pad_states(dhT);
  }
  const int64_t Np = a.Bm.size(2);
  const naju_scan_desc d = describe(a, flags);
  // (the padding of fewer than 16 states, and with it the checkpoints' layout, depends on NAJU_B200_FORM)
  const int64_t want = std::max<int64_t>(static_cast<int64_t>(naju_b200_ckpt_bytes(&d)), 256);
  TORCH_CHECK(ckpt.numel() == want, "checkpoint buffer of ", ckpt.numel(), " bytes where this call's layout has ", want,
              ": NAJU_B200_FORM has changed since the forward, or the buffer belongs to another call");
  c10::cuda::CUDAGuard guard(a.u.device());
  const auto f32 = a.u.options().dtype(at::kFloat);
  BwdOut o;
  // (a time-contiguous u gets its gradient in the same layout: naju_b200.h, naju_scan_desc)
  o.du = d.u_sd > 1 ? at::empty_strided(a.u.sizes(), a.u.strides(), a.u.options()) : at::empty({B, T, D}, a.u.options());
  o.dfl = at::empty({B, T, D}, a.fl.options());
  o.dil = at::empty({B, T, D}, a.fl.options());
  o.dB = at::empty({B, T, Np}, a.Bm.options());
  o.dC = at::empty({B, T, Np}, a.Bm.options());
  o.dD = at::empty({D}, f32);
  if (want_dh0) o.dh0 = at::empty({B, D, Np}, f32);
  Tensor scratch = workspace(naju_b200_bwd_scratch_bytes(&d), a.u.device());
  const Tensor dy = as_type(dy_in, a.u.scalar_type()).contiguous();
  void* st = stream_of(a.u);
  check(naju_b200_bwd(&d, ptr(a.u), ptr(a.fl), ptr(a.il), ptr(a.Bm), ptr(a.Cm), fptr(a.D), fptr(h0), ptr(dy), fptr(dhT),
                      ptr(ckpt), mptr(o.du), mptr(o.dfl), mptr(o.dil), mptr(o.dB), mptr(o.dC), mfptr(o.dD), mfptr(o.dh0),
                      mptr(scratch), st),
        "naju_b200_bwd");
  if (env_on("NAJU_B200_CHECK_STATUS") && a.u.numel() > 0) check_status(scratch, st, g_form_bwd, "naju_b200_bwd");
  if (Np != N) {
    o.dB = o.dB.narrow(-1, 0, N).contiguous();
    o.dC = o.dC.narrow(-1, 0, N).contiguous();
    if (o.dh0.defined()) o.dh0 = o.dh0.narrow(-1, 0, N).contiguous();
  }
  return o;
}

// ------------------------------------------------------------------------------ autograd
// Counterpart of _NajuCudaFn (naju/cuda/__init__.py:38-63) as a native autograd function: the prepared inputs and
// the forward's checkpoints are saved, the gradients come back in each input's own type.
static_assert(static_cast<int>(at::ScalarType::NumOptions) <= 64, "a type fits six bits");

struct NajuScan : public torch::autograd::Function<NajuScan> {
  static variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& u, const Tensor& fl, const Tensor& il,
                               const Tensor& Bm, const Tensor& Cm, const Tensor& D, const std::optional<Tensor>& h0_in,
                               bool want_final) {
    const Tensor h0 = h0_in.has_value() ? *h0_in : Tensor();
    const Tensor* in[7] = {&u, &fl, &il, &Bm, &Cm, &D, &h0};
    const int flags = call_flags();
    Args a;
    Tensor ph0;
    const FwdOut o = run(u, fl, il, Bm, Cm, D, h0, want_final, flags, a, ph0);
    ctx->save_for_backward({a.u, a.fl, a.il, a.Bm, a.Cm, a.D, ph0, o.ckpt});
    ctx->set_materialize_grads(false);
    // One number for what is not a tensor: the forward's flags (they decide how the checkpoints are laid out), whether the final state was
    // asked for, the inputs' types (six bits each).
    int64_t meta = flags | (want_final ? 1 << 8 : 0);
    for (int i = 0; i < 7; ++i)
      if (in[i]->defined()) meta |= static_cast<int64_t>(in[i]->scalar_type()) << (16 + 6 * i);
    ctx->saved_data["meta"] = meta;
    return want_final ? variable_list{o.y, o.hT} : variable_list{o.y};
  }

  static variable_list backward(torch::autograd::AutogradContext* ctx, const variable_list& grads) {
    const variable_list s = ctx->get_saved_variables();
    const int64_t meta = ctx->saved_data["meta"].toInt();
    const Args a{s[0], s[1], s[2], s[3], s[4], s[5]};
    const Tensor& h = s[6];
    const Tensor dy = grads[0].defined() ? grads[0] : at::zeros_like(a.u);
    Tensor dhT;
    if ((meta & (1 << 8)) != 0 && grads.size() > 1 && grads[1].defined())
      dhT = state_arg(grads[1], a.u.size(0), a.u.size(2), a.Bm.size(2), "dhT");
    const bool want_dh0 = h.defined() && ctx->needs_input_grad(6);
    BwdOut o;
    {
      at::AutoDispatchBelowADInplaceOrView below;
      o = naju_backward(a, h, dy, dhT, s[7], want_dh0, static_cast<int>(meta & 0xFF));
    }
    variable_list out(8);
    const Tensor* g[7] = {&o.du, &o.dfl, &o.dil, &o.dB, &o.dC, &o.dD, &o.dh0};
    for (size_t i = 0; i < 7; ++i)
      if (g[i]->defined() && ctx->needs_input_grad(i)) out[i] = as_type(*g[i], static_cast<at::ScalarType>(meta >> (16 + 6 * i) & 63));
    return out;
  }

  static FwdOut run(const Tensor& u, const Tensor& fl, const Tensor& il, const Tensor& Bm, const Tensor& Cm, const Tensor& D,
                    const Tensor& h0, bool want_final, int flags, Args& a, Tensor& ph0) {
    // Nothing in here is recorded.  (A tensor that needs no conversion is the caller's own, with its version counter, so that a
    // change in place before the backward is noticed.  A detach() in here would not share the counter.)
    at::AutoDispatchBelowADInplaceOrView below;
    a = prepare(u, fl, il, Bm, Cm, D);
    ph0 = state_arg(h0, a.u.size(0), a.u.size(2), a.Bm.size(2), "h0");
    return naju_forward(a, ph0, want_final, false, flags);
  }
};

std::tuple<Tensor, Tensor> scan(const Tensor& u, const Tensor& fl, const Tensor& il, const Tensor& Bm, const Tensor& Cm,
                                const Tensor& D, const Tensor& h0, bool want_final) {
  const Tensor* in[7] = {&u, &fl, &il, &Bm, &Cm, &D, &h0};
  if (c10::AutogradState::get_tls_state().get_fw_grad_mode())
    for (const Tensor* t : in)
      TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(/*level=*/0).defined(),
                                  "the scan has no forward-mode derivative (jvp): use reverse mode");
  bool grad = false;
  if (at::GradMode::is_enabled())
    for (const Tensor* t : in) grad = grad || (t->defined() && t->requires_grad());
  if (grad) {
    const variable_list o = NajuScan::apply(u, fl, il, Bm, Cm, D, h0.defined() ? std::optional<Tensor>(h0) : std::nullopt, want_final);
    return {o[0], want_final ? o[1] : Tensor()};
  }
  Args a;
  Tensor ph0;
  const FwdOut o = NajuScan::run(u, fl, il, Bm, Cm, D, h0, want_final, call_flags(), a, ph0);
  return {o.y, o.hT};
}

// ------------------------------------------------------------------------------ decode step
// A row operand of the step as the kernel takes it: inner stride 1, rows at least a row apart.  Rows that overlap or repeat (an operand
// broadcast over the batch) are copied; with one row only the stride means nothing.
Tensor step_rows(const Tensor& t) {
  const auto size = t.sizes(), stride = t.strides();
  const bool ok = stride[1] == 1 && (size[0] == 1 || stride[0] >= size[1]) &&
                  reinterpret_cast<uintptr_t>(t.data_ptr()) % t.element_size() == 0;
  return ok ? t : t.contiguous();
}

// state [B,D,N] fp32 is updated in place; u, f_logit, i_logit [B,D]; B, C [B,N].
Tensor step(const Tensor& state, const Tensor& u, const Tensor& fl, const Tensor& il, const Tensor& Bm, const Tensor& Cm,
            const Tensor& D) {
  TORCH_CHECK(state.is_cuda(), "naju_b200 step needs CUDA tensors (there is no CPU fallback)");
  TORCH_CHECK(state.scalar_type() == at::kFloat && state.is_contiguous() && state.dim() == 3,
              "state must be a contiguous fp32 [B, D, N] tensor");
  TORCH_CHECK(u.is_cuda(), "naju_b200 scan needs CUDA tensors (there is no CPU fallback)");
  const int64_t B = state.size(0), Dc = state.size(1), N = state.size(2);
  TORCH_CHECK_VALUE(u.dim() == 2 && u.size(0) == B && u.size(1) == Dc && fl.sizes() == u.sizes() && il.sizes() == u.sizes(),
                    "u_t, f_logit_t, i_logit_t must all be [B, D]");
  TORCH_CHECK_VALUE(Bm.dim() == 2 && Bm.sizes() == Cm.sizes() && Bm.size(0) == B && Bm.size(1) == N,
                    "B_t and C_t must both be [B, N] matching the state");
  TORCH_CHECK_VALUE(D.dim() == 1 && D.size(0) == Dc, "D_skip must be [D]");
  TORCH_CHECK(N >= 1 && N <= 128, "d_state must be in 1..128");
  TORCH_CHECK(dtype_code(u.scalar_type()) >= 0, "unsupported dtype ", u.scalar_type());
  at::AutoDispatchBelowADInplaceOrView below;
  c10::cuda::CUDAGuard guard(state.device());
  const auto gdt = gate_type(u, fl, il), bdt = bc_type(Bm, Cm);
  const Tensor pu = step_rows(u), pf = step_rows(as_type(fl, gdt)), pi = step_rows(as_type(il, gdt)), pB = step_rows(as_type(Bm, bdt)),
               pC = step_rows(as_type(Cm, bdt)),
               pD = as_type(D, at::kFloat).contiguous();
  naju_scan_desc d{};
  d.B = static_cast<int32_t>(B); d.T = 1; d.D = static_cast<int32_t>(Dc); d.N = static_cast<int32_t>(N);
  d.act_dtype = dtype_code(pu.scalar_type());
  d.gate_dtype = dtype_code(gdt);
  d.bc_dtype = dtype_code(bdt);
  d.u_sb = d.fl_sb = d.il_sb = Dc;   // (one row: its stride means nothing)
  d.bm_sb = d.cm_sb = N;
  if (B > 1) {
    d.u_sb = pu.stride(0); d.fl_sb = pf.stride(0); d.il_sb = pi.stride(0);
    d.bm_sb = pB.stride(0); d.cm_sb = pC.stride(0);
  }
  Tensor y = at::empty({B, Dc}, pu.options());
  check(naju_b200_step(&d, static_cast<float*>(state.data_ptr()), ptr(pu), ptr(pf), ptr(pi), ptr(pB), ptr(pC), fptr(pD),
                       mptr(y), stream_of(state)),
        "naju_b200_step");
  return y;
}

// ------------------------------------------------------------------------------ Python boundary
const Tensor& tensor_arg(PyObject* o, const char* name) {
  TORCH_CHECK_TYPE(THPVariable_Check(o), name, " must be a tensor, got ", Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}

PyObject* py_scan(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n == 8, "scan takes 8 arguments");
  const Tensor &u = tensor_arg(args[0], "u"), &fl = tensor_arg(args[1], "f_logit"), &il = tensor_arg(args[2], "i_logit"),
               &Bm = tensor_arg(args[3], "B"), &Cm = tensor_arg(args[4], "C"), &D = tensor_arg(args[5], "D_skip");
  const Tensor h0 = args[6] == Py_None ? Tensor() : tensor_arg(args[6], "h0");
  const bool want_final = PyObject_IsTrue(args[7]) == 1;
  std::tuple<Tensor, Tensor> r;
  {
    pybind11::gil_scoped_release nogil;
    r = scan(u, fl, il, Bm, Cm, D, h0, want_final);
  }
  if (!want_final) return THPVariable_Wrap(std::move(std::get<0>(r)));
  return PyTuple_Pack(2, THPObjectPtr(THPVariable_Wrap(std::get<0>(r))).get(),
                      THPObjectPtr(THPVariable_Wrap(std::get<1>(r))).get());
  END_HANDLE_TH_ERRORS
}

PyObject* py_step(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n == 7, "step takes 7 arguments");
  const Tensor &state = tensor_arg(args[0], "state"), &u = tensor_arg(args[1], "u_t"),
               &fl = tensor_arg(args[2], "f_logit_t"), &il = tensor_arg(args[3], "i_logit_t"),
               &Bm = tensor_arg(args[4], "B_t"), &Cm = tensor_arg(args[5], "C_t"), &D = tensor_arg(args[6], "D_skip");
  Tensor y;
  {
    pybind11::gil_scoped_release nogil;
    y = step(state, u, fl, il, Bm, Cm, D);
  }
  return PyTuple_Pack(2, THPObjectPtr(THPVariable_Wrap(std::move(y))).get(), args[0]);
  END_HANDLE_TH_ERRORS
}

PyMethodDef kFast[] = {
    {"scan", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_scan)), METH_FASTCALL,
     "scan(u, f_logit, i_logit, B, C, D_skip, h0 or None, want_final) -> y or (y, hT), differentiable"},
    {"step", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_step)), METH_FASTCALL,
     "step(state, u_t, f_logit_t, i_logit_t, B_t, C_t, D_skip) -> (y_t, state)"},
    {nullptr, nullptr, 0, nullptr}};

using OptTensor = std::optional<Tensor>;
Tensor opt(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }
py::bytes desc_bytes(const naju_scan_desc& d) { return py::bytes(reinterpret_cast<const char*>(&d), sizeof(d)); }
OptTensor ret(const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; }

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  PyModule_AddFunctions(m.ptr(), kFast);
  m.def("version", []() { return naju_b200_version(); });
  m.def("time_contig", &time_contig);
  m.def("prepare", [](const Tensor& u, const Tensor& fl, const Tensor& il, const Tensor& Bm, const Tensor& Cm, const Tensor& D) {
    const Args a = prepare(u, fl, il, Bm, Cm, D.detach());
    return std::make_tuple(a.u, a.fl, a.il, a.Bm, a.Cm, a.D);
  });
  m.def("describe", [](const Tensor& u, const Tensor& fl, const Tensor& il, const Tensor& Bm, const Tensor& Cm) {
    const naju_scan_desc d = describe({u, fl, il, Bm, Cm, Tensor()}, call_flags());
    return desc_bytes(d);
  });
  m.def("state_arg", [](const OptTensor& h, int64_t B, int64_t D, int64_t N, const std::string& name) {
    const Tensor t = opt(h);
    return ret(state_arg(t.defined() ? t.detach() : t, B, D, N, name.c_str()));
  });
  m.def("forward", [](const Tensor& u, const Tensor& fl, const Tensor& il, const Tensor& Bm, const Tensor& Cm, const Tensor& D,
                      const OptTensor& h0, bool want_final, bool want_decay) {
    at::NoGradGuard ng;
    const FwdOut o = naju_forward({u, fl, il, Bm, Cm, D}, opt(h0), want_final, want_decay, call_flags());
    return std::make_tuple(o.y, ret(o.hT), ret(o.pT), o.ckpt, desc_bytes(o.desc));
  });
  m.def("backward", [](int flags, const Tensor& u, const Tensor& fl, const Tensor& il, const Tensor& Bm, const Tensor& Cm,
                       const Tensor& D, const OptTensor& h0, const Tensor& dy, const OptTensor& dhT, const Tensor& ckpt,
                       bool want_dh0) {
    at::NoGradGuard ng;
    const BwdOut o = naju_backward({u, fl, il, Bm, Cm, D}, opt(h0), dy, opt(dhT), ckpt, want_dh0, flags);
    return std::make_tuple(o.du, o.dfl, o.dil, o.dB, o.dC, o.dD, ret(o.dh0));
  });
  m.def("forms", []() { return std::make_pair(g_form_fwd.load(), g_form_bwd.load()); });
  m.def("take_guarded", []() {
    std::lock_guard<std::mutex> lock(g_guard_mutex);
    auto out = std::move(g_guarded);
    g_guarded.clear();
    return out;
  });
}
