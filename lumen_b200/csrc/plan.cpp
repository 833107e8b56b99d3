// The compiled program: an ordered list of steps over the caller's inputs, outputs and ONE workspace, the
// counterpart of the reference's DevicePlan / StepBase / execute loop (lumen/plan/mod.rs:78-148,
// lumen/plan/step/mod.rs:27-76, lumen/plan/run.rs:247-427). Placement (live ranges packed into the workspace at
// 256-byte aligned offsets) is decided by the host-side compiler; this file holds the prepared steps - each
// already bound to its generated kernel or library kernel - and the run loop, which only turns offsets into
// pointers and queues launches on the caller's stream. It never allocates, synchronises or waits.
//
// Plan text:
//   module <k> ... endmodule        fusion bodies in the graph text format, referred to by index
//   plan <n_inputs> <n_outputs> <workspace_bytes>
//   t <id> <dtype> <base> <byte_offset> <rank> <shape...> <strides...>     base: i<k> | o<k> | w
//   s <kind> <label> <args...>
//   end
//
// Collectives are steps too (lumen/plan/step/triton.rs:122-177): `s all_reduce <label> <tensor> <op>` queues NCCL's
// all-reduce of a (bucket of) gradient(s) on the plan's side stream once everything queued before it has finished,
// and `s wait <label> <k>` makes the compute stream wait for the k-th collective of the plan (the device_wait of
// lumen/distributed/nccl.rs:279-307, :532-565: side stream + one event per collective). Nothing blocks the host.
#include <chrono>
#include <cstring>
#include <map>
#include <mutex>
#include <memory>
#include <sstream>

#include "fused.h"
#include "gemm.h"

struct lb_comm;

namespace lb {
bool gemm(const lb_tensor& a, const lb_tensor& b, const lb_tensor& d, int epilogue, int kernel_choice, void* stream,
          void* scratch, size_t scratch_bytes, const lb_tensor* aux, const GemmTuning* tuning, SimtProblem* held = nullptr);
bool gemm_held(const lb_tensor& a, const lb_tensor& b, SimtProblem& q);
int gemm_launches(const lb_tensor& a, const lb_tensor& b, size_t scratch_bytes, int kernel_choice, const GemmTuning* tuning);
int gemm_model_splits(long long M, long long N, long long K, long long batch);
void fill_noise(void* ptr, size_t bytes, void* stream);
void transpose_2d(const lb_tensor& in, const lb_tensor& out, void* stream);
void strided_copy(const lb_tensor& in, const lb_tensor& out, void* stream);
void attention_forward(const lb_attn_desc& desc, const lb_tensor& q, const lb_tensor& k, const lb_tensor& v, const lb_tensor& o,
                       const lb_tensor* lse, void* stream);
void attention_backward(const lb_attn_desc& desc, const lb_tensor& q, const lb_tensor& k, const lb_tensor& v, const lb_tensor& o,
                        const lb_tensor& d_o, const lb_tensor& lse, const lb_tensor& delta, const lb_tensor& dq, const lb_tensor& dk,
                        const lb_tensor& dv, void* stream, const lb_tensor* dq_acc, void* scratch, size_t scratch_bytes);
void scatter_add_rows(const lb_tensor& x, const lb_tensor& ids, const lb_tensor& updates, const lb_tensor& out, void* scratch,
                      bool x_is_zero, bool deterministic, void* stream);
size_t scatter_add_scratch_bytes(long long rows, long long width, long long tokens, bool deterministic);
int scatter_add_launches(long long rows, long long tokens, bool deterministic);
void comm_all_reduce(lb_comm* c, const void* send, void* recv, size_t count, int dtype, int op, void* stream);
int comm_world(const lb_comm* c);

namespace {

struct View {
    char base_kind = 'w';  // 'i', 'o' or 'w'
    int base_index = 0;
    size_t offset = 0;
    lb_tensor t{};
};

enum Kind { FUSION, MULTI, GEMM, ATTN_FWD, ATTN_BWD, SCATTER_ADD, COPY, FILL, TRANSPOSE, ALL_REDUCE, WAIT };

struct Step {
    Kind kind;
    std::string label;
    std::vector<int> args;  // view ids (-1 = absent)
    lb_fusion* fusion = nullptr;
    int scratch = -1;
    int aux = -1;  // gemm: tensor id of the epilogue operand
    int epilogue = 0;
    lb_attn_desc attn{};
    int fill_byte = 0;
    GemmTuning tuning{};   // gemm: what the autotuner picked (zeros: the library's own choices)
    int tuned_kernel = 0;  // gemm: 0 = choose, 3 = the one-CTA kernel
};

}  // namespace
}  // namespace lb

struct lb_plan {
    int n_inputs = 0, n_outputs = 0;
    size_t workspace_bytes = 0;
    std::vector<lb::View> views;
    std::vector<lb::Step> steps;
    std::string json;
    std::string text;  // the plan text this plan was parsed from
    // collectives: the communicator (borrowed), the side stream they run on and, per collective, the event the compute
    // stream records before it and the event the side stream records after it. Created on first use.
    int n_collectives = 0;
    lb_comm* comm = nullptr;
    cudaStream_t side = nullptr;
    std::vector<cudaEvent_t> ready, done;
    ~lb_plan() {
        for (auto e : ready) cudaEventDestroy(e);
        for (auto e : done) cudaEventDestroy(e);
        if (side) cudaStreamDestroy(side);
    }
};

namespace lb {
namespace {

lb_tensor bind(const lb_plan& p, int id, void* ws, void* const* in, void* const* out) {
    if (id < 0 || id >= (int)p.views.size()) fail(LB_ERR_INVALID, format("plan: tensor %d is not defined", id));
    const View& v = p.views[id];
    char* base = v.base_kind == 'w' ? (char*)ws : v.base_kind == 'i' ? (char*)in[v.base_index] : (char*)out[v.base_index];
    lb_tensor t = v.t;
    t.ptr = base + v.offset;
    return t;
}

size_t view_bytes(const lb_tensor& t) {
    size_t n = 1;
    for (int d = 0; d < t.rank; d++) n *= (size_t)t.shape[d];
    return n * dtype_size(t.dtype);
}

std::unique_ptr<lb_plan> parse_plan(const std::string& text) {
    auto plan = std::make_unique<lb_plan>();
    std::vector<lb_fusion*> modules;
    std::vector<std::string> module_texts;
    std::istringstream lines(text);
    std::string line, module_text;
    bool in_module = false, seen_plan = false, ended = false;
    std::ostringstream json;
    json << "[";
    while (std::getline(lines, line)) {
        if (in_module) {
            if (line == "endmodule") {
                modules.push_back(compile_fusion(module_text)), module_texts.push_back(module_text);
                in_module = false;
            } else {
                module_text += line + "\n";
            }
            continue;
        }
        std::istringstream ts(line);
        std::vector<std::string> tok;
        for (std::string t; ts >> t;) tok.push_back(t);
        if (tok.empty()) continue;
        if (tok[0] == "module") {
            in_module = true;
            module_text.clear();
        } else if (tok[0] == "plan" && tok.size() == 4) {
            plan->n_inputs = std::stoi(tok[1]);
            plan->n_outputs = std::stoi(tok[2]);
            plan->workspace_bytes = std::stoull(tok[3]);
            seen_plan = true;
        } else if (tok[0] == "t" && tok.size() >= 6) {
            int id = std::stoi(tok[1]);
            View v;
            v.t.dtype = dtype_from_name(tok[2]);
            v.base_kind = tok[3][0];
            if (v.base_kind != 'w') v.base_index = std::stoi(tok[3].substr(1));
            if (v.base_kind != 'w' && v.base_kind != 'i' && v.base_kind != 'o') fail(LB_ERR_INVALID, "plan: bad tensor base " + tok[3]);
            if (v.base_kind == 'i' && v.base_index >= plan->n_inputs) fail(LB_ERR_INVALID, "plan: input index out of range");
            if (v.base_kind == 'o' && v.base_index >= plan->n_outputs) fail(LB_ERR_INVALID, "plan: output index out of range");
            v.offset = std::stoull(tok[4]);
            v.t.rank = std::stoi(tok[5]);
            if (v.t.rank < 0 || v.t.rank > LB_MAX_RANK || (int)tok.size() != 6 + 2 * v.t.rank) fail(LB_ERR_INVALID, "plan: bad tensor line: " + line);
            for (int d = 0; d < v.t.rank; d++) {
                v.t.shape[d] = std::stoll(tok[6 + d]);
                v.t.stride[d] = std::stoll(tok[6 + v.t.rank + d]);
            }
            if ((int)plan->views.size() <= id) plan->views.resize(id + 1);
            plan->views[id] = v;
        } else if (tok[0] == "s" && tok.size() >= 3) {
            Step s;
            const std::string& kind = tok[1];
            s.label = tok[2];
            auto ints = [&](size_t from, size_t count) {
                if (tok.size() < from + count) fail(LB_ERR_INVALID, "plan: short step line: " + line);
                for (size_t k = 0; k < count; k++) s.args.push_back(std::stoi(tok[from + k]));
            };
            if (kind == "fusion") {
                s.kind = FUSION;
                int m = std::stoi(tok.at(3));
                if (m < 0 || m >= (int)modules.size()) fail(LB_ERR_INVALID, "plan: fusion refers to an undefined module");
                s.fusion = modules[m];
                s.scratch = std::stoi(tok.at(4));
                ints(6, std::stoul(tok.at(5)));
                if (s.fusion->scratch_bytes && s.scratch < 0) fail(LB_ERR_INVALID, "plan: fusion " + s.label + " needs scratch");
                // (a text written by a library whose kernels cut the same module into fewer slices: those of at most sixteen warps an SM still can)
                auto too_little = [&] { return s.scratch >= 0 && (s.scratch >= (int)plan->views.size() || view_bytes(plan->views[s.scratch].t) < s.fusion->scratch_bytes); };
                if (too_little()) s.fusion = compile_fusion("option sixteen_warps\n" + module_texts[m]);
                if (too_little())
                    fail(LB_ERR_INVALID, "plan: the scratch of fusion " + s.label + " is smaller than its kernel needs: lower the module again");
            } else if (kind == "multi") {  // s multi <label> <module> <n_groups> <tensor ids, group after group>
                s.kind = MULTI;
                int m = std::stoi(tok.at(3));
                if (m < 0 || m >= (int)modules.size()) fail(LB_ERR_INVALID, "plan: multi refers to an undefined module");
                s.fusion = modules[m];
                s.aux = std::stoi(tok.at(4));
                const int per = s.fusion->kernel.n_inputs + s.fusion->kernel.n_outputs;
                if (!s.fusion->kernel.multi || s.aux < 1) fail(LB_ERR_INVALID, "plan: a multi step needs a module compiled with option multi and at least one group");
                ints(5, (size_t)s.aux * per);
            } else if (kind == "gemm") {
                s.kind = GEMM;
                ints(3, 3);
                s.epilogue = std::stoi(tok.at(6));
                s.scratch = tok.size() > 7 ? std::stoi(tok[7]) : -1;
                s.aux = tok.size() > 8 ? std::stoi(tok[8]) : -1;  // operand of an add / mask epilogue
            } else if (kind == "attn_fwd" || kind == "attn_bwd") {
                s.kind = kind == "attn_fwd" ? ATTN_FWD : ATTN_BWD;
                // attn_bwd: q k v o dO lse delta dq dk dv [dq accumulator: the single-kernel form with atomic dQ]
                size_t n = s.kind == ATTN_FWD ? 5 : (tok.size() >= 17 ? 11 : 10);
                ints(3, n);
                s.attn.scale = (float)std::strtod(tok.at(3 + n).c_str(), nullptr);
                s.attn.causal = std::stoi(tok.at(4 + n));
                s.attn.causal_offset = std::stoll(tok.at(5 + n));
            } else if (kind == "scatter_add") {
                s.kind = SCATTER_ADD;
                ints(3, 5);  // x (-1: zeros), ids, updates, out, scratch
                s.epilogue = tok.size() > 8 ? std::stoi(tok[8]) : 0;  // 1: deterministic (sorted) form, 0: float32 atomics
            } else if (kind == "transpose") {
                s.kind = TRANSPOSE;
                ints(3, 2);  // dense [R, C] source, dense [C, R] destination
            } else if (kind == "all_reduce") {
                s.kind = ALL_REDUCE;
                ints(3, 1);  // the dense tensor reduced in place
                s.epilogue = std::stoi(tok.at(4));  // 0 sum, 1 prod, 2 max, 3 min
                s.aux = plan->n_collectives++;      // its number among the plan's collectives
            } else if (kind == "wait") {
                s.kind = WAIT;
                s.aux = std::stoi(tok.at(3));
                if (s.aux < 0 || s.aux >= plan->n_collectives) fail(LB_ERR_INVALID, "plan: wait refers to a collective that is not queued before it");
            } else if (kind == "copy") {
                s.kind = COPY;
                ints(3, 2);
            } else if (kind == "fill") {
                s.kind = FILL;
                ints(3, 1);
                s.fill_byte = std::stoi(tok.at(4));
            } else {
                fail(LB_ERR_UNSUPPORTED, "plan: no kernel for step kind " + kind);
            }
            json << (plan->steps.empty() ? "" : ", ") << "{\"kind\": \"" << kind << "\", \"label\": \"" << s.label << "\"}";
            plan->steps.push_back(std::move(s));
        } else if (tok[0] == "end") {
            ended = true;
        } else {
            fail(LB_ERR_INVALID, "plan: cannot parse '" + line + "'");
        }
    }
    if (!seen_plan || !ended) fail(LB_ERR_INVALID, "plan text needs a 'plan' line and an 'end' line");
    json << "]";
    plan->json = json.str();
    return plan;
}

static bool row_major(const lb_tensor& t) {
    int64_t expect = 1;
    for (int d = t.rank - 1; d >= 0; d--) {
        if (t.shape[d] != 1 && t.stride[d] != expect) return false;
        expect *= t.shape[d];
    }
    return true;
}

// How a copy step moves its bytes: 0 one contiguous block; 1 rows of a rank-2 view with unit inner strides that are
// further apart on either side (a 2-d copy); 2 anything else (the strided copy kernel).
int copy_form(const lb_tensor& src, const lb_tensor& dst) {
    if (row_major(src) && row_major(dst)) return 0;
    if (src.rank == 2 && dst.rank == 2 && src.stride[1] == 1 && dst.stride[1] == 1 && src.stride[0] >= src.shape[1] && dst.stride[0] >= dst.shape[1]) return 1;
    return 2;
}

// The side stream and events of the plan's collectives, made on the first run that reaches one.
void prepare_collectives(lb_plan& p) {
    if (!p.comm) fail(LB_ERR_INVALID, "plan: it holds collectives; bind a communicator with lb_plan_set_comm before running it");
    if (p.side) return;
    LB_CUDA(cudaStreamCreateWithFlags(&p.side, cudaStreamNonBlocking));
    for (int k = 0; k < p.n_collectives; k++) {
        cudaEvent_t a = nullptr, b = nullptr;
        LB_CUDA(cudaEventCreateWithFlags(&a, cudaEventDisableTiming));
        LB_CUDA(cudaEventCreateWithFlags(&b, cudaEventDisableTiming));
        p.ready.push_back(a), p.done.push_back(b);
    }
}

// Products of float32 operands (always the CUDA cores') that follow one another and of which none reads or writes what another writes:
// the two gradients of a linear layer, and the like. They are queued together (gemm_simt_many), at the latest before the
// next step of another kind.
struct Bytes {
    uintptr_t begin, end;
    explicit Bytes(const lb_tensor& t) {
        long long low = 0, high = 1;
        for (int d = 0; d < t.rank; d++) (t.stride[d] < 0 ? low : high) += (t.shape[d] - 1) * t.stride[d];
        begin = (uintptr_t)t.ptr + low * (long long)dtype_size(t.dtype), end = (uintptr_t)t.ptr + high * (long long)dtype_size(t.dtype);
    }
    bool meets(const Bytes& o) const { return begin < o.end && o.begin < end; }
};
struct Products {
    std::vector<SimtProblem> held;
    std::vector<Bytes> read, written;
    static bool takes(const Step& s, const lb_tensor& a) { return s.kind == GEMM && a.dtype == LB_F32; }
    bool independent(const lb_tensor& a, const lb_tensor& b, const lb_tensor& d, const lb_tensor* aux) const {
        const Bytes x(a), y(b), z(d), u(aux ? *aux : a);
        for (const Bytes& w : written)
            if (w.meets(x) || w.meets(y) || w.meets(z) || w.meets(u)) return false;
        for (const Bytes& r : read)
            if (r.meets(z)) return false;
        return true;
    }
    void add(const lb_tensor& a, const lb_tensor& b, const lb_tensor& d, const lb_tensor* aux, const SimtProblem& q) {
        held.push_back(q);
        read.emplace_back(a), read.emplace_back(b), written.emplace_back(d);
        if (aux) read.emplace_back(*aux);
    }
    int queue(int sms, bool launch, cudaStream_t s) {
        if (held.empty()) return 0;
        const int n = gemm_simt_many(held.data(), (int)held.size(), sms, launch, s);
        held.clear(), read.clear(), written.clear();
        return n;
    }
};

void run(const lb_plan& p, void* ws, void* const* in, void* const* out, int first, int last, void* stream) {
    if (first < 0 || last > (int)p.steps.size() || first > last) fail(LB_ERR_INVALID, "plan: step range out of bounds");
    std::vector<lb_tensor> tensors;
    Products products;
    auto queue = [&] {
        if (!products.held.empty()) products.queue(device_info().sms, true, (cudaStream_t)stream);  // (asking for the device takes the host 0.1 us)
    };
    for (int k = first; k < last; k++) {
        const Step& s = p.steps[k];
        auto T = [&](int i) { return bind(p, s.args.at(i), ws, in, out); };
        if (s.kind == GEMM && Products::takes(s, T(0))) {
            const lb_tensor a = T(0), b = T(1), d = T(2), other = s.aux >= 0 ? bind(p, s.aux, ws, in, out) : lb_tensor{};
            const lb_tensor* aux = s.aux >= 0 ? &other : nullptr;
            if (!products.independent(a, b, d, aux)) queue();
            SimtProblem q{};
            if (gemm(a, b, d, s.epilogue, s.tuned_kernel, stream, nullptr, 0, aux, &s.tuning, &q)) products.add(a, b, d, aux, q);
            continue;
        }
        queue();
        switch (s.kind) {
            case FUSION: {
                tensors.clear();
                for (int id : s.args) tensors.push_back(bind(p, id, ws, in, out));
                void* scratch = s.scratch >= 0 ? bind(p, s.scratch, ws, in, out).ptr : nullptr;
                launch_fusion(s.fusion, tensors.data(), (int)tensors.size(), scratch, stream);
                break;
            }
            case MULTI: {
                tensors.clear();
                for (int id : s.args) tensors.push_back(bind(p, id, ws, in, out));
                launch_fusion_multi(s.fusion, tensors.data(), s.aux, stream);
                break;
            }
            case GEMM: {
                void* scratch = nullptr;
                size_t bytes = 0;
                if (s.scratch >= 0) {
                    lb_tensor sc = bind(p, s.scratch, ws, in, out);
                    scratch = sc.ptr, bytes = view_bytes(sc);
                }
                lb_tensor aux{};
                if (s.aux >= 0) aux = bind(p, s.aux, ws, in, out);
                gemm(T(0), T(1), T(2), s.epilogue, s.tuned_kernel, stream, scratch, bytes, s.aux >= 0 ? &aux : nullptr, &s.tuning);
                break;
            }
            case ATTN_FWD: {
                lb_tensor lse = T(4);
                attention_forward(s.attn, T(0), T(1), T(2), T(3), &lse, stream);
                break;
            }
            case ATTN_BWD: {
                lb_tensor acc{};
                if (s.args.size() > 10) acc = T(10);
                attention_backward(s.attn, T(0), T(1), T(2), T(3), T(4), T(5), T(6), T(7), T(8), T(9), stream, s.args.size() > 10 ? &acc : nullptr, nullptr, 0);
                break;
            }
            case SCATTER_ADD: {
                lb_tensor outp = T(3);
                lb_tensor x = s.args[0] >= 0 ? T(0) : outp;
                lb_tensor ids = T(1), scratch = T(4);
                long long tokens = 1;
                for (int d = 0; d < ids.rank; d++) tokens *= ids.shape[d];
                if (view_bytes(scratch) < scatter_add_scratch_bytes(outp.shape[0], outp.shape[1], tokens, s.epilogue != 0))
                    fail(LB_ERR_INVALID, "plan: scatter_add scratch is too small");
                scatter_add_rows(x, ids, T(2), outp, scratch.ptr, s.args[0] < 0, s.epilogue != 0, stream);
                break;
            }
            case TRANSPOSE: transpose_2d(T(0), T(1), stream); break;
            case ALL_REDUCE: {
                lb_plan& mp = const_cast<lb_plan&>(p);  // lazily made stream and events; the step list is not touched
                prepare_collectives(mp);
                lb_tensor t = T(0);
                size_t count = 1;
                for (int d = 0; d < t.rank; d++) count *= (size_t)t.shape[d];
                LB_CUDA(cudaEventRecord(mp.ready[s.aux], (cudaStream_t)stream));
                LB_CUDA(cudaStreamWaitEvent(mp.side, mp.ready[s.aux], 0));
                comm_all_reduce(mp.comm, t.ptr, t.ptr, count, t.dtype, s.epilogue, mp.side);
                LB_CUDA(cudaEventRecord(mp.done[s.aux], mp.side));
                break;
            }
            case WAIT: {
                if (!p.side) fail(LB_ERR_INVALID, "plan: a wait ran before its collective (run the range that queues it first)");
                LB_CUDA(cudaStreamWaitEvent((cudaStream_t)stream, p.done[s.aux], 0));
                break;
            }
            case COPY: {
                lb_tensor src = T(0), dst = T(1);
                const size_t size = dtype_size(src.dtype);
                switch (copy_form(src, dst)) {
                    case 0: LB_CUDA(cudaMemcpyAsync(dst.ptr, src.ptr, view_bytes(src), cudaMemcpyDeviceToDevice, (cudaStream_t)stream)); break;
                    case 1:  // rows of a matrix into (or out of) rows further apart: a column block of a wider matrix
                        if (src.shape[0] && src.shape[1])
                            LB_CUDA(cudaMemcpy2DAsync(dst.ptr, (size_t)dst.stride[0] * size, src.ptr, (size_t)src.stride[0] * size, (size_t)src.shape[1] * size,
                                                      (size_t)src.shape[0], cudaMemcpyDeviceToDevice, (cudaStream_t)stream));
                        break;
                    default: strided_copy(src, dst, stream); break;  // any other pair of views, element by element
                }
                break;
            }
            case FILL: {
                lb_tensor dst = T(0);
                LB_CUDA(cudaMemsetAsync(dst.ptr, s.fill_byte, view_bytes(dst), (cudaStream_t)stream));
                break;
            }
        }
    }
    queue();
}

}  // namespace
}  // namespace lb

extern "C" {

int lb_plan_create(const char* text, lb_plan** out) {
    return lb::guarded([&] {
        if (!text || !out) lb::fail(LB_ERR_INVALID, "lb_plan_create: null argument");
        auto plan = lb::parse_plan(text);
        plan->text = text;
        *out = plan.release();
    });
}
void lb_plan_destroy(lb_plan* plan) { delete plan; }
size_t lb_plan_workspace_bytes(const lb_plan* plan) { return plan ? plan->workspace_bytes : 0; }
size_t lb_plan_workspace_alignment(const lb_plan*) { return 256; }
int lb_plan_num_steps(const lb_plan* plan) { return plan ? (int)plan->steps.size() : -1; }
const char* lb_plan_steps_json(const lb_plan* plan) { return plan ? plan->json.c_str() : "[]"; }
const char* lb_plan_text(const lb_plan* plan) { return plan ? plan->text.c_str() : ""; }

// A step range recorded once as a CUDA graph and replayed with one launch. The range is recorded on a private
// stream (the caller's may be the legacy default stream, which cannot be captured); nothing runs while recording.
struct lb_graph {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    ~lb_graph() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
    }
};

int lb_plan_capture(const lb_plan* plan, void* workspace, void* const* inputs, int n_inputs, void* const* outputs,
                    int n_outputs, int first_step, int last_step, lb_graph** out) {
    return lb::guarded([&] {
        if (!plan || !out) lb::fail(LB_ERR_INVALID, "lb_plan_capture: null argument");
        if (n_inputs != plan->n_inputs || n_outputs != plan->n_outputs)
            lb::fail(LB_ERR_INVALID, lb::format("the plan takes %d inputs and %d outputs, got %d and %d", plan->n_inputs,
                                                plan->n_outputs, n_inputs, n_outputs));
        if (plan->workspace_bytes && (!workspace || ((uintptr_t)workspace & 255) != 0))
            lb::fail(LB_ERR_INVALID, "lb_plan_capture: the workspace must be 256-byte aligned");
        cudaStream_t side = nullptr;
        LB_CUDA(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
        auto g = std::make_unique<lb_graph>();
        cudaError_t err = cudaStreamBeginCapture(side, cudaStreamCaptureModeThreadLocal);
        if (err != cudaSuccess) {
            cudaStreamDestroy(side);
            lb::fail(LB_ERR_CUDA, lb::format("cudaStreamBeginCapture: %s", cudaGetErrorString(err)));
        }
        std::string problem;
        try {
            lb::run(*plan, workspace, inputs, outputs, first_step, last_step < 0 ? (int)plan->steps.size() : last_step, side);
        } catch (const std::exception& e) {
            problem = e.what();
        }
        err = cudaStreamEndCapture(side, &g->graph);  // always ends the capture, also after a failed step
        cudaStreamDestroy(side);
        if (!problem.empty()) lb::fail(LB_ERR_CUDA, "lb_plan_capture: " + problem);
        if (err != cudaSuccess) lb::fail(LB_ERR_CUDA, lb::format("cudaStreamEndCapture: %s", cudaGetErrorString(err)));
        LB_CUDA(cudaGraphInstantiate(&g->exec, g->graph, 0));
        *out = g.release();
    });
}

int lb_graph_launch(const lb_graph* graph, void* stream) {
    return lb::guarded([&] {
        if (!graph || !graph->exec) lb::fail(LB_ERR_INVALID, "lb_graph_launch: null graph");
        LB_CUDA(cudaGraphLaunch(graph->exec, (cudaStream_t)stream));
    });
}

void lb_graph_destroy(lb_graph* graph) { delete graph; }

int lb_plan_autotune(lb_plan* plan, void* workspace, void* const* inputs, int n_inputs, void* const* outputs, int n_outputs,
                     void* stream, char* report, size_t report_bytes) {
    return lb::guarded([&] {
        using namespace lb;
        if (!plan) fail(LB_ERR_INVALID, "lb_plan_autotune: null plan");
        if (n_inputs != plan->n_inputs || n_outputs != plan->n_outputs) fail(LB_ERR_INVALID, "lb_plan_autotune: wrong number of inputs or outputs");
        if (plan->workspace_bytes && (!workspace || ((uintptr_t)workspace & 255) != 0)) fail(LB_ERR_INVALID, "lb_plan_autotune: the workspace must be 256-byte aligned");
        cudaStream_t s = (cudaStream_t)stream;
        struct Pick { GemmTuning tuning; int kernel; double us, default_us; int candidates; };
        static std::mutex mutex;
        static std::map<std::string, Pick> picks;  // by shape, majors, dtypes, epilogue: shared across plans
        std::ostringstream json;
        json << "[";
        bool first_entry = true, warmed = false;
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        LB_CUDA(cudaEventCreate(&e0));
        LB_CUDA(cudaEventCreate(&e1));
        if (plan->workspace_bytes) fill_noise(workspace, plan->workspace_bytes, stream);
        for (Step& st : plan->steps) {
            if (st.kind != GEMM) continue;
            lb_tensor a = bind(*plan, st.args.at(0), workspace, inputs, outputs), b = bind(*plan, st.args.at(1), workspace, inputs, outputs);
            lb_tensor d = bind(*plan, st.args.at(2), workspace, inputs, outputs);
            if (a.rank != 2 || b.rank != 2 || (a.dtype != LB_BF16 && a.dtype != LB_F16)) continue;
            if (plan->views[st.args.at(2)].base_kind == 'i') continue;  // never write a caller's input while tuning
            const long long M = a.shape[0], K = a.shape[1], N = b.shape[1];
            if ((double)M * N * K < 1073741824.0) continue;  // tuned from 2^30 multiply-adds on
            void* scratch = nullptr;
            size_t bytes = 0;
            if (st.scratch >= 0) {
                lb_tensor sc = bind(*plan, st.scratch, workspace, inputs, outputs);
                scratch = sc.ptr, bytes = view_bytes(sc);
            }
            lb_tensor aux{};
            if (st.aux >= 0) aux = bind(*plan, st.aux, workspace, inputs, outputs);
            const std::string key = format("%lld %lld %lld a%lld.%lld b%lld.%lld %d>%d e%d s%zu", M, N, K, (long long)a.stride[0], (long long)a.stride[1],
                                           (long long)b.stride[0], (long long)b.stride[1], a.dtype, d.dtype, st.epilogue, bytes);
            Pick pick{};
            bool known = false;
            {
                std::lock_guard<std::mutex> lock(mutex);
                auto it = picks.find(key);
                if (it != picks.end()) pick = it->second, known = true;
            }
            if (!known) {
                struct Candidate { GemmTuning t; int kernel; };
                std::vector<Candidate> cands;
                const int model = gemm_model_splits(M, N, K, 1);
                std::vector<int> split_options = {0};  // 0: the cost model's own choice
                for (int sp : {1, model / 2, model * 2})
                    if (sp >= 1 && sp != model && (sp == 1 || (size_t)sp * M * N * 4 <= bytes) && (K + 63) / 64 / sp >= 8) split_options.push_back(sp);
                for (int sp : split_options)
                    for (int gm : {0, 4, 16}) cands.push_back({{sp, gm}, 0});
                if (M > 128) cands.push_back({{0, 0}, 3});
                auto run_one = [&](const Candidate& c) {
                    gemm(a, b, d, st.epilogue, c.kernel, stream, scratch, bytes, st.aux >= 0 ? &aux : nullptr, &c.t);
                };
                if (!warmed) {  // reach sustained clocks before the first candidate is timed
                    auto t0 = std::chrono::steady_clock::now();
                    while (std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count() < 0.2) {
                        for (int r = 0; r < 8; r++) run_one(cands[0]);
                        LB_CUDA(cudaStreamSynchronize(s));
                    }
                    warmed = true;
                }
                double best = 1e30;
                for (size_t ci = 0; ci < cands.size(); ci++) {
                    for (int r = 0; r < 5; r++) run_one(cands[ci]);
                    LB_CUDA(cudaEventRecord(e0, s));
                    for (int r = 0; r < 10; r++) run_one(cands[ci]);
                    LB_CUDA(cudaEventRecord(e1, s));
                    LB_CUDA(cudaEventSynchronize(e1));
                    float ms = 0.0f;
                    LB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
                    const double us = ms * 100.0;  // per run
                    if (ci == 0) pick.default_us = us;
                    if (us < best * 0.99 || ci == 0) {  // a candidate has to win by a percent to displace an earlier one
                        if (us < best) best = us;
                        pick.tuning = cands[ci].t, pick.kernel = cands[ci].kernel, pick.us = us;
                    }
                }
                pick.candidates = (int)cands.size();
                std::lock_guard<std::mutex> lock(mutex);
                picks[key] = pick;
            }
            st.tuning = pick.tuning, st.tuned_kernel = pick.kernel;
            json << (first_entry ? "" : ", ") << "{\"label\": \"" << st.label << "\", \"m\": " << M << ", \"n\": " << N << ", \"k\": " << K
                 << ", \"candidates\": " << pick.candidates << ", \"picked\": {\"kernel\": " << pick.kernel << ", \"splits\": " << pick.tuning.splits
                 << ", \"group_m\": " << pick.tuning.group_m << "}, \"us\": " << pick.us << ", \"default_us\": " << pick.default_us << "}";
            first_entry = false;
        }
        json << "]";
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        LB_CUDA(cudaStreamSynchronize(s));
        if (report && report_bytes) snprintf(report, report_bytes, "%s", json.str().c_str());
    });
}

int lb_plan_set_comm(lb_plan* plan, lb_comm* comm) {
    return lb::guarded([&] {
        if (!plan) lb::fail(LB_ERR_INVALID, "lb_plan_set_comm: null plan");
        plan->comm = comm;
    });
}
int lb_plan_num_collectives(const lb_plan* plan) { return plan ? plan->n_collectives : -1; }

int lb_plan_kernel_launches(const lb_plan* plan) {
    if (!plan) return -1;
    int n = 0;
    const int rc = lb::guarded([&] {  // a step may name a tensor that the plan does not define
        lb::Products products;  // told apart by where they lie in the workspace, which input and which output they are
        const int sms = lb::sm_count_hint();
        for (const lb::Step& s : plan->steps) {
            auto placed = [&](int id) {
                const lb::View& v = plan->views.at((size_t)id);
                lb_tensor t = v.t;
                const uintptr_t base = v.base_kind == 'w' ? 1 : 2 + 2 * (uintptr_t)v.base_index + (v.base_kind == 'o');
                t.ptr = (void*)((base << 44) + v.offset);
                return t;
            };
            auto place = [&](int i) { return placed(s.args.at(i)); };
            if (s.kind == lb::GEMM && lb::Products::takes(s, place(0))) {
                const lb_tensor a = place(0), b = place(1), d = place(2), other = s.aux >= 0 ? placed(s.aux) : lb_tensor{};
                const lb_tensor* aux = s.aux >= 0 ? &other : nullptr;
                if (!products.independent(a, b, d, aux)) n += products.queue(sms, false, nullptr);
                lb::SimtProblem q{};
                if (lb::gemm_held(a, b, q)) products.add(a, b, d, aux, q);
                continue;
            }
            n += products.queue(sms, false, nullptr);
            switch (s.kind) {
                case lb::FUSION: n += s.fusion && s.fusion->kernel.empty ? 0 : (s.scratch >= 0 ? 2 : 1); break;  // partial sums + finalize
                case lb::MULTI: n += s.fusion && s.fusion->kernel.multi_max_groups > 0 ? (s.aux + s.fusion->kernel.multi_max_groups - 1) / s.fusion->kernel.multi_max_groups : 1; break;
                case lb::GEMM: {  // split-K partial tiles + reduction, or one kernel
                    auto operand = [&](int i) {
                        const lb::View& v = plan->views.at((size_t)s.args.at(i));
                        lb_tensor t = v.t;
                        t.ptr = (void*)v.offset;
                        return t;
                    };
                    const size_t bytes = s.scratch >= 0 ? lb::view_bytes(plan->views.at((size_t)s.scratch).t) : 0;
                    n += lb::gemm_launches(operand(0), operand(1), bytes, s.tuned_kernel, &s.tuning);
                    break;
                }
                case lb::ATTN_FWD: n += 1; break;
                case lb::ATTN_BWD: n += 3; break;  // delta, then dK/dV and dQ - or the single kernel and the rounding of dQ
                case lb::SCATTER_ADD: {
                    const lb_tensor &ids = plan->views.at((size_t)s.args.at(1)).t, &out = plan->views.at((size_t)s.args.at(3)).t;
                    long long tokens = 1;
                    for (int d = 0; d < ids.rank; d++) tokens *= ids.shape[d];
                    n += lb::scatter_add_launches(out.shape[0], tokens, s.epilogue != 0);
                    break;
                }
                case lb::TRANSPOSE: n += 1; break;
                case lb::COPY: n += lb::copy_form(plan->views.at((size_t)s.args.at(0)).t, plan->views.at((size_t)s.args.at(1)).t) == 2 ? 1 : 0; break;
                default: break;  // block and 2-d copies, fills, collectives and waits launch no kernel of this library
            }
        }
        n += products.queue(sms, false, nullptr);
    });
    return rc == LB_OK ? n : -1;
}

size_t lb_scatter_add_scratch_bytes(int64_t rows, int64_t width, int64_t updates, int deterministic) {
    return lb::scatter_add_scratch_bytes(rows, width, updates, deterministic != 0);
}

int lb_scatter_add_rows(const lb_tensor* x, const lb_tensor* ids, const lb_tensor* updates, const lb_tensor* out, void* scratch,
                        size_t scratch_bytes, int deterministic, void* stream) {
    return lb::guarded([&] {
        if (!ids || !updates || !out) lb::fail(LB_ERR_INVALID, "lb_scatter_add_rows: null argument");
        if (out->rank != 2) lb::fail(LB_ERR_UNSUPPORTED, "lb_scatter_add_rows: a [rows, width] result");
        long long tokens = 1;
        for (int d = 0; d < ids->rank; d++) tokens *= ids->shape[d];
        if (scratch_bytes < lb::scatter_add_scratch_bytes(out->shape[0], out->shape[1], tokens, deterministic != 0))
            lb::fail(LB_ERR_INVALID, "lb_scatter_add_rows: scratch smaller than lb_scatter_add_scratch_bytes");
        lb::scatter_add_rows(x ? *x : *out, *ids, *updates, *out, scratch, x == nullptr, deterministic != 0, stream);
    });
}

int lb_plan_run(const lb_plan* plan, void* workspace, void* const* inputs, int n_inputs, void* const* outputs, int n_outputs,
                int first_step, int last_step, void* stream) {
    return lb::guarded([&] {
        if (!plan) lb::fail(LB_ERR_INVALID, "lb_plan_run: null plan");
        if (n_inputs != plan->n_inputs || n_outputs != plan->n_outputs)
            lb::fail(LB_ERR_INVALID, lb::format("the plan takes %d inputs and %d outputs, got %d and %d", plan->n_inputs,
                                                plan->n_outputs, n_inputs, n_outputs));
        if (plan->workspace_bytes && (!workspace || ((uintptr_t)workspace & 255) != 0))
            lb::fail(LB_ERR_INVALID, "lb_plan_run: the workspace must be 256-byte aligned");
        lb::run(*plan, workspace, inputs, outputs, first_step, last_step < 0 ? (int)plan->steps.size() : last_step, stream);
    });
}
}
