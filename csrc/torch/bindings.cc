// Thin PyTorch layer: the communicator and its collectives over torch tensors on
// the current CUDA stream, buffer utilities, topology and tuning queries.
// The functional torch.ops.yali.* operators are registered from Python on top of
// these entry points (yali_b200/ops/registry.py).
//
// Parity: the reference has no framework layer (its README.md:199-203 lists the
// C++ headers as the only interface); this file is an addition.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <ATen/cuda/EmptyTensor.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include <memory>
#include <string>
#include <vector>

#include "comm/communicator.h"
#include "comm/topology.h"
#include "ops/buffer_ops.h"
#include "ops/fused_linear.h"
#include "ops/host_pipeline.h"
#include "ops/tuning.h"

namespace py = pybind11;
using namespace yali;

namespace {

Dtype ToDtype(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return Dtype::FP32;
        case at::kHalf: return Dtype::FP16;
        case at::kBFloat16: return Dtype::BF16;
        default: TORCH_CHECK(false, "yali: unsupported dtype ", t, " (fp32, fp16, bf16 only)");
    }
}

KernelMode ToMode(const std::string& s) {
    KernelMode m;
    TORCH_CHECK(ParseKernelMode(s.c_str(), &m), "yali: unknown kernel mode '", s, "'");
    return m;
}

void Throw(Result r, const std::string& what) {
    if (r == Result::Success) return;
    std::string msg = std::string("yali: ") + GetErrorString(r) + (what.empty() ? "" : ": " + what);
    if (r == Result::Timeout) throw std::runtime_error("YaliTimeout: " + msg);
    throw std::runtime_error(msg);
}

class PyComm {
   public:
    static std::shared_ptr<PyComm> SingleProcess(std::vector<int> devices, uint64_t heap_bytes, bool want_mc,
                                                 int64_t timeout_ms) {
        auto p = std::make_shared<PyComm>();
        CommOptions o;
        o.heap_bytes = heap_bytes;
        o.want_multicast = want_mc;
        o.timeout_ms = timeout_ms;
        std::string err;
        Throw(Communicator::CreateSingleProcess(devices, o, &p->c_, &err), err);
        return p;
    }
    static std::shared_ptr<PyComm> Emulated(int world, int device, uint64_t heap_bytes, int64_t timeout_ms) {
        auto p = std::make_shared<PyComm>();
        CommOptions o;
        o.heap_bytes = heap_bytes;
        o.want_multicast = false;
        o.timeout_ms = timeout_ms;
        std::string err;
        Throw(Communicator::CreateEmulated(world, device, o, &p->c_, &err), err);
        return p;
    }
    static std::shared_ptr<PyComm> FromEnv(int device, uint64_t heap_bytes, bool want_mc, int64_t timeout_ms) {
        auto p = std::make_shared<PyComm>();
        Result r = Result::Success;
        std::string err;
        std::unique_ptr<Bootstrap> bs;
        {
            py::gil_scoped_release nogil;
            bs = MakeEnvBootstrap(&r, &err);
        }
        if (!bs) Throw(r == Result::Success ? Result::BootstrapError : r, err);
        if (device < 0) {
            int ndev = 0;
            TORCH_CHECK(cudaGetDeviceCount(&ndev) == cudaSuccess && ndev > 0, "yali: no CUDA device");
            device = bs->local_rank() % ndev;
        }
        CommOptions o;
        o.heap_bytes = heap_bytes;
        o.want_multicast = want_mc;
        o.timeout_ms = timeout_ms;
        {
            py::gil_scoped_release nogil;
            r = Communicator::CreateMultiProcess(std::move(bs), device, o, &p->c_, &err);
        }
        Throw(r, err);
        return p;
    }

    void Close() {
        py::gil_scoped_release nogil;
        host_pipe_.reset();
        c_.reset();
    }
    Communicator& c() {
        TORCH_CHECK(c_ != nullptr, "yali: communicator is closed");
        return *c_;
    }

    int world() { return c().world(); }
    int nlocal() { return c().nlocal(); }
    int rank(int i) { return c().rank_of(i); }
    int device(int i) { return c().device_of(i); }
    bool emulated() { return c().emulated(); }
    bool has_multicast() { return c().has_multicast(); }
    std::string heap_kind() { return c().heap_kind(); }
    uint64_t launches() { return c().last_call().launches; }
    py::dict layout() {
        const HeapLayout& l = c().layout();
        py::dict d;
        d["total_bytes"] = l.total_bytes;
        d["flash_cap"] = l.flash_cap;
        d["ring_bytes"] = l.ring_bytes;
        d["nvls_cap"] = l.nvls_cap;
        d["gemm_cap"] = l.gemm_cap;
        d["user_bytes"] = l.user_bytes;
        return d;
    }
    py::dict last_call() {
        const LastCallInfo& l = c().last_call();
        py::dict d;
        d["variant"] = VariantName(l.variant);
        d["kernel"] = l.kernel;
        d["ctas"] = l.ctas;
        d["slot_bytes"] = l.slot_bytes;
        d["stages"] = l.stages;
        d["flags"] = l.flags;
        d["launches"] = l.launches;
        return d;
    }

    void SetTrace(bool on) { c().SetTrace(on); }
    // Device-side timeline of local rank `local_index`: (traced calls so far, [(start_ns, end_ns), ...])
    // for the most recent calls, oldest first.  Synchronise before reading.
    py::tuple ReadTrace(int local_index, int max_entries) {
        std::vector<uint64_t> buf(static_cast<size_t>(std::max(max_entries, 1)) * 2);
        uint64_t calls = 0;
        const int n = c().ReadTrace(local_index, buf.data(), max_entries, &calls);
        py::list out;
        for (int k = 0; k < n; ++k) out.append(py::make_tuple(buf[2 * k], buf[2 * k + 1]));
        return py::make_tuple(calls, out);
    }

    void CheckTensors(const std::vector<at::Tensor>& ts, const char* what, at::ScalarType* dt, int64_t* numel) {
        TORCH_CHECK(static_cast<int>(ts.size()) == c().nlocal(), "yali: expected ", c().nlocal(), " ", what,
                    " tensors (one per local rank), got ", ts.size());
        for (int i = 0; i < c().nlocal(); ++i) {
            const at::Tensor& t = ts[i];
            TORCH_CHECK(t.is_cuda(), "yali: ", what, "[", i, "] is not a CUDA tensor");
            TORCH_CHECK(t.is_contiguous(), "yali: ", what, "[", i, "] is not contiguous");
            TORCH_CHECK(t.get_device() == c().device_of(i), "yali: ", what, "[", i, "] lives on GPU ", t.get_device(),
                        ", rank ", c().rank_of(i), " owns GPU ", c().device_of(i));
            if (i == 0) {
                *dt = t.scalar_type();
                *numel = t.numel();
            } else {
                TORCH_CHECK(t.scalar_type() == *dt && t.numel() == *numel, "yali: ", what,
                            " tensors differ in dtype or size");
            }
        }
    }
    std::vector<cudaStream_t> Streams() {
        std::vector<cudaStream_t> s(c().nlocal());
        for (int i = 0; i < c().nlocal(); ++i) s[i] = at::cuda::getCurrentCUDAStream(c().device_of(i)).stream();
        return s;
    }

    void AllReduce(std::vector<at::Tensor> send, std::vector<at::Tensor> recv, const std::string& mode,
                   c10::optional<double> scale, int ctas, int slot_bytes, int skip_rank) {
        at::ScalarType sd, rd;
        int64_t sn, rn;
        CheckTensors(send, "send", &sd, &sn);
        CheckTensors(recv, "recv", &rd, &rn);
        TORCH_CHECK(sn == rn, "yali: send and recv differ in size");
        OpOptions o;
        o.mode = ToMode(mode);
        o.ctas = ctas;
        o.slot_bytes = slot_bytes;
        o.skip_rank = skip_rank;
        if (scale.has_value() || sd != rd) {
            o.epilogue = kEpiScaleCast;
            o.scale = static_cast<float>(scale.value_or(1.0));
        }
        std::vector<const void*> s(send.size());
        std::vector<void*> r(recv.size());
        for (size_t i = 0; i < send.size(); ++i) {
            s[i] = send[i].data_ptr();
            r[i] = recv[i].data_ptr();
        }
        auto st = Streams();
        c10::cuda::OptionalCUDAGuard guard(c().device_of(0));
        Result res = c().AllReduce(s.data(), r.data(), sn, ToDtype(sd), ToDtype(rd), o, st.data());
        Throw(res, c().last_error());
    }

    // ---- the calls a program makes, straight from Python objects ----
    // A collective argument is a tensor (one local rank) or a sequence of one tensor per local rank.  Everything from
    // here to the launch stays in C++ and allocates nothing but the outputs: for small messages the time per
    // call is the host's, and building lists, optionals and vectors of tensors for eight ranks took longer
    // than the kernel ran (28 us a call for the all-reduce + RMSNorm of 16 rows over eight ranks).
    struct Args {
        const at::Tensor* t[kMaxRanks];
        PyObject* obj[kMaxRanks];
        py::object held;  // a list made of another kind of sequence
        const at::Tensor& operator[](int i) const { return *t[i]; }
    };
    // False: `o` is None (where that is allowed).
    bool Read(PyObject* o, const char* what, Args* a, bool optional = false) {
        if (optional && o == Py_None) return false;
        const int n = c().nlocal();
        if (THPVariable_Check(o)) {
            if (n != 1)
                throw py::value_error(std::string(what) + ": this communicator drives " + std::to_string(n) +
                                      " ranks; pass one tensor per rank");
            a->obj[0] = o;
            a->t[0] = &THPVariable_Unpack(o);
            return true;
        }
        if (!PyList_Check(o) && !PyTuple_Check(o)) {
            a->held = py::reinterpret_steal<py::object>(PySequence_List(o));
            if (!a->held) throw py::error_already_set();
            o = a->held.ptr();
        }
        const Py_ssize_t len = PySequence_Fast_GET_SIZE(o);
        if (len != n)
            throw py::value_error(std::string(what) + ": expected " + std::to_string(n) + " tensors, got " + std::to_string(len));
        PyObject** items = PySequence_Fast_ITEMS(o);
        for (int i = 0; i < n; ++i) {
            TORCH_CHECK_TYPE(THPVariable_Check(items[i]), "yali: ", what, "[", i, "] is not a tensor");
            a->obj[i] = items[i];
            a->t[i] = &THPVariable_Unpack(items[i]);
        }
        return true;
    }
    void CheckArgs(const Args& a, const char* what, at::ScalarType* dt, int64_t* numel) {
        const int n = c().nlocal();
        for (int i = 0; i < n; ++i) {
            const at::Tensor& t = a[i];
            TORCH_CHECK(t.is_cuda(), "yali: ", what, "[", i, "] is not a CUDA tensor");
            TORCH_CHECK(t.is_contiguous(), "yali: ", what, "[", i, "] is not contiguous");
            TORCH_CHECK(t.get_device() == c().device_of(i), "yali: ", what, "[", i, "] lives on GPU ", t.get_device(),
                        ", rank ", c().rank_of(i), " owns GPU ", c().device_of(i));
            if (i == 0) {
                *dt = t.scalar_type();
                *numel = t.numel();
            } else {
                TORCH_CHECK(t.scalar_type() == *dt && t.numel() == *numel, "yali: ", what,
                            " tensors differ in dtype or size");
            }
        }
    }
    // The outputs of a call: the caller's, or new ones of this shape per local rank.
    static constexpr uint64_t kSharedOutputBytes = 4ull << 20;
    struct Outputs {
        Args a;
        at::Tensor fresh[kMaxRanks];
        bool given = false;
    };
    void Out(PyObject* o, const char* what, const Args& like, c10::IntArrayRef sizes, at::ScalarType dt, Outputs* r) {
        r->given = Read(o, what, &r->a, true);
        if (r->given) return;
        const int n = c().nlocal();
        // Several small outputs on one GPU are pieces of one allocation: a call of 8 ranks spent 6 of its 10.7 us on taking
        // and giving back eight blocks (16 x 4096 bf16).  Each tensor keeps the whole block alive, hence the limit: calls
        // whose outputs are larger take longer on the device than on the host.
        const uint64_t bytes = static_cast<uint64_t>(c10::multiply_integers(sizes)) * c10::elementSize(dt);
        const uint64_t piece = (bytes + 511) / 512 * 512;
        bool one_gpu = n > 1 && piece * n <= kSharedOutputBytes;
        for (int i = 0; i < n; ++i) one_gpu = one_gpu && like[i].is_cuda() && like[i].get_device() == like[0].get_device();
        if (one_gpu) {
            const at::TensorBase block =
                at::detail::empty_cuda({static_cast<int64_t>(piece * n)}, at::kByte, like[0].device(), c10::nullopt);
            for (int i = 0; i < n; ++i) {
                r->fresh[i] = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(block.storage()), c10::DispatchKeySet(c10::DispatchKey::CUDA),
                                                                       c10::scalarTypeToTypeMeta(dt));
                c10::TensorImpl* t = r->fresh[i].unsafeGetTensorImpl();
                t->set_storage_offset(static_cast<int64_t>(piece * i / c10::elementSize(dt)));
                t->set_sizes_contiguous(sizes);
                r->a.t[i] = &r->fresh[i];
            }
            return;
        }
        for (int i = 0; i < n; ++i) {
            if (like[i].is_cuda()) r->fresh[i] = at::Tensor(at::detail::empty_cuda(sizes, dt, like[i].device(), c10::nullopt));
            else r->fresh[i] = at::empty(sizes, like[i].options().dtype(dt));  // CheckArgs says what is wrong
            r->a.t[i] = &r->fresh[i];
        }
    }
    // What the Python call returns: a tensor where one was given, else a list.
    py::object Returned(PyObject* like, Outputs& r) {
        auto one = [&](int i) {
            if (r.given) return py::reinterpret_borrow<py::object>(r.a.obj[i]);
            return py::reinterpret_steal<py::object>(THPVariable_Wrap(std::move(r.fresh[i])));
        };
        if (THPVariable_Check(like)) return one(0);
        py::list l(c().nlocal());
        for (int i = 0; i < c().nlocal(); ++i) PyList_SET_ITEM(l.ptr(), i, one(i).release().ptr());
        return l;
    }
    struct StreamTable {
        cudaStream_t s[kMaxRanks];
    };
    StreamTable CurrentStreams() {
        StreamTable t;
        for (int i = 0; i < c().nlocal(); ++i)
            t.s[i] = i > 0 && c().device_of(i) == c().device_of(0)
                         ? t.s[0]
                         : at::cuda::getCurrentCUDAStream(c().device_of(i)).stream();
        return t;
    }
    // An argument that is no tensor; what does not convert is a TypeError, as for arguments that pybind11 converts.
    template <typename T>
    static T Cast(const py::object& o, const char* what) {
        try {
            return py::cast<T>(o);
        } catch (const py::cast_error&) {
            throw py::type_error(std::string(what) + ": cannot use an object of type " + Py_TYPE(o.ptr())->tp_name);
        }
    }
    static KernelMode ModeOf(const py::object& mode) {
        static PyObject* const auto_name = PyUnicode_InternFromString("auto");
        if (mode.ptr() == auto_name) return KernelMode::Auto;
        return ToMode(Cast<std::string>(mode, "mode"));
    }
    void Finish(Result r) {
        if (r != Result::Success) Throw(r, c().last_error());
    }

    py::object CallAllReduce(const py::object& send, const py::object& recv, const py::object& mode, const py::object& scale,
                             const py::object& out_dtype, int ctas, int slot_bytes, int skip_rank) {
        Args s;
        Outputs r;
        at::ScalarType sd, rd;
        int64_t sn, rn;
        Read(send.ptr(), "send", &s);
        // (Outputs of the caller's have a type already.)
        const at::ScalarType want = out_dtype.is_none() || !recv.is_none() ? s[0].scalar_type() : Cast<at::ScalarType>(out_dtype, "out_dtype");
        Out(recv.ptr(), "recv", s, s[0].sizes(), want, &r);
        CheckArgs(s, "send", &sd, &sn);
        CheckArgs(r.a, "recv", &rd, &rn);
        TORCH_CHECK(sn == rn, "yali: send and recv differ in size");
        OpOptions o;
        o.mode = ModeOf(mode);
        o.ctas = ctas;
        o.slot_bytes = slot_bytes;
        o.skip_rank = skip_rank;
        if (!scale.is_none() || sd != rd) {
            o.epilogue = kEpiScaleCast;
            o.scale = scale.is_none() ? 1.0f : static_cast<float>(Cast<double>(scale, "scale"));
        }
        const void* sp[kMaxRanks];
        void* rp[kMaxRanks];
        for (int i = 0; i < c().nlocal(); ++i) {
            sp[i] = s[i].data_ptr();
            rp[i] = r.a[i].data_ptr();
        }
        const StreamTable st = CurrentStreams();
        c10::cuda::OptionalCUDAGuard guard(c().device_of(0));
        Finish(c().AllReduce(sp, rp, sn, ToDtype(sd), ToDtype(rd), o, st.s));
        return Returned(send.ptr(), r);
    }

    py::object CallRmsNorm(const py::object& x, const py::object& weight, const py::object& residual, double eps,
                           const py::object& out, const py::object& residual_out, const py::object& mode, int ctas) {
        Args s, w, res, ro;
        Outputs r;
        at::ScalarType sd, rd, wd, d;
        int64_t sn, rn, wn, m;
        Read(x.ptr(), "x", &s);
        Read(weight.ptr(), "weight", &w);
        Out(out.ptr(), "out", s, s[0].sizes(), s[0].scalar_type(), &r);
        const bool has_res = Read(residual.ptr(), "residual", &res, true);
        const bool has_ro = Read(residual_out.ptr(), "residual_out", &ro, true);
        CheckArgs(s, "send", &sd, &sn);
        CheckArgs(r.a, "recv", &rd, &rn);
        CheckArgs(w, "weight", &wd, &wn);
        TORCH_CHECK(sd == rd && sd == wd && sn == rn, "yali: rmsnorm tensors must agree in dtype and size");
        TORCH_CHECK(wn > 0 && sn % wn == 0, "yali: input size is not a multiple of the hidden size");
        OpOptions o;
        o.mode = ModeOf(mode);
        o.ctas = ctas;
        o.epilogue = kEpiResidualRmsNorm;
        o.hidden = static_cast<int>(wn);
        o.eps = static_cast<float>(eps);
        const void *sp[kMaxRanks], *wp[kMaxRanks], *resp[kMaxRanks];
        void *rp[kMaxRanks], *rop[kMaxRanks];
        if (has_res) {
            CheckArgs(res, "residual", &d, &m);
            TORCH_CHECK(d == sd && m == sn, "yali: residual must match the input");
            o.residual = resp;
        }
        if (has_ro) {
            CheckArgs(ro, "residual_out", &d, &m);
            TORCH_CHECK(d == sd && m == sn, "yali: residual_out must match the input");
            o.residual_out = rop;
        }
        for (int i = 0; i < c().nlocal(); ++i) {
            sp[i] = s[i].data_ptr();
            rp[i] = r.a[i].data_ptr();
            wp[i] = w[i].data_ptr();
            if (has_res) resp[i] = res[i].data_ptr();
            if (has_ro) rop[i] = ro[i].data_ptr();
        }
        o.weight = wp;
        const StreamTable st = CurrentStreams();
        c10::cuda::OptionalCUDAGuard guard(c().device_of(0));
        Finish(c().AllReduce(sp, rp, sn, ToDtype(sd), ToDtype(rd), o, st.s));
        return Returned(x.ptr(), r);
    }

    // Reduce-scatter (rs): send is the full message, recv ShardElems(numel, world) elements per rank; all-gather: send is a
    // shard per rank, recv `count` elements.
    py::object CallHalf(const py::object& send, int64_t count, const py::object& recv, int ctas, int slot_bytes, bool rs) {
        Args s;
        Outputs r;
        at::ScalarType sd, rd;
        int64_t sn, rn;
        Read(send.ptr(), "send", &s);
        const int64_t full = rs ? s[0].numel() : count;
        TORCH_CHECK(full >= 0, "yali: count must not be negative, got ", full);
        const int64_t shard = c().world() > 1 ? static_cast<int64_t>(ShardElems(full, c().world())) : full;
        const int64_t size[1] = {rs ? shard : full};
        Out(recv.ptr(), "recv", s, c10::IntArrayRef(size, 1), s[0].scalar_type(), &r);
        CheckArgs(s, "send", &sd, &sn);
        CheckArgs(r.a, "recv", &rd, &rn);
        TORCH_CHECK(sd == rd, "yali: dtype mismatch");
        const int64_t owned = static_cast<int64_t>(ShardElems(rs ? sn : rn, c().world()));
        TORCH_CHECK((rs ? rn : sn) >= owned || c().world() == 1, "yali: ", rs ? "recv" : "send",
                    " needs shard_elems(count, world) elements");
        OpOptions o;
        o.ctas = ctas;
        o.slot_bytes = slot_bytes;
        const void* sp[kMaxRanks];
        void* rp[kMaxRanks];
        for (int i = 0; i < c().nlocal(); ++i) {
            sp[i] = s[i].data_ptr();
            rp[i] = r.a[i].data_ptr();
        }
        const StreamTable st = CurrentStreams();
        c10::cuda::OptionalCUDAGuard guard(c().device_of(0));
        Finish(rs ? c().ReduceScatter(sp, rp, sn, ToDtype(sd), o, st.s) : c().AllGather(sp, rp, rn, ToDtype(sd), o, st.s));
        return Returned(send.ptr(), r);
    }

    // out = RMSNorm(residual + sum_r x_r @ w_r^T) * norm_weight.
    py::object FusedLinear(const py::object& x, const py::object& w, const py::object& norm_weight, const py::object& out,
                           const py::object& residual, const py::object& residual_out, double eps, int force_oneshot,
                           int ctas, const py::object& trace, int nvls, int decode) {
        Args xa, wa, na, res, ro, ta;
        Outputs r;
        at::ScalarType d;
        int64_t n;
        Read(x.ptr(), "x", &xa);
        Read(w.ptr(), "w", &wa);
        Read(norm_weight.ptr(), "norm_weight", &na);
        TORCH_CHECK(xa[0].dim() == 2 && wa[0].dim() == 2, "yali: x [T,K], w [N,K], out [T,N]");
        const int64_t T = xa[0].size(0), K = xa[0].size(1), N = wa[0].size(0);
        const int64_t sizes[2] = {T, N};
        Out(out.ptr(), "out", xa, c10::IntArrayRef(sizes, 2), at::kBFloat16, &r);
        const bool has_res = Read(residual.ptr(), "residual", &res, true);
        const bool has_ro = Read(residual_out.ptr(), "residual_out", &ro, true);
        const std::pair<const Args*, const char*> all[] = {{&xa, "x"}, {&wa, "w"}, {&na, "norm_weight"}, {&r.a, "out"}};
        for (const auto& p : all) {
            CheckArgs(*p.first, p.second, &d, &n);
            TORCH_CHECK(d == at::kBFloat16, "yali: fused linear takes bf16 tensors");
        }
        TORCH_CHECK(r.a[0].dim() == 2, "yali: x [T,K], w [N,K], out [T,N]");
        TORCH_CHECK(wa[0].size(1) == K && r.a[0].size(0) == T && r.a[0].size(1) == N && na[0].numel() == N,
                    "yali: fused linear shape mismatch");
        const int nl = c().nlocal();
        FusedLinearDesc descs[kMaxRanks];
        for (int i = 0; i < nl; ++i) {
            descs[i].x = xa[i].data_ptr();
            descs[i].w = wa[i].data_ptr();
            descs[i].norm_weight = na[i].data_ptr();
            descs[i].out = r.a[i].data_ptr();
        }
        if (has_res) {
            CheckArgs(res, "residual", &d, &n);
            TORCH_CHECK(d == at::kBFloat16 && n == T * N, "yali: residual must be bf16 [T,N]");
            for (int i = 0; i < nl; ++i) descs[i].residual = res[i].data_ptr();
        }
        if (has_ro) {
            CheckArgs(ro, "residual_out", &d, &n);
            TORCH_CHECK(d == at::kBFloat16 && n == T * N, "yali: residual_out must be bf16 [T,N]");
            for (int i = 0; i < nl; ++i) descs[i].residual_out = ro[i].data_ptr();
        }
        FusedLinearOptions o;
        o.force_oneshot = force_oneshot;
        o.ctas = ctas;
        o.nvls = nvls;
        o.decode = decode;
        o.eps = static_cast<float>(eps);
        unsigned long long* tr[kMaxRanks] = {};
        if (Read(trace.ptr(), "trace", &ta, true)) {
            for (int i = 0; i < nl; ++i) {
                TORCH_CHECK(ta[i].scalar_type() == at::kLong && ta[i].numel() >= 8 && ta[i].is_cuda(),
                            "yali: trace tensors are int64 CUDA tensors with 8 elements");
                tr[i] = reinterpret_cast<unsigned long long*>(ta[i].data_ptr());
            }
            o.trace = tr;
        }
        const StreamTable st = CurrentStreams();
        c10::cuda::OptionalCUDAGuard guard(c().device_of(0));
        Finish(FusedLinearAllReduceRmsNorm(c(), descs, static_cast<uint32_t>(T), static_cast<uint32_t>(N),
                                           static_cast<uint32_t>(K), o, st.s));
        return Returned(x.ptr(), r);
    }

    // One tensor per local rank, at the same offset of every rank's heap.  The tensors alias
    // heap memory: they stay valid until the communicator is closed.
    std::vector<at::Tensor> SymmEmpty(std::vector<int64_t> shape, at::ScalarType dtype) {
        int64_t n = 1;
        for (int64_t d : shape) n *= d;
        std::vector<void*> ptrs;
        Throw(c().SymmAlloc(static_cast<uint64_t>(n) * c10::elementSize(dtype), &ptrs), c().last_error());
        std::vector<at::Tensor> out;
        for (int i = 0; i < c().nlocal(); ++i) {
            auto opts = at::TensorOptions().dtype(dtype).device(at::kCUDA, c().device_of(i));
            out.push_back(at::from_blob(ptrs[i], shape, [](void*) {}, opts));
        }
        return out;
    }
    void SymmReset() {
        if (host_pipe_) host_pipe_->Invalidate();
        c().SymmReset();
    }

    // dst = scale * sum over ranks of src, both in pinned host memory; copies and all-reduce
    // overlap chunk by chunk (ops/host_pipeline.h).
    void AllReduceHost(const py::object& src, const py::object& dst, int64_t chunk_bytes, const py::object& scale,
                       const py::object& mode, bool copies_only) {
        const int nl = c().nlocal();
        Args sa, da;
        Read(src.ptr(), "src", &sa);
        Read(dst.ptr(), "dst", &da);
        const at::ScalarType d = sa[0].scalar_type();
        const int64_t n = sa[0].numel();
        const void* s[kMaxRanks];
        void* r[kMaxRanks];
        for (int i = 0; i < nl; ++i) {
            for (const at::Tensor* t : {&sa[i], &da[i]}) {
                if (t->is_cuda() || !t->is_contiguous() || !t->is_pinned())
                    throw py::value_error("all_reduce_host takes contiguous tensors in pinned host memory");
                TORCH_CHECK(t->scalar_type() == d && t->numel() == n, "yali: src and dst must agree in size and dtype");
            }
            s[i] = sa[i].data_ptr();
            r[i] = da[i].data_ptr();
        }
        OpOptions o;
        o.mode = ModeOf(mode);
        if (!scale.is_none()) {
            o.epilogue = kEpiScaleCast;
            o.scale = static_cast<float>(Cast<double>(scale, "scale"));
        }
        if (!host_pipe_) host_pipe_ = std::make_unique<HostPipeline>(c());
        const StreamTable st = CurrentStreams();
        c10::cuda::OptionalCUDAGuard guard(c().device_of(0));
        Finish(host_pipe_->AllReduce(s, r, static_cast<uint64_t>(n), ToDtype(d), o,
                                     static_cast<uint64_t>(chunk_bytes <= 0 ? 0 : std::max<int64_t>(chunk_bytes, 4096)), st.s,
                                     copies_only));
    }

    void Sync() {
        auto st = Streams();
        Result r;
        {
            py::gil_scoped_release nogil;
            r = c().Sync(st.data());
        }
        Throw(r, c().last_error());
    }
    void Check() { Throw(c().Check(), c().last_error()); }
    void Reset() {
        Result r;
        {
            py::gil_scoped_release nogil;
            r = c().Reset();
        }
        Throw(r, c().last_error());
    }
    void Barrier() {
        Result r;
        {
            py::gil_scoped_release nogil;
            r = c().Barrier();
        }
        Throw(r, c().last_error());
    }
    std::string Status() { return c().DescribeStatus(); }

    // Host-side collectives over the control plane (small Python objects, test plumbing).
    py::bytes AllgatherBytes(const std::string& mine) {
        Bootstrap* bs = c().bootstrap();
        if (!bs) return py::bytes(mine);
        std::string out(mine.size() * bs->world(), '\0');
        Result r;
        {
            py::gil_scoped_release nogil;
            r = bs->allgather(mine.data(), &out[0], mine.size());
        }
        Throw(r, bs->last_error());
        return py::bytes(out);
    }

    std::unique_ptr<Communicator> c_;
    std::unique_ptr<HostPipeline> host_pipe_;
};

void FillRandomT(at::Tensor t, int dist, uint64_t seed) {
    TORCH_CHECK(t.is_cuda() && t.is_contiguous(), "yali: fill_random needs a contiguous CUDA tensor");
    c10::cuda::CUDAGuard g(t.device());
    cudaError_t e = FillRandom(t.data_ptr(), t.numel(), ToDtype(t.scalar_type()), dist, seed,
                               at::cuda::getCurrentCUDAStream().stream());
    TORCH_CHECK(e == cudaSuccess, "yali: fill_random: ", cudaGetErrorString(e));
}

void FillConstantT(at::Tensor t, double v) {
    TORCH_CHECK(t.is_cuda() && t.is_contiguous(), "yali: fill_constant needs a contiguous CUDA tensor");
    c10::cuda::CUDAGuard g(t.device());
    cudaError_t e = FillConstant(t.data_ptr(), t.numel(), ToDtype(t.scalar_type()), static_cast<float>(v),
                                 at::cuda::getCurrentCUDAStream().stream());
    TORCH_CHECK(e == cudaSuccess, "yali: fill_constant: ", cudaGetErrorString(e));
}

py::dict ValidateSumT(at::Tensor out, at::ScalarType in_dtype, int dist, uint64_t seed_base, int world, double scale,
                      c10::optional<double> rtol, c10::optional<double> atol, uint64_t index_offset) {
    TORCH_CHECK(out.is_cuda() && out.is_contiguous(), "yali: validate_sum needs a contiguous CUDA tensor");
    c10::cuda::CUDAGuard g(out.device());
    double rt, at_;
    DefaultTolerance(ToDtype(out.scalar_type()), world, &rt, &at_);
    if (std::fabs(scale) > 1.0) at_ *= std::fabs(scale);
    if (rtol.has_value()) rt = *rtol;
    if (atol.has_value()) at_ = *atol;
    ValidateReport h = {0ull, ~0ull, 0.0};
    ValidateReport* d = nullptr;
    TORCH_CHECK(cudaMalloc(reinterpret_cast<void**>(&d), sizeof(h)) == cudaSuccess, "yali: cudaMalloc failed");
    cudaStream_t s = at::cuda::getCurrentCUDAStream().stream();
    cudaMemcpyAsync(d, &h, sizeof(h), cudaMemcpyHostToDevice, s);
    cudaError_t e = ValidateSumAsync(out.data_ptr(), out.numel(), index_offset, ToDtype(in_dtype),
                                     ToDtype(out.scalar_type()), dist, seed_base, world, static_cast<float>(scale), rt,
                                     at_, d, s);
    cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, s);
    cudaError_t e2 = cudaStreamSynchronize(s);
    cudaFree(d);
    TORCH_CHECK(e == cudaSuccess && e2 == cudaSuccess, "yali: validate_sum failed: ",
                cudaGetErrorString(e != cudaSuccess ? e : e2));
    py::dict r;
    r["mismatches"] = h.mismatches;
    r["first_mismatch"] = h.mismatches ? py::cast(h.first_mismatch) : py::none();
    r["max_abs_err"] = h.max_abs_err;
    r["rtol"] = rt;
    r["atol"] = at_;
    return r;
}

py::dict TopologyDict() {
    TopologyInfo t = QueryTopology();
    py::dict d;
    d["device_count"] = t.device_count;
    d["all_pairs_connected"] = t.AllPairsConnected();
    d["connected_pairs"] = t.ConnectedPairs();
    py::list mc, fab, names;
    for (int i = 0; i < t.device_count; ++i) {
        mc.append(static_cast<bool>(t.multicast_supported[i]));
        fab.append(static_cast<bool>(t.fabric_handle_supported[i]));
        names.append(t.names[i]);
    }
    d["multicast_supported"] = mc;
    d["fabric_handle_supported"] = fab;
    d["names"] = names;
    return d;
}

}  // namespace

PYBIND11_MODULE(_C, m) {
    m.doc() = "yali_b200 native bindings";
    py::class_<PyComm, std::shared_ptr<PyComm>>(m, "Comm")
        .def_static("single_process", &PyComm::SingleProcess, py::arg("devices"), py::arg("heap_bytes") = 0,
                    py::arg("want_multicast") = true, py::arg("timeout_ms") = -1)
        .def_static("emulated", &PyComm::Emulated, py::arg("world"), py::arg("device") = 0, py::arg("heap_bytes") = 0,
                    py::arg("timeout_ms") = -1)
        .def_static("from_env", &PyComm::FromEnv, py::arg("device") = -1, py::arg("heap_bytes") = 0,
                    py::arg("want_multicast") = true, py::arg("timeout_ms") = -1)
        .def("close", &PyComm::Close)
        .def_property_readonly("world", &PyComm::world)
        .def_property_readonly("nlocal", &PyComm::nlocal)
        .def("rank", &PyComm::rank, py::arg("local_index") = 0)
        .def("device", &PyComm::device, py::arg("local_index") = 0)
        .def_property_readonly("is_emulated", &PyComm::emulated)
        .def_property_readonly("has_multicast", &PyComm::has_multicast)
        .def_property_readonly("heap_kind", &PyComm::heap_kind)
        .def_property_readonly("launches", &PyComm::launches)
        .def("layout", &PyComm::layout)
        .def("last_call", &PyComm::last_call)
        .def("set_trace", &PyComm::SetTrace, py::arg("on"))
        .def("read_trace", &PyComm::ReadTrace, py::arg("local_index") = 0, py::arg("max_entries") = 4096)
        .def("all_reduce", &PyComm::AllReduce, py::arg("send"), py::arg("recv"), py::arg("mode") = "auto",
             py::arg("scale") = py::none(), py::arg("ctas") = 0, py::arg("slot_bytes") = 0, py::arg("skip_rank") = -1)
        .def("call_all_reduce", &PyComm::CallAllReduce)
        .def("call_all_reduce_rmsnorm", &PyComm::CallRmsNorm)
        .def("call_half", &PyComm::CallHalf)
        .def("fused_linear", &PyComm::FusedLinear)
        .def("symm_empty", &PyComm::SymmEmpty, py::arg("shape"), py::arg("dtype"))
        .def("symm_reset", &PyComm::SymmReset)
        .def("all_reduce_host", &PyComm::AllReduceHost, py::arg("src"), py::arg("dst"), py::arg("chunk_bytes") = 0,
             py::arg("scale") = py::none(), py::arg("mode") = "auto", py::arg("copies_only") = false)
        .def("sync", &PyComm::Sync)
        .def("check", &PyComm::Check)
        .def("reset", &PyComm::Reset)
        .def("barrier", &PyComm::Barrier)
        .def("status", &PyComm::Status)
        .def("allgather_bytes", &PyComm::AllgatherBytes)
        .def("raw", [](PyComm& p) { return reinterpret_cast<uintptr_t>(&p.c()); });

    m.def("fill_random", &FillRandomT, py::arg("tensor"), py::arg("dist"), py::arg("seed"));
    m.def("fill_constant", &FillConstantT, py::arg("tensor"), py::arg("value"));
    m.def("validate_sum", &ValidateSumT, py::arg("out"), py::arg("in_dtype"), py::arg("dist"), py::arg("seed_base"),
          py::arg("world"), py::arg("scale") = 1.0, py::arg("rtol") = py::none(), py::arg("atol") = py::none(),
          py::arg("index_offset") = 0);
    m.def("topology", &TopologyDict);
    m.def("shard_elems", [](uint64_t count, int world) { return ShardElems(count, world); });
}
