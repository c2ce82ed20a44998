// The call path between Python and the C ABI: one native function per entry point that a training or serving loop calls
// every step. capi.py and host.py keep the signatures, the documentation and the checks of set-up calls; what a step pays
// for is here. For a small tensor the host, not the GPU, is what bounds a call: the same call through ctypes spent 8 us on
// attribute look-ups of its tensors, argument conversions and torch.cuda.current_stream(), against 2.4 us of GPU time for
// batch norm + ReLU of one 64x32x32 image. Reading the tensors' addresses and extents from the objects themselves and the
// stream from c10 costs a few tens of nanoseconds.
//
// The interpreter's lock is released around every call into the library, as ctypes does: a launch can block while the
// stream's queue is full, and other threads keep enqueueing on theirs. torch's functions throw (no usable device, a tensor without
// storage), and so may an allocation: every function of the module runs inside guarded(), which makes a Python error of it.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <c10/cuda/CUDAStream.h>

#include "../../../include/nnf_b200.h"

#include <vector>

extern "C"
{
	// the flat interface of the layer objects (host/nnf_layers.cpp)
	const char * nnfh_last_error(void);
	int nnfh_tester_forward(void *, void *, void *, const void * const *, int, const void * const *, int, unsigned int);
	int nnfh_updater_forward(void *, void *, void *, const void * const *, int, const void * const *, int, void *, size_t, void *, void *, unsigned int);
	int nnfh_forward(void *, void *, void * const *, int, const void * const *, int, const void * const *, int, void *, size_t, void *, void *, unsigned int);
	int nnfh_backward_data(void *, void *, unsigned int, void *, const void *, const void * const *, int, const void * const *, int, const void *, const void *,
		const void *, int, unsigned int);
	int nnfh_backward_weights(void *, void *, void * const *, int, const void * const *, int, const void *, void *, size_t, unsigned int);
	int nnfh_backward_data_and_weights(void *, void *, void * const *, int, const void *, void * const *, int, const void * const *, int,
		const void * const *, int, const void *, void *, size_t, void *, int, unsigned int);
}

namespace
{
	PyObject * g_error_type = nullptr;   // capi.NnfError
	PyObject * g_act_type = nullptr, * g_pool_type = nullptr;   // capi.Act, capi.Pool
	PyObject * ctypes_type(const nnf_act&) { return g_act_type; }
	PyObject * ctypes_type(const nnf_pool&) { return g_pool_type; }

	struct extents
	{
		int64_t n = 0, c = 0, h = 1, w = 1, hw = 1;
	};

	// a reference that is given back however the scope is left
	struct owned
	{
		PyObject * object;
		~owned() { Py_XDECREF(object); }
	};

	// Reads the positional arguments of one call in order. The first conversion that fails leaves its exception set, and
	// the rest of the reads return zeros without looking at their argument: nothing may call into Python, or clear an exception,
	// while one is set.
	class arguments
	{
	public:
		// `streamed`: the last argument is the stream. It is read before the others, as a caller without a device hears of that
		// before it hears of anything else.
		arguments(PyObject * const * a, Py_ssize_t n, bool streamed) : a(a), n(n)
		{
			if (streamed && n > 0)
				read_stream(a[n - 1]);
		}

		bool ok() const { return good; }

		PyObject * next()
		{
			if (i >= n)
				fail(PyExc_TypeError, "missing argument");
			return good ? a[i++] : Py_None;
		}

		// a tensor's address (None: null; an int: itself)
		template <bool CHECKED = true>
		void * address_of(PyObject * o)
		{
			if (!good || o == Py_None)
				return nullptr;
			if (THPVariable_Check(o))
			{
				const at::Tensor& t = THPVariable_Unpack(o);
				if (CHECKED && !(t.is_cuda() && t.is_contiguous()))
					fail(PyExc_AssertionError, "tensors must be contiguous CUDA tensors");
				return good ? t.data_ptr() : nullptr;
			}
			if (CHECKED && PyLong_Check(o))
				return address_in(o);
			// an object that answers as a tensor does (storage, a wrapper)
			if (CHECKED && !(truth(member(o, "is_cuda")) && truth(result(o, "is_contiguous"))))
				fail(PyExc_AssertionError, "tensors must be contiguous CUDA tensors");
			const owned p{good ? result(o, "data_ptr") : nullptr};
			return p.object && p.object != Py_None ? address_in(p.object) : nullptr;
		}
		float * ptr() { return static_cast<float *>(address_of(next())); }
		void * raw() { return address_of(next()); }
		void * loose() { return address_of<false>(next()); }

		// the number of elements of a tensor
		int64_t numel(PyObject * o)
		{
			if (!good || THPVariable_Check(o))
				return good ? THPVariable_Unpack(o).numel() : 0;
			return count(result(o, "numel"));
		}

		// a tensor's address and its extents [n][c][h...][w]
		float * ptr(extents& e, bool planes = false)
		{
			PyObject * o = next();
			float * p = static_cast<float *>(address_of(o));
			if (!good)
				return nullptr;
			if (THPVariable_Check(o))
			{
				const auto s = THPVariable_Unpack(o).sizes();
				set_extents(e, s.data(), s.size(), planes);
				return p;
			}
			std::vector<int64_t> s;
			const owned shape{member(o, "shape")};
			sequence(shape.object, [&](PyObject * d) { s.push_back(PyLong_AsLongLong(d)); good = !PyErr_Occurred(); });
			set_extents(e, s.data(), s.size(), planes);
			return p;
		}

		void set_extents(extents& e, const int64_t * s, size_t dims, bool planes)
		{
			if (planes && dims != 4)
				fail(PyExc_ValueError, "a tensor [n][c][h][w] is expected");
			else if (dims < 2)
				fail(PyExc_IndexError, "a tensor [n][c][...] is expected");
			if (!good)
				return;
			e.n = s[0];
			e.c = s[1];
			for (size_t d = 2; d < dims; ++d)
				e.hw *= s[d];
			if (planes)
			{
				e.h = s[2];
				e.w = s[3];
			}
		}

		// a working buffer and its size in bytes (None: none of 0 bytes)
		template <bool CHECKED = true>
		void * buffer(size_t& bytes)
		{
			PyObject * o = next();
			bytes = 0;
			void * p = address_of<CHECKED>(o);
			if (!good || o == Py_None)
				return p;
			if (THPVariable_Check(o))
				bytes = THPVariable_Unpack(o).nbytes();
			else if (!PyLong_Check(o))
				bytes = size_t(count(result(o, "numel")) * count(result(o, "element_size")));
			return p;
		}

		double number()
		{
			return number(next());
		}

		double number(PyObject * o)
		{
			if (!good)
				return 0.0;
			const double v = PyFloat_CheckExact(o) ? PyFloat_AS_DOUBLE(o) : PyFloat_AsDouble(o);
			if (v == -1.0 && PyErr_Occurred())
				good = false;
			return v;
		}

		long long integer()
		{
			PyObject * o = next();
			const long long v = good ? PyLong_AsLongLong(o) : 0;
			if (v == -1 && PyErr_Occurred())
				good = false;
			return v;
		}

		int flag()
		{
			PyObject * o = next();
			const int v = good ? PyObject_IsTrue(o) : 0;
			if (v < 0)
				good = false;
			return v;
		}

		void * handle()
		{
			PyObject * o = next();
			if (o == Py_None)
				return nullptr;
			void * p = PyLong_AsVoidPtr(o);
			if (p == nullptr && PyErr_Occurred())
				good = false;
			return p;
		}

		nnf_stream_t stream()
		{
			next();
			return given_stream;
		}

		// the fields of one ctypes structure: an object of the type itself, as other bytes of its size may hold any address
		template <class T>
		void structure(PyObject * o, T& out)
		{
			if (!good)
				return;
			PyObject * const type = ctypes_type(out);
			const int is = type ? PyObject_IsInstance(o, type) : 0;
			if (is == 0)
				fail(PyExc_TypeError, "an activation (Act) or a pooling geometry (Pool) is expected");
			Py_buffer b;
			if (is <= 0 || PyObject_GetBuffer(o, &b, PyBUF_SIMPLE) != 0)
			{
				good = false;
				return;
			}
			if (b.len == (Py_ssize_t)sizeof(T))
				memcpy(&out, b.buf, sizeof(T));
			else
				fail(PyExc_TypeError, "a structure of another size");
			PyBuffer_Release(&b);
		}

		// an activation chain of any length (the library refuses those that are too long)
		std::vector<nnf_act>& acts()
		{
			PyObject * o = next();
			chain.clear();
			if (o == Py_None)
				return chain;
			sequence(o, [&](PyObject * item) { nnf_act a = {}; structure(item, a); chain.push_back(a); });
			return chain;
		}

		template <bool CHECKED>
		void addresses(std::vector<void *>& out)
		{
			PyObject * o = next();
			out.clear();
			if (o != Py_None)
				sequence(o, [&](PyObject * item) { out.push_back(address_of<CHECKED>(item)); });
		}

		template <class F>
		void sequence(PyObject * o, F f)
		{
			const owned s{good ? PySequence_Fast(o, "a sequence is expected") : nullptr};
			if (!s.object)
			{
				good = false;
				return;
			}
			for (Py_ssize_t k = 0; k < PySequence_Fast_GET_SIZE(s.object) && good; ++k)
				f(PySequence_Fast_GET_ITEM(s.object, k));
		}

		void fail(PyObject * type, const char * text)
		{
			if (good && type)   // null: the exception is set already
				PyErr_SetString(type, text);
			good = false;
		}

	private:
		void * address_in(PyObject * number)
		{
			void * p = PyLong_AsVoidPtr(number);
			if (p == nullptr && PyErr_Occurred())
				good = false;
			return p;
		}

		PyObject * member(PyObject * o, const char * name)
		{
			PyObject * v = good ? PyObject_GetAttrString(o, name) : nullptr;
			good = v != nullptr;
			return v;
		}

		PyObject * result(PyObject * o, const char * name)
		{
			PyObject * v = good ? PyObject_CallMethod(o, name, nullptr) : nullptr;
			good = v != nullptr;
			return v;
		}

		// take the reference that they are given
		bool truth(PyObject * o)
		{
			const owned v{o};
			const int t = v.object ? PyObject_IsTrue(v.object) : 0;
			good = good && t >= 0;
			return t > 0;
		}

		long long count(PyObject * o)
		{
			const owned v{o};
			const long long n = v.object ? PyLong_AsLongLong(v.object) : 0;
			good = good && !(n == -1 && PyErr_Occurred());
			return n;
		}

		// torch's current stream unless one is given (an object with a cuda_stream, or the stream's address)
		void read_stream(PyObject * o)
		{
			if (o == Py_None)
			{
				given_stream = (nnf_stream_t)c10::cuda::getCurrentCUDAStream().stream();
				return;
			}
			PyObject * v = PyObject_GetAttrString(o, "cuda_stream");
			if (!v && PyErr_ExceptionMatches(PyExc_AttributeError))
			{
				PyErr_Clear();
				v = PyNumber_Long(o);
			}
			given_stream = v ? (nnf_stream_t)PyLong_AsVoidPtr(v) : nullptr;
			Py_XDECREF(v);
			good = !PyErr_Occurred();
		}

		PyObject * const * a;
		Py_ssize_t n, i = 0;
		bool good = true;
		nnf_stream_t given_stream = nullptr;
		std::vector<nnf_act> chain;
	};

	// runs f without the interpreter's lock, which is taken again if f throws, too
	template <class F>
	int without_lock(F f)
	{
		int status;
		PyThreadState * const state = PyEval_SaveThread();
		try
		{
			status = f();
		}
		catch (const std::exception&)
		{
			PyEval_RestoreThread(state);
			throw;
		}
		PyEval_RestoreThread(state);
		return status;
	}

	// (what is no std::exception is none of torch's or the library's: the unwinding of a thread that is being ended passes through)
	template <PyObject * (*F)(PyObject *, PyObject * const *, Py_ssize_t)>
	PyObject * guarded(PyObject * self, PyObject * const * args, Py_ssize_t nargs)
	{
		try
		{
			return F(self, args, nargs);
		}
		catch (const std::exception&)
		{
			PyErr_Clear();   // an exception is translated with none set
			torch::translate_exception_to_python(std::current_exception());
		}
		return nullptr;
	}

	// calls the library without the interpreter's lock; a status raises NnfError with the library's text
	template <class F>
	PyObject * call(const arguments& a, F f)
	{
		if (!a.ok())
			return nullptr;
		const int status = without_lock(f);
		if (status == 0)
			Py_RETURN_NONE;
		PyObject * e = PyObject_CallFunction(g_error_type ? g_error_type : PyExc_RuntimeError, "is", status, nnf_last_error_string());
		if (e)
		{
			PyErr_SetObject((PyObject *)Py_TYPE(e), e);
			Py_DECREF(e);
		}
		return nullptr;
	}

	// the same for the layer objects, whose errors host.py raises
	template <class F>
	PyObject * call_object(const arguments& a, F f)
	{
		if (!a.ok())
			return nullptr;
		const nnf_stream_t stream = (nnf_stream_t)c10::cuda::getCurrentCUDAStream().stream();
		const int status = without_lock([&] { return f(stream); });
		return PyLong_FromLong(status);
	}

	#define NNF_NATIVE(name) PyObject * name(PyObject *, PyObject * const * args, Py_ssize_t nargs)
	#define NNF_READ arguments a(args, nargs, true)
	#define NNF_READ_OBJECT arguments a(args, nargs, false)   // the layer objects run on torch's current stream

	// (gamma, beta, mean, invsigma) or None
	struct bn_arrays
	{
		const float * gamma = nullptr, * beta = nullptr, * mean = nullptr, * invsigma = nullptr;

		explicit bn_arrays(arguments& a)
		{
			PyObject * o = a.next();
			if (o == Py_None)
				return;
			const float * p[4] = {};
			int k = 0;
			a.sequence(o, [&](PyObject * item) { const float * v = static_cast<const float *>(a.address_of(item)); if (k < 4) p[k] = v; ++k; });
			if (k != 4)
				a.fail(PyExc_ValueError, "batch norm takes (gamma, beta, mean, invsigma)");
			gamma = p[0]; beta = p[1]; mean = p[2]; invsigma = p[3];
		}
	};

	NNF_NATIVE(bn_infer_act)   // y, x, bias, bn, residual, add_alpha, acts, stream
	{
		NNF_READ;
		extents e;
		float * y = a.ptr();
		const float * x = a.ptr(e), * bias = a.ptr();
		const bn_arrays bn(a);
		const float * residual = a.ptr();
		const float alpha = (float)a.number();
		const auto& acts = a.acts();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return !bias ? nnf_bn_infer_act(s, y, x, bn.gamma, bn.beta, bn.mean, bn.invsigma, residual, alpha, acts.data(), (int)acts.size(), e.n, e.c, e.hw)
			: nnf_bias_bn_infer_act(s, y, x, bias, bn.gamma, bn.beta, bn.mean, bn.invsigma, residual, alpha, acts.data(), (int)acts.size(), e.n, e.c, e.hw); });
	}

	NNF_NATIVE(act_fwd)   // y, x, act, stream
	{
		NNF_READ;
		extents e;
		nnf_act act = {};
		float * y = a.ptr();
		const float * x = a.ptr(e);
		a.structure(a.next(), act);
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_act_fwd(s, y, x, &act, e.n, e.c, e.hw); });
	}

	NNF_NATIVE(act_bwd)   // dx, dy, neurons, act, add_to_destination, stream
	{
		NNF_READ;
		extents e;
		nnf_act act = {};
		float * dx = a.ptr();
		const float * dy = a.ptr(e), * neurons = a.ptr();
		a.structure(a.next(), act);
		const int add = a.flag();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_act_bwd(s, dx, dy, neurons, &act, e.n, e.c, e.hw, add); });
	}

	NNF_NATIVE(prelu_bwd_weights)   // dslope, dy, x, workspace, stream
	{
		NNF_READ;
		extents e;
		float * dslope = a.ptr();
		const float * dy = a.ptr(), * x = a.ptr(e);
		size_t bytes;
		void * ws = a.buffer(bytes);
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_prelu_bwd_weights(s, dslope, dy, x, e.n, e.c, e.hw, ws, bytes); });
	}

	NNF_NATIVE(add_fwd)   // y, inputs, alpha, stream
	{
		NNF_READ;
		PyObject * const t = a.next();
		float * y = static_cast<float *>(a.address_of(t));
		const int64_t count = a.numel(t);
		std::vector<void *> in;
		a.addresses<true>(in);
		const float alpha = (float)a.number();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_add_fwd(s, y, (const float * const *)in.data(), (int)in.size(), alpha, count); });
	}

	NNF_NATIVE(add_bwd)   // dx, dy, alpha, add_to_destination, stream
	{
		NNF_READ;
		float * dx = a.ptr();
		PyObject * const t = a.next();
		const float * dy = static_cast<const float *>(a.address_of(t));
		const int64_t count = a.numel(t);
		const float alpha = (float)a.number();
		const int add = a.flag();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_add_bwd(s, dx, dy, alpha, count, add); });
	}

	NNF_NATIVE(softmax_fwd)   // y, x, stream
	{
		NNF_READ;
		extents e;
		float * y = a.ptr();
		const float * x = a.ptr(e);
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_softmax_fwd(s, y, x, e.n, e.c, e.hw); });
	}

	NNF_NATIVE(softmax_bwd)   // dx, dy, y, add_to_destination, stream
	{
		NNF_READ;
		extents e;
		float * dx = a.ptr();
		const float * dy = a.ptr(), * y = a.ptr(e);
		const int add = a.flag();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_softmax_bwd(s, dx, dy, y, e.n, e.c, e.hw, add); });
	}

	NNF_NATIVE(maxpool_fwd)   // y, argmax, x, pool, stream
	{
		NNF_READ;
		extents e;
		nnf_pool pool = {};
		float * y = a.ptr();
		uint32_t * argmax = static_cast<uint32_t *>(a.raw());
		const float * x = a.ptr(e, true);
		a.structure(a.next(), pool);
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_maxpool_fwd(s, y, argmax, x, e.n, e.c, e.h, e.w, &pool); });
	}

	NNF_NATIVE(maxpool_bwd)   // dx, dy, argmax, pool, add_to_destination, stream
	{
		NNF_READ;
		extents e;
		nnf_pool pool = {};
		float * dx = a.ptr(e, true);
		const float * dy = a.ptr();
		const uint32_t * argmax = static_cast<const uint32_t *>(a.raw());
		a.structure(a.next(), pool);
		const int add = a.flag();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_maxpool_bwd(s, dx, dy, argmax, e.n, e.c, e.h, e.w, &pool, add); });
	}

	NNF_NATIVE(bn_add_relu_maxpool_fwd)   // z, pooled, argmax, x, residual, bn, relu_slope, pool, stream
	{
		NNF_READ;
		extents e;
		nnf_pool pool = {};
		float * z = a.ptr(), * pooled = a.ptr();
		uint32_t * argmax = static_cast<uint32_t *>(a.raw());
		const float * x = a.ptr(e, true), * residual = a.ptr();
		const bn_arrays bn(a);
		const float slope = (float)a.number();
		a.structure(a.next(), pool);
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_bn_add_relu_maxpool_fwd(s, z, pooled, argmax, x, residual, bn.gamma, bn.beta, bn.mean, bn.invsigma, slope, e.n, e.c, e.h, e.w, &pool); });
	}

	NNF_NATIVE(bn_add_relu_maxpool_bwd)   // dx, dresidual, dpooled, argmax, z, gamma, invsigma, relu_slope, pool, stream
	{
		NNF_READ;
		extents e;
		nnf_pool pool = {};
		float * dx = a.ptr(), * dresidual = a.ptr();
		const float * dpooled = a.ptr();
		const uint32_t * argmax = static_cast<const uint32_t *>(a.raw());
		const float * z = a.ptr(e, true), * gamma = a.ptr(), * invsigma = a.ptr();
		const float slope = (float)a.number();
		a.structure(a.next(), pool);
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_bn_add_relu_maxpool_bwd(s, dx, dresidual, dpooled, argmax, z, gamma, invsigma, slope, e.n, e.c, e.h, e.w, &pool); });
	}

	NNF_NATIVE(bn_train_stats)   // sums, x, workspace, stream
	{
		NNF_READ;
		extents e;
		float * sums = a.ptr();
		const float * x = a.ptr(e);
		size_t bytes;
		void * ws = a.buffer(bytes);
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_bn_train_stats(s, sums, x, e.n, e.c, e.hw, ws, bytes); });
	}

	NNF_NATIVE(bn_train_stats_static)   // sums, x, stream
	{
		NNF_READ;
		extents e;
		float * sums = a.ptr();
		const float * x = a.ptr(e);
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_bn_train_stats_static(s, sums, x, e.n, e.c, e.hw); });
	}

	NNF_NATIVE(bn_train_apply_act)   // y, saved, x, gamma, beta, sums, count_total, eps, acts, stream
	{
		NNF_READ;
		extents e;
		float * y = a.ptr(), * saved = a.ptr();
		const float * x = a.ptr(e), * gamma = a.ptr(), * beta = a.ptr(), * sums = a.ptr();
		const double count = a.number();
		const float eps = (float)a.number();
		const auto& acts = a.acts();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_bn_train_apply_act(s, y, saved, x, gamma, beta, sums, count, eps, acts.data(), (int)acts.size(), e.n, e.c, e.hw); });
	}

	NNF_NATIVE(bn_train_fwd)   // y, saved, sums, x, gamma, beta, eps, acts, workspace, stream
	{
		NNF_READ;
		extents e;
		float * y = a.ptr(), * saved = a.ptr(), * sums = a.ptr();
		const float * x = a.ptr(e), * gamma = a.ptr(), * beta = a.ptr();
		const float eps = (float)a.number();
		const auto& acts = a.acts();
		size_t bytes;
		void * ws = a.buffer(bytes);
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_bn_train_fwd(s, y, saved, sums, x, gamma, beta, eps, acts.data(), (int)acts.size(), e.n, e.c, e.hw, ws, bytes); });
	}

	NNF_NATIVE(bn_train_bwd)   // dx, bsums, dy, x, gamma, beta, saved, acts, 5 gradients, mean, invsigma, entry_count, add_to_destination, workspace, stream
	{
		NNF_READ;
		extents e;
		float * dx = a.ptr(), * bsums = a.ptr();
		const float * dy = a.ptr(), * x = a.ptr(e), * gamma = a.ptr(), * beta = a.ptr(), * saved = a.ptr();
		const auto& acts = a.acts();
		float * gg = a.ptr(), * gb = a.ptr(), * gm = a.ptr(), * gi = a.ptr(), * gs = a.ptr();
		const float * mean = a.ptr(), * invsigma = a.ptr();
		const float entries = (float)a.number();
		const int add = a.flag();
		size_t bytes;
		void * ws = a.buffer(bytes);
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_bn_train_bwd(s, dx, bsums, dy, x, gamma, beta, saved, acts.data(), (int)acts.size(), gg, gb, gm, gi, gs, mean, invsigma, entries, e.n, e.c, e.hw, add, ws, bytes); });
	}

	NNF_NATIVE(bn_train_bwd_stats)   // bsums, gsums, dy, x, gamma, beta, saved, acts, workspace, stream
	{
		NNF_READ;
		extents e;
		float * bsums = a.ptr(), * gsums = a.ptr();
		const float * dy = a.ptr(), * x = a.ptr(e), * gamma = a.ptr(), * beta = a.ptr(), * saved = a.ptr();
		const auto& acts = a.acts();
		size_t bytes;
		void * ws = a.buffer(bytes);
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_bn_train_bwd_stats(s, bsums, gsums, dy, x, gamma, beta, saved, acts.data(), (int)acts.size(), e.n, e.c, e.hw, ws, bytes); });
	}

	NNF_NATIVE(bn_train_bwd_apply)   // dx, dy, x, gamma, beta, saved, gsums, bsums, count_total, acts, 5 gradients, mean, invsigma, entry_count, add, stream
	{
		NNF_READ;
		extents e;
		float * dx = a.ptr();
		const float * dy = a.ptr(), * x = a.ptr(e), * gamma = a.ptr(), * beta = a.ptr(), * saved = a.ptr(), * gsums = a.ptr(), * bsums = a.ptr();
		const double count = a.number();
		const auto& acts = a.acts();
		float * gg = a.ptr(), * gb = a.ptr(), * gm = a.ptr(), * gi = a.ptr(), * gs = a.ptr();
		const float * mean = a.ptr(), * invsigma = a.ptr();
		const float entries = (float)a.number();
		const int add = a.flag();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_bn_train_bwd_apply(s, dx, dy, x, gamma, beta, saved, gsums, bsums, count, acts.data(), (int)acts.size(), gg, gb, gm, gi, gs, mean, invsigma, entries, e.n, e.c, e.hw, add); });
	}

	NNF_NATIVE(avgpool_fwd)   // y, x, win_w, win_h, mult, stream
	{
		NNF_READ;
		extents e;
		float * y = a.ptr();
		const float * x = a.ptr(e, true);
		const int ww = (int)a.integer(), wh = (int)a.integer();
		const float mult = (float)a.number();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_avgpool_fwd(s, y, x, e.n, e.c, e.h, e.w, ww, wh, mult); });
	}

	NNF_NATIVE(avgpool_bwd)   // dx, dy, win_w, win_h, mult, add_to_destination, stream
	{
		NNF_READ;
		extents e;
		float * dx = a.ptr(e, true);
		const float * dy = a.ptr();
		const int ww = (int)a.integer(), wh = (int)a.integer();
		const float mult = (float)a.number();
		const int add = a.flag();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_avgpool_bwd(s, dx, dy, e.n, e.c, e.h, e.w, ww, wh, mult, add); });
	}

	NNF_NATIVE(bn_add_relu_avgpool_fwd)   // z, pooled, x, residual, bn, relu_slope, win_w, win_h, mult, stream
	{
		NNF_READ;
		extents e;
		float * z = a.ptr(), * pooled = a.ptr();
		const float * x = a.ptr(e, true), * residual = a.ptr();
		const bn_arrays bn(a);
		const float slope = (float)a.number();
		const int ww = (int)a.integer(), wh = (int)a.integer();
		const float mult = (float)a.number();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_bn_add_relu_avgpool_fwd(s, z, pooled, x, residual, bn.gamma, bn.beta, bn.mean, bn.invsigma, slope, e.n, e.c, e.h, e.w, ww, wh, mult); });
	}

	NNF_NATIVE(bn_add_relu_avgpool_bwd)   // dx, dresidual, dpooled, z, gamma, invsigma, relu_slope, win_w, win_h, mult, stream
	{
		NNF_READ;
		extents e;
		float * dx = a.ptr(), * dresidual = a.ptr();
		const float * dpooled = a.ptr(), * z = a.ptr(e, true), * gamma = a.ptr(), * invsigma = a.ptr();
		const float slope = (float)a.number();
		const int ww = (int)a.integer(), wh = (int)a.integer();
		const float mult = (float)a.number();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_bn_add_relu_avgpool_bwd(s, dx, dresidual, dpooled, z, gamma, invsigma, slope, e.n, e.c, e.h, e.w, ww, wh, mult); });
	}

	NNF_NATIVE(accuracy_fwd)   // out, predicted, targets, mask, top_n, stream
	{
		NNF_READ;
		extents e;
		float * out = a.ptr();
		const float * predicted = a.ptr(e), * targets = a.ptr(), * mask = a.ptr();
		const int top_n = (int)a.integer();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_accuracy_fwd(s, out, predicted, targets, mask, top_n, e.n, e.c, e.hw); });
	}

	// err, predicted, targets, mask, scale, stream
	template <int (*F)(nnf_stream_t, float *, const float *, const float *, const float *, float, int64_t, int64_t, int64_t)>
	NNF_NATIVE(loss_fwd)
	{
		NNF_READ;
		extents e;
		float * err = a.ptr();
		const float * predicted = a.ptr(e), * targets = a.ptr(), * mask = a.ptr();
		const float scale = (float)a.number();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return F(s, err, predicted, targets, mask, scale, e.n, e.c, e.hw); });
	}

	// dpredicted, predicted, targets, mask, scale, add_to_destination, stream
	template <int (*F)(nnf_stream_t, float *, const float *, const float *, const float *, float, int64_t, int64_t, int64_t, int)>
	NNF_NATIVE(loss_bwd)
	{
		NNF_READ;
		extents e;
		float * d = a.ptr();
		const float * predicted = a.ptr(e), * targets = a.ptr(), * mask = a.ptr();
		const float scale = (float)a.number();
		const int add = a.flag();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return F(s, d, predicted, targets, mask, scale, e.n, e.c, e.hw, add); });
	}

	NNF_NATIVE(softmax_nll_fwd)   // probs, err, logits, targets, mask, scale, stream
	{
		NNF_READ;
		extents e;
		float * probs = a.ptr(), * err = a.ptr();
		const float * logits = a.ptr(e), * targets = a.ptr(), * mask = a.ptr();
		const float scale = (float)a.number();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_softmax_nll_fwd(s, probs, err, logits, targets, mask, scale, e.n, e.c, e.hw); });
	}

	// The fields of one chunk's dict. A step hands over hundreds of chunks, so the dict is walked once and its keys, which are interned
	// strings in nearly every program, are told apart by address; other strings are compared. (Seven look-ups per chunk took
	// 110 ns, three times the GPU's time for a network of small layers; the walk takes 60.) Any other mapping, a subclass of dict among
	// them, is asked through its own item and get.
	enum part_field { kData, kGradient, kLearningRate, kUpdateAccum, kPrevUpd, kPrevUpd2, kWeightDecay, kPartFields };
	struct part_keys
	{
		PyObject * key[kPartFields];
		part_keys()
		{
			static const char * const names[kPartFields] = {"data", "gradient", "learning_rate", "update_accum", "prev_upd", "prev_upd2", "weight_decay"};
			for (int k = 0; k < kPartFields; ++k)
				key[k] = PyUnicode_InternFromString(names[k]);
		}
	};

	NNF_NATIVE(apply_gradient)   // parts, momentum_type, momentum, momentum2, normalizer, iteration_id, stream
	{
		static const part_keys keys;
		NNF_READ;
		std::vector<nnf_opt_part> parts;
		PyObject * list = a.next();
		if (PyList_Check(list))
			parts.reserve((size_t)PyList_GET_SIZE(list));
		auto add = [&](PyObject * const (&v)[kPartFields])
		{
			auto address = [&](int k) { return v[k] ? a.address_of(v[k]) : nullptr; };
			nnf_opt_part p = {};
			p.data = static_cast<float *>(address(kData));
			p.gradient = static_cast<float *>(address(kGradient));
			p.prev_upd = static_cast<float *>(address(kPrevUpd));
			p.prev_upd2 = static_cast<float *>(address(kPrevUpd2));
			p.update_accum = static_cast<double *>(address(kUpdateAccum));
			p.learning_rate = (float)a.number(v[kLearningRate]);
			p.weight_decay = v[kWeightDecay] ? (float)a.number(v[kWeightDecay]) : 0.0F;
			p.elem_count = a.numel(v[kData]);
			if (a.ok())
				parts.push_back(p);
		};
		auto add_mapping = [&](PyObject * d)
		{
			PyObject * v[kPartFields] = {};
			owned asked[kPartFields] = {};
			for (int k = 0; k < kPartFields; ++k)
			{
				const bool required = k <= kLearningRate;
				asked[k].object = required ? PyObject_GetItem(d, keys.key[k]) : PyObject_CallMethod(d, "get", "O", keys.key[k]);
				if (!asked[k].object)
				{
					a.fail(nullptr, nullptr);
					return;
				}
				v[k] = required || asked[k].object != Py_None ? asked[k].object : nullptr;
			}
			add(v);
		};
		a.sequence(list, [&](PyObject * d)
		{
			if (!PyDict_CheckExact(d))
			{
				add_mapping(d);
				return;
			}
			PyObject * v[kPartFields] = {};
			PyObject * key, * value;
			for (Py_ssize_t pos = 0; PyDict_Next(d, &pos, &key, &value);)
			{
				int k = 0;
				while (k < kPartFields && key != keys.key[k])
					++k;
				if (k == kPartFields && PyUnicode_Check(key))
					for (k = 0; k < kPartFields && PyUnicode_Compare(key, keys.key[k]) != 0; ++k) {}
				if (k < kPartFields)
					v[k] = value;
			}
			for (int k : {kData, kGradient, kLearningRate})
				if (!v[k])
				{
					PyErr_SetObject(PyExc_KeyError, keys.key[k]);   // as d[key] does
					a.fail(nullptr, nullptr);
					return;
				}
			add(v);
		});
		const int type = (int)a.integer();
		const float m1 = (float)a.number(), m2 = (float)a.number(), normalizer = (float)a.number();
		const unsigned int iteration = (unsigned int)a.integer();
		const nnf_stream_t s = a.stream();
		return call(a, [&] { return nnf_apply_gradient(s, parts.data(), (int)parts.size(), type, m1, m2, normalizer, iteration); });
	}

	// ---- layer objects (host.py) ---------------------------------------------------------------------
	NNF_NATIVE(tester_forward)   // handle, output, data, inputs, entry_count
	{
		NNF_READ_OBJECT;
		std::vector<void *> data, in;
		void * h = a.handle(), * out = a.loose();
		a.addresses<false>(data);
		a.addresses<false>(in);
		const unsigned int n = (unsigned int)a.integer();
		return call_object(a, [&](nnf_stream_t s) { return nnfh_tester_forward(h, s, out, data.data(), (int)data.size(), in.data(), (int)in.size(), n); });
	}

	NNF_NATIVE(updater_forward)   // handle, output, data, inputs, working, fixed, per_entry, entry_count
	{
		NNF_READ_OBJECT;
		std::vector<void *> data, in;
		void * h = a.handle(), * out = a.loose();
		a.addresses<false>(data);
		a.addresses<false>(in);
		size_t bytes;
		void * ws = a.buffer<false>(bytes), * fixed = a.loose(), * per_entry = a.loose();
		const unsigned int n = (unsigned int)a.integer();
		return call_object(a, [&](nnf_stream_t s) { return nnfh_updater_forward(h, s, out, data.data(), (int)data.size(), in.data(), (int)in.size(), ws, bytes, fixed, per_entry, n); });
	}

	NNF_NATIVE(object_forward)   // handle, outputs, data, inputs, working, fixed, per_entry, entry_count
	{
		NNF_READ_OBJECT;
		std::vector<void *> out, data, in;
		void * h = a.handle();
		a.addresses<false>(out);
		a.addresses<false>(data);
		a.addresses<false>(in);
		size_t bytes;
		void * ws = a.buffer<false>(bytes), * fixed = a.loose(), * per_entry = a.loose();
		const unsigned int n = (unsigned int)a.integer();
		return call_object(a, [&](nnf_stream_t s) { return nnfh_forward(h, s, out.data(), (int)out.size(), data.data(), (int)data.size(), in.data(), (int)in.size(), ws, bytes, fixed, per_entry, n); });
	}

	NNF_NATIVE(object_backward_data)   // handle, input_index, input_errors, output_errors, data, input_neurons, output_neurons, fixed, per_entry, add, entry_count
	{
		NNF_READ_OBJECT;
		std::vector<void *> data, in;
		void * h = a.handle();
		const unsigned int index = (unsigned int)a.integer();
		void * ie = a.loose(), * oe = a.loose();
		a.addresses<false>(data);
		a.addresses<false>(in);
		void * on = a.loose(), * fixed = a.loose(), * per_entry = a.loose();
		const int add = a.flag();
		const unsigned int n = (unsigned int)a.integer();
		return call_object(a, [&](nnf_stream_t s) { return nnfh_backward_data(h, s, index, ie, oe, data.data(), (int)data.size(), in.data(), (int)in.size(), on, fixed, per_entry, add, n); });
	}

	NNF_NATIVE(object_backward_weights)   // handle, gradient, input_neurons, output_errors, working, entry_count
	{
		NNF_READ_OBJECT;
		std::vector<void *> gradient, in;
		void * h = a.handle();
		a.addresses<false>(gradient);
		a.addresses<false>(in);
		void * oe = a.loose();
		size_t bytes;
		void * ws = a.buffer<false>(bytes);
		const unsigned int n = (unsigned int)a.integer();
		return call_object(a, [&](nnf_stream_t s) { return nnfh_backward_weights(h, s, gradient.data(), (int)gradient.size(), in.data(), (int)in.size(), oe, ws, bytes, n); });
	}

	NNF_NATIVE(object_backward_data_and_weights)   // handle, input_errors, output_errors, gradient, data, input_neurons, output_neurons, working, fixed, add, entry_count
	{
		NNF_READ_OBJECT;
		std::vector<void *> ie, gradient, data, in;
		void * h = a.handle();
		a.addresses<false>(ie);
		void * oe = a.loose();
		a.addresses<false>(gradient);
		a.addresses<false>(data);
		a.addresses<false>(in);
		void * on = a.loose();
		size_t bytes;
		void * ws = a.buffer<false>(bytes), * fixed = a.loose();
		const int add = a.flag();
		const unsigned int n = (unsigned int)a.integer();
		return call_object(a, [&](nnf_stream_t s) { return nnfh_backward_data_and_weights(h, s, ie.data(), (int)ie.size(), oe, gradient.data(), (int)gradient.size(),
			data.data(), (int)data.size(), in.data(), (int)in.size(), on, ws, bytes, fixed, add, n); });
	}

	PyObject * set_types(PyObject *, PyObject * types)   // (NnfError, Act, Pool)
	{
		PyObject * error, * act, * pool;
		if (!PyArg_ParseTuple(types, "OOO", &error, &act, &pool))
			return nullptr;
		Py_XSETREF(g_error_type, Py_NewRef(error));
		Py_XSETREF(g_act_type, Py_NewRef(act));
		Py_XSETREF(g_pool_type, Py_NewRef(pool));
		Py_RETURN_NONE;
	}

	#define NNF_ENTRY(name) {#name, (PyCFunction)(void (*)(void))guarded<name>, METH_FASTCALL, nullptr}
	#define NNF_ENTRY_AS(name, ...) {name, (PyCFunction)(void (*)(void))guarded<__VA_ARGS__>, METH_FASTCALL, nullptr}
	PyMethodDef g_methods[] = {
		NNF_ENTRY(bn_infer_act), NNF_ENTRY(act_fwd), NNF_ENTRY(act_bwd), NNF_ENTRY(prelu_bwd_weights), NNF_ENTRY(add_fwd), NNF_ENTRY(add_bwd),
		NNF_ENTRY(softmax_fwd), NNF_ENTRY(softmax_bwd), NNF_ENTRY(maxpool_fwd), NNF_ENTRY(maxpool_bwd), NNF_ENTRY(bn_add_relu_maxpool_fwd),
		NNF_ENTRY(bn_add_relu_maxpool_bwd), NNF_ENTRY(bn_train_stats), NNF_ENTRY(bn_train_stats_static), NNF_ENTRY(bn_train_apply_act),
		NNF_ENTRY(bn_train_fwd), NNF_ENTRY(bn_train_bwd), NNF_ENTRY(bn_train_bwd_stats), NNF_ENTRY(bn_train_bwd_apply), NNF_ENTRY(avgpool_fwd),
		NNF_ENTRY(avgpool_bwd), NNF_ENTRY(bn_add_relu_avgpool_fwd), NNF_ENTRY(bn_add_relu_avgpool_bwd), NNF_ENTRY(accuracy_fwd),
		NNF_ENTRY_AS("nll_fwd", loss_fwd<nnf_nll_fwd>), NNF_ENTRY_AS("nll_bwd", loss_bwd<nnf_nll_bwd>),
		NNF_ENTRY_AS("cross_entropy_fwd", loss_fwd<nnf_cross_entropy_fwd>), NNF_ENTRY_AS("cross_entropy_bwd", loss_bwd<nnf_cross_entropy_bwd>),
		NNF_ENTRY(softmax_nll_fwd), NNF_ENTRY_AS("softmax_nll_bwd", loss_bwd<nnf_softmax_nll_bwd>), NNF_ENTRY(apply_gradient),
		NNF_ENTRY(tester_forward), NNF_ENTRY(updater_forward), NNF_ENTRY(object_forward), NNF_ENTRY(object_backward_data),
		NNF_ENTRY(object_backward_weights), NNF_ENTRY(object_backward_data_and_weights),
		{"set_types", set_types, METH_VARARGS, nullptr},
		{nullptr, nullptr, 0, nullptr}};

	PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", "Call path between Python and the C ABI.", -1, g_methods, nullptr, nullptr, nullptr, nullptr};
}

PyMODINIT_FUNC PyInit__native(void)
{
	return PyModule_Create(&g_module);
}
