// Host-side walks over the parameters of a DLR-Net, native because a net has four tensors per layer (about 570) and a decode
// step visits every net: the same walk in Python costs 655 us per forward through ParameterList indexing, and still 80 us
// written with map(); the forward itself is about 110 us of GPU time.
//
//   in_order(dict, n)        whether the keys of a dict are "0", "1", ... "n-1", in this order
//   snapshot(dicts)          bytes: storage address and in-place version of every tensor of the dicts, in order
//   unchanged(bytes, dicts)  whether snapshot(dicts) would return the same bytes (no, if it would refuse the dicts, and for
//                            anything but bytes)
//   layers(dicts)            what the fold kernel needs of the four parameter dicts (V, U, gains, alphas; keys "0", "1", ...)
//   state_layers(dict)       the same of a state dict (keys Vs.i, Us.i, rms_w.i, alphas.i, an _orig_mod. prefix allowed)
//
// The last two return (L, r, d, device index, matrices are bf16, alphas are bf16, addresses of V, U, gain, alpha as four
// bytes objects), or None for anything but complete layers of contiguous bf16 or fp32 tensors of one shape on one GPU; the
// caller then takes the general way through torch operations.  A C++ exception becomes a Python one: the address of a tensor
// without storage (under a functorch transform) is a RuntimeError, as it is for Tensor.data_ptr().
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstring>
#include <string>
#include <vector>

#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

namespace {

struct Word {
    uint64_t address, version;
};

// (raises for an inference tensor, whose edits leave no trace)
Word word_of(PyObject* o) {
    const at::Tensor& t = THPVariable_Unpack(o);
    return Word{reinterpret_cast<uint64_t>(t.const_data_ptr()), t.unsafeGetTensorImpl()->version_counter().current_version()};
}

// "0", "1", ... as text, and whether a key is the one that is due.
struct Count {
    char text[24];
    char* at = text + sizeof(text) - 1;

    Count() { *at = '0'; }

    bool is(PyObject* key) {
        char* const end = text + sizeof(text);
        const bool same = PyUnicode_CheckExact(key) && PyUnicode_IS_COMPACT_ASCII(key) && PyUnicode_GET_LENGTH(key) == end - at &&
                          std::memcmp(PyUnicode_1BYTE_DATA(key), at, size_t(end - at)) == 0;
        char* c = end - 1;
        while (c >= at && *c == '9') *c-- = '0';
        if (c < at) *--at = '1';
        else ++*c;
        return same;
    }
};

// Calls f on every tensor of a tuple of dicts; f returns false to stop.  False if stopped, on something else than a tensor
// and on keys that are not in order (the dict of a list with an entry that is not a plain parameter).
template <class F>
bool for_each_tensor(PyObject* dicts, F f) {
    const Py_ssize_t n = PyTuple_GET_SIZE(dicts);
    for (Py_ssize_t i = 0; i < n; ++i) {
        PyObject *key, *value;
        Py_ssize_t pos = 0;
        PyObject* d = PyTuple_GET_ITEM(dicts, i);
        if (!PyDict_Check(d)) return false;
        Count count;
        while (PyDict_Next(d, &pos, &key, &value))
            if (!count.is(key) || !THPVariable_Check(value) || !f(value)) return false;
    }
    return true;
}

PyObject* snapshot(PyObject*, PyObject* dicts) {
    HANDLE_TH_ERRORS
    if (!PyTuple_Check(dicts)) {
        PyErr_SetString(PyExc_TypeError, "snapshot takes a tuple of dicts of tensors, keys \"0\", \"1\", ... in order");
        return nullptr;
    }
    std::vector<Word> words;
    if (!for_each_tensor(dicts, [&](PyObject* o) { words.push_back(word_of(o)); return true; })) {
        PyErr_SetString(PyExc_TypeError, "snapshot takes a tuple of dicts of tensors, keys \"0\", \"1\", ... in order");
        return nullptr;
    }
    return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(words.data()), Py_ssize_t(words.size() * sizeof(Word)));
    END_HANDLE_TH_ERRORS
}

PyObject* unchanged(PyObject*, PyObject* args) {
    HANDLE_TH_ERRORS
    PyObject *snap, *dicts;
    if (!PyArg_ParseTuple(args, "OO!", &snap, &PyTuple_Type, &dicts)) return nullptr;
    if (!PyBytes_Check(snap)) Py_RETURN_FALSE;
    const char* at = PyBytes_AS_STRING(snap);
    const char* end = at + PyBytes_GET_SIZE(snap);
    const bool same = for_each_tensor(dicts, [&](PyObject* o) {
        const Word w = word_of(o);
        if (end - at < Py_ssize_t(sizeof(Word)) || std::memcmp(at, &w, sizeof(Word)) != 0) return false;
        at += sizeof(Word);
        return true;
    });
    return PyBool_FromLong(same && at == end);
    END_HANDLE_TH_ERRORS
}

struct Group {
    std::vector<PyObject*> at;      // borrowed, by layer

    bool put(long i, PyObject* o) {
        if (i < 0 || i > 65535 || !THPVariable_Check(o)) return false;
        if (size_t(i) >= at.size()) at.resize(size_t(i) + 1, nullptr);
        if (at[size_t(i)]) return false;
        at[size_t(i)] = o;
        return true;
    }
};

// Layer number at the end of a key, -1 if there is none.
long number(const char* s) {
    if (*s < '0' || *s > '9') return -1;
    long n = 0;
    for (; *s >= '0' && *s <= '9'; ++s) {
        n = 10 * n + (*s - '0');
        if (n > 65535) return -1;
    }
    return *s ? -1 : n;
}

PyObject* in_order(PyObject*, PyObject* args) {
    HANDLE_TH_ERRORS
    PyObject* d;
    Py_ssize_t n;
    if (!PyArg_ParseTuple(args, "O!n", &PyDict_Type, &d, &n)) return nullptr;
    PyObject *key, *value;
    Py_ssize_t pos = 0;
    Count count;
    bool same = PyDict_GET_SIZE(d) == n;
    while (same && PyDict_Next(d, &pos, &key, &value)) same = count.is(key);
    return PyBool_FromLong(same);
    END_HANDLE_TH_ERRORS
}

PyObject* describe(const Group (&g)[4]) {
    const size_t L = g[0].at.size();
    if (L == 0) Py_RETURN_NONE;
    int64_t r = 0, d = 0;
    int device = -1;
    bool bf16[2] = {false, false};
    std::vector<uint64_t> address[4];
    for (int k = 0; k < 4; ++k) {
        if (g[k].at.size() != L) Py_RETURN_NONE;
        address[k].reserve(L);
        for (size_t i = 0; i < L; ++i) {
            if (!g[k].at[i]) Py_RETURN_NONE;
            const at::Tensor& t = THPVariable_Unpack(g[k].at[i]);
            if (!t.has_storage()) Py_RETURN_NONE;
            if (k == 0 && i == 0) {
                if (t.dim() != 2 || !t.is_cuda()) Py_RETURN_NONE;
                r = t.size(0);
                d = t.size(1);
                device = t.get_device();
                bf16[0] = t.scalar_type() == at::kBFloat16;
            }
            if (k == 3 && i == 0) bf16[1] = t.scalar_type() == at::kBFloat16;
            const at::ScalarType want = bf16[k == 3] ? at::kBFloat16 : at::kFloat;
            if (!t.is_cuda() || t.get_device() != device || t.scalar_type() != want || t.layout() != at::kStrided || !t.is_contiguous() ||
                t.is_conj() || t.is_neg())
                Py_RETURN_NONE;
            const bool shaped = k == 0 ? t.dim() == 2 && t.size(0) == r && t.size(1) == d
                              : k == 1 ? t.dim() == 2 && t.size(0) == d && t.size(1) == r
                              : k == 2 ? t.dim() == 1 && t.size(0) == d
                                       : t.numel() == 1;
            if (!shaped) Py_RETURN_NONE;
            const void* data = t.const_data_ptr();
            if (!data) Py_RETURN_NONE;                 // (a fake tensor)
            address[k].push_back(reinterpret_cast<uint64_t>(data));
        }
    }
    auto bytes = [&](int k) {
        return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(address[k].data()), Py_ssize_t(L * sizeof(uint64_t)));
    };
    return Py_BuildValue("nnniOONNNN", Py_ssize_t(L), Py_ssize_t(r), Py_ssize_t(d), device, bf16[0] ? Py_True : Py_False,
                         bf16[1] ? Py_True : Py_False, bytes(0), bytes(1), bytes(2), bytes(3));
}

PyObject* layers(PyObject*, PyObject* dicts) {
    HANDLE_TH_ERRORS
    if (!PyTuple_Check(dicts) || PyTuple_GET_SIZE(dicts) != 4) {
        PyErr_SetString(PyExc_TypeError, "layers takes a tuple of four dicts");
        return nullptr;
    }
    Group g[4];
    for (int k = 0; k < 4; ++k) {
        PyObject *key, *value;
        Py_ssize_t pos = 0;
        PyObject* d = PyTuple_GET_ITEM(dicts, k);
        if (!PyDict_Check(d)) Py_RETURN_NONE;
        while (PyDict_Next(d, &pos, &key, &value)) {
            const char* s = PyUnicode_Check(key) ? PyUnicode_AsUTF8(key) : nullptr;
            if (!s) {
                PyErr_Clear();
                Py_RETURN_NONE;
            }
            if (!g[k].put(number(s), value)) Py_RETURN_NONE;
        }
    }
    return describe(g);
    END_HANDLE_TH_ERRORS
}

PyObject* state_layers(PyObject*, PyObject* sd) {
    HANDLE_TH_ERRORS
    if (!PyDict_Check(sd)) Py_RETURN_NONE;
    static const struct { const char* name; size_t n; } kNames[4] = {{"Vs.", 3}, {"Us.", 3}, {"rms_w.", 6}, {"alphas.", 7}};
    Group g[4];
    PyObject *key, *value;
    Py_ssize_t pos = 0;
    while (PyDict_Next(sd, &pos, &key, &value)) {
        const char* s = PyUnicode_Check(key) ? PyUnicode_AsUTF8(key) : nullptr;
        if (!s) {
            PyErr_Clear();
            Py_RETURN_NONE;
        }
        if (std::strncmp(s, "_orig_mod.", 10) == 0) s += 10;
        for (int k = 0; k < 4; ++k)
            if (std::strncmp(s, kNames[k].name, kNames[k].n) == 0) {
                if (!g[k].put(number(s + kNames[k].n), value)) Py_RETURN_NONE;      // (no layer number either)
            }
    }
    return describe(g);
    END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {{"in_order", in_order, METH_VARARGS, nullptr},
                          {"snapshot", snapshot, METH_O, nullptr},
                          {"unchanged", unchanged, METH_VARARGS, nullptr},
                          {"layers", layers, METH_O, nullptr},
                          {"state_layers", state_layers, METH_O, nullptr},
                          {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&kModule); }
