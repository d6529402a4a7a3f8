// _param_watch: "has any of these parameters changed since the plan was built?" for a whole module tree in one call.
//
// A plan (parameter structs with raw pointers, packed weights) is valid as long as every parameter is the same object
// contents: same address and same version counter. Asked tensor by tensor from Python this costs 0.3 - 0.5 us per
// parameter, 300 us for the 624 parameters of a 24-block diffusion stack; here it is about 10 ns each.
#include <torch/csrc/autograd/python_variable.h>

#include <memory>
#include <vector>

namespace {

struct Slot {
    PyObject *dict, *name;   // a module's _parameters and a key of it (owned references)
    const void* ptr;
    uint32_t version;
};
struct Watch {
    std::vector<Slot> slots;
    ~Watch() {
        for (Slot& s : slots) {
            Py_DECREF(s.dict);
            Py_DECREF(s.name);
        }
    }
};

// 0: read, 1: there is nothing that can be watched (missing, no storage, no version counter)
int read(const Slot& s, const void** ptr, uint32_t* version) {
    PyObject* o = PyDict_GetItemWithError(s.dict, s.name);   // borrowed
    if (o == nullptr || !THPVariable_Check(o)) {
        PyErr_Clear();
        return 1;
    }
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.has_storage() || t.is_inference()) return 1;
    *ptr = t.const_data_ptr();
    *version = t.unsafeGetTensorImpl()->version_counter().current_version();
    return 0;
}

const char* kName = "openfold3_b200.param_watch";
void destroy(PyObject* cap) { delete static_cast<Watch*>(PyCapsule_GetPointer(cap, kName)); }

// make([(dict, name), ...]) -> handle, or None when one of them cannot be watched
PyObject* make(PyObject*, PyObject* list) {
    if (!PyList_Check(list)) {
        PyErr_SetString(PyExc_TypeError, "a list of (dict, name) is wanted");
        return nullptr;
    }
    auto w = std::make_unique<Watch>();
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(list); ++i) {
        PyObject* it = PyList_GET_ITEM(list, i);
        if (!PyTuple_Check(it) || PyTuple_GET_SIZE(it) != 2 || !PyDict_Check(PyTuple_GET_ITEM(it, 0))) {
            PyErr_SetString(PyExc_TypeError, "a list of (dict, name) is wanted");
            return nullptr;
        }
        Slot s{PyTuple_GET_ITEM(it, 0), PyTuple_GET_ITEM(it, 1), nullptr, 0};
        if (read(s, &s.ptr, &s.version)) Py_RETURN_NONE;
        Py_INCREF(s.dict);
        Py_INCREF(s.name);
        w->slots.push_back(s);
    }
    return PyCapsule_New(w.release(), kName, destroy);
}

// changed(handle) -> bool
PyObject* changed(PyObject*, PyObject* cap) {
    Watch* w = static_cast<Watch*>(PyCapsule_GetPointer(cap, kName));
    if (w == nullptr) return nullptr;
    for (const Slot& s : w->slots) {
        const void* p;
        uint32_t v;
        if (read(s, &p, &v) || p != s.ptr || v != s.version) Py_RETURN_TRUE;
    }
    Py_RETURN_FALSE;
}

PyMethodDef kMethods[] = {{"make", make, METH_O, nullptr}, {"changed", changed, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_param_watch", nullptr, -1, kMethods};

}  // namespace

PyMODINIT_FUNC PyInit__param_watch(void) { return PyModule_Create(&kModule); }
