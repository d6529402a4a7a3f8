// _param_watch: "has anything changed that this plan was built from?" for a whole module tree in one call.
//
// A plan (parameter structs with raw pointers, packed weights, sizes) is valid as long as every parameter has the same
// address and version counter, every module the same children and parameters, and every constant that was read is the same
// object. Asked one by one from Python this costs 0.3 - 0.5 us each, 300 us for the 624 parameters of a 24-block diffusion
// stack alone; here it is about 10 ns each.
#include <torch/csrc/autograd/python_variable.h>

#include <exception>
#include <memory>
#include <vector>

namespace {

// The references are borrowed: the list that make() returns beside the handle owns them (it is visible to the garbage
// collector, which a capsule's contents are not: a module tree may refer to itself).
struct Item {
    PyObject *key, *value;
    const void* ptr = nullptr;   // of a parameter
    uint32_t version = 0;
};
struct Content {
    PyObject* dict;
    size_t first;      // into items
    Py_ssize_t count;
    bool params;       // a module's _parameters: tensors and Nones
};
struct Attr {
    PyObject *dict, *name, *value;   // value null: not there
};
struct Watch {
    std::vector<Item> items;
    std::vector<Content> contents;
    std::vector<Attr> attrs;
};

// False: there is nothing that can be watched (no tensor, no storage or address, no version counter).
bool read(PyObject* o, const void** ptr, uint32_t* version) {
    if (!THPVariable_Check(o)) return false;
    try {   // (a tensor without memory of its own, as tracing makes them, may throw when it is asked for its address)
        const at::Tensor& t = THPVariable_Unpack(o);
        if (!t.has_storage() || t.is_inference()) return false;
        *ptr = t.const_data_ptr();
        *version = t.unsafeGetTensorImpl()->version_counter().current_version();
    } catch (const std::exception&) {
        return false;
    }
    return true;
}

const char* kName = "openfold3_b200.param_watch";
void destroy(PyObject* cap) { delete static_cast<Watch*>(PyCapsule_GetPointer(cap, kName)); }

// make(params [dict, ...], contents [dict, ...], attrs [(dict, name), ...]) -> (handle, objects to be kept with it), or None
// when a parameter cannot be watched. Watched: keys and values of each dict, address and version of each tensor of `params`,
// the value (or absence) of each of `attrs`.
PyObject* make(PyObject*, PyObject* args) {
    PyObject *params, *contents, *attrs;
    if (!PyArg_ParseTuple(args, "O!O!O!", &PyList_Type, &params, &PyList_Type, &contents, &PyList_Type, &attrs)) return nullptr;
    auto w = std::make_unique<Watch>();
    struct Ref {
        PyObject* p;
        ~Ref() { Py_XDECREF(p); }
    } kept{PyList_New(0)};
    if (kept.p == nullptr) return nullptr;
    auto keep = [&](PyObject* o) { return PyList_Append(kept.p, o) == 0; };
    for (PyObject* list : {params, contents}) {
        for (Py_ssize_t i = 0; i < PyList_GET_SIZE(list); ++i) {
            PyObject* d = PyList_GET_ITEM(list, i);
            if (!PyDict_Check(d)) {
                PyErr_SetString(PyExc_TypeError, "a list of dicts is wanted");
                return nullptr;
            }
            w->contents.push_back({d, w->items.size(), PyDict_GET_SIZE(d), list == params});
            if (!keep(d)) return nullptr;
            Py_ssize_t pos = 0;
            Item it;
            while (PyDict_Next(d, &pos, &it.key, &it.value)) {
                if (list == params && it.value != Py_None && !read(it.value, &it.ptr, &it.version)) Py_RETURN_NONE;
                w->items.push_back(it);
                if (!keep(it.key) || !keep(it.value)) return nullptr;
            }
        }
    }
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(attrs); ++i) {
        PyObject *it = PyList_GET_ITEM(attrs, i), *d, *n;
        if (!PyArg_ParseTuple(it, "O!O", &PyDict_Type, &d, &n)) return nullptr;
        PyObject* v = PyDict_GetItemWithError(d, n);   // borrowed
        if (v == nullptr && PyErr_Occurred()) return nullptr;
        w->attrs.push_back({d, n, v});
        if (!keep(d) || !keep(n) || (v != nullptr && !keep(v))) return nullptr;
    }
    Ref cap{PyCapsule_New(w.get(), kName, destroy)};
    if (cap.p == nullptr) return nullptr;
    w.release();
    return PyTuple_Pack(2, cap.p, kept.p);
}

// changed(handle) -> bool
PyObject* changed(PyObject*, PyObject* cap) {
    Watch* w = static_cast<Watch*>(PyCapsule_GetPointer(cap, kName));
    if (w == nullptr) return nullptr;
    for (const Content& c : w->contents) {
        if (PyDict_GET_SIZE(c.dict) != c.count) Py_RETURN_TRUE;
        Py_ssize_t pos = 0;
        PyObject *key, *value;
        for (const Item* want = w->items.data() + c.first; PyDict_Next(c.dict, &pos, &key, &value); ++want) {
            if (key != want->key || value != want->value) Py_RETURN_TRUE;
            if (!c.params || value == Py_None) continue;
            const void* p;
            uint32_t v;
            if (!read(value, &p, &v) || p != want->ptr || v != want->version) Py_RETURN_TRUE;
        }
    }
    for (const Attr& a : w->attrs) {
        PyObject* v = PyDict_GetItemWithError(a.dict, a.name);
        if (v == nullptr && PyErr_Occurred()) return nullptr;
        if (v != a.value) Py_RETURN_TRUE;
    }
    Py_RETURN_FALSE;
}

PyMethodDef kMethods[] = {{"make", make, METH_VARARGS, nullptr}, {"changed", changed, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_param_watch", nullptr, -1, kMethods};

}  // namespace

PyMODINIT_FUNC PyInit__param_watch(void) { return PyModule_Create(&kModule); }
