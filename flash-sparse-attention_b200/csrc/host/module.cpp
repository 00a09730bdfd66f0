// The extension module (fsa/lib/_fsa_host.so).
#include "host_common.h"

PYBIND11_MODULE(_fsa_host, m) {
    fsa_host::bind_sel(m);
    fsa_host::bind_decode(m);
    fsa_host::bind_layer(m);
}
