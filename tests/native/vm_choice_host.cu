// Test harness only: the engine's choice of VMs (vm_choice.cuh) compiled for
// the host.  The product never loads this library.
#include "../../gagp_b200/csrc/vm_choice.cuh"

extern "C" {
int host_exact_possible(const gagp_grammar* g, int fuel) { return gb::exact_possible(g, fuel); }
int host_bytecode_bound(const gagp_grammar* g) { return gb::bytecode_bound(g, g->max_nodes - g->fixed_nodes); }
}
