// Takes one of a net's events of its second stream away, or puts it back: what a CUDA call that fails looks like from there.
// (Compiled without access control.)
#include "../../cnet_b200/host/cnet.h"

extern "C" void* swap_side_event(void* net, int join, void* event) {
	cnet_b200::CNet* n = static_cast<cnet_b200::CNet*>(net);         // (the first member of the C handle)
	void*& at = join ? n->ev_side_join_ : n->ev_side_fork_;
	void* was = at;
	at = event;
	return was;
}
