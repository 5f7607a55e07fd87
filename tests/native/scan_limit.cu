// The engine with one entry point more: the number of looks a wait of the prefix scan may take (0: every wait gives
// up at once, as if the tile it waits for never came).
#include "../../woo_gb300/csrc/wdem_api.cu"
extern "C" void scan_limit_set(wdem_handle* h, int looks) { h->cs.scanLooks = looks; }
