extern "C" const char* pb_abi() { return "cc65064b7c93"; }
